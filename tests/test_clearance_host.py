"""The clearance grid by its kernel's own code (asc_clear.cuh) as host C++:
every cell's byte is the distance, in voxels and the maximum norm, from the
cell's span [2c, 2c + 2] to the nearest voxel above the threshold, at most 15;
at sizes around the cells, the blocks of 32 voxels and a warp's 64."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def hc(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hc") / "libhost_clear.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "host_clear.cpp")], check=True)
    lib = C.CDLL(so)
    lib.hc_grid.restype = None
    lib.hc_grid.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_float, C.c_void_p]
    return lib


def distances(above):
    d = np.where(above, 0, 15).astype(np.int32)
    for axis in range(3):
        n = d.shape[axis]
        v = np.arange(n)
        out = []
        for c in range((n + 1) // 2):
            off = np.maximum(np.maximum(2 * c - v, v - 2 * c - 2), 0).reshape([-1 if a == axis else 1 for a in range(3)])
            out.append(np.maximum(d, off).min(axis))
        d = np.stack(out, axis)
    return d


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (33, 31, 64), (40, 66, 35), (15, 66, 98)])  # depth, height, width
@pytest.mark.parametrize("storage", [0, 2, 3])  # u16, bfloat16, FP32
def test_every_cell_holds_its_distance(hc, shape, storage):
    rng = np.random.default_rng(sum(shape))
    for density in (0.0, 2e-3, 0.2):
        vol = np.where(rng.random(shape) < density, 200, 100)
        if density == 2e-3:
            vol[-1, -1, -1] = 200  # the corner, whose copies past the edge are no voxels
        words = vol.astype(np.float32).view(np.uint32) if storage else vol.astype(np.uint32)
        words = np.ascontiguousarray(words >> 16 if storage == 2 else words)
        got = np.full([(n + 1) // 2 for n in shape], 255, np.uint8)
        hc.hc_grid(words.ctypes.data, shape[2], shape[1], shape[0], storage, 150.0, got.ctypes.data)
        assert np.array_equal(got, distances(vol > 150)), density
