"""A march block's sample pairs, whose taps are not clamped, give the bits of
the clamped samples one at a time, for every ray that ray_setup cuts to the
volume's box; rays on longer axes than the bound holds for take the latter.
The kernels' code (asc_march.cuh) as host C++."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from autoscoper_gb300 import scene as S
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def hb(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hb") / "libhost_block.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "host_block.cpp")], check=True)
    lib = C.CDLL(so)
    lib.hb_blocks.restype = None
    lib.hb_blocks.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_float,
                              C.c_float, C.c_int, C.c_int, C.c_void_p]
    return lib


def blocks(hb, vol, storage, m, vp, step, cutoff, w, h):
    words = vol.astype(np.float32).view(np.uint32) if storage else vol.astype(np.uint32)
    if storage == 2:  # bfloat16: the upper half of integers of at most 8 bits
        words = words >> 16
    words = np.ascontiguousarray(words)
    nz, ny, nx = vol.shape
    counts = (C.c_longlong * 3)()
    mf, vpf = np.ascontiguousarray(m, np.float32), np.ascontiguousarray(vp, np.float32)
    hb.hb_blocks(words.ctypes.data, nx, ny, nz, storage, mf.ctypes.data, vpf.ctypes.data, step, cutoff, w, h, counts)
    return list(counts)


@pytest.mark.parametrize("storage", [0, 2, 3])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 5, 2), (48, 40, 56)])
def test_pairs_equal_clamped_samples(hb, storage, dims):
    sc = S.make_scene([dims], 1.0, (40, 36), 0.8, filters="sobel", seed=3)
    tr = O.Tracker(sc)
    rng = np.random.default_rng(5)
    vol = rng.integers(0, 256 if storage == 2 else 65536, dims[::-1])
    seen = 0
    for i in range(3):
        pose = S.perturb(sc.truth[0], rng, 3.0, 20.0).astype(np.float64)
        ok, m, vp, w, h = tr.view_setup(0, i % 2, pose)
        n, outside, differ = blocks(hb, vol, storage, m, vp, sc.ray[i % 2][0].step, 0.3 / (257 if storage == 2 else 1),
                                    w, h)
        assert outside == 0 and differ == 0
        seen += n
    assert seen > 0


def test_long_axes_are_clamped(hb):
    """An axis of more than 2^16 voxels: no ray takes the unclamped pairs."""
    rng = np.random.default_rng(6)
    vol = rng.integers(0, 65536, (1, 1, 65537))
    # a camera 3 units before the unit box, looking along -z (volume z in [-1, 0])
    m = np.float32([[1, 0, 0, 0.5], [0, 1, 0, 0.5], [0, 0, 1, 3.0]])
    n, outside, differ = blocks(hb, vol, 0, m, [-0.2, -0.2, 0.4, 0.4], 0.05, 0.1, 9, 7)
    assert n > 0 and outside > 0 and differ == 0
