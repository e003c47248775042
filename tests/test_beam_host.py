"""What the ray caster skips, by its own code (asc_rays.cuh) as host C++ with a
warp's lanes side by side: images with skipping equal those that sample every
ray from end to end, bit for bit, and the samples marched stay near those of
fine pixels however coarse the pixels are and however long the volume is."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from autoscoper_gb300 import scene as S
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def hr(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("hr") / "libhost_beam.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "cpp", "host_beam.cpp")], check=True)
    lib = C.CDLL(so)
    lib.hr_cast.restype = None
    lib.hr_cast.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_float, C.c_float,
                            C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    return lib


def cast(hr, vol, m, vp, step, cutoff, w, h, skip):
    nz, ny, nx = vol.shape
    out, counts = np.zeros((h, w), np.float32), (C.c_longlong * 4)()
    mf, vpf = np.ascontiguousarray(m, np.float32), np.ascontiguousarray(vp, np.float32)
    hr.hr_cast(vol.ctypes.data, nx, ny, nz, skip, mf.ctypes.data, vpf.ctypes.data, step, cutoff, w, h, out.ctypes.data,
               counts)
    return out, list(counts)


def lone_voxels(rng, shape):
    vol = np.full(shape, 100, np.uint16)
    vol[rng.random(shape) < 0.003] = 900
    d, h, w = shape
    vol[d // 3:2 * d // 3, h // 3:2 * h // 3, w // 3:2 * w // 3] = 1500
    vol.reshape(-1)[[0, -1]] = 900
    return vol


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 2, 61), (40, 36, 44), (75, 33, 90)])  # depth, height, width
@pytest.mark.parametrize("scale", [(1.0, 1.0, 1.0), (0.2, 1.0, 2.5)])
def test_skipping_changes_no_bit(hr, shape, scale):
    rng = np.random.default_rng(sum(shape))
    sc = S.make_scene([shape], 1.0, (64, 64), 1.0, filters="none", seed=3)
    sc.volumes[0] = S.Volume(lone_voxels(rng, shape), scale)
    sc.pivots[0] = S.pivot_matrix(sc.volumes[0])
    tr = O.Tracker(sc)
    vol = np.ascontiguousarray(tr.vd[0].data, np.uint16)
    seen = 0
    for k, (w, h, step) in enumerate([(41, 30, 0.4), (17, 9, 0.7), (8, 5, 3.1), (3, 3, 0.11), (1, 1, 0.5)]):
        # nearer to the camera, farther from it, almost in it
        at = np.zeros(3)
        at[k % 2] = (0.0, 300.0, -4000.0, 0.0, 580.0)[k]
        ok, m, vp, _, _ = tr.view_setup(0, k % 2, S.pose_centered_at(sc.volumes[0], at, rng.uniform(-180, 180, 3)))
        if not ok:
            continue
        full, n = cast(hr, vol, m, vp, step, 400 / 65535.0, w, h, 0)
        skip, marched = cast(hr, vol, m, vp, step, 400 / 65535.0, w, h, 1)
        assert n[1] == n[0] == marched[0]
        assert full.tobytes() == skip.tobytes()
        seen += int(full.any())
    assert seen >= 2


def ellipsoid(n):
    ax = np.arange(n) - (n - 1) / 2
    r2 = (ax / (0.31 * n)) ** 2
    vol = np.full((n, n, n), 200, np.uint16)
    vol[r2[None, None, :] + r2[None, :, None] + r2[:, None, None] <= 1] = 1500
    return vol


@pytest.mark.parametrize("n", [160, 224])
def test_coarse_pixels_keep_their_skipping(hr, n):
    """One volume at 1 to 8 voxels a pixel: the marched share of the samples is
    that of the finest pixels within a tenth (the ellipsoid fills an eighth of
    the box)."""
    sc = S.make_scene([(8, 8, 8)], 0.5, (64, 64), 1.0, filters="none", seed=5)
    sc.volumes[0] = S.Volume(ellipsoid(n), (0.5,) * 3)
    sc.pivots[0] = S.pivot_matrix(sc.volumes[0])
    tr = O.Tracker(sc)
    vol = np.ascontiguousarray(tr.vd[0].data, np.uint16)
    ok, m, _, _, _ = tr.view_setup(0, 0, S.pose_centered_at(sc.volumes[0], (0, 0, 0), (12, -7, 20)))
    half = 3 ** 0.5 * n * 0.5 / 2 / 300  # the turned box from 600 mm
    share = {}
    for voxels in (1, 2, 3, 3.5, 4, 5, 6, 8):
        px = int(2 * half * 300 / 0.5 / voxels)
        args = (hr, vol, m, [-half, -half, 2 * half, 2 * half], 0.25, 400 / 65535.0, px, px)
        img, c = cast(*args, 1)
        share[voxels] = c[1] / c[0]
        if voxels > 3:
            assert img.any() and img.tobytes() == cast(*args, 0)[0].tobytes()
    assert share[1] < 0.2
    assert all(s <= 1.1 * share[1] for s in share.values()), share


def test_long_volumes_keep_their_skipping(hr):
    """Rays along 3000 voxels, whose 64 intervals are longer than any clearance
    can answer for: two occupied stretches of 60 voxels are marched to the
    march blocks' granularity (64 samples at either end of each)."""
    vol = np.full((12, 12, 3000), 100, np.uint16)
    vol[3:9, 3:9, 700:760] = 900
    vol[3:9, 3:9, 2100:2160] = 900
    # a camera on the x axis, 2 box lengths before the unit box, looking along x
    m = np.float32([[0, 0, -1, -2.0], [1, 0, 0, 0.5], [0, 1, 0, -0.5]])
    vp = [-0.2, -0.2, 0.4, 0.4]
    full, n = cast(hr, vol, m, vp, 0.5 / 3000, 400 / 65535.0, 9, 7, 0)
    skip, c = cast(hr, vol, m, vp, 0.5 / 3000, 400 / 65535.0, 9, 7, 1)
    assert full.any() and full.tobytes() == skip.tobytes()
    # each stretch of 120 samples and a block of 64 at either end, on every ray
    assert 0 < c[1] <= full.size * 2 * (120 + 2 * 64)
