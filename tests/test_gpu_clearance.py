"""Skipping by the clearance grid changes no bit: the ray caster's images and
the engine's costs with skipping on equal those that sample every ray from end
to end, at the sizes where grid cells, grid blocks (32 voxels) and beams
(8 x 4 pixels) are cut, for pixels and steps from much finer to much coarser
than a voxel, and for rays along the axes."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, geometry as G, scene as S

pytestmark = pytest.mark.gpu


def both(f):
    try:
        L.call("asc_set_option", L.ASC_OPT_EMPTY_SKIP, 0)
        full = f()
    finally:
        L.call("asc_set_option", L.ASC_OPT_EMPTY_SKIP, 1)
    return full, f()


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (31, 32, 33), (64, 17, 16), (63, 65, 70)])  # depth, height, width
@pytest.mark.parametrize("storage", [L.ASC_STORE_U16, L.ASC_STORE_F32])
def test_raycast_skips_nothing_that_counts(shape, storage):
    rng = np.random.default_rng(sum(shape))
    data = np.full(shape, 100, np.uint16)
    data[rng.random(shape) < 0.004] = 900  # lone voxels anywhere, the faces among them
    data.reshape(-1)[[0, -1]] = 900
    d, h, w = shape
    data[d // 3:2 * d // 3, h // 3:2 * h // 3, w // 3:2 * w // 3] = 1500
    vol = api.DeviceVolume(S.Volume(data, (1.0, 1.0, 1.0)), storage)
    size = float(max(shape))
    seen = False
    for k, (step, width, height) in enumerate([(0.5, 61, 47), (0.07 * size, 33, 9), (3.3, 8, 100), (0.21, 5, 3)]):
        for angles in ((0, 0, 0), (90, 0, 90), tuple(rng.uniform(-180, 180, 3))):
            pose = G.from_xyzypr([0, 0, 0, *angles])
            eye = G.translate(G.identity(), [0, 0, 3.0 * size])
            centre = G.point(pose, np.array([w / 2.0, h / 2.0, -d / 2.0]))
            pose = G.translate(pose, -centre)
            imv = G.row_matrix(G.inverse(G.mul(G.inverse(eye), pose)))
            vp = [-0.5, -0.5, 1.0, 1.0] if k % 2 == 0 else [-0.31, -0.42, 0.83, 0.77]
            full, skip = both(lambda: api.raycast(vol, imv, vp, step, 50.0, 400 / 65535.0, width, height).to_host())
            assert np.array_equal(full, skip), (shape, step, angles)
            seen |= bool(full.any())
    assert seen


@pytest.mark.parametrize("render", [(96, 80), (17, 233)])
def test_engine_skips_nothing_that_counts(render):
    sc = S.make_scene([(33, 47, 62), (30, 64, 31)], 1.0, render, 96.0 / render[0], filters="none", seed=9,
                      bone_offsets=[(0, 0, -9), (3, -2, 12)])
    api.render_targets(sc)
    rng = np.random.default_rng(3)
    bones = rng.integers(0, 2, 33).astype(np.int32)
    man = rng.uniform(-6, 6, (33, 6))
    full, skip = both(lambda: api.Engine(sc, max_items=33).eval(bones, man))
    assert np.array_equal(full[0], skip[0]) and np.array_equal(full[1], skip[1])


def test_engine_counts_the_reference_samples():
    """asc_engine_counters: the reference's samples from the crops' records
    (the rays that meet nothing among them), the marched ones a part of them."""
    import ctypes as C
    from oracle import oracle as O
    sc = S.make_scene([(40, 36, 44)], 1.0, (96, 96), 1.0, filters="sobel", seed=4)
    api.render_targets(sc)
    eng = api.Engine(sc, max_items=2)
    eng.eval([0], np.zeros((1, 6)))
    out = (C.c_ulonglong * 4)()
    for _ in range(2):  # asking twice counts once
        L.call("asc_engine_counters", eng.handle, out)
    tr = O.Tracker(sc)
    want = 0
    for v in range(2):
        ok, m, vp, w, h = tr.view_setup(0, v, tr.compose(0, np.zeros(6)))
        rp = sc.ray[v][0]
        want += int(O.raycast(tr.vd[0], m, np.float32(vp).astype(np.float64), float(np.float32(rp.step)), 1.0,
                              float(np.float32(rp.cutoff)), w, h, want_samples=True)[1].sum())
    assert out[0] == want
    assert 0 < out[2] <= min(out[0], out[3])
