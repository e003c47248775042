"""The filter / NCC kernel over its chains' halo: at least the resident blocks
per SM that a tile and three square stage buffers with its halo
leave room for (three up to a halo of 12, two up to 22), and the costs of chains of
every halo against the plain per-operator form, both within the NCC bar of
FP64."""
import ctypes as C

import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S

pytestmark = pytest.mark.gpu

RADIUS = {1: 0.4, 2: 0.7, 3: 1.0, 4: 1.4, 5: 1.7, 6: 2.0, 8: 2.7, 15: 5.0}  # of a blur of 2 k + 1 taps


def chain(halo):
    """Sobel, then blurs of both kinds, down to the halo: continuous filters, so
    that rounding decides nothing (Contrast has a step at a mean of 0.01,
    Sharpen at its threshold)."""
    out = []
    if halo > 2:
        out = [S.Filter.sobel(1.0, 0.3)]
        halo -= 1
    if halo > 22:
        out.append(S.Filter.sharpen(RADIUS[15], 1.0, 0.0))
        halo -= 15
    while halo:
        r = min(halo, 6) if halo != 8 else 8
        out.append(S.Filter.gaussian(RADIUS[r]) if len(out) % 2 else S.Filter.sharpen(RADIUS[r], 1.5, 0.0))
        halo -= r
    return out


@pytest.fixture(scope="module")
def scene():
    sc = S.make_scene([(40, 48, 56)], 1.0, (131, 117), 0.9, filters="none", seed=7)
    api.render_targets(sc)
    return sc


@pytest.mark.parametrize("halo", [0, 1, 2, 3, 7, 8, 10, 12, 13, 17, 20, 21, 22, 23, 30, 42])
def test_blocks_and_costs(scene, halo):
    ch = chain(halo)
    assert len(ch) <= 8
    for v in scene.views:
        v.drr_filters = v.rad_filters = ch
    eng = api.Engine(scene, max_items=6)
    cfg, blocks = L.LaunchConfig(), C.c_int()
    L.call("asc_engine_get_launch", eng.handle, C.byref(cfg), C.byref(blocks))
    assert blocks.value >= (3 if halo <= 12 else 2 if halo <= 22 else 1)
    man = np.random.default_rng(halo).uniform(-3, 3, (6, 6))
    _, got = eng.eval(np.zeros(6, np.int32), man)
    _, ref = eng.eval(np.zeros(6, np.int32), man, plain=True)
    assert (np.abs(got - ref) <= 2e-5 * np.maximum(np.abs(1.0 - ref), 1e-2)).all()
