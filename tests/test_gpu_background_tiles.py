"""The fused filter / NCC kernel's background mask, whose film-plane mapping is
tabulated per tile column and row in the radiograph's tables: crops cut around
one and two tiles, chains with and without a halo (where the tables lie), and
background images of other sizes than the radiograph.  Against the plain
per-operator form of the same evaluation, which maps every pixel by itself:
both hold the NCC bar to FP64, so they lie within twice that bar."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S

pytestmark = pytest.mark.gpu

CHAINS = {
    "none": [],
    "sobel": [S.Filter.sobel()],
    "gauss13+sharpen7": [S.Filter.gaussian(radius=2.0), S.Filter.sharpen(radius=1.0)],
}


def bar(ncc):
    return 2e-5 * max(abs(ncc), 1e-2)


@pytest.mark.parametrize("chain", list(CHAINS))
@pytest.mark.parametrize("threshold", [0.0, 0.4])
@pytest.mark.parametrize("render,size", [((45, 131), (45, 131)), ((98, 96), (31, 257)), ((143, 53), (7, 5))])
def test_background_matches_the_plain_operators(chain, threshold, render, size):
    w, h = render
    sc = S.make_scene([(30, 33, 41)], 1.0, render, 120.0 / max(w, h), filters="none", seed=11, bone_offsets=[(2, 0, 1)])
    yy, xx = np.mgrid[0:size[1], 0:size[0]]
    for i, v in enumerate(sc.views):
        v.drr_filters = CHAINS[chain]
        v.rad_filters = CHAINS[chain]
        v.background = (0.5 + 0.5 * np.sin(9.0 * xx / size[0] + i) * np.cos(7.0 * yy / size[1])).astype(np.float32)
        v.bg_threshold = threshold
    api.render_targets(sc)
    rng = np.random.default_rng(len(chain))
    n = 9
    man = np.concatenate([rng.uniform(-12, 12, (n, 3)), rng.uniform(-8, 8, (n, 3))], 1)
    for coverage in (L.ASC_SUM_TREE, L.ASC_SUM_FULL):
        eng = api.Engine(sc, max_items=n, coverage=coverage)
        _, got = eng.eval(np.zeros(n, np.int32), man)
        _, want = eng.eval(np.zeros(n, np.int32), man, plain=True)
        for a, b in zip(got.ravel(), want.ravel()):
            assert a == b or abs(a - b) <= bar(1.0 - b), (a, b)
