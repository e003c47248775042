"""The fused filter / NCC kernel where its tiles and four-column units are cut:
crops of every width modulo 4 around one and two tiles, chains of each halo (the
rows and columns around a tile), every Gaussian kernel size with its own code
and the general one, and the reference's partial sums at sizes that drop pixels.
Against the plain per-operator form of the same evaluation, which runs other
kernels: both hold the NCC bar to FP64, so they lie within twice that bar."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S

pytestmark = pytest.mark.gpu

CHAINS = {
    "none": [],
    "contrast5": [S.Filter.contrast_filter(alpha=1.5, beta=0.7, size=5)],
    "contrast+sobel": [S.Filter.contrast_filter(alpha=2.5, beta=0.9), S.Filter.sobel(blend=0.3)],
    "gauss3": [S.Filter.gaussian(radius=0.4)],
    "gauss5": [S.Filter.gaussian(radius=0.7), S.Filter.sobel()],
    "sharpen11": [S.Filter.sharpen(radius=1.7, contrast=2.0, threshold=0.01), S.Filter.sobel()],
    "gauss13+sharpen7": [S.Filter.gaussian(radius=2.0), S.Filter.sharpen(radius=1.0)],
    "gauss17": [S.Filter.gaussian(radius=2.7)],
}


def bar(ncc):
    return 2e-5 * max(abs(ncc), 1e-2)


@pytest.mark.parametrize("chain", list(CHAINS))
@pytest.mark.parametrize("render", [(45, 131), (98, 96), (143, 53)])
def test_tiles_match_the_plain_operators(chain, render):
    w, h = render
    sc = S.make_scene([(30, 33, 41)], 1.0, render, 120.0 / max(w, h), filters="none", seed=11, bone_offsets=[(2, 0, 1)])
    for v in sc.views:
        v.drr_filters = CHAINS[chain]
        v.rad_filters = CHAINS[chain]
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
