"""A background mask under the SAD cost (the fused kernel masks the DRR, then
k_sad sums over the pixels left): batched and plain against the FP64 oracle,
per view within 1e-5 of the SAD and FP32's partial sums, for background images
of other sizes than the radiograph; and the threshold matters."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coverage", [L.ASC_SUM_TREE, L.ASC_SUM_FULL])
@pytest.mark.parametrize("size", [(112, 112), (31, 57)])
def test_background_under_sad_matches_the_oracle(size, coverage):
    sc = S.make_scene([(40, 48, 56), (36, 30, 44)], 1.0, (112, 112), 0.9, filters="sobel", seed=19,
                      bone_offsets=[(0, 0, -12), (4, -3, 14)])
    sc.cf_model = 1
    w, h = size
    yy, xx = np.mgrid[0:h, 0:w]
    for i, v in enumerate(sc.views):
        v.background = (0.5 + 0.5 * np.sin(16.0 * xx / w + i) * np.cos(10.0 * yy / h)).astype(np.float32)
        v.bg_threshold = 0.4
    api.render_targets(sc)
    tr = O.Tracker(sc, tree=coverage == L.ASC_SUM_TREE)
    rng = np.random.default_rng(23)
    n = 8
    bones = rng.integers(0, 2, n).astype(np.int32)
    man = rng.uniform(-2, 2, (n, 6))
    eng = api.Engine(sc, max_items=n, coverage=coverage)
    want = np.array([tr.track_frame(int(bones[k]), tr.compose(int(bones[k]), man[k])) for k in range(n)])
    for plain in (False, True):
        cost, got = eng.eval(bones, man, plain=plain)
        assert (np.abs(got - want) <= 1e-5 * want + 2e-6).all(), (plain, np.abs(got / want - 1).max())
        assert np.allclose(cost, got.sum(1), rtol=1e-15)
    for v in sc.views:
        v.bg_threshold = -1.0
    _, free = api.Engine(sc, max_items=n, coverage=coverage).eval(bones, man)
    assert (free > 1.01 * want).all()  # the mask leaves out pixels that the DRR's keeps
