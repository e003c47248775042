"""Contrast filters over images that hold infinities and NaN: inside, on the
border and at the edges of the 32-pixel tiles, against the FP64 oracle's
formula: the same infinities, zeros and NaN, and the finite pixels within the
filters' usual bound.  And the fused chain against the plain operators where a
first contrast makes infinities (0 to a negative power) that a second one
reads and a blur takes back to [0, 1]."""
import numpy as np
import pytest

from autoscoper_gb300 import api, scene as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("size", [1, 2, 3, 4, 5, 7])
def test_contrast_of_infinities(value, size):
    x = np.random.default_rng(size).uniform(0.1, 1, (75, 83)).astype(np.float32)
    for y, c in ((0, 0), (74, 82), (0, 40), (37, 0), (31, 31), (32, 64), (50, 20), (51, 21)):
        x[y, c] = value
    dx = api.DeviceArray.from_host(x)
    for alpha, beta in ((1.7, 0.6), (0.5, 0.5), (0.2, 1.5), (1.0, -0.5), (0.0, 0.0)):
        f = S.Filter.contrast_filter(alpha, beta, size=size)
        with np.errstate(invalid="ignore"):
            ref = O.apply_filter(f, x)
        got = api.apply_filter(f, dx).to_host()
        fin = np.isfinite(ref)
        assert np.array_equal(got[~fin], ref[~fin].astype(np.float32), equal_nan=True), (alpha, beta)
        assert np.abs(got[fin] - ref[fin]).max() < 3e-5 * max(1.0, np.abs(ref[fin]).max()), (alpha, beta)


def test_fused_chain_of_infinities_matches_the_plain_operators():
    sc = S.make_scene([(40, 36, 44)], 1.0, (101, 97), 1.0, filters="none", seed=4)
    api.render_targets(sc)
    for v in sc.views:
        v.drr_filters = [S.Filter.contrast_filter(1.0, -0.5), S.Filter.contrast_filter(0.5, 0.0), S.Filter.gaussian(1.0)]
        v.rad_filters = [S.Filter.gaussian(1.0)]
    eng = api.Engine(sc, max_items=4)
    man = np.random.default_rng(1).uniform(-2, 2, (4, 6))
    _, got = eng.eval(np.zeros(4, np.int32), man)
    _, ref = eng.eval(np.zeros(4, np.int32), man, plain=True)
    assert np.isfinite(ref).all()
    assert (np.abs(got - ref) <= 2e-5 * np.maximum(np.abs(1.0 - ref), 1e-2)).all()
