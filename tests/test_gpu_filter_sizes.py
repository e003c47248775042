"""The plain filters at every kernel size with code of its own and at sizes of
the general kernel, on images cut around the 32-pixel tiles, against the FP64
oracle.  Two FP32 passes of K <= 31 taps summing to 1 on values below 1 err by
less than 2 K 2^-24 < 4e-6; Sharpen doubles the difference to the blur."""
import numpy as np
import pytest

from autoscoper_gb300 import api, scene as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (31, 33), (64, 32), (5, 71), (97, 3)])
def test_filters_of_every_size(shape):
    x = np.random.default_rng(shape[0]).uniform(0, 1, shape).astype(np.float32)
    dx = api.DeviceArray.from_host(x)
    for radius in (0.4, 0.7, 1.0, 1.4, 1.7, 2.0, 2.7, 5.0):  # 3, 5, 7, 9, 11, 13, 17, 31 taps
        got = api.apply_filter(S.Filter.gaussian(radius), dx).to_host()
        assert np.abs(got - O.apply_filter(S.Filter.gaussian(radius), x)).max() < 4e-6, radius
        f = S.Filter.sharpen(radius, 1.0, 0.0)
        assert np.abs(api.apply_filter(f, dx).to_host() - O.apply_filter(f, x)).max() < 8e-6, radius
    for size in (1, 2, 3, 4, 5, 6, 7):
        f = S.Filter.contrast_filter(1.7, 0.6, size=size)
        ref = O.apply_filter(f, x)
        assert np.abs(api.apply_filter(f, dx).to_host() - ref).max() < 3e-5 * max(1.0, np.abs(ref).max()), size
