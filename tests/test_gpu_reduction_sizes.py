"""asc_ncc and asc_hdist where the sums over their 4096-pixel chunks change form
(NCC: one wave of 304 blocks of 1024 threads, or blocks of 256; SAD: one warp
up to 64 chunks, then the block), with the last chunk full and ragged, against NumPy in 64 bits.  NCC: compensated sums and FP64, 1e-10.
SAD: FP32 sums of 4096 values a chunk (16 a thread, then 8 levels), below 24 x
2^-24 of the sum, and FP32 means, another 2 x 2^-24: 2e-6."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [63 * 4096, 64 * 4096 - 5, 64 * 4096, 64 * 4096 + 1, 65 * 4096, 304 * 4096,
                               304 * 4096 + 1, 305 * 4096 - 1, 307 * 4096 + 33, 1025 * 4096 + 7])
def test_merge_of_every_form(n):
    rng = np.random.default_rng(n)
    f, g = (rng.uniform(0, 1, (1, n)).astype(np.float32) for _ in range(2))
    g = (0.6 * f + 0.4 * g + np.linspace(0, 3, n, dtype=np.float32)).astype(np.float32)  # chunks of unlike means
    m = (rng.uniform(0, 1, (1, n)) > 0.4).astype(np.float32)
    m[0, 4096 * 5:4096 * 7] = 0  # chunks without a pixel
    F, G, M = f.astype(np.float64), g.astype(np.float64), m.astype(np.float64)
    df, dg, dm = (api.DeviceArray.from_host(x) for x in (f, g, m))
    # the means run over every pixel and count the mask's, the sums over the mask's
    mf, mg = F.sum() / M.sum(), G.sum() / M.sum()
    a, b = (F - mf)[m > 0.5], (G - mg)[m > 0.5]
    want = (a * b).sum() / np.sqrt((a * a).sum() * (b * b).sum())
    sad = np.abs(a - b).sum()
    for _ in range(2):  # the scratch is in order after a call
        assert abs(api.ncc(df, dg, dm, L.ASC_SUM_FULL) - want) < 1e-10
        assert abs(api.hdist(df, dg, dm, L.ASC_SUM_FULL) - sad) < 2e-6 * sad
