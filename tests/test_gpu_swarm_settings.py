"""A swarm run depends on its own arguments and the options in force, not on
the iteration that an earlier run of the same engine captured."""
import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    sc = S.make_scene([(40, 36, 44)], 1.0, (96, 96), 1.0, filters="sobel", seed=4)
    api.render_targets(sc)
    sc.poses = [S.perturb(sc.truth[0], np.random.default_rng(2), 4.0, 4.0)]  # the best is not where a particle starts
    return sc


@pytest.mark.parametrize("seed", [2**53, 2**63])
def test_seeds_that_round_to_one_double(scene, seed):
    used = api.Engine(scene, max_items=12)
    used.pso(12, 4, seed=seed)
    got = used.pso(12, 4, seed=seed + 1)
    want = api.Engine(scene, max_items=12).pso(12, 4, seed=seed + 1)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def _marched(eng):
    import ctypes as C
    out = (C.c_ulonglong * 4)()
    L.call("asc_engine_counters", eng.handle, out)
    return out[2]


def test_skipping_switched_off_is_off_for_a_swarm(scene):
    eng = api.Engine(scene, max_items=12)
    skip = eng.pso(12, 2, seed=5)
    few = _marched(eng)
    try:
        L.call("asc_set_option", L.ASC_OPT_EMPTY_SKIP, 0)
        full = eng.pso(12, 2, seed=5)
        every = _marched(eng)
    finally:
        L.call("asc_set_option", L.ASC_OPT_EMPTY_SKIP, 1)
    assert np.array_equal(skip[0], full[0]) and np.array_equal(skip[1], full[1])
    assert every > 2 * few  # about seven eighths of the phantom's box lies below the cutoff
