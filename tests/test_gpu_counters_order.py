"""The work counters of an evaluation that is still queued on a stream of the
caller's: asked for at once, they are those of that evaluation, as after a
wait; and the phase times alone count no samples."""
import ctypes as C

import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, scene as S

pytestmark = pytest.mark.gpu


def _counters(eng):
    out, n = (C.c_ulonglong * 4)(), C.c_int()
    L.call("asc_engine_counters", eng.handle, out)
    L.call("asc_engine_exact_rays", eng.handle, C.byref(n))
    return out[0], out[1], out[2], n.value


def test_counters_follow_a_queued_evaluation():
    sc = S.make_scene([(64, 60, 72)], 0.8, (256, 256), 0.5, filters="chain", seed=4)
    api.render_targets(sc)
    n = 64
    eng = api.Engine(sc, max_items=n)
    rng = np.random.default_rng(3)
    few = api.DeviceArray.from_host(rng.uniform(-1, 1, (4, 6)))
    many = api.DeviceArray.from_host(rng.uniform(-3, 3, (n, 6)))
    bones = api.DeviceArray.from_host(np.zeros(n, np.int32))
    cost = api.DeviceArray(n, np.float64)
    s = C.c_void_p()
    L.call("asc_stream_create", C.byref(s))
    try:
        want = {}
        for k, m in ((4, few), (n, many)):
            eng.eval_device(k, bones, m, cost, s)
            L.call("asc_stream_sync", s)
            want[k] = _counters(eng)
        assert want[4][0] < want[n][0]
        for k, m in ((4, few), (n, many), (4, few)):
            for _ in range(10):  # a queue of the other batch before it
                eng.eval_device(n + 4 - k, bones, many if k == 4 else few, cost, s)
            eng.eval_device(k, bones, m, cost, s)
            assert _counters(eng) == want[k]
        L.call("asc_engine_profile", eng.handle, 1)
        eng.eval_device(n, bones, many, cost, s)
        ms, pixels = (C.c_float * 3)(), C.c_ulonglong()
        L.call("asc_engine_stats", eng.handle, ms, None, C.byref(pixels))
        assert min(ms) > 0 and pixels.value == want[n][1]
    finally:
        L.call("asc_stream_sync", s)
        L.call("asc_stream_destroy", s)


def test_counters_follow_a_graph():
    """An evaluation captured into a graph of the caller's leaves no event of its
    own; after a replay and a wait the counters are its."""
    torch = pytest.importorskip("torch")
    sc = S.make_scene([(40, 36, 44)], 1.0, (96, 96), 1.0, filters="sobel", seed=4)
    api.render_targets(sc)
    eng = api.Engine(sc, max_items=8)
    man = np.random.default_rng(3).uniform(-1, 1, (8, 6))
    want_cost, _ = eng.eval(np.zeros(8, np.int32), man)
    want = _counters(eng)
    bones, mans = api.DeviceArray.from_host(np.zeros(8, np.int32)), api.DeviceArray.from_host(man)
    cost = api.DeviceArray(8, np.float64)
    g = torch.cuda.CUDAGraph()
    L.call("asc_device_sync")
    with torch.cuda.graph(g):
        eng.eval_device(8, bones, mans, cost, torch.cuda.current_stream().cuda_stream)
    eng.eval(np.zeros(2, np.int32), np.zeros((2, 6)))
    g.replay()
    torch.cuda.synchronize()
    assert _counters(eng) == want
    assert np.array_equal(cost.to_host(), want_cost)
