"""asc_raycast on one volume from several streams, threads and graphs, with
cutoffs in turn: every image equals the one cast alone, bit for bit, though
the volume keeps one clearance grid and builds it anew for each cutoff."""
import ctypes as C
import threading

import numpy as np
import pytest

from autoscoper_gb300 import _lib as L
from autoscoper_gb300 import api, geometry as G, scene as S

pytestmark = pytest.mark.gpu

W, H = 120, 90
CUTOFFS = [c / 65535.0 for c in (300, 600, 1100, 150)]


@pytest.fixture(scope="module")
def volume():
    rng = np.random.default_rng(1)
    data = S.phantom((60, 72, 66), seed=2)
    data[rng.random(data.shape) < 0.002] = 1000
    return api.DeviceVolume(S.Volume(data, (1.0, 1.0, 1.0)))


def _imv():
    pose = G.from_xyzypr([0, 0, 0, 20, -35, 50])
    eye = G.translate(G.identity(), [0, 0, 200.0])
    pose = G.translate(pose, -G.point(pose, np.array([33.0, 36.0, -30.0])))
    return G.row_matrix(G.inverse(G.mul(G.inverse(eye), pose)))


def _cast(vol, cutoff, out, stream):
    m = np.ascontiguousarray(_imv(), np.float64)
    vp = np.array([-0.5, -0.4, 1.0, 0.8], np.float32)
    L.call("asc_raycast", vol.handle, m.ctypes.data_as(C.POINTER(C.c_double)), vp.ctypes.data_as(C.POINTER(C.c_float)),
           0.5, 60.0, cutoff, 1, out.ptr, W, H, stream)


@pytest.fixture(scope="module")
def alone(volume):
    imgs = []
    for c in CUTOFFS:
        out = api.DeviceArray((H, W))
        _cast(volume, c, out, None)
        imgs.append(out.to_host())
    assert all(not np.array_equal(imgs[0], i) for i in imgs[1:])
    return imgs


def test_a_captured_cast_keeps_its_grid(volume, alone):
    torch = pytest.importorskip("torch")
    graphs, outs = [], []
    for k in (0, 1, 1):  # a grid that was built before, one that was not, one that another graph reads
        if k == 0:
            _cast(volume, CUTOFFS[0], api.DeviceArray((H, W)), None)
        outs.append(api.DeviceArray((H, W)))
        graphs.append(torch.cuda.CUDAGraph())
        L.call("asc_device_sync")
        with torch.cuda.graph(graphs[-1]):
            _cast(volume, CUTOFFS[k], outs[-1], torch.cuda.current_stream().cuda_stream)
    for c in (2, 1, 3):
        out = api.DeviceArray((H, W))
        _cast(volume, CUTOFFS[c], out, None)
        for g in graphs:
            g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.to_host(), alone[c])
        for o, k in zip(outs, (0, 1, 1)):
            assert np.array_equal(o.to_host(), alone[k])


def test_streams_and_threads_cast_side_by_side(volume, alone):
    def work(first, results):
        streams = []
        for _ in range(3):  # with both threads more streams than the volume remembers
            s = C.c_void_p()
            L.call("asc_stream_create", C.byref(s))
            streams.append(s)
        outs = [(k % 4, api.DeviceArray((H, W))) for k in range(first, first + 24)]
        for n, (k, out) in enumerate(outs):
            _cast(volume, CUTOFFS[k], out, streams[n % 3])
        for s in streams:
            L.call("asc_stream_sync", s)
            L.call("asc_stream_destroy", s)
        results.extend((k, out.to_host()) for k, out in outs)

    for _ in range(4):
        results = []
        threads = [threading.Thread(target=work, args=(i, results)) for i in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(results) == 48
        for k, img in results:
            assert np.array_equal(img, alone[k])
