"""A server that has run dry keeps a small engine for its next requests, without
the caller's stream: that may have been destroyed by then."""
import ctypes

import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def _drain(srv):
    for _ in range(200):
        if not srv.round():
            return srv.poll()
    raise AssertionError("the server does not finish")


@pytest.mark.parametrize("second", ["own", "new"])
def test_idle_server_outlives_the_callers_stream(native, second):
    import torch
    rt = torch.cuda.cudart()
    torch.cuda.init()
    reqs = [scenes.random_cluster(0, n=40), scenes.settling_box(n_side=4, max_iterations=200)]
    srv = native.NativeServer(precision=native.DV_PREC_FP64)
    for k, sc in enumerate(reqs):
        ptr = 0
        if k == 0 or second == "new":
            s = ctypes.c_void_p()
            assert int(rt.cudaStreamCreate(ctypes.addressof(s))) == 0
            ptr = s.value
        srv.set_stream(ptr)
        rid = srv.submit(sc, 7)
        assert [r["status"] for r in _drain(srv)] == [0]
        if ptr:
            assert int(rt.cudaStreamDestroy(ptr)) == 0
        g = native.NativeScene.from_scene(sc)
        g.step(7)
        for got, want in zip(srv.result_state(rid), g.state()):
            assert np.array_equal(got, want)
        g.close()
    srv.close()
