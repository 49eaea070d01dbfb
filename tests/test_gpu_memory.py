"""Device memory that engines hold: a scene whose contact buffers have grown holds
what one created for those contacts holds, an idle server holds no more than its
budget, and a scene served from parked memory has the same bits."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture()
def used():
    """Device bytes in use since the fixture's start, the modules loaded."""
    import gc

    import torch
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    gc.collect()  # scenes that earlier tests left behind

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    return lambda start=None: free() if start is None else start - free()


def _crowd(n=1500, spread=1.0):
    sc = scenes.crowd(n, max_iterations=1)
    sc.pos[:] = sc.pos.mean(axis=0) + spread * (sc.pos - sc.pos.mean(axis=0))
    return sc


def test_grown_scene_holds_what_a_fresh_one_does(native, used):
    def held(steps):
        # contacts grow from some 300,000 to 992,079 where the state is drawn together
        sc = _crowd()
        start = used()
        g = native.NativeScene.from_scene(sc)
        for spread in steps:
            g.set_state(_crowd(spread=spread).pos, np.zeros_like(sc.pos))
            g.step(1, raise_on_error=False)
        nc = g.stats()["num_contacts"]
        out = used(start)
        g.close()
        return out, nc
    held([1.0])  # loads what a step loads
    fresh, nc0 = held([1.0])
    grown, nc1 = held([1.8, 1.0])
    assert nc0 == nc1 > 900000
    # 464 bytes per slot and 1.24 million slots; the buffers before took over 100 MB
    assert grown < fresh + 50 * MB, (grown / MB, fresh / MB)


def test_idle_server_holds_no_more_than_its_budget(native, used):
    # a crowd's contacts outgrow the estimate per body by far
    sc = _crowd(800)

    def burst(srv, n=3):
        ids = [srv.submit(sc, 2) for _ in range(n)]
        while srv.round():
            pass
        srv.poll()
        return ids
    warm = native.NativeServer(precision=native.DV_PREC_FP64)
    burst(warm)
    warm.close()
    start = used()
    for budget in (40e6, 4e9):
        srv = native.NativeServer(precision=native.DV_PREC_FP64, hbm_budget_bytes=budget)
        burst(srv)
        assert used(start) <= min(budget, 1 << 30) + 4 * MB, (budget, used(start) / MB)
        ids = burst(srv, 1)
        g = native.NativeScene.from_scene(sc)
        g.step(2)
        for x, y in zip(srv.result_state(ids[0]), g.state()):
            assert np.array_equal(x, y)
        g.close()
        srv.close()
    assert used(start) <= 4 * MB


def test_resident_scene_stays_within_its_estimate(native, used):
    """1.5 million bodies far apart: 96 MB for the blocks' granularity (some 45
    blocks of 2 MB at most); the estimate is 3.5 GB."""
    n = 1_500_000
    sc = scenes.free_balls(n)
    small = native.NativeServer(precision=native.DV_PREC_FP64)
    small.submit(scenes.free_balls(3), 2)
    while small.round():
        pass
    small.close()
    start = used()
    srv = native.NativeServer(precision=native.DV_PREC_FP64, hbm_budget_bytes=2.4e3 * n)
    srv.submit(sc, 9)  # more than a round
    assert srv.round()
    estimate = srv.stats()["bytes_in_use"]
    held = used(start)
    srv.close()
    assert held <= estimate + 96 * MB, (held / n, estimate / n)
