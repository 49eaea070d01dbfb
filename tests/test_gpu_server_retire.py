"""A request over the partner limit is retired (DV_ERR_ARG, no steps done) also
where its scene is the only one in the engine, and the requests behind it are
served."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def _drain(srv):
    for _ in range(200):
        if not srv.round():
            return {r["id"]: r for r in srv.poll()}
    raise AssertionError("the server does not finish")


@pytest.mark.parametrize("solver", [1, 5, 6])
@pytest.mark.parametrize("max_active", [4096, 1])
def test_lone_request_over_the_partner_limit_is_retired(native, max_active, solver):
    bad = scenes.raspberry(8193, ballast=8200)
    bad.params["solver"] = solver
    good = scenes.random_cluster(0, n=40)
    srv = native.NativeServer(precision=native.DV_PREC_FP64, max_active=max_active)
    first = srv.submit(bad, 4)
    if max_active == 1:
        second = srv.submit(good, 5)
        got = _drain(srv)
    else:
        got = _drain(srv)
        second = srv.submit(good, 5)
        got.update(_drain(srv))
    assert got[first]["status"] == 1 and got[first]["nsteps"] == 0
    assert got[second]["status"] == 0 and got[second]["nsteps"] == 5
    g = native.NativeScene.from_scene(good)
    g.step(5)
    for x, y in zip(srv.result_state(second), g.state()):
        assert np.array_equal(x, y)
    g.close()
    srv.close()
