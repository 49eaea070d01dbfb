"""The PGS sweep updates contacts in rounds, each when it is next for both of
its bodies: the same bits as the oracle's sweep, contact by contact, where all
contacts share a body, where windows of 256 end inside a body's contacts, and
where impulses overflow at a fixed body (its velocity then turns to NaN, and
the sweep keeps the fixed bodies' order too)."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def _overflow(speed):
    sc = scenes.random_cluster(11, n=64)
    first = int(np.argmax(sc.fixed == 0))
    sc.vel[first:first + 3] = speed
    return sc


@pytest.mark.parametrize("make,iterations", [
    (lambda: scenes.raspberry(255), 5), (lambda: scenes.raspberry(257), 5),
    (lambda: scenes.raspberry(600), 4), (lambda: scenes.crowd(300), 4),
    (lambda: scenes.settling_box(n_side=7, spacing=0.1), 20),
    (lambda: _overflow(1e160), 3), (lambda: _overflow(1e308), 3)])
def test_sweep_in_rounds_equals_the_oracle(native, oracle_mod, make, iterations):
    sc = make()
    sc.params.update(solver=6, max_iterations=iterations)
    g = native.NativeScene.from_scene(sc)
    o = oracle_mod.OracleScene(sc)
    g.step(1, raise_on_error=False)
    try:
        o.step(1)
    except Exception:
        pass
    assert g.stats()["num_contacts"] == o.stats()["num_contacts"] > 0
    assert np.array_equal(g.gamma(), o.gamma(), equal_nan=True)
    assert np.array_equal(g.state()[1], o.state()[1], equal_nan=True)
    g.close()
