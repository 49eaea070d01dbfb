"""A PGS sweep that starts again in the strict order, on scenes whose team has
several members (one per 256 bodies): the same bits as the oracle's sweep,
at the first iteration and at later ones."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,speed", [(500, 1e160), (900, 1e160), (900, 1e308), (2500, 1e308)])
def test_restarted_sweep_of_a_team_equals_the_oracle(native, oracle_mod, n, speed):
    sc = scenes.random_cluster(11, n=n)
    first = int(np.argmax(sc.fixed == 0))
    sc.vel[first:first + 3] = speed
    sc.params.update(solver=6, max_iterations=4)
    g = native.NativeScene.from_scene(sc)
    o = oracle_mod.OracleScene(sc)
    g.step(1, raise_on_error=False)
    try:
        o.step(1)
    except Exception:
        pass
    assert g.stats()["num_contacts"] == o.stats()["num_contacts"] > 256
    assert np.array_equal(g.gamma(), o.gamma(), equal_nan=True)
    assert np.array_equal(g.state()[1], o.state()[1], equal_nan=True)
    g.close()
