"""Bilateral rows added one by one past the sizes at which their arrays grow (16
rows, then by doubling) and past the tile of rows that every scene has room for
(512): the same bits as the oracle, and the rows' impulses."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16, 17, 35, 512, 513, 700])
def test_many_rows_equal_the_oracle(native, oracle_mod, rows):
    sc = scenes.random_cluster(5, n=720, max_iterations=12)
    first = int(np.argmax(sc.fixed == 0))
    sc.bilateral = [(3 * (first + i), -1, 0.0, 0.0) for i in range(rows)]
    g = native.NativeScene.from_scene(sc)
    o = oracle_mod.OracleScene(sc)
    for _ in range(2):
        g.step(1)
        o.step(1)
    assert g.stats()["num_contacts"] == o.stats()["num_contacts"] > 0
    for x, y in zip(g.state(), o.state()):
        assert np.array_equal(x, y)
    assert np.array_equal(g.gamma(), o.gamma())
    assert len(g.bilateral_gamma()) == rows
    g.close()
