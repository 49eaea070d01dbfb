"""The rounds of a PGS sweep end: one whose counts never come up stops with an
error bit that a step reports as a timeout, and the device stays usable."""
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def test_sweep_without_a_next_contact_ends(native):
    assert native.selftest_stalled_sweep(0) == (0, 0)
    assert native.selftest_stalled_sweep(1) == (1, 1)  # the barrier-timeout bit
    sc = scenes.ball_on_ground()
    sc.params.update(solver=6, max_iterations=20)
    g = native.NativeScene.from_scene(sc)
    g.step(2)
    assert g.stats()["num_contacts"] == 1 and g.stats()["status"] == 0
    g.close()
