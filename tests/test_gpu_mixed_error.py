"""Mixed precision with FP64 refinement, a solver error in the FP32 phase: a plain
scene's step ends with the error and leaves positions, velocities and contact
forces as they were; a scene of a batch reports its error and is updated, as
without refinement."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(refine):
    # a pile whose solve backtracks: with no backtracks allowed it ends in an error
    sc = scenes.random_cluster(7, n=200)
    sc.params.update(max_backtracks=0, refine_iterations=refine)
    return sc


def test_plain_scene_stays(native):
    g = native.NativeScene.from_scene(_scene(50), precision=native.DV_PREC_MIXED)
    before = (*g.state(), g.fcontact())
    assert g.step(1, raise_on_error=False) == 4 and g.stats()["status"] == 4
    assert g.stats()["num_contacts"] > 0
    for x, y in zip((*g.state(), g.fcontact()), before):
        assert np.array_equal(x, y)
    g.close()


@pytest.mark.parametrize("refine", [0, 50])
def test_scene_of_a_batch_is_updated(native, refine):
    sc = _scene(refine)
    b = native.NativeBatch([sc, scenes.ball_on_ground()], precision=native.DV_PREC_MIXED)
    before = b.state(0)
    b.step(1)
    assert b.scene_stats()[0]["status"] == 4 and b.scene_stats()[1]["status"] == 0
    assert not np.array_equal(b.state(0)[0], before[0])
    b.close()
