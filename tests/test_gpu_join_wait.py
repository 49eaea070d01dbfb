"""The wait of a team that forms ends after its limit, and the limit starts again
while other teams make progress."""
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passes", [0, 1, 12])
def test_join_wait_runs_out_after_the_last_progress(native, passes):
    timed_out, after, bits = native.selftest_bounded_join(40, passes)
    assert timed_out == 1 and bits == 1  # the barrier timeout
    if passes:
        # 12 passes are three limits: without them the wait would have ended before
        assert 39.0 <= after <= 60.0, after
    b = native.NativeBatch([scenes.ball_on_ground(), scenes.random_cluster(0, n=40)])
    b.step(2)
    assert [s["status"] for s in b.scene_stats()] == [0, 0]
    b.close()


def test_join_selftest_rejects_bad_arguments(native):
    for limit, passes in ((0, 1), (501, 1), (40, -1), (40, 101)):
        with pytest.raises(native.DvError):
            native.selftest_bounded_join(limit, passes)
