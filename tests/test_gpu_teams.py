"""Teams of the solve kernel: scenes whose tiles are fewer than, as many as and
more than the grid's CTAs, with several scenes per CTA and several CTAs per
scene, give the bits of the same scenes stepped alone."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu

# spheres on a lattice: 1, 2, ... tiles of 512 contacts, one scene without contacts
SIZES = (1, 7, 130, 180, 40, 900, 343, 2)


def _scenes():
    out = [scenes.random_cluster(20 + i, n=n, max_iterations=60) for i, n in enumerate(SIZES)]
    out.insert(3, scenes.free_balls(5))
    out.append(scenes.ball_on_ground())
    for sc in out:
        sc.params["tolerance"] = 1e-6
        sc.params["refine_iterations"] = 40
    return out


@pytest.fixture(scope="module")
def alone(native):
    got = {}
    for precision in (0, 1):
        for i, sc in enumerate(_scenes()):
            g = native.NativeScene.from_scene(sc, precision=precision)
            g.step(3)
            got[precision, i] = (*g.state(), g.stats()["iterations"])
            g.close()
    return got


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid,chunk,contiguous", [(1, 1, 0), (2, 1, 0), (3, 2, 0), (5, 1, 1),
                                                   (9, 1, 0), (64, 1, 0), (0, 4, 0)])
def test_batch_equals_alone_in_every_grid(native, alone, precision, grid, chunk, contiguous):
    scs = _scenes()
    b = native.NativeBatch(scs, precision=precision)
    b.set_launch(grid=grid, chunk=chunk, contiguous=contiguous)
    b.step(3)
    stats = b.scene_stats()
    for i in range(len(scs)):
        p, v = b.state(i)
        assert np.array_equal(p, alone[precision, i][0]) and np.array_equal(v, alone[precision, i][1])
        assert stats[i]["iterations"] == alone[precision, i][2]
    b.close()
