"""Collision detection in its forms -- engines of few and of many bodies, spheres
whose partners are kept from the count pass and those that are searched again,
bodies that are second in many contacts: contact lists and one step equal the
oracle's bit for bit."""
import numpy as np
import pytest

from dvide_b200 import scenes

pytestmark = pytest.mark.gpu


def _reversed(sc):
    """The same scene with its bodies in reverse order."""
    for name in ("pos", "vel", "mass", "geom", "fixed", "family"):
        setattr(sc, name, getattr(sc, name)[::-1].copy())
    return sc


def _cluster(nb):
    return scenes.random_cluster(nb, n=nb - 5, max_iterations=15)


@pytest.mark.parametrize("make", [
    # kept partners end at 8, the warp's list at 128
    *[lambda n=n: scenes.crowd(n, max_iterations=10) for n in (7, 8, 9, 31, 33, 127, 130)],
    # the crowded sphere last: second in all its contacts; 24 is one thread's longest run
    *[lambda n=n: _reversed(scenes.crowd(n, max_iterations=10)) for n in (23, 24, 25, 26, 200)],
    lambda: _reversed(scenes.raspberry(1500, max_iterations=5)),
    lambda: _reversed(scenes.raspberry(1500, ballast=5000, max_iterations=5)),
    lambda: _reversed(scenes.random_cluster(4, n=216, max_iterations=10)),
    # the line between the forms, 6,144 bodies
    lambda: _cluster(6143), lambda: _cluster(6144), lambda: _cluster(6145)])
def test_contacts_and_a_step_equal_the_oracle(native, oracle_mod, make):
    sc = make()
    g = native.NativeScene.from_scene(sc)
    o = oracle_mod.OracleScene(sc)
    g.collide()
    o.collide()
    for x, y in zip(g.contacts(), o.contacts()):
        assert np.array_equal(x, y)
    assert g.num_contacts()[1] == o.stats()["num_possible"]
    g.step(2)
    o.step(2)
    assert g.stats()["num_contacts"] == o.stats()["num_contacts"] > 0
    assert np.array_equal(g.state()[0], o.state()[0])
    assert np.array_equal(g.state()[1], o.state()[1])
    g.close()


def test_families_and_many_small_scenes(native):
    """Pairs of one family never touch; a batch of one-body to 40-body scenes
    (short form) equals the same scenes inside a batch of over 6,144 bodies."""
    scs = [scenes.random_cluster(30 + i, n=1 + i, max_iterations=20) for i in range(0, 40, 3)]
    scs[5].family[:] = 3
    few = native.NativeBatch(scs)
    many = native.NativeBatch(scs + [_cluster(6500)])
    for b in (few, many):
        b.step(3)
    assert few.scene_stats()[5]["num_contacts"] == 0
    for i in range(len(scs)):
        for x, y in zip(few.state(i), many.state(i)):
            assert np.array_equal(x, y)
        assert few.scene_stats()[i] == many.scene_stats()[i]


def test_frames_keep_the_mode_of_their_detection(native, oracle_mod):
    """Frames and forces are those of the step, also after the mode is changed."""
    sc = scenes.random_cluster(6, n=60)
    sc.params["fp64_narrowphase"] = 1
    g = native.NativeScene.from_scene(sc)
    o = oracle_mod.OracleScene(sc)
    g.step(1)
    o.step(1)
    forces = g.contact_forces()
    g.set_params(fp64_narrowphase=0)
    assert np.array_equal(g.frames(), o.frames())
    for x, y in zip(g.contact_forces(), forces):
        assert np.array_equal(x, y)
    g.close()
