"""Worlds of more than 1024 bodies step on thread-block clusters, as many CTAs a world as the number of such worlds
leaves room for, and on one CTA a world past that. A world's results do not depend on which: the same world alone,
among a few and among many big worlds gives the same bits, pairs, contacts and events."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch

# One body past the limit and well past it; chains of contacts, contacts solved one at a time, swept shapes, a mesh.
WORLDS = {
    "pyramid": lambda: scenes.pyramid(45, seed=1),
    "planar": lambda: scenes.planar(n=1022, cols=24, spheres=16, seed=2, sphere_height=(4.0, 30.0), floor="halfspace",
                                    restitution=0.2),
    "terrain": lambda: scenes.terrain(cells=64, cols=8, levels=17, top=20.0, seed=3, cylinders=True),
}


def _run(world, copies, steps):
    batch = Batch([world] * copies + [scenes.pyramid(3, seed=9)])
    dt = float(np.float32(1.0 / 60.0))
    for _ in range(steps):
        batch.step_checked(dt)
    out = [batch.world_states(0), batch.candidates(0), [bytes(c) for c in batch.contacts(0)], batch.contact_events(0),
           batch.solver_counts(0), batch.world_states(copies)]
    batch.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(WORLDS))
def test_big_worlds_do_not_depend_on_their_cluster(kind):
    world = WORLDS[kind]()
    assert len(world.bodies) > 1024
    alone = _run(world, 1, 40)
    # 16, 8, 2 CTAs a world on 148 SMs, and one CTA a world.
    for copies in (12, 40, 76):
        other = _run(world, copies, 40)
        for a, b in ((alone[0], other[0]), (alone[5], other[5])):
            for key in a:
                assert np.array_equal(np.asarray(a[key]).view(np.uint32), np.asarray(b[key]).view(np.uint32)), (copies, key)
        assert np.array_equal(alone[1], other[1])
        assert alone[2:5] == other[2:5]


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 3])
def test_a_world_at_the_limit_is_not_a_big_one(copies):
    # 1024 bodies exactly, alone and beside a world that is one body larger: both step as they do alone.
    def world(bodies):
        return scenes.planar(n=bodies - 1, cols=24, spheres=0, seed=2, floor="halfspace")
    at, above = world(1024), world(1025)
    assert (len(at.bodies), len(above.bodies)) == (1024, 1025)
    for other in (at, above):
        got = _run(at, copies, 10), _run(other, copies, 10)
        batch = Batch([at] * copies + [other] * copies)
        for _ in range(10):
            batch.step_checked(float(np.float32(1.0 / 60.0)))
        for k, alone in ((0, got[0]), (copies, got[1])):
            state = batch.world_states(k)
            for key in state:
                assert np.array_equal(np.asarray(state[key]).view(np.uint32), np.asarray(alone[0][key]).view(np.uint32)), key
            assert np.array_equal(batch.candidates(k), alone[1])
        batch.close()
