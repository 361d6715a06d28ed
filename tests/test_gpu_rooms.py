"""The world substep with rooms for contact records (batches whose contacts outweigh their bodies) against the flat
solve, which has none: the same bits, where a color fills part of a warp, one round of a CTA's warps or several, with
struck contacts and contacts solved one at a time among them."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch


def _rolling(world):
    world.shapes["rolling_resistance"][1::5] = 0.1
    return world


SETS = {
    "walls": lambda: scenes.config5(3, seed=2).worlds,
    "pyramid": lambda: [scenes.pyramid(40, seed=1)],
    "rolling": lambda: [_rolling(scenes.pyramid(12, seed=3)), scenes.config5(1, seed=5).worlds[0]],
}


@pytest.mark.gpu
@pytest.mark.parametrize("threads,big", [(32, 0), (128, 0), (256, 1000), (512, 0)])
@pytest.mark.parametrize("kind", list(SETS))
def test_rooms_give_the_flat_solve_s_bits(kind, threads, big):
    worlds = SETS[kind]()
    dt = float(np.float32(1.0 / 60.0))
    states = []
    for shape in ((threads, big, 32768), (256, -1, 0)):
        batch = Batch(worlds)
        batch.set_launch("substep", *shape)
        most = 0.0
        for _ in range(24):
            batch.step_checked(dt)
            work = batch.work_counts()
            most = max(most, work["active_contacts"] / work["bodies"])
        assert most >= 2.0, "the contacts never outweigh the bodies here: the rooms did not run"
        states.append(batch.states())
        batch.close()
    for key in states[0]:
        assert np.array_equal(states[0][key].view(np.uint32), states[1][key].view(np.uint32)), key
