"""Snapshots copy the contacts that the worlds hold, several CTAs a world or several worlds a CTA: steps after a restore
give the bits of the steps after the save, for worlds with no contacts, with few and with many."""
import numpy as np
import pytest

from parity import states_bitwise_equal
from twofold_b200 import scenes
from twofold_b200.world import Batch


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 2, 150, 1300])
def test_steps_after_a_restore_are_the_steps_after_the_save(copies):
    kinds = [scenes.pyramid(8, seed=1), scenes.single("boxes", n=1, seed=1), scenes.jointed(3)]
    batch = Batch([kinds[k % 3] for k in range(copies)])
    dt = float(np.float32(1.0 / 60.0))
    for _ in range(12):
        batch.step_checked(dt)
    batch.save_state(0)
    for _ in range(9):
        batch.step_checked(dt)
    first = batch.states(), [[bytes(c) for c in batch.contacts(k)] for k in range(min(copies, 3))]
    batch.restore_state(0)
    for _ in range(9):
        batch.step_checked(dt)
    assert states_bitwise_equal(first[0], batch.states())
    assert first[1] == [[bytes(c) for c in batch.contacts(k)] for k in range(min(copies, 3))]
    batch.close()
