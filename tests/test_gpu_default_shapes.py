"""Batches on both sides of the lines of the substep's default shape: the solve the default takes gives the bits of
the other one (exact: both do the same operations in the same order)."""
import numpy as np
import pytest

from parity import states_bitwise_equal
from twofold_b200 import scenes
from twofold_b200.world import Batch


def _jointed(n):
    shared = [scenes.jointed(s) for s in range(8)]
    return scenes.Scene("jointed", [shared[k % 8] for k in range(n)])


# 592 and 1184 are 4 and 8 worlds an SM on 148.
SCENES = {
    "jointed below": (lambda: _jointed(1183), False),
    "jointed at": (lambda: _jointed(1184), True),
    "uneven few": (lambda: scenes.config4(591, seed=2), False),
    "uneven": (lambda: scenes.config4(592, seed=2), True),
    "uneven many": (lambda: scenes.config4(1184, seed=2), False),
}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(SCENES))
def test_default_substep_shapes_give_the_same_bits(kind):
    make, flat = SCENES[kind]
    sc = make()
    default, other = Batch.from_scene(sc), Batch.from_scene(sc)
    other.set_launch("substep", *((128, 32, 32768) if flat else (256, -1, 0)))
    dt = float(np.float32(1.0 / 60.0))
    for batch in (default, other):
        batch.step_checked(dt, 24)
    assert (default.launch("substep")["big_bodies"] == 0xFFFFFFFF) == flat
    assert states_bitwise_equal(default.states(), other.states())
    assert all(np.array_equal(default.candidates(w), other.candidates(w)) for w in range(0, len(sc.worlds), 97))
    default.close()
    other.close()
