"""Direct steps of few worlds launch each kernel while the one before still runs; steps by graph and of more worlds do
not. Both give the same bits."""
import numpy as np
import pytest

from parity import states_bitwise_equal
from twofold_b200 import scenes
from twofold_b200.world import Batch

KINDS = {
    "boxes": lambda: [scenes.single("boxes", n=8, seed=1)],
    "pyramid": lambda: [scenes.pyramid(10, seed=1), scenes.hulls(24, seed=2)],
    "jointed": lambda: [scenes.jointed(s) for s in range(74)],
    "planar": lambda: [scenes.planar(n=300, cols=16, spheres=4, seed=2)],
    "falling": lambda: [scenes.hulls(60, seed=5)] * 3,
}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(KINDS))
def test_direct_steps_give_the_bits_of_steps_by_graph(kind):
    worlds = KINDS[kind]()
    direct, graph = Batch(worlds), Batch(worlds)
    dt = float(np.float32(1.0 / 60.0))
    for steps in (1, 30, 29):
        direct.step_checked(dt, steps)
        graph.step_checked(dt, steps, graph=True)
    assert states_bitwise_equal(direct.states(), graph.states())
    for k in range(min(len(worlds), 3)):
        assert [bytes(c) for c in direct.contacts(k)] == [bytes(c) for c in graph.contacts(k)]
        assert np.array_equal(direct.candidates(k), graph.candidates(k))
    assert direct.device_flags() == 0
