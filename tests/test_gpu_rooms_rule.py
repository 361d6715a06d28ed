"""Batches on both sides of the lines past which the world substep takes its launch with rooms, at the default shapes:
contacts of one point and of four, colors that fit the rooms and that do not, worlds that fill an SM each, a second round
and a third, worlds past the ones that get a warp. Against the flat solve, which has no rooms: the same bits."""
import numpy as np
import pytest

from test_gpu_joint_chains import _chains
from twofold_b200 import abi, scenes
from twofold_b200.world import Batch

DT = float(np.float32(1.0 / 60.0))


def _block(geometry, side, seed):
    """A block of touching unit boxes or balls, side in each direction, on a half-space."""
    n = side ** 3
    b, s = scenes._bodies(n + 1), scenes._shapes(n + 1)
    scenes._ground(b, s)
    k = np.arange(n)
    at = np.stack([k % side, 0.5 + 1.001 * (k // side ** 2), k // side % side], axis=1) * (1.001, 1.0, 1.001)
    b["position"][1:] = (at + np.random.default_rng(seed).uniform(-1e-4, 1e-4, (n, 3))).astype(np.float32)
    s["geometry"][1:] = geometry
    return scenes.World(b, s, np.arange(n + 1))


def _sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


SETS = {
    "balls": lambda: [_block(abi.TF_SPHERE, 6, 1), _block(abi.TF_SPHERE, 8, 2)],
    "boxes": lambda: [_block(abi.TF_BOX, 5, 1)],
    "balls among boxes": lambda: [_block(abi.TF_SPHERE, 4, 1), _block(abi.TF_BOX, 4, 2), _chains([3, 3])],
    "colors at the lanes": lambda: [scenes.pyramid(31, seed=1), scenes.pyramid(33, seed=2)],
    "a round": lambda: [scenes.pyramid(9, seed=k % 5) for k in range(_sms())],
    "two rounds": lambda: [scenes.pyramid(9, seed=k % 5) for k in range(_sms() + 1)],
    "two rounds of dense worlds": lambda: [_block(abi.TF_BOX, 5, k % 2) for k in range(_sms() + 1)],
    "two full rounds": lambda: [_block(abi.TF_BOX, 3, k % 5) for k in range(2 * _sms())],
    "three rounds": lambda: [scenes.pyramid(9, seed=k % 5) for k in range(2 * _sms() + 1)],
    "a warp or a CTA": lambda: [scenes.pyramid(13 if k % 2 else 14, seed=k % 5) for k in range(8 * _sms())],
}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(SETS))
def test_default_substep_against_the_flat_solve(kind):
    worlds = SETS[kind]()
    states = []
    for shape in (None, (256, -1, 0)):
        batch = Batch(worlds)
        if shape:
            batch.set_launch("substep", *shape)
        for _ in range(8):
            batch.step_checked(DT)
        states.append(batch.states())
        batch.close()
    for key in states[0]:
        assert np.array_equal(states[0][key].view(np.uint32), states[1][key].view(np.uint32)), key
