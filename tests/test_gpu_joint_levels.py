"""Joints solved level by level: a level holds more joints of one kind than a warp has lanes, chains make many levels,
and joints created in an order that crosses them (each body met by joints far apart in index order). Worlds that
differ only in how many threads step them give the same bits: one warp, a CTA, the flat solve, a cluster."""
import numpy as np
import pytest

from twofold_b200 import abi, scenes
from twofold_b200.world import Batch


def _ropes(ropes, links, extra=0, seed=0):
    """`ropes` chains of `links` boxes hung from the world by point joints, every third neighbour pair tied by a
    distance joint too, the joints created in a shuffled order; `extra` loose boxes."""
    rng = np.random.default_rng(seed)
    n = ropes * links + extra
    b, s = scenes._bodies(n + 1), scenes._shapes(n + 1)
    scenes._ground(b, s)
    s["half_extents"][1:] = (0.15, 0.1, 0.1)
    joints = []
    for r in range(ropes):
        for k in range(links):
            i = 1 + r * links + k
            b["position"][i] = (0.4 * (k + 1), 6.0 + 0.05 * (r % 7), 0.8 * r)
            prev = None if k == 0 else abi.tf_id(i - 1, 0)
            joints.append(abi.joint_desc(abi.TF_JOINT_POINT, abi.tf_id(i, 0), prev, anchor=(0.4 * k + 0.2, 6.0, 0.8 * r)))
            if k and k % 3 == 0:
                joints.append(abi.joint_desc(abi.TF_JOINT_DISTANCE, abi.tf_id(i, 0), prev, anchor=(0.4 * k, 6.0, 0.8 * r),
                                             anchor_b=(0.4 * (k + 1), 6.0, 0.8 * r), hertz=3.0, damping_ratio=0.4))
    for x in range(extra):
        b["position"][1 + ropes * links + x] = (0.3 * (x % 40), 8.0 + 0.5 * (x // 40), 0.8 * (x % 9))
    w = scenes.World(b, s, np.arange(n + 1))
    w.joints = [joints[i] for i in rng.permutation(len(joints))]
    return w


def _run(worlds, shape, steps=20):
    batch = Batch(worlds)
    if shape:
        batch.set_launch(None, *shape[0])
        batch.set_launch("substep", *shape[1])
    dt = float(np.float32(1.0 / 60.0))
    for _ in range(steps):
        batch.step_checked(dt)
    out = [batch.world_states(0), [bytes(batch.joint_info(0, abi.tf_id(j, 0))) for j in range(len(worlds[0].joints))]]
    batch.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("ropes,links,extra", [(1, 40, 0), (70, 1, 0), (40, 5, 0), (33, 3, 1000)])
def test_joint_levels_do_not_depend_on_the_threads(ropes, links, extra):
    world = _ropes(ropes, links, extra)
    warp = _run([world], ((32, 0, 0), (32, 0, 0)))
    assert np.isfinite(warp[0]["p"]).all()
    for shape in (((256, 0, 0), (256, 0, 32768)), ((128, 0, 0), (256, -1, 0)), None):
        other = _run([world], shape)
        for key in warp[0]:
            assert np.array_equal(np.asarray(warp[0][key]).view(np.uint32), np.asarray(other[0][key]).view(np.uint32)), (shape, key)
        assert warp[1] == other[1], shape
