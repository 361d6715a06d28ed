"""A world whose joints are nearly all one chain is solved joint after joint, others level by level: the same chain alone,
beside a chain short enough to stay on the one side of that line, and beside chains that put it on the other gives the
same bits, whatever number of threads steps the world."""
import numpy as np
import pytest

from test_gpu_joint_levels import _run
from twofold_b200 import abi, scenes


def _chains(lengths):
    """Chains of boxes hung from the world by point joints, far apart, the first one first in every list."""
    n = sum(lengths)
    b, s = scenes._bodies(n + 1), scenes._shapes(n + 1)
    scenes._ground(b, s)
    s["half_extents"][1:] = (0.15, 0.1, 0.1)
    joints, i = [], 1
    for r, length in enumerate(lengths):
        for k in range(length):
            b["position"][i] = (0.4 * (k + 1), 40.0, 5.0 * r)
            joints.append(abi.joint_desc(abi.TF_JOINT_POINT, abi.tf_id(i, 0), None if k == 0 else abi.tf_id(i - 1, 0),
                                         anchor=(0.4 * k + 0.2, 40.0, 5.0 * r)))
            i += 1
    w = scenes.World(b, s, np.arange(n + 1))
    w.joints = joints
    return w


# 3 x joints against 4 x levels: 36 and 48, 45 and 48, 48 and 48 (the first by levels), far past it, a hundred levels.
@pytest.mark.gpu
@pytest.mark.parametrize("first,others", [(12, [3]), (12, [4]), (12, [12, 12, 5]), (1, []), (100, [2])])
def test_a_chain_does_not_depend_on_the_others(first, others):
    for shape in (((32, 0, 0), (32, 0, 0)), ((128, 0, 0), (256, -1, 0)), None):
        alone, beside = _run([_chains([first])], shape), _run([_chains([first] + others)], shape)
        assert np.isfinite(alone[0]["p"]).all()
        for key in alone[0]:
            a, b = np.asarray(alone[0][key]), np.asarray(beside[0][key])[:first + 1]
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (shape, key)
        assert alone[1] == beside[1][:first], shape
