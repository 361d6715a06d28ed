"""The broadphase of worlds up to 1024 bodies at the edges of its blocks of 32, in worlds that take a warp and in
worlds that take a CTA, staged and not, against the pair rules restated in numpy float32 (exact: keys are integers)."""
import numpy as np
import pytest

from test_gpu_pair_tiles import _expected
from test_zz_no_alloc import DT, _pair_inputs, _sphere_world
from twofold_b200 import scenes
from twofold_b200.world import Batch

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 255, 256, 257, 1000, 1024]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [None, (32, 0, 0), (64, 2000, 16384), (256, 40, 65536), (512, 0, 98304)])
def test_candidates_at_the_edges_of_the_blocks(shape):
    # About four pairs a body: a block of rows has more than a queue holds.
    worlds = [_sphere_world(n, 0.42 * max(n, 2) ** (1.0 / 3.0), n) for n in SIZES]
    for w in worlds:
        w.bodies["awake"][::7] = 0
    sc = scenes.Scene("spheres", worlds)
    batch = Batch.from_scene(sc)
    if shape:
        batch.set_launch("broadphase", *shape)
    batch.step_checked(float(DT))
    for k, w in enumerate(worlds):
        expected = _expected(*_pair_inputs(w, sc.settings))
        assert np.array_equal(batch.candidates(k), expected), SIZES[k]
