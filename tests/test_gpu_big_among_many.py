"""A few worlds of more than 1024 bodies in a batch of many small ones: the big ones have clusters with more threads a CTA
than the batch's own shape, beside launches that give the others a warp or a CTA. Each world steps as it does alone."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch

DT = float(np.float32(1.0 / 60.0))


def _states(worlds, which, steps=12):
    batch = Batch(worlds)
    for _ in range(steps):
        batch.step_checked(DT)
    out = [(batch.world_states(k), batch.candidates(k), batch.solver_counts(k)) for k in which]
    batch.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("many", [591, 1184])
def test_big_worlds_among_many_small_ones(many):
    big = [scenes.pyramid(45, seed=1),
           scenes.planar(n=1040, cols=24, spheres=16, seed=2, sphere_height=(4.0, 30.0), floor="halfspace")]
    small = scenes.config4(16, seed=3, min_bodies=4, max_bodies=150).worlds
    assert min(len(w.bodies) for w in big) > 1024
    together = _states([big[0]] + [small[k % 16] for k in range(many - 1)] + [big[1]], [0, many] + list(range(1, 17)))
    alone = _states([big[0]], [0]) + _states([big[1]], [0]) + _states(small, range(16))
    for k, ((a, pairs_a, counts_a), (b, pairs_b, counts_b)) in enumerate(zip(alone, together)):
        for key in a:
            assert np.array_equal(np.asarray(a[key]).view(np.uint32), np.asarray(b[key]).view(np.uint32)), (k, key)
        assert np.array_equal(pairs_a, pairs_b) and counts_a == counts_b, k
