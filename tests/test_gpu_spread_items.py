"""The pair collisions and refreshes take a list of pairs a lane each, a few lanes of each warp or one, by its length
and the grid; convex pairs that are collided anew wait in a queue first. A world's results do not depend on any of it:
the same worlds alone, among a few and among many, on small and on large CTAs, give the same bits."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch


def _run(worlds, threads, steps, at):
    batch = Batch(worlds)
    for kernel in ("collide", "refresh"):
        batch.set_launch(kernel, threads, 0, 0)
    for _ in range(steps):
        batch.step_checked(float(np.float32(1.0 / 60.0)))
    out = [(batch.world_states(k), batch.candidates(k), [bytes(c) for c in batch.contacts(k)], batch.contact_events(k))
           for k in at]
    batch.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("copies,threads", [(1, 32), (1, 256), (5, 64), (40, 256), (300, 32), (900, 256)])
def test_results_do_not_depend_on_how_pairs_are_spread(copies, threads):
    # Struck walls (kept and new convex pairs, refreshes of both kinds), falling hulls, boxes beside each other.
    kinds = [scenes.config5(1, seed=4).worlds[0], scenes.hulls(12, seed=2), scenes.single("boxes", n=8, seed=1)]
    steps = 26
    alone = [_run([w], 128, steps, [0])[0] for w in kinds]
    many = _run([kinds[k % 3] for k in range(3 * copies)], threads, steps, [0, 1, 2, 3 * copies - 3, 3 * copies - 1])
    for got, want in zip(many, [alone[0], alone[1], alone[2], alone[0], alone[2]]):
        for key in got[0]:
            assert np.array_equal(np.asarray(got[0][key]).view(np.uint32), np.asarray(want[0][key]).view(np.uint32)), key
        assert np.array_equal(got[1], want[1])
        assert got[2:] == want[2:]
