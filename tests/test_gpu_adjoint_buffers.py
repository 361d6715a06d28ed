"""A run's buffers are kept from one recorded tape to the next: tapes of more and of fewer contact operations than the
buffers were made for, forward runs alone in between, and the other precision, against a batch whose buffers are new. The
same operations on the same inputs, so the same bits; in float the friction gradients are sums of atomics whose order may
change: a few hundred terms of either sign, 1e-7 x 300 of their size."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch

DT = float(np.float32(1.0 / 60.0))
STEPS = 6


def _run(batch, shapes, precision, forwards=1):
    batch.tape_record(DT, STEPS)
    for _ in range(forwards):
        final = batch.adjoint_forward(precision)
    grad = np.random.default_rng(1).normal(size=final.shape)
    return (final,) + tuple(batch.adjoint_backward(grad, shapes))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
def test_kept_buffers_give_what_new_ones_give(precision):
    # Boxes in the air, then on the ground and on one another: no operation, some, more, and none again.
    worlds = [scenes.single("boxes", n=12, seed=k) for k in range(3)] + [scenes.pyramid(2, seed=4)]
    shapes = sum(len(w.shapes) for w in worlds)
    kept = Batch(worlds)
    kept.save_state()
    other = 96 - precision
    for skip, forwards, precisions in ((0, 1, [precision]), (20, 2, [precision]), (30, 1, [precision]), (70, 1, [other, precision]),
                                       (4, 1, [precision]), (50, 3, [precision])):
        for p in precisions:
            results = []
            for fresh in (False, True):
                batch = Batch(worlds) if fresh else kept
                if not fresh:
                    kept.restore_state()
                for _ in range(skip):
                    batch.step_checked(DT)
                results.append(_run(batch, shapes, p, 1 if fresh else forwards))
                if fresh:
                    batch.close()
            for a, b in zip(results[0][:3], results[1][:3]):
                assert np.array_equal(a, b), (skip, p)
            a, b = results[0][3], results[1][3]
            assert np.array_equal(a, b) if p == 64 else np.abs(a - b).max() <= 3e-5 * np.abs(b).max(), (skip, p)
