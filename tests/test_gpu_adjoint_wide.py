"""The model and its adjoint in double with a CTA a world (few worlds) against a warp a world (many): the same rows in
the same order, rounded in another association, so the gradients agree to double's rounding times what contacts amplify
(under a million over these steps, measured as float's distance from double): 1e-16 x 1e6 x 10."""
import numpy as np
import pytest

from twofold_b200 import scenes
from twofold_b200.world import Batch

STEPS = 12


def _gradients(worlds, n_bodies, n_shapes):
    batch = Batch(worlds)
    batch.tape_record(1.0 / 60.0, STEPS)
    final = batch.adjoint_forward(64)
    grad = np.zeros_like(final)
    grad[:n_bodies] = np.random.default_rng(3).normal(size=(n_bodies, 13))
    gi, gm, gf = batch.adjoint_backward(grad, sum(len(w.shapes) for w in worlds))
    again = batch.adjoint_forward(64)
    assert np.array_equal(final, again), "a second forward on the kept buffers differs"
    batch.close()
    return final[:n_bodies], gi[:n_bodies], gm[:n_bodies], gf[:n_shapes]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["impact", "pyramid", "mixed"])
def test_wide_walks_match_a_warp_a_world(kind):
    worlds = {"impact": lambda: scenes.config5(3, seed=2).worlds,
              "pyramid": lambda: [scenes.pyramid(9, seed=1), scenes.pyramid(1, seed=2)],
              "mixed": lambda: [scenes.hulls(20, seed=1), scenes.single("boxes", n=12, seed=12), scenes.single("sphere_on_ground", restitution=0.5,
                                                                                   position=(0.0, 0.52, 0.0))]}[kind]()
    bodies, shapes = sum(len(w.bodies) for w in worlds), sum(len(w.shapes) for w in worlds)
    wide = _gradients(worlds, bodies, shapes)
    many = _gradients(worlds + [scenes.single("box_on_ground")] * 640, bodies, shapes)
    for a, b in zip(wide, many):
        scale = max(float(np.linalg.norm(b)), 1e-30)
        assert float(np.linalg.norm(a - b)) / scale <= 1e-9
