"""The friction gradients of a CTA's walk in double, where a shape has many contacts (a floor under every ball), few or
none, the floor before the balls or behind them, and the contacts' two shares each fill a warp, less or more. Against the
warp's walk, which adds every share where it arises: the same shares in another order, so the tolerance of
test_gpu_adjoint_wide. And the same bits every time."""
import numpy as np
import pytest

from test_gpu_adjoint_wide import _gradients
from twofold_b200 import abi, scenes


def _balls(n, floor_first):
    rng = np.random.default_rng(n)
    b, s = scenes._bodies(n + 1), scenes._shapes(n + 1)
    floor, balls = (0, np.arange(1, n + 1)) if floor_first else (n, np.arange(n))
    b["type"][floor] = abi.TF_STATIC
    b["position"][floor] = (0.0, -0.5, 0.0)
    s["half_extents"][floor] = (40.0, 0.5, 40.0)
    k = np.arange(n)
    b["position"][balls] = np.stack([1.5 * (k % 12) - 9.0, np.full(n, 0.499), 1.5 * (k // 12) - 9.0], 1)
    b["linear_velocity"][balls] = rng.uniform(-2.0, 2.0, (n, 3)) * (1.0, 0.0, 1.0)
    s["geometry"][balls], s["radius"][balls] = abi.TF_SPHERE, 0.5
    s["friction"] = rng.uniform(0.1, 0.9, n + 1)
    s["friction"][balls[::5]] = 0.0
    return scenes.World(b, s, np.arange(n + 1))


@pytest.mark.gpu
@pytest.mark.parametrize("n,floor_first", [(1, True), (15, False), (16, True), (17, False), (150, True), (150, False)])
def test_friction_gradients_of_a_floor(n, floor_first):
    worlds = [_balls(n, floor_first), scenes.pyramid(4, seed=n)]
    bodies, shapes = sum(len(w.bodies) for w in worlds), sum(len(w.shapes) for w in worlds)
    wide, again = (_gradients(worlds, bodies, shapes) for _ in range(2))
    many = _gradients(worlds + [scenes.single("box_on_ground")] * 640, bodies, shapes)
    floor = 0 if floor_first else n
    if n > 1:  # the only ball of the smallest case has no friction
        assert wide[3][floor] != 0.0
    for a, b, c in zip(wide, many, again):
        scale = max(float(np.linalg.norm(b)), 1e-30)
        assert float(np.linalg.norm(a - b)) / scale <= 1e-9
        assert np.array_equal(a, c)
