"""The broadphase of worlds of more than 1024 bodies where its grid takes another form: some bodies wide along the second
axis, more than a sixteenth of them, widths within a few ulps of an eighth of the axis, one row and one layer of bodies,
wide bodies whose runs take several warps, bounds that reach infinity. Against the pair rules restated in numpy float32
(exact: keys are integers), for worlds that have a cluster of 16 CTAs each and for worlds that have one CTA each."""
import numpy as np
import pytest

from test_gpu_pair_tiles import _expected
from test_zz_no_alloc import DT, _pair_inputs, _sphere_world
from twofold_b200 import scenes
from twofold_b200.world import Batch

F32 = np.float32


def _span(n):
    return 0.42 * n ** (1.0 / 3.0)  # half the side of a cube with about four pairs a body


def _some_wide():
    w = _sphere_world(1500, _span(1500), 1)
    w.shapes["radius"][10:1500:75] = 0.4 * _span(1500)
    return w


def _many_wide():
    w = _sphere_world(4000, _span(4000), 2)
    w.shapes["radius"][::10] = 1.2  # 2.4 of about 15
    return w


def _at_an_eighth():
    # Two bodies hold the axes' ends; a hundred static ones are as wide as an eighth of the second axis, give or take
    # eight ulps: growth 0.02 and slack 0.001 (and a millionth of the coordinate) at either side of a sphere.
    n, reach = 2000, 9.0
    w = _sphere_world(n, _span(n), 3)
    b, s = w.bodies, w.shapes
    b["position"][:2] = [(0, 0, -reach), (0, 0, reach)]
    s["radius"][:2] = 0.5
    edge = np.arange(7, n, 19)[:100]
    b["type"][edge] = b["type"][0]
    b["linear_velocity"][edge] = b["angular_velocity"][edge] = 0.0
    b["linear_velocity"][:2] = b["angular_velocity"][:2] = 0.0
    b["type"][:2] = b["type"][0]
    eighth = 2.0 * (reach + 0.5 + 0.02 + 1e-3 + 1e-6 * (reach + 0.5)) / 8.0
    z = np.abs(b["position"][edge, 2].astype(np.float64))
    slack = 1e-3 + 1e-6 * np.maximum(z, eighth / 2.0)  # the mean of the two ends'
    steps = np.random.default_rng(3).integers(-8, 9, len(edge))
    s["radius"][edge] = (eighth * (1.0 + steps * 2.0 ** -24) / 2.0 - 0.02 - slack).astype(F32)
    return w


def _row():
    w = _sphere_world(1100, 300.0, 4)
    w.bodies["position"][:, 1:] = 0.0
    return w


def _layer():
    w = _sphere_world(1300, 13.0, 5)
    w.bodies["position"][:, 1] = 0.0
    return w


def _long_runs():
    # Wide bodies that cover all of x as well: three parts of a thousand records each.
    w = _sphere_world(2600, _span(2600), 6)
    w.shapes["radius"][[0, 1300, 2599]] = 1.5 * _span(2600)
    return w


def _infinite():
    # Two bodies that collide with nothing, one whose bounds reach past the largest float and one that stands there.
    w = _sphere_world(1200, _span(1200), 7)
    b, s = w.bodies, w.shapes
    for i, at, r in ((100, 2.5e38, 2.5e38), (1000, -3.0e38, 1.0e38)):
        b["type"][i] = b["type"][0]
        b["linear_velocity"][i] = b["angular_velocity"][i] = 0.0
        b["position"][i] = (at, at, at)
        s["radius"][i] = r
        s["category"][i] = s["mask"][i] = 0
    return w


KINDS = [_some_wide, _many_wide, _at_an_eighth, _row, _layer, _long_runs, _infinite]


@pytest.mark.gpu
def test_pairs_of_big_worlds():
    worlds = [kind() for kind in KINDS]
    settings = scenes.Scene("spheres", worlds).settings
    expected = []
    with np.errstate(over="ignore"):
        for w in worlds:
            keys = _expected(*_pair_inputs(w, settings))
            lone = np.flatnonzero(w.shapes["mask"] == 0)
            a, b = (keys >> np.uint64(32)).astype(np.int64), (keys & np.uint64(0xFFFFFFFF)).astype(np.int64)
            expected.append(keys[~np.isin(a, lone) & ~np.isin(b, lone)])
    for copies in (1, 12):
        batch = Batch.from_scene(scenes.Scene("spheres", worlds * copies))
        batch.step_checked(float(DT))
        for k in range(len(worlds) * copies):
            assert np.array_equal(batch.candidates(k), expected[k % len(worlds)]), (copies, KINDS[k % len(worlds)].__name__)
        batch.close()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [31, 32, 33, 70])
def test_pairs_where_the_worlds_share_the_warps(count):
    # Worlds are taken 32 at a time, each one's items from where the last one's ended: sizes and wide bodies differ.
    worlds = []
    for k in range(count):
        w = _sphere_world(1025 + 37 * (k % 5), _span(1025), 20 + k % 5)
        if k % 5 == 2:
            w.shapes["radius"][5:1025:100] = 0.5 * _span(1025)
        worlds.append(w)
    scene = scenes.Scene("spheres", worlds)
    expected = [_expected(*_pair_inputs(w, scene.settings)) for w in worlds[:5]]
    batch = Batch.from_scene(scene)
    batch.step_checked(float(DT))
    for k in range(count):
        assert np.array_equal(batch.candidates(k), expected[k % 5]), k
    batch.close()
