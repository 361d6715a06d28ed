"""Which shapes the continuous pass sweeps: those that moved further than half their inner extent past what the step's
start let expect. A thin box, prism and disk pushed from rest, free and locked to a plane: the inner extent of a shape in
its plane leaves out the directions along the plane's normal, so a shape that is thin along it alone is not swept. One
pair each, a ball inside the swept bounds and out of the way. In the library and in its checking build, where a body that
was read in parts has odd values in the others."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from twofold_b200 import abi, build, scenes
from twofold_b200.world import Batch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DT = float(np.float32(1.0 / 60.0))
MOVE = 0.1  # against half of 0.02 and half of 0.5
SHAPES = ("box", "prism", "disk")
# Thin axis, locked plane's normal (None: free), direction of the push, whether it is swept.
CASES = [("z", None, "z", True), ("z", None, "y", True), ("z", "z", "y", False), ("z", "z", "x", False),
         ("y", "y", "x", False), ("y", None, "x", True), ("y", "z", "y", True), ("y", "z", "x", True)]
AXES = {"x": 0, "y": 1, "z": 2}
TURNED = scenes.GROUND_ROTATION  # z to y


def _world(shape, thin, normal, push):
    b, s = scenes._bodies(2), scenes._shapes(2)
    b["gravity_scale"] = 0.0
    if shape == "box":
        half = np.full(3, 0.5)
        half[AXES[thin]] = 0.02
        s["geometry"][1], s["half_extents"][1] = abi.TF_BOX, half
    elif shape == "disk":
        s["geometry"][1], s["radius"][1], s["half_height"][1] = abi.TF_CYLINDER, 0.5, 0.02
    else:
        s["geometry"][1], s["z_min"][1], s["z_max"][1] = abi.TF_PRISM, -0.02, 0.02
    if shape != "box" and thin == "y":
        b["rotation"][1] = TURNED
    if normal:
        b["locks"][1] = abi.TF_LOCK_PLANAR
        if normal == "y":
            b["lock_frame"][1] = TURNED
    at = np.full(3, 0.98)
    at[AXES[thin]] = 0.0
    b["type"][0], b["position"][0] = abi.TF_STATIC, at
    s["geometry"][0], s["radius"][0] = abi.TF_SPHERE, 0.5
    w = scenes.World(b, s, np.arange(2), meta={"push": AXES[push]})
    if shape == "prism":
        scenes._set_points(w, 1, [(-0.5, -0.5), (0.5, -0.5), (0.5, 0.5), (-0.5, 0.5)])
    return w


def swept_pairs():
    worlds = [_world(shape, thin, normal, push) for shape in SHAPES for thin, normal, push, _ in CASES]
    batch = Batch(worlds)
    forces = np.zeros((2 * len(worlds), 3), np.float32)
    steps = 4  # substeps: an acceleration a moves a body from rest a h^2 (1 + 2 + 3 + 4)
    for k, w in enumerate(worlds):
        forces[2 * k + 1, w.meta["push"]] = batch.mass(k, 1)[0] * MOVE / (10.0 * (DT / steps) ** 2)
    batch.add_forces(forces)
    batch.step_checked(DT)
    moved = [float(np.abs(batch.world_states(k)["p"][1]).max()) for k in range(len(worlds))]
    assert np.allclose(moved, MOVE, rtol=0.05), moved
    return [int(batch.profile(k).swept_pairs) for k in range(len(worlds))]


EXPECTED = [int(swept) for _ in SHAPES for _, _, _, swept in CASES]


@pytest.mark.gpu
def test_shapes_that_are_swept():
    assert swept_pairs() == EXPECTED


@pytest.mark.gpu
@pytest.mark.skipif(not os.path.exists(build.CHECKED_OUT), reason="checked build missing")
def test_shapes_that_are_swept_in_the_checking_build():
    code = ("import sys, json; sys.path[:0] = [{0!r}, {0!r} + '/tests']\nimport test_gpu_fast_shapes as t\n"
            "print(json.dumps(t.swept_pairs()))").format(ROOT)
    res = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, TWOFOLD_B200_LIB=build.CHECKED_OUT),
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert json.loads(res.stdout.splitlines()[-1]) == EXPECTED
