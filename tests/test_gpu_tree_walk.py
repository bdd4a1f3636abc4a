"""The warps' common walk over the broad-phase trees on a B200: query counts
that are no multiple of a warp, trees of a few primitives, large primitives
kept out of the tree, and a stack too small for the walk (CIPC_WALK_STACK, read
once per process), which hands subtrees to single lanes.  The contact sets, the
step bounds and the intersection flag must be those of the spatial hash, which
shares no tree code, bit for bit, whatever the stack."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import hashlib, json, os, sys
import numpy as np
sys.path.insert(0, os.path.join(sys.argv[1], "cpu-ipc_b200"))
import cipc
out = {}
for name, sc, squeeze in (("cubes_1", cipc.scene_two_cubes(1, gap=0.002), 1.0), ("cubes_4", cipc.scene_two_cubes(4, gap=0.002), 1.0),
                          ("cloth_5", cipc.scene_cloth_drape(5, 1), 1.0), ("cloth_33", cipc.scene_cloth_drape(33, 4), 1.0),
                          ("pile_3", cipc.scene_pile(3, 5, seed=2), 0.2)):
    x = np.array(sc["x"])
    rng = np.random.default_rng(7)
    free = sc["btype"] == 0
    if name.startswith("cloth"):
        x[free, 1] -= 0.1 - 8e-4          # onto the cube
    x[free] += 2e-4 * np.sin(40 * x[free] + 1.0)
    d = 0.05 * squeeze * rng.standard_normal(x.shape) * free[:, None]
    for backend in ("lbvh", "spatial-hash"):
        g = cipc.Simulator(sc)
        g.set_broad_phase(backend)
        g.set("x", x)
        sets = g.collision_sets()
        out[name + " " + backend] = [{k: [len(v), hashlib.sha256(np.ascontiguousarray(v).tobytes()).hexdigest()] for k, v in sets.items()},
                                     g.step_bounds(d, 1.0), g.intersected()]
        g.close()
print(json.dumps(out))
"""


def _run(stack=None, **more):
    env = {**os.environ, **more}
    env.pop("CIPC_WALK_STACK", None)
    if stack:
        env["CIPC_WALK_STACK"] = str(stack)
    r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_walk_finds_the_hash_grids_sets_for_any_stack():
    default = _run()
    for name in {k.split()[0] for k in default}:
        assert default[name + " lbvh"] == default[name + " spatial-hash"], name
    assert any(v[0]["self_active"][0] for v in default.values())
    assert any(v[0]["ccd"][0] > 1000 for v in default.values())
    for stack in (32, 40, 100):
        assert _run(stack) == default, stack


def test_joint_sort_orders_the_lists_as_their_own_sorts():
    """The lists packed and sorted together, and each sorted by its own keys, as in
    scenes too large for the joint sort (both backends share the packing, so the
    hash grid cannot show a mistake in it)."""
    assert _run(CIPC_SETS_APART="1") == _run()
