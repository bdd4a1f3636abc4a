"""The streaming PCG (systems whose rows do not fit the chip's shared memory).

A child process with CIPC_PCG_NOCACHE=1 sends systems of every size to that
kernel: tiles of 8 rows with a remainder, rows from one block (the diagonal)
to 41, more than one round of a lane's columns, fewer tiles than SMs and more
than a block's warps take at once, data within and beyond L2, and the
recurrence vectors in shared memory and, in a system too large for that, in
global memory (it is then beyond L2 as well).  The solver promises
|b - A x| <= tol |b| in FP64 for the matrix it holds (rounded to FP32 in mixed
mode), so the residual is compared with the tolerance itself.
"""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r'''
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import scipy.sparse as sp
import torch
import cipc

# past 128 tiles on every SM the recurrence vectors leave shared memory
LARGE = torch.cuda.get_device_properties(0).multi_processor_count * 128 * 8 + 8 * 37 + 3


def system(nv, width, seed):
    """Diagonally dominant symmetric blocks: a ring of neighbours, and every
    97th row joined to `width` more."""
    rng = np.random.default_rng(seed)
    i = np.arange(nv)
    far = [(i, (i + d) % nv) for d in (1, 2, 5)] + [(i[::97], (i[::97] + 3 * d + 7) % nv) for d in range(width)]
    p, q = np.concatenate([a for a, _ in far]), np.concatenate([b for _, b in far])
    lo, hi = np.minimum(p, q), np.maximum(p, q)
    key = np.unique(lo[lo != hi].astype(np.int64) * nv + hi[lo != hi])
    p, q = key // nv, key % nv
    B = rng.standard_normal((len(p), 3, 3))
    D = np.tile(np.eye(3), (nv, 1, 1))
    weight = np.abs(B).sum(2).max(1) + np.abs(B).sum(1).max(1)
    np.add.at(D, p, weight[:, None, None] * np.eye(3))
    np.add.at(D, q, weight[:, None, None] * np.eye(3))
    rows, cols = np.concatenate([p, q, i]), np.concatenate([q, p, i])
    blocks = np.concatenate([B, B.transpose(0, 2, 1), D])
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nv))]).astype(np.int32)
    return rp, cols[order].astype(np.int32), np.ascontiguousarray(blocks[order]), rng.standard_normal(3 * nv)


for nv, width in ((1, 0), (7, 2), (8, 1), (9, 3), (131, 12), (1201, 37), (9473, 30), (19001, 9), (150011, 9), (LARGE, 9)):
    rp, ci, va, b = system(nv, width, nv)
    for precision in ("fp64", "mixed"):
        x, it, rr = cipc.pcg_bsr(rp, ci, va, b, precision=precision, tol=1e-6)
        held = va.astype(np.float32).astype(np.float64) if precision == "mixed" else va
        A = sp.bsr_matrix((held, ci, rp), shape=(3 * nv, 3 * nv))
        res = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        assert res <= 1e-6 * (1 + 1e-6) + 1e-15, (nv, precision, res)
print("systems ok")
'''

FACTOR = r'''
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import cipc
out, iters = [], []
for precision in ("fp64", "mixed"):
    for precond in ("jacobi", "fsai"):
        sim = cipc.Simulator(cipc.scene_two_cubes(4, gap=0.002), precision=precision, precond=precond)
        steps = [sim.step() for _ in range(4)]
        iters.append([sum(s["pcgIterations"] for s in steps), sum(s["newtonIterations"] + 1 for s in steps)])
        assert sim.precond_stats()["fallbacks"] == 0
        assert len(sim.collision_sets()["self_active"]) > 0
        out.append(sim.get("x"))
        sim.close()
np.savez(sys.argv[2], x=np.stack(out), iters=iters)
'''


SOLVE = r'''
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import cipc
out = {}
for cells in map(int, sys.argv[3].split(",")):
    scene = cipc.scene_two_cubes(cells, gap=0.0015)  # closer than the barrier's distance
    x = np.array(scene["x"])
    x += 2e-4 * np.sin(7 * x[:, [1, 2, 0]] + 1.0) * (1 + x[:, 1:2])
    for precision in sys.argv[4].split(","):
        sim = cipc.Simulator(scene, precision=precision, precond="fsai")
        sim.set("x", x)
        sim.set_kappa(1e4)
        assert len(sim.collision_sets()["self_active"]) > 0
        sim.friction_init()
        sim.assemble()
        _, it, _ = sim.solve()
        assert sim.precond_stats()["fallbacks"] == 0
        out["%d %s" % (cells, precision)] = it
        sim.close()
np.savez(sys.argv[2], **out)
'''


def _child(code, *args, **env):
    pkg = os.path.join(os.path.dirname(HERE), "cpu-ipc_b200")
    r = subprocess.run([sys.executable, "-c", code, pkg, *args], env={**os.environ, **env}, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout + r.stderr


@pytest.mark.gpu
def test_systems_of_all_shapes():
    said = _child(CHILD, CIPC_PCG_NOCACHE="1", CIPC_DEBUG_PCG="1")
    assert "systems ok" in said
    ran = set(re.findall(r"streaming launch: .* state in shared memory (\d), beyond L2 (\d)", said))
    assert ran == {("1", "0"), ("1", "1"), ("0", "1")}
    assert "block-CSR launch" not in said and "single-pass launch" not in said


STREAM = {"CIPC_PCG_NOCACHE": "1"}
UNPACKED = {"CIPC_PCG_NOCACHE": "1", "CIPC_PCG_NOPACK": "1"}


@pytest.mark.gpu
def test_scenes_step_alike_in_both_kernels(tmp_path):
    """Steps of two cubes with contacts, block-Jacobi and a factor (in FP16 and
    in FP32 tiles), in the streaming and in the single-pass kernel: both stop
    at a residual of 1e-6, which moved the trajectories by 3.1e-7 of the
    scene's size in the learned factor's own comparison with the oracle.  A
    wrong factor would still reach that residual, in more iterations or through
    block-Jacobi: no solve falls back, and the iterations of the four steps agree
    to 2 % with FP32 tiles (the same factor) and to 3 a solve with FP16 ones, whose
    rounding costs so much where stiff contacts leave the scaled matrix nearly
    singular."""
    got = {}
    for name, env in (("cached", {}), ("stream", STREAM), ("unpacked", UNPACKED)):
        path = str(tmp_path / (name + ".npz"))
        _child(FACTOR, path, **env)
        got[name] = np.load(path)
    size = np.linalg.norm(np.ptp(got["cached"]["x"][0].reshape(-1, 3), axis=0))
    for name in ("stream", "unpacked"):
        assert np.abs(got[name]["x"] - got["cached"]["x"]).max() < 1e-6 * size, name
        (its, solves), ref = got[name]["iters"].T, got["cached"]["iters"][:, 0]
        assert np.all(np.abs(its - ref) <= (0.02 * ref if name == "unpacked" else np.maximum(0.02 * ref, 3 * solves))), (name, its, ref)


@pytest.mark.gpu
def test_factor_tiles_precondition_as_the_rows_do(tmp_path):
    """One Newton system with contacts and the exact factor, from the same
    positions: 10,648 rows in the single-pass kernel and in tiles, 21,296 (more
    than one tile a warp, within L2) and 101,306 (beyond L2) in tiles and, FP64, in
    the textbook kernel over the slot-aligned factor.  FP32 tiles hold the same
    factor, so only the order of sums differs; FP16 rounds its entries by 2^-11,
    which moves the preconditioned condition number by about 2^-9 and its root, the
    number of iterations, by 0.1 %.  A wrong slot, a diagonal block that is not
    transposed or a dropped contact block costs iterations."""
    runs = {"rows": ("17", "fp64,mixed", {}), "stream": ("17,21,36", "fp64,mixed", STREAM), "unpacked": ("17,21,36", "fp64,mixed", UNPACKED),
            "textbook": ("21,36", "fp64", {"CIPC_PCG_CLASSIC": "1"})}
    its = {}
    for name, (cells, precisions, env) in runs.items():
        path = str(tmp_path / (name + ".npz"))
        said = _child(SOLVE, path, cells, precisions, CIPC_DEBUG_PCG="1", **env)
        its[name] = {k: int(v) for k, v in np.load(path).items()}
        ran = set(re.findall(r"streaming launch: .* beyond L2 (\d)", said))
        assert ran == ({"0", "1"} if env.get("CIPC_PCG_NOCACHE") else set())
        assert ("single-pass launch" in said) == (name == "rows")
    for name in ("stream", "unpacked"):
        for key, it in its[name].items():
            ref = its["rows"].get(key, its["textbook"].get(key, its["unpacked"][key]))
            assert abs(it - ref) <= 2 + 0.01 * ref, (name, key, it, ref)
