"""The streaming PCG (systems whose rows do not fit the chip's shared memory).

A child process with CIPC_PCG_NOCACHE=1 sends systems of every size to that
kernel: tiles of 8 rows with a remainder, rows from one block (the diagonal)
to 41, more than one round of a lane's columns, fewer tiles than SMs and more
than a block's warps take at once, data within and beyond L2, and the
recurrence vectors in shared and in global memory.  The solver promises
|b - A x| <= tol |b| in FP64 for the matrix it holds (rounded to FP32 in mixed
mode), so the residual is compared with the tolerance itself.
"""
import os
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
import cipc


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


for nv, width in ((1, 0), (7, 2), (8, 1), (9, 3), (131, 12), (1201, 37), (9473, 30), (19001, 9), (150011, 9)):
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
out = []
for precision in ("fp64", "mixed"):
    for precond in ("jacobi", "fsai"):
        sim = cipc.Simulator(cipc.scene_two_cubes(4, gap=0.002), precision=precision, precond=precond)
        for _ in range(4):
            sim.step()
        out.append(sim.get("x"))
        sim.close()
np.save(sys.argv[2], np.stack(out))
'''


def _child(code, *args, **env):
    pkg = os.path.join(os.path.dirname(HERE), "cpu-ipc_b200")
    r = subprocess.run([sys.executable, "-c", code, pkg, *args], env={**os.environ, **env}, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.gpu
def test_systems_of_all_shapes():
    assert "systems ok" in _child(CHILD, CIPC_PCG_NOCACHE="1")


@pytest.mark.gpu
def test_scenes_step_alike_in_both_kernels(tmp_path):
    """Steps of two cubes with contacts, block-Jacobi and a factor (in FP16 and
    in FP32 tiles), in the streaming and in the single-pass kernel: both stop
    at a residual of 1e-6, which moved the trajectories by 3.1e-7 of the
    scene's size in the learned factor's own comparison with the oracle."""
    got = {}
    for name, env in (("cached", {}), ("stream", {"CIPC_PCG_NOCACHE": "1"}), ("unpacked", {"CIPC_PCG_NOCACHE": "1", "CIPC_PCG_NOPACK": "1"})):
        path = str(tmp_path / (name + ".npy"))
        _child(FACTOR, path, **env)
        got[name] = np.load(path)
    size = np.linalg.norm(np.ptp(got["cached"][0].reshape(-1, 3), axis=0))
    for name in ("stream", "unpacked"):
        assert np.abs(got[name] - got["cached"]).max() < 1e-6 * size, name
