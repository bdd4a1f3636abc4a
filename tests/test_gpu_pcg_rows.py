"""The block-CSR streaming PCG: systems whose rows differ so much that tiles of 8
rows would be mostly padding.  The child's solves name their kernel on stderr;
the solver promises |b - A x| <= tol |b| in FP64 for the matrix it holds (rounded
to FP32 in mixed mode), so the residual is compared with the tolerance itself."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import numpy as np
import scipy.sparse as sp
sys.path[:0] = [sys.argv[1] + "/cpu-ipc_b200", sys.argv[1] + "/tests"]
import cipc
from fake_runtime import hub_system

for nv, every, degree in ((9, 8, 2), (513, 8, 62), (1601, 16, 98), (40011, 8, 76), (40013, 3, 120)):
    rp, ci, va, _ = hub_system(nv, every, degree)
    rng = np.random.default_rng(nv)
    row = np.repeat(np.arange(nv), np.diff(rp))
    up = row < ci
    B = rng.standard_normal((int(up.sum()), 3, 3))
    order = np.lexsort((row[up], ci[up]))  # the lower blocks by row are the upper ones by column
    va[up] = B
    va[row > ci] = B[order].transpose(0, 2, 1)
    size = np.abs(va).sum(2).max(1)
    weight = np.zeros(nv)
    np.add.at(weight, row, size)
    va[row == ci] = (weight + 0.1)[:, None, None] * np.eye(3)
    b = rng.standard_normal(3 * nv)
    for precision in ("fp64", "mixed"):
        x, it, rr = cipc.pcg_bsr(rp, ci, va, b, precision=precision, tol=1e-6)
        held = va.astype(np.float32).astype(np.float64) if precision == "mixed" else va
        A = sp.bsr_matrix((held, ci, rp), shape=(3 * nv, 3 * nv))
        assert abs(A - A.T).max() == 0
        res = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        assert res <= 1e-6 * (1 + 1e-6) + 1e-15, (nv, precision, res)
print("systems ok")
"""


@pytest.mark.gpu
def test_systems_with_long_rows():
    env = {**os.environ, "CIPC_PCG_NOCACHE": "1", "CIPC_DEBUG_PCG": "1"}
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "systems ok" in r.stdout, r.stdout + r.stderr[-2000:]
    assert r.stderr.count("block-CSR launch") == 8  # the first system's rows suit tiles
