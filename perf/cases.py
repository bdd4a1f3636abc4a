"""What a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public Python binding (cpu-ipc_b200/cipc.py) or, for
device pointers, the C entry point it binds:

  step        one whole time step of a scene restored from a host state
  newton      one Newton system: gradient and Hessian assembly, then the linear solve
  contact     the line search's queries at new positions: contact sets, energy,
              intersection test, step bounds along a direction
  train       loss and weight gradient of the learned preconditioner on a Newton system
  pcg         the stand-alone block-CSR solver on host arrays
  pcg_device  the allocation-free solver on device arrays
  accd        additive continuous collision detection on a batch of candidate pairs

Scenes are the ones of the benchmark configurations (stacked cubes, cloth drape,
pile of cubes, twisted cylinder) in several sizes.  A scene's state is made from
the seed: bodies resting on one another at a fraction of the barrier distance, in
general position, smoothly deformed, with a smooth velocity field.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cpu-ipc_b200"))

import cipc  # noqa: E402

WEIGHTS = os.path.join(cipc.HERE, "weights", "pile_64x12_seeds0-49.bin")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the small example scene, whole steps: launches and host waits count
        {"name": "step_cubes_5", "kind": "step", "scene": "cubes", "a": 5, "b": 0, "precision": "fp64", "precond": "jacobi"},
        # the headline workload, whole steps of a pile (279,936 tetrahedra)
        {"name": "step_pile_27x12", "kind": "step", "scene": "pile", "a": 27, "b": 12, "precision": "mixed", "precond": "learned"},
        # a Newton system of a small odd-sized cloth
        {"name": "newton_cloth_37", "kind": "newton", "scene": "cloth", "a": 37, "b": 7, "precision": "fp64", "precond": "jacobi"},
        # the cloth-drape configuration
        {"name": "newton_cloth_128", "kind": "newton", "scene": "cloth", "a": 128, "b": 10, "precision": "mixed", "precond": "fsai"},
        # the pile configuration with the learned factor
        {"name": "newton_pile_64x12", "kind": "newton", "scene": "pile", "a": 64, "b": 12, "precision": "mixed", "precond": "learned"},
        # the plain FP64 method on a twisted cylinder of 188,325 tetrahedra
        {"name": "newton_twist_13x81", "kind": "newton", "scene": "twist", "a": 13, "b": 81, "precision": "fp64", "precond": "jacobi"},
        # the queries of a line-search trial
        {"name": "contact_cloth_128", "kind": "contact", "scene": "cloth", "a": 128, "b": 10, "precision": "fp64", "precond": "jacobi"},
        {"name": "contact_pile_27x12", "kind": "contact", "scene": "pile", "a": 27, "b": 12, "precision": "mixed", "precond": "jacobi"},
        # one training evaluation of the network (forward, loss, backward)
        {"name": "train_pile_8x12", "kind": "train", "scene": "pile", "a": 8, "b": 12, "precision": "mixed", "precond": "learned"},
        # the stand-alone solver as a linear-solver backend of a host program
        {"name": "pcg_30011_mixed", "kind": "pcg", "nv": 30011, "precision": "mixed", "tol": 1e-6},
        # the same on device arrays that the caller owns
        {"name": "pcg_device_5003", "kind": "pcg_device", "nv": 5003, "precision": "fp64", "tol": 1e-6},
        # a broad phase's candidates checked on their own
        {"name": "accd_40009", "kind": "accd", "n": 40009, "edges": 0.6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "newton", "newton", "contact", "contact", "train", "pcg", "pcg_device", "accd"])
    if kind == "pcg":
        return {"kind": kind, "nv": _log(rng, 200, 60000), "precision": rng.choice(["fp64", "mixed"]), "tol": rng.choice([1e-6, 1e-8])}
    if kind == "pcg_device":
        return {"kind": kind, "nv": _log(rng, 100, cipc.NOALLOC_MAX_ROWS), "precision": "fp64", "tol": rng.choice([1e-6, 1e-8])}
    if kind == "accd":
        return {"kind": kind, "n": _log(rng, 64, 200000), "edges": round(rng.random(), 3)}
    scene = rng.choice(["cubes", "cloth", "pile"] + (["twist"] if kind != "contact" else []))
    if scene == "cubes":
        a, b = rng.randint(2, 12), 0
    elif scene == "cloth":
        a, b = _log(rng, 12, 128), rng.randint(4, 10)
    elif scene == "pile":
        a, b = _log(rng, 2, 40), rng.randint(4, 12)
    else:
        a, b = rng.randint(3, 12), rng.randint(12, 80)
    precision = rng.choice(["fp64", "mixed"])
    precond = "learned" if kind == "train" else rng.choice(["jacobi", "learned", "fsai"])
    return {"kind": kind, "scene": scene, "a": a, "b": b, "precision": precision, "precond": precond}


# ---------------------------------------------------------------------------
# scenes and states
# ---------------------------------------------------------------------------
def _scene(case, seed):
    a, b = case["a"], case["b"]
    if case["scene"] == "cubes":
        return cipc.scene_two_cubes(a)
    if case["scene"] == "cloth":
        return cipc.scene_cloth_drape(a, b)
    if case["scene"] == "pile":
        return cipc.scene_pile(a, b, seed=seed)
    # a radial layers, b axial ones, as many angular ones as make the cells even
    return cipc.scene_twist(a, 2 * a + 5, b)


def _modes(rng, x, length, amplitude, count=3):
    """A smooth vector field at x: a few Fourier modes with waves of about `length`."""
    u = np.zeros_like(x)
    for _ in range(count):
        k = rng.standard_normal(3) * (2 * math.pi / length) * 0.5
        u += np.sin(x @ k + rng.uniform(0, 2 * math.pi))[:, None] * rng.standard_normal(3)
    return u * (amplitude / math.sqrt(count))


def _turn(rng, p, tilt):
    """p turned about the vertical through the origin and tilted a little."""
    t = rng.uniform(0, 2 * math.pi)
    c, s = math.cos(t), math.sin(t)
    q = p @ np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]]).T
    tx, tz = rng.uniform(-tilt, tilt, 2)
    return q @ np.array([[1, tz, 0], [-tz, 1, tx], [0, -tx, 1]]).T


def _stack(rng, x, bodies, size, gap, floor, spots):
    """Bodies (vertex ranges, local shapes) set in columns on the floor, `gap` apart."""
    tilt = 0.25 * gap / size
    for k, (first, local) in enumerate(bodies):
        cx, cz = spots[k % len(spots)]
        level = k // len(spots)
        y = floor + gap * (level + 1) + size * (level + 0.5)
        x[first:first + len(local)] = _turn(rng, local, tilt) + np.array([cx, y, cz])


def _state(case, scene, seed):
    """Positions, velocities and kappa of a scene in contact."""
    rng = np.random.default_rng([seed, 77])
    x = np.array(scene["x"])
    free = scene["btype"] == 0
    dhat = scene["params"]["relDhat"] * float(np.linalg.norm(np.subtract(scene["bbox_max"], scene["bbox_min"])))
    # a step starts near rest; within a step the trial positions are further off
    quiet = case["kind"] == "step"
    gap = dhat * (rng.uniform(0.94, 1.0) if quiet else rng.uniform(0.85, 0.95))
    bend = 0.1 if quiet else 1.0
    velocity = _modes(rng, x, 0.7, 0.02 if quiet else 0.2) + np.array([0.0, -0.05 if quiet else -0.2, 0.0])
    if case["scene"] == "cubes":
        local, _ = cipc.cube_mesh(case["a"], 1.0)
        n = len(local)
        _stack(rng, x, [(0, local), (n, local)], 1.0, gap, -1.0, [(0.0, 0.0)])
        x += _modes(rng, x, 1.5, 4e-3 * bend) * (1 - np.exp(-(x[:, 1:2] + 1.0) / 0.5))
    elif case["scene"] == "pile":
        local, _ = cipc.cube_mesh(case["b"], 0.2)
        n, floor = len(local), -0.98
        columns = -(-case["a"] // 4)
        side = math.ceil(math.sqrt(columns))
        at = [-0.75 + (i + 0.5) * 1.5 / side for i in range(side)]
        spots = [(at[i % side], at[i // side]) for i in range(columns)]
        bodies = [(k * n, local) for k in range(case["a"])]
        _stack(rng, x, bodies, 0.2, gap, floor, spots)
        x[free] += (_modes(rng, x, 0.5, 1.5e-3 * bend) * (1 - np.exp(-np.maximum(x[:, 1:2] - floor, 0.0) / 0.1)))[free]
    elif case["scene"] == "cloth":
        r = np.maximum(np.maximum(np.abs(x[:, 0]), np.abs(x[:, 2])) - 0.26, 0.0)
        y = 0.25 + gap + 0.2 * gap * np.sin(9 * x[:, 0] + rng.uniform(0, 6)) * np.sin(8 * x[:, 2] + rng.uniform(0, 6)) - 0.1 * bend * r * r / (r + 0.1)
        drift = _modes(rng, x, 0.4, 6e-4 * bend)
        x[free, 1] = y[free]
        x[free, 0] += drift[free, 0]
        x[free, 2] += drift[free, 2]
    else:
        turn = rng.uniform(0.2, 0.5) * math.pi * x[:, 0] / 0.5
        c, s = np.cos(turn), np.sin(turn)
        x[:, 1], x[:, 2] = c * x[:, 1] - s * x[:, 2], s * x[:, 1] + c * x[:, 2]
        x += _modes(rng, x, 0.4, 1e-3 * bend) * free[:, None]
        velocity = _modes(rng, x, 0.4, 0.1)
    velocity[~free] = 0.0
    return x, velocity


_surfaces = {}  # the collision surface of a mesh, as a host program has it in hand


def _simulator(case, scene):
    key = (case["scene"], case["a"], case["b"])
    sim = cipc.Simulator(scene, precision=case["precision"], precond=case["precond"], surface=_surfaces.get(key))
    _surfaces.setdefault(key, sim.surface())
    if case["precond"] == "learned":
        sim.set_precond_weights(np.fromfile(WEIGHTS, np.float32))
    return sim


def _kappa(sim):
    """The barrier stiffness a step starts from (suggestKappa)."""
    s = sim.scalars()
    hhat, bbox2 = s["Hhat"], s["bboxDiag2"]
    d = 1e-16 * bbox2
    t = d - hhat
    hb = (math.log(d / hhat) * -2.0 - t * 4.0 / d) + (t * t) / (d * d)
    return 1e13 * s["meanMass"] / (4e-16 * bbox2 * hb)


# ---------------------------------------------------------------------------
# block-CSR systems and candidate pairs
# ---------------------------------------------------------------------------
def _system(case, seed):
    """An SPD block-CSR system on the device: springs over the 15-point
    neighbourhood of a lattice, the pattern of a tetrahedral mesh, plus mass.
    Returns row pointers, columns, blocks (n x 3 x 3) and right-hand side."""
    nv = case["nv"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m = max(2, math.ceil(nv ** (1 / 3)))
    v = torch.arange(nv, device="cuda")
    i, j, k = v // (m * m), (v // m) % m, v % m
    rows, cols, blocks = [], [], []
    diag = torch.eye(3, dtype=torch.float64, device="cuda").expand(nv, 3, 3) * (0.05 + 0.1 * torch.rand(nv, 1, 1, generator=gen, device="cuda", dtype=torch.float64))
    diag = diag.clone()
    for d in ((0, 0, 1), (0, 1, 0), (0, 1, 1), (1, 0, 0), (1, 0, 1), (1, 1, 0), (1, 1, 1)):
        far = v + d[0] * m * m + d[1] * m + d[2]
        keep = (j + d[1] < m) & (k + d[2] < m) & (far < nv)
        p, q = v[keep], far[keep]
        n = torch.randn(len(p), 3, generator=gen, device="cuda", dtype=torch.float64) * 0.3 + torch.tensor(d, dtype=torch.float64, device="cuda")
        n = n / n.norm(dim=1, keepdim=True)
        stiff = torch.exp(torch.randn(len(p), 1, 1, generator=gen, device="cuda", dtype=torch.float64))
        blk = stiff * (n[:, :, None] * n[:, None, :] + 0.1 * torch.eye(3, dtype=torch.float64, device="cuda"))
        diag.index_add_(0, p, blk)
        diag.index_add_(0, q, blk)
        rows += [p, q]
        cols += [q, p]
        blocks += [-blk, -blk]
    rows, cols, blocks = torch.cat(rows + [v]), torch.cat(cols + [v]), torch.cat(blocks + [diag])
    order = torch.argsort(rows * nv + cols)
    ptr = torch.zeros(nv + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=nv), 0)
    b = torch.randn(3 * nv, generator=gen, device="cuda", dtype=torch.float64)
    return ptr.to(torch.int32), cols[order].to(torch.int32), blocks[order].contiguous(), b


def _pairs(case, seed):
    """Candidate pairs at the sizes and distances of a contact phase: features
    of about a centimetre within a few millimetres, moving about as far."""
    rng = np.random.default_rng([seed, 5])
    n = case["n"]
    kind = (rng.random(n) < case["edges"]).astype(np.int32)
    x = rng.standard_normal((n, 4, 3)) * 0.008
    split = np.where(kind[:, None] == 0, np.array([[1, 0, 0, 0]]), np.array([[1, 1, 0, 0]]))
    away = rng.standard_normal((n, 3))
    away /= np.linalg.norm(away, axis=1, keepdims=True)
    x += split[:, :, None] * (away * 10 ** rng.uniform(-3.5, -1.5, (n, 1)))[:, None, :]
    d = rng.standard_normal((n, 4, 3)) * 0.002 - split[:, :, None] * (away * 10 ** rng.uniform(-3.5, -1.5, (n, 1)))[:, None, :]
    return kind, x, d


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        rp, ci, va, b = (t.cpu().numpy() for t in _system(case, seed))
        return dict(case=case, args=(rp, ci, va, b), precision=case["precision"], tol=case["tol"])
    if kind == "pcg_device":
        rp, ci, va, b = _system(case, seed)
        return dict(case=case, args=(rp, ci, va, b), tol=case["tol"], sol=torch.zeros_like(b), lib=cipc.lib())
    if kind == "accd":
        return dict(case=case, args=_pairs(case, seed))
    scene = _scene(case, seed)
    sim = _simulator(case, scene)
    x, v = _state(case, scene, seed)
    dt = scene["params"]["dt"]
    down = np.array([0.0, -9.8 * dt * dt if scene["params"]["apply_gravity"] else 0.0, 0.0])
    kappa = _kappa(sim)
    s = dict(case=case, sim=sim, kappa=kappa, x=x, vel=v, xtilde=x + dt * v + down, direction=-dt * v)
    sim.set_kappa(kappa)
    s["counts"] = (ctypes.c_longlong * 4)()
    if kind == "step":
        return s
    if kind == "contact":
        # the host's own buffers for the sets, as large as they can get
        room = 6 * sim.nsv + 1024
        s["sets"] = {"self_active": np.full((room, 4), -1, np.int32), "self_ee": np.full((room // 4, 4), -1, np.int32),
                     "ee_ie": np.full((room // 4, 2), -1, np.int32), "ground": np.full(sim.nsv, -1, np.int32)}
    # within a step: the positions have moved since its start
    sim.set("x", x)
    sim.set("vprev", x - 0.3 * dt * v)
    sim.set("xtilde", x + 0.7 * dt * v + down)
    sim.collision_sets()
    sim.friction_init()
    if kind == "train":
        sim.assemble()
        s["weights"] = np.fromfile(WEIGHTS, np.float32)
        s["seed"] = seed
    return s


def _collision_sets(sim, counts, into=None):
    """Contact sets at the current positions; into the host's buffers if it asks for them."""
    sim._chk(sim.L.cipc_gpu_build_collision_sets(sim.h, counts))
    if into is None:
        return
    if counts[0] > len(into["self_active"]) or counts[1] > len(into["self_ee"]):
        raise ValueError("more contacts than the buffers hold: %s" % list(counts))
    at = {k: v.ctypes.data_as(ctypes.POINTER(ctypes.c_int)) for k, v in into.items()}
    sim._chk(sim.L.cipc_gpu_get_active_sets(sim.h, at["self_active"], at["self_ee"], at["ee_ie"], None, at["ground"]))


def run(s):
    kind = s["case"]["kind"]
    if kind == "pcg":
        sol, _, _ = cipc.pcg_bsr(*s["args"], precision=s["precision"], tol=s["tol"])
        return {"sol": sol}
    if kind == "pcg_device":
        rp, ci, va, b = s["args"]
        it, rr = ctypes.c_int(0), ctypes.c_double(0)
        rc = s["lib"].cipc_gpu_pcg_bsr_noalloc(len(rp) - 1, rp.data_ptr(), ci.data_ptr(), va.data_ptr(), b.data_ptr(), s["sol"].data_ptr(),
                                               s["tol"], 10000, torch.cuda.current_stream().cuda_stream, ctypes.byref(it), ctypes.byref(rr))
        if rc != cipc.CIPC_OK:
            raise cipc.CipcError(rc, "pcg_bsr_noalloc")
        return {"sol": s["sol"]}
    if kind == "accd":
        return {"toi": cipc.accd(*s["args"])}
    sim = s["sim"]
    if kind == "train":
        sim.set_precond_weights(s["weights"])
        loss, grad = sim.precond_loss(nprobes=4, seed=s["seed"], grad=True)
        return {"loss": loss, "grad": grad}
    if kind == "newton":
        grad, collisions = sim.assemble()
        direction, _, _ = sim.solve()
        return {"grad": grad, "collisions": collisions, "direction": direction}
    if kind == "contact":
        sim.set("x", s["x"])
        _collision_sets(sim, s["counts"], s["sets"])
        energy = sim.energy(s["kappa"])
        hit = sim.intersected()
        bounds = sim.step_bounds(s["direction"])
        return {"sets": s["sets"], "energy": energy, "intersected": hit, "bounds": bounds}
    # a whole step from a state that the host uploads, read back by the host
    sim.set("x", s["x"])
    sim.set("vprev", s["x"])
    sim.set("vel", s["vel"])
    sim.set("xtilde", s["xtilde"])
    _collision_sets(sim, s["counts"])
    sim.set_kappa(s["kappa"])
    sim.step()
    return {"x": sim.get("x"), "vel": sim.get("vel")}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(case):
    """Vertices, tetrahedra, triangles and matrix blocks of a scene."""
    a, b = case["a"], case["b"]
    if case["scene"] == "cubes":
        nv, nt, nf = 2 * (a + 1) ** 3, 12 * a ** 3, 0
    elif case["scene"] == "cloth":
        nv, nt, nf = a * a + (b + 1) ** 3, 6 * b ** 3, 2 * (a - 1) ** 2
    elif case["scene"] == "pile":
        nv, nt, nf = a * (b + 1) ** 3 + 20, 6 * a * b ** 3, 10
    else:
        ang = 2 * a + 5
        nv, nt, nf = (1 + a * ang) * (b + 1), 3 * b * ang * (2 * a - 1), 0
    return nv, nt, nf, 14 * nv


def work(case):
    """Inputs read once and outputs written once; floating-point operations of
    the elements and of a solve of about 150 iterations."""
    kind = case["kind"]
    if kind in ("pcg", "pcg_device"):
        nv, nb = case["nv"], 14 * case["nv"]
        return {"bytes": 76.0 * nb + 52.0 * nv, "flops": 150.0 * (18 * nb + 60 * nv)}
    if kind == "accd":
        return {"bytes": 204.0 * case["n"], "flops": 2000.0 * case["n"]}
    nv, nt, nf, nb = _sizes(case)
    value = 4 if case["precision"] == "mixed" else 8
    elements = {"bytes": 112.0 * nt + 60.0 * nf + 120.0 * nv, "flops": 3500.0 * nt + 1500.0 * nf}
    solve = {"bytes": nb * (9.0 * value + 4) + 72.0 * nv, "flops": 150.0 * (18 * nb + 60 * nv)}
    if kind == "contact":
        return {"bytes": 112.0 * nt + 60.0 * nf + 200.0 * nv, "flops": 150.0 * nt + 100.0 * nf + 1000.0 * nv}
    if kind == "train":
        # six 64-to-32 layers over edges and vertices, forward and twice that backward
        return {"bytes": solve["bytes"], "flops": 3.0 * 3 * 2 * 64 * 32 * (nb / 2 + nv)}
    rounds = 4 if kind == "step" else 1  # Newton iterations of a step
    return {k: rounds * (elements[k] + solve[k]) for k in ("bytes", "flops")}


def tolerance(case):
    """About four times what another order of the sums, another recurrence of the
    conjugate gradients or the unpacked factor gave on listed and drawn cases."""
    kind = case["kind"]
    if kind in ("pcg", "pcg_device"):  # 3.2e-6 at a residual of 1e-6: where the iteration stops
        return {"rel": 13 * case["tol"], "max": 60 * case["tol"]}
    if kind == "accd":
        return {"rel": 1e-10, "max": 1e-8}
    if kind == "train":  # layer inputs round to 16 bits: 1e-3 against a 64-bit network
        return {"rel": 4e-3, "max": 4e-2}
    if kind == "contact":
        return {"rel": 1e-11, "max": 1e-9, "differ": 0.0}
    if kind == "newton":  # 1.8e-4 and 1.4e-3, the solve's stop at 1e-6 on a cloth
        return {"rel": 7e-4, "max": 6e-3, "differ": 0.0}
    return {"rel": 2e-4, "max": 1.4e-2}  # 4.8e-5 and 3.5e-3 in a step's velocities


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _exact_pcg(case, seed):
    rp, ci, va, b = _system(case, seed)
    nv = case["nv"]
    if case["kind"] == "pcg" and case["precision"] == "mixed":
        va = va.float().double()  # the solver's matrix is the one rounded to 32 bits
    rows = torch.repeat_interleave(torch.arange(nv, device="cuda"), (rp[1:] - rp[:-1]).long())
    cols = ci.long()
    jacobi = torch.linalg.inv(va[rows == cols])

    def times(u):
        y = torch.zeros(nv, 3, dtype=torch.float64, device="cuda")
        return y.index_add_(0, rows, torch.bmm(va, u.view(nv, 3)[cols][:, :, None])[:, :, 0]).view(-1)

    def pre(u):
        return torch.bmm(jacobi, u.view(nv, 3, 1)).view(-1)

    x = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual
        r = b - times(x)
        z = pre(r)
        p, rz = z.clone(), r @ z
        stop = 1e-15 * b.norm()
        for _ in range(1500):
            ap = times(p)
            alpha = rz / (p @ ap)
            x = x + alpha * p
            r = r - alpha * ap
            if r.norm() < stop:
                break
            z = pre(r)
            rz, old = r @ z, rz
            p = z + (rz / old) * p
    return x


def _segment(p, a, b):
    """Squared distance of p to the segment a-b."""
    e = b - a
    t = (((p - a) * e).sum(1) / (e * e).sum(1)).clip(0, 1)
    return ((p - a - t[:, None] * e) ** 2).sum(1)


def _distance(kind, x):
    """Squared distances of points to triangles (kind 0) and of edges (kind 1)."""
    a, b, c, d = x[:, 0], x[:, 1], x[:, 2], x[:, 3]
    # point a, triangle b c d
    best = np.minimum(np.minimum(_segment(a, b, c), _segment(a, c, d)), _segment(a, d, b))
    n = np.cross(c - b, d - b)
    n2 = (n * n).sum(1)
    h = ((a - b) * n).sum(1)
    foot = a - (h / n2)[:, None] * n
    inside = np.ones(len(x), bool)
    for p, q in ((b, c), (c, d), (d, b)):
        inside &= (np.cross(q - p, foot - p) * n).sum(1) >= 0
    pt = np.where(inside, np.minimum(best, h * h / n2), best)
    # edges a-b, c-d
    best = np.minimum(np.minimum(_segment(a, c, d), _segment(b, c, d)), np.minimum(_segment(c, a, b), _segment(d, a, b)))
    u, v, w = b - a, d - c, a - c
    uu, uv, vv, uw, vw = ((p * q).sum(1) for p, q in ((u, u), (u, v), (v, v), (u, w), (v, w)))
    den = uu * vv - uv * uv
    s, t = (uv * vw - vv * uw) / den, (uu * vw - uv * uw) / den
    n = np.cross(u, v)
    h = (w * n).sum(1)
    inside = (s > 0) & (s < 1) & (t > 0) & (t < 1)
    ee = np.where(inside, np.minimum(best, h * h / (n * n).sum(1)), best)
    return np.where(kind == 0, pt, ee)


def _exact_accd(case, seed, eta=0.2):
    """The additive advancement on exact distances: steps of (1 - eta) d / L until
    the distance is under eta times the first one, L the largest closing motion."""
    kind, x, d = _pairs(case, seed)
    d = d - d.mean(1, keepdims=True)
    size = np.sqrt((d * d).sum(2))
    reach = np.where(kind == 0, size[:, 0] + size[:, 1:].max(1), size[:, :2].max(1) + size[:, 2:].max(1))
    toi = np.ones(case["n"])
    at, t = np.arange(case["n"]), np.zeros(case["n"])
    x, d2 = x.copy(), _distance(kind, x)
    goal = eta * np.sqrt(d2)
    for _ in range(10000):
        if not len(at):
            break
        step = (1 - eta) * np.sqrt(d2) / reach[at]
        x = x + step[:, None, None] * d[at]
        d2 = _distance(kind[at], x)
        touched = (t > 0) & (np.sqrt(d2) < goal)
        toi[at[touched]] = np.minimum(t[touched], 1.0)
        t = t + step
        stay = ~touched & (t <= 1.0)
        at, t, x, d2, goal = at[stay], t[stay], x[stay], d2[stay], goal[stay]
    return toi


def _exact_gradient(case, seed):
    """Inertia and Stable Neo-Hookean gradient of a scene without contacts."""
    scene = _scene(case, seed)
    x, v = _state(case, scene, seed)
    p = scene["params"]
    dt = p["dt"]
    target = x + 0.7 * dt * v
    X, T = torch.from_numpy(scene["x"]).cuda(), torch.from_numpy(scene["tets"].astype(np.int64)).cuda()
    x, target = torch.from_numpy(x).cuda(), torch.from_numpy(target).cuda()
    rest = torch.stack([X[T[:, i]] - X[T[:, 0]] for i in (1, 2, 3)], 2)
    vol = torch.linalg.det(rest).abs() / 6
    inv = torch.linalg.inv(rest)
    lame1 = p["E"] / (2 * (1 + p["nu"]))
    lame2 = p["E"] * p["nu"] / ((1 + p["nu"]) * (1 - 2 * p["nu"]))
    mu, lam = 4 * lame1 / 3, lame2 + 5 * lame1 / 6
    mass = torch.zeros(len(X), dtype=torch.float64, device="cuda")
    for i in range(4):
        mass.index_add_(0, T[:, i], vol * (p["density"] / 4))
    F = torch.stack([x[T[:, i]] - x[T[:, 0]] for i in (1, 2, 3)], 2) @ inv
    cof = torch.stack([torch.linalg.cross(F[:, :, 1], F[:, :, 2]), torch.linalg.cross(F[:, :, 2], F[:, :, 0]), torch.linalg.cross(F[:, :, 0], F[:, :, 1])], 2)
    i2, J = (F * F).sum((1, 2)), torch.linalg.det(F)
    P = (mu * (1 - 1 / (i2 + 1)))[:, None, None] * F + (lam * (J - 1 - 0.75 * mu / lam))[:, None, None] * cof
    force = (vol * dt * dt)[:, None, None] * (P @ inv.transpose(1, 2))
    g = mass[:, None] * (x - target)
    for i in range(3):
        g.index_add_(0, T[:, i + 1], force[:, :, i])
        g.index_add_(0, T[:, 0], -force[:, :, i])
    return g


def exact(case, seed):
    """Solutions of the given systems, times of impact, and the gradient of a
    scene without contacts.  What a solve or step to a relative tolerance of
    1e-6 stops at has no value of its own in 64 bits, nor have the contact sets'
    bounds and energies outside this repository's pipeline."""
    kind = case["kind"]
    if kind in ("pcg", "pcg_device"):
        return {"sol": _exact_pcg(case, seed)}
    if kind == "accd":
        return {"toi": _exact_accd(case, seed)}
    if kind == "newton" and case["scene"] == "twist":
        return {"grad": _exact_gradient(case, seed), "collisions": None, "direction": None}
    return None
