"""Timed cases of the elastic-wave time loop, through the engine's public entry points.

A case is one program that keeps an ``Engine`` over one or several meshes and advances it chunk
by chunk: every pass steps ``steps`` time steps and takes that chunk's output (the receiver
traces, and where the case says so the velocity fields or the whole wave field).  The plan (mesh,
medium, sources, receivers, the engine itself) is made by ``prepare``; a run whose wavelet table
is used up starts again with ``reset``, as the next run of such a program does.

Meshes are jittered grids of triangles with random diagonals, the kind of mesh the benchmark
configurations use; the medium, sources, receivers, wavelet and the wave field a pass starts from
come from the seed.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("discontinuous-galerkin-method_b200")

# the P2 nodes on the reference triangle, in the order of the operator files
_NODES = np.array([[1.0, -1.0], [0.0, 0.0], [-1.0, 1.0], [0.0, -1.0], [-1.0, 0.0], [-1.0, -1.0]])
# work of one element and shot over one step (both half steps), the operators' zeros left out
_FLOPS = 1250.0
# time per element-shot-step of each arithmetic against FP32, about: what draw() takes for cost
_COST = {"fp32": 1.0, "fp32_kahan": 1.7, "fp64": 4.0, "fp64_ref": 12.0}


def _case(name, precision, nx, nz, shots, steps, medium="layered", receivers=101, meshes=1, call="step", fields=0):
    return {"name": name, "precision": precision, "nx": nx, "nz": nz, "shots": shots, "steps": steps,
            "medium": medium, "receivers": receivers, "meshes": meshes, "call": call, "fields": fields}


def listed():
    return [
        # a driver that keeps the reference's own loop: one wavelet sample in, one step, every step
        _case("tiny_fp64_stepwise", "fp64", 16, 16, 1, 20, "homogeneous", 17, call="stepwise"),
        # the small meshes models are tried out on: a few shots, chunks of 25 steps
        _case("small_fp32_3shots", "fp32", 41, 37, 3, 25, "layered", 38),
        # the plain configuration: 20,000 elements, traces and Vx/Vz kept every 200 steps
        _case("square_fp64", "fp64", 100, 100, 1, 200, "homogeneous", 101, fields=2),
        # the same with the reference's own operators and operation order (a drop-in check run)
        _case("square_fp64_ref", "fp64_ref", 100, 100, 1, 200, "homogeneous", 101, fields=2),
        # a few shots on a mid-size mesh, an odd element and shot count
        _case("mid_fp32_5shots", "fp32", 171, 143, 5, 100, "layered", 101),
        # coupled water/elastic slope at its full size, FP32, two snapshots while it steps
        _case("slope_fp32_snapshots", "fp32", 660, 294, 1, 600, "slope", 301, call="snapshots"),
        # the same model in FP64: the run an FP32 one is checked against
        _case("slope_fp64", "fp64", 660, 294, 1, 50, "slope", 301),
        # two million elements, compensated FP32 (long runs), whole wave field kept at the end
        _case("random2m_kahan", "fp32_kahan", 1000, 1000, 1, 100, "random", 501),
        # the multi-shot batch: 200,000 elements, 64 shots, chunks of 100 steps
        _case("multishot64_fp32", "fp32", 400, 250, 64, 100, "layered", 201),
        # a shot count that is no power of two
        _case("multishot24_fp32", "fp32", 190, 130, 24, 100, "layered", 151),
        # 16 shots, compensated FP32
        _case("multishot16_kahan", "fp32_kahan", 300, 170, 16, 100, "layered", 201),
        # uneven meshes in one context, 1-8 shots each, their own media and time steps
        _case("uneven12_fp32", "fp32", 0, 0, 0, 50, "layered", 41, meshes=12),
    ]


def draw(rng):
    precision = rng.choice(["fp32", "fp32", "fp32", "fp32_kahan", "fp64", "fp64", "fp64_ref"])
    steps = int(round(math.exp(rng.uniform(math.log(10), math.log(200)))))
    call = rng.choice(["step", "step", "step", "stepwise", "snapshots"])
    fields = rng.choice([0, 0, 2])
    receivers = rng.randrange(5, 400)
    medium = rng.choice(["homogeneous", "layered", "slope", "random"])
    budget = 6.0e8 / _COST[precision]
    if rng.random() < 0.2:
        meshes = rng.randrange(2, 13)
        while _elements_shots(meshes) * steps > budget and steps > 10:
            steps = max(10, steps // 2)
        while _elements_shots(meshes) * steps > budget and meshes > 2:
            meshes -= 1
        call = "step" if call == "snapshots" else call
        c = _case("", precision if precision != "fp64_ref" else "fp64", 0, 0, 0, steps, "layered", min(receivers, 41),
                  meshes, call, 0)
    else:
        K = math.exp(rng.uniform(math.log(300), math.log(1.2e6)))
        shots = 1 if rng.random() < 0.45 else int(round(math.exp(rng.uniform(math.log(2), math.log(128)))))
        while K * shots * steps > budget and steps > 10:
            steps = max(10, steps // 2)
        while K * shots * steps > budget and shots > 1:
            shots = max(1, shots // 2)
        K = min(K, budget / (shots * steps))
        aspect = math.exp(rng.uniform(math.log(0.5), math.log(2.5)))
        nx = max(8, int(round(math.sqrt(K / 2 * aspect))))
        nz = max(8, int(round(K / 2 / nx)))
        c = _case("", precision, nx, nz, shots, steps, medium, receivers, 1, call, fields if K < 5e5 else 0)
    del c["name"]
    return c


# ---- meshes and media ----------------------------------------------------------------------


def _uneven(count):
    """(cells along an edge, shots) of the meshes of an uneven batch: element counts log-uniform
    in 5,000 - 500,000, 1 to 8 shots."""
    rng = np.random.default_rng(5)
    out = []
    for _ in range(count):
        K = float(np.exp(rng.uniform(np.log(5000.0), np.log(500000.0))))
        out.append((max(4, int(round(math.sqrt(K / 2)))), int(rng.integers(1, 9))))
    return out


def _elements_shots(meshes):
    return sum(2 * n * n * s for n, s in _uneven(meshes))


def _parts(case):
    """(nx, nz, shots) of every mesh of the case."""
    if case["meshes"] > 1:
        return [(n, n, s) for n, s in _uneven(case["meshes"])]
    return [(case["nx"], case["nz"], case["shots"])]


@functools.lru_cache(maxsize=2)
def _grid(nx, nz, curved):
    """A jittered grid of 20 m cells, each cut into two triangles along a random diagonal, the
    vertex each triangle starts with random; `curved`: the top follows a sine.  The mesh belongs
    to the case: seeds share it."""
    rng = np.random.default_rng(nx * 100003 + nz)
    h = 20.0
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(nz + 1), indexing="xy")
    x, z = i * h, j * h
    inner = (i > 0) & (i < nx) & (j > 0) & (j < nz)
    x = x + np.where(inner, rng.uniform(-0.1 * h, 0.1 * h, x.shape), 0.0)
    z = z + np.where(inner, rng.uniform(-0.1 * h, 0.1 * h, x.shape), 0.0)
    if curved:
        z = z * (1.0 - 0.07 * (1.0 - np.sin(2 * np.pi * x / (nx * h) * 4)) / 2)
    points = np.stack([x.ravel(), z.ravel()], 1)
    ci, cj = (v.ravel() for v in np.meshgrid(np.arange(nx), np.arange(nz), indexing="xy"))
    a = cj * (nx + 1) + ci
    b, d = a + 1, a + nx + 1
    c = d + 1
    cell = cj * nx + ci
    flip = rng.integers(0, 2, nx * nz)
    f = flip[:, None] == 1
    first = np.where(f, np.stack([a, b, d], 1), np.stack([a, b, c], 1))
    second = np.where(f, np.stack([b, c, d], 1), np.stack([a, c, d], 1))
    down = np.where(cj > 0, 2 * (cell - nx) + 1, -1)
    up = np.where(cj < nz - 1, 2 * (cell + nx), -1)
    r = np.minimum(cell + 1, nx * nz - 1)
    right = np.where(ci < nx - 1, 2 * r + (1 - flip[r]), -1)
    le = np.maximum(cell - 1, 0)
    left = np.where(ci > 0, 2 * le + flip[le], -1)
    one, two = 2 * cell, 2 * cell + 1
    # the neighbour opposite each vertex
    n_first = np.where(f, np.stack([two, left, down], 1), np.stack([right, two, down], 1))
    n_second = np.where(f, np.stack([up, one, right], 1), np.stack([up, left, one], 1))
    K = 2 * nx * nz
    tris = np.stack([first, second], 1).reshape(K, 3)
    neigh = np.stack([n_first, n_second], 1).reshape(K, 3)
    turn = (np.arange(3)[None, :] + rng.integers(0, 3, K)[:, None]) % 3
    tris, neigh = np.take_along_axis(tris, turn, 1), np.take_along_axis(neigh, turn, 1)
    marks = np.where(inner, 0, 1).ravel()
    return pkg.meshgen.Mesh(points, tris.astype(np.int64), neigh.astype(np.int64), np.ones(K, np.int64), marks)


def _setup(case, seed, k, nx, nz, shots):
    """Mesh k of the case with the seed's medium, sources and receivers: the arrays the engine
    takes, as the host set-up makes them, and the mesh's set-up."""
    rng = np.random.default_rng([seed, k])
    mesh = _grid(nx, nz, case["medium"] == "slope")
    width, height = nx * 20.0, nz * 20.0
    cen = mesh.centroids()
    depth = 1.0 - cen[:, 1] / height
    if case["medium"] == "homogeneous":
        vp = np.full(mesh.K, rng.uniform(2800.0, 3200.0))
    elif case["medium"] == "random":
        g = np.zeros(mesh.K)
        for _ in range(6):
            q = rng.normal(0.0, 2 * np.pi / 400.0, 2)
            g += np.cos(cen @ q + rng.uniform(0, 2 * np.pi))
        vp = 3500.0 * np.exp(0.06 * g)
    else:
        layers = np.sort(rng.uniform(1500.0, 4500.0, 4))
        vp = layers[np.clip((depth * 4).astype(int), 0, 3)]
    vs, rho = vp / math.sqrt(3.0), pkg.workloads.gardner(vp)
    if case["medium"] == "slope":  # water on top
        wet = depth < 0.25
        vp, vs, rho = np.where(wet, 1500.0, vp), np.where(wet, 0.0, vs), np.where(wet, 1000.0, rho)
    inner = np.nonzero(mesh.markers == 0)[0]
    src = mesh.points[rng.choice(inner, shots)]
    R = case["receivers"]
    top = np.arange((nx + 1) * nz, (nx + 1) * (nz + 1))
    ids = np.concatenate([top[np.linspace(0, nx, R - R // 2).astype(int)], rng.choice(inner, R // 2)])
    b = 0.05 * min(width, height)
    w = pkg.workloads.Workload("perf", mesh, vp, vs, rho, 15.0, (b, b, width - 2 * b, height - 2 * b), src,
                               mesh.points[ids], _table(case))
    return pkg.host.build_setup(w, full=case["precision"] == "fp64_ref")


def _table(case):
    """Length of the wavelet table: a run of about a thousand steps, whole chunks."""
    return case["steps"] * max(2, 1000 // case["steps"])


def _waves(setup, seed, k):
    """A wave field to start from: up to four sets of five fields (K, 6), plane waves of 8 to 30
    cells' length; shot s starts from set s % (number of sets), scaled by 1 + s/64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.as_tensor(setup.Point, device=dev)[torch.as_tensor(setup.Triangle, device=dev) - 1]  # (K, 3, 2)
    rs = torch.as_tensor(_NODES, device=dev)
    shape = torch.stack([-(rs[:, 0] + rs[:, 1]) / 2, (1 + rs[:, 0]) / 2, (1 + rs[:, 1]) / 2], 1)  # (6, 3)
    at = torch.einsum("iv,kvc->kic", shape, p)
    A = torch.as_tensor(setup.A, device=dev)
    imp = torch.sqrt(A[:, 2] / A[:, 0])[:, None]  # rho * vp
    solid = (A[:, 4] > 0)[:, None]
    sets = []
    for q in range(min(4, setup.n_shots)):
        rng = np.random.default_rng([seed, k, q])
        f = []
        for n in range(5):
            g = torch.zeros(at.shape[:2], dtype=torch.float64, device=dev)
            for _ in range(2):
                length, angle, phase = rng.uniform(160.0, 600.0), rng.uniform(0, 2 * np.pi), rng.uniform(0, 2 * np.pi)
                g += torch.sin((at[..., 0] * math.cos(angle) + at[..., 1] * math.sin(angle)) * (2 * np.pi / length) + phase)
            g *= 1e-3
            f.append(g if n < 2 else g * imp)
        f[3] = torch.where(solid, f[3], f[2])  # a fluid carries pressure only
        f[4] = torch.where(solid, f[4], torch.zeros_like(f[4]))
        sets.append([v.cpu().numpy() for v in f])
    return sets


_FIELDS = ("Vx", "Vz", "Txx", "Tzz", "Txz")


def prepare(case, seed):
    T, meshes, waves = _table(case), [], []
    for k, (nx, nz, shots) in enumerate(_parts(case)):
        s = _setup(case, seed, k, nx, nz, shots)
        meshes.append(pkg.engine.mesh_from_setup(s, with_ref_ops=case["precision"] == "fp64_ref"))
        waves.append(_waves(s, seed, k))
    e = pkg.engine.Engine(meshes, case["precision"])
    for k, sets in enumerate(waves):
        S = e.info[k]["S"]
        for s in range(S):
            for n, f in enumerate(_FIELDS):
                v = sets[s % len(sets)][n]
                e.load(f, v if s == 0 else v * (1.0 + s / 64.0), k, s)
    values = case["steps"] * sum(i["S"] * i["R"] for i in e.info)
    pin = torch.cuda.is_available()
    out = [torch.empty(values, dtype=torch.float64, pin_memory=pin) for _ in range(2)]
    return {"case": case, "engine": e, "table": T, "out": out, "wavelet": [m["wavelet"] for m in meshes]}


def run(state):
    case, e, n = state["case"], state["engine"], state["case"]["steps"]
    if e.steps_done + n > state["table"]:
        e.reset()
    t0 = e.steps_done
    answer = {}
    # an FP32 run's results are kept in FP32
    keep = (lambda v: v) if case["precision"].startswith("fp64") else (
        lambda v: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32))
    if case["call"] == "stepwise":
        for t in range(t0, t0 + n):
            for k, w in enumerate(state["wavelet"]):
                e.set_wavelet(t, w[t:t + 1], k)
            e.step(1)
    elif case["call"] == "snapshots":
        every = max(1, n // 2)
        shots = []
        e.step_snapshots(n - n % every, every, lambda step, vx, vz: shots.append((keep(vx), keep(vz))))
        if n % every:
            e.step(n % every)
        answer["snapshots"] = shots
    else:
        e.step(n)
    x, z = state["out"]
    e.fetch_traces(t0, n, pkg.engine.ALL_MESHES, out_x=x, out_z=z)
    answer["x"], answer["z"] = keep(x), keep(z)
    if case["fields"]:
        for f in _FIELDS[:case["fields"]]:
            answer[f] = keep(e.fetch(f))
    return answer


def work(case):
    """A pass's bytes: the wave field read and written once a step where it cannot stay in the
    126 MB L2 from one step to the next, else once; the geometry, material and face codes the
    same way; the traces once.  Kahan carries a compensation per value."""
    w = 8 if case["precision"].startswith("fp64") else 4
    n, bytes_, flops = case["steps"], 0.0, 0.0
    for nx, nz, shots in _parts(case):
        K = 2.0 * nx * nz
        state = 30.0 * K * shots * w * (2 if case["precision"] == "fp32_kahan" else 1)
        const = K * (8.0 * w + 16.0)
        times = n if state + const > 126e6 else 1
        bytes_ += times * (2 * state + const) + 2.0 * n * case["receivers"] * shots * w
        flops += n * K * shots * _FLOPS
    return {"bytes": bytes_, "flops": flops}


# ---- the same steps in 64 bits, by plain torch ------------------------------------------------


def _exact_mesh(case, seed, k, nx, nz, shots, want):
    s = _setup(case, seed, k, nx, nz, shots)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    K, S, n = s.K, shots, case["steps"]
    ops = {q: t64(v) for q, v in s.ops.items()}
    Dr, Ds = ops["Vr"] @ ops["inverV"], ops["Vs"] @ ops["inverV"]
    lift = t64(s.arrays["S"])  # (3, 6, 3)
    X = t64(s.Point)[torch.as_tensor(s.Triangle, device=dev) - 1]
    r, q = (X[:, 1] - X[:, 0]) / 2, (X[:, 2] - X[:, 0]) / 2
    J = r[:, 0] * q[:, 1] - q[:, 0] * r[:, 1]
    rx, rz, sx, sz = q[:, 1] / J, -q[:, 0] / J, -r[:, 1] / J, r[:, 0] / J
    nx_ = torch.stack([-sx / 2, (rx + sx) / 2, -rx / 2])[:, None, :, None]  # (3, 1, K, 1)
    nz_ = torch.stack([-sz / 2, (rz + sz) / 2, -rz / 2])[:, None, :, None]
    g = lambda v: v[None, :, None]  # noqa: E731
    rx, rz, sx, sz = g(rx), g(rz), g(sx), g(sz)
    A = t64(s.A)
    irho, l2m, lam, mu = g(A[:, 0]), g(A[:, 2]), g(A[:, 3]), g(A[:, 4])
    # a node of the wave field is row node * K + element
    nb = torch.as_tensor(s.Neighbor, device=dev) - 1
    nn = torch.as_tensor(s.Node_Neighbor, device=dev).reshape(K, 3, 3) - 1
    far = (nn * K + nb[:, :, None]).permute(1, 2, 0).reshape(-1)
    inside = t64(s.Edge_flag).T[:, None, :, None]
    face = torch.as_tensor(s.ibe, device=dev).reshape(9) - 1
    sponge = t64(s.absorb_fun).T[:, :, None]  # (6, K, 1)
    rec = torch.as_tensor(np.asarray(s.receiver).reshape(-1, 2), device=dev) - 1
    rec = rec[:, 1] * K + rec[:, 0]
    se = torch.as_tensor(np.asarray(s.source).reshape(-1, 2)[:, 0], device=dev) - 1
    fun, wavelet = t64(np.asarray(s.fun).reshape(S, 6)), t64(s.wavelet)
    shot = torch.arange(S, device=dev)
    sets = _waves(s, seed, k)
    U = [torch.stack([t64(sets[m % len(sets)][f]).T * (1.0 + m / 64.0) for m in range(S)], 2) for f in range(5)]
    dt = s.dt

    def jump(v):  # (3 faces, 3 nodes, K, S)
        out = v.reshape(6 * K, S)[far].reshape(3, 3, K, S) * inside
        return out - v[face].reshape(3, 3, K, S)

    def mat(M, v):
        return (M @ v.reshape(v.shape[0], -1)).reshape(M.shape[0], K, S)

    L = lift.permute(1, 0, 2).reshape(6, 9)
    tx, tz, snaps = [], [], []
    every = max(1, n // 2)
    for t in range(n):
        for f in range(5):
            U[f] *= sponge
        vx, vz, xx, zz, xz = U
        vz[:, se, shot] += fun.T * wavelet[t]
        jx, jz, jm = jump(xx), jump(zz), jump(xz)
        hx = mat(L, (nx_ * jx + nz_ * jm).reshape(9, K, S))
        hz = mat(L, (nz_ * jz + nx_ * jm).reshape(9, K, S))
        del jx, jz, jm
        hx += mat(Dr, rx * xx + rz * xz) + mat(Ds, sx * xx + sz * xz)
        hz += mat(Dr, rx * xz + rz * zz) + mat(Ds, sx * xz + sz * zz)
        vx += dt * irho * hx
        vz += dt * irho * hz
        del hx, hz
        ju, jw = jump(vx), jump(vz)
        ru, su, rw, sw = mat(Dr, vx), mat(Ds, vx), mat(Dr, vz), mat(Ds, vz)
        ex = rx * ru + sx * su + mat(L, (nx_ * ju).reshape(9, K, S))
        ez = rz * rw + sz * sw + mat(L, (nz_ * jw).reshape(9, K, S))
        em = rx * rw + sx * sw + rz * ru + sz * su + mat(L, (nz_ * ju + nx_ * jw).reshape(9, K, S))
        del ju, jw, ru, su, rw, sw
        xx += dt * (l2m * ex + lam * ez)
        zz += dt * (lam * ex + l2m * ez)
        xz += dt * mu * em
        del ex, ez, em
        tx.append(vx.reshape(6 * K, S)[rec].T.clone())
        tz.append(vz.reshape(6 * K, S)[rec].T.clone())
        if case["call"] == "snapshots" and (t + 1) % every == 0 and t + 1 <= n - n % every:
            snaps.append(tuple(v[:, :, 0].T.clone() for v in (vx, vz)))
    traces = [torch.stack(v, 1).reshape(-1) for v in (tx, tz)]
    fields = [U[f][:, :, 0].T.reshape(-1).clone() for f in range(want)]
    return traces, snaps, fields


def exact(case, seed):
    if sum(2.0 * nx * nz * s for nx, nz, s in _parts(case)) * case["steps"] > 2e9:
        return None
    x, z, answer = [], [], {}
    for k, (nx, nz, shots) in enumerate(_parts(case)):
        (tx, tz), snaps, fields = _exact_mesh(case, seed, k, nx, nz, shots, case["fields"] if k == 0 else 0)
        x.append(tx.cpu())
        z.append(tz.cpu())
        if k == 0:
            if case["call"] == "snapshots":
                answer["snapshots"] = [(vx.cpu().numpy(), vz.cpu().numpy()) for vx, vz in snaps]
            for f, v in zip(_FIELDS, fields):
                answer[f] = v.cpu().numpy()
    answer["x"], answer["z"] = torch.cat(x), torch.cat(z)
    return answer
