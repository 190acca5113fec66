"""The work a program has this solver do, as cases that can be timed and checked.

Every case is one pass through the public entry points (GpuOperator, its
resident state, BatchRunner) on a mesh, materials and fields of the kinds the
configurations of this repository use: PEC cavities, a dielectric sphere in a
jittered box, a lossy slab in a box graded toward one face, a waveguide with
absorbing ends, batches of small cavities of mixed order.

``exact`` is a separate f64 implementation in plain torch: its own reference
element, geometry, face matching, flux, time steppers; only the meshes and the
inputs are shared with ``prepare``.
"""
from __future__ import annotations

import functools
import itertools
import math

import numpy as np
import torch

from rapidfem_b200 import _native as nat
from rapidfem_b200 import batch as B
from rapidfem_b200 import gpu as G
from rapidfem_b200 import operator as O

# ------------------------------------------------------------------ the cases


def _case(name, kind, order, nx, ny, nz, mesh="box", **more):
    return {"name": name, "kind": kind, "order": order, "nx": nx, "ny": ny, "nz": nz, "mesh": mesh, **more}


def listed():
    return [
        # a small sweep point: 4^3 cells at order 2, LSERK4 from torch memory to
        # torch memory (a parameter study steps thousands of these)
        _case("cavity_small_n2", "lserk", 2, 4, 4, 4, steps=20),
        # the plain configuration: the 8^3 PEC cavity at order 3
        _case("cavity_n3", "lserk", 3, 8, 8, 8, steps=50),
        # the large single instance: the 48^3 jittered box with the dielectric
        # sphere at order 4 (139 M DOFs)
        _case("sphere_n4_large", "lserk", 4, 48, 48, 48, mesh="jitter", steps=5),
        # order 5 on an odd-sized box whose element count fills no whole tile
        _case("sphere_n5_odd", "lserk", 5, 13, 17, 11, mesh="jitter", steps=10),
        # the stiff lossy slab at order 3, a point source sampled at the stage
        # times (how the explicit runs of the driven configuration are made)
        _case("slab_n3_stages", "stages", 3, 24, 24, 24, mesh="graded", steps=20),
        # a waveguide section with absorbing ends driven by a source pattern,
        # two modal amplitudes recorded per step: the whole host call, host
        # arrays in and out
        _case("waveguide_n3_host", "functionals", 3, 20, 9, 51, mesh="guide", steps=40),
        # uneven cavities of orders 2-5 as one captured batch
        _case("batch_mixed", "batch", 0, 4, 0, 12, count=24, steps=10),
        # one right-hand side on device arrays, as a program with its own time
        # stepper or eigensolver calls it
        _case("rhs_n3", "apply", 3, 21, 19, 23, mesh="jitter"),
        # one accepted exponential (Krylov) step of the stiff driven slab
        _case("slab_n3_etd", "etd", 3, 24, 24, 24, mesh="graded", m=48),
        # the adaptive Runge-Kutta transient, trajectory recorded to the host
        _case("cavity_n3_adaptive", "kcl", 3, 10, 10, 10, mesh="jitter", steps=4),
        # the double-precision transient of the plain configuration
        _case("cavity_n3_f64", "f64", 3, 8, 8, 8, steps=50),
        # the CUDA-core FP32 engine at order 4: the check every tensor-core run
        # is compared with
        _case("sphere_n4_fp32", "lserk", 4, 20, 20, 20, mesh="jitter", steps=5, engine="fp32"),
    ]


def draw(rng):
    kind = rng.choice(["lserk", "lserk", "lserk", "stages", "functionals", "batch", "apply", "etd", "kcl", "f64"])
    if kind == "batch":
        lo = rng.randint(3, 6)
        return {"kind": kind, "order": 0, "nx": lo, "ny": 0, "nz": lo + rng.randint(2, 8), "mesh": "box",
                "count": rng.randint(5, 32), "steps": 2 * rng.randint(1, 6)}
    order = rng.randint(1, 5)
    # the number of elements is spread over its logarithm, up to a size that
    # costs about what the listed case of the kind costs
    top = {"lserk": 2.5e7, "stages": 2.5e7, "functionals": 6e6, "apply": 5e7, "etd": 1e7, "kcl": 1e6, "f64": 1e6}[kind]
    np_ = (order + 1) * (order + 2) * (order + 3) // 6
    n_hex = math.exp(rng.uniform(math.log(8), math.log(top / (36 * np_))))
    side = n_hex ** (1 / 3)
    nx, ny = (max(2, round(side * rng.uniform(0.7, 1.4))) for _ in range(2))
    nz = max(2, round(n_hex / (nx * ny)))
    mesh = "guide" if kind == "functionals" else rng.choice(["box", "jitter", "graded"])
    c = {"kind": kind, "order": order, "nx": nx, "ny": ny, "nz": nz, "mesh": mesh}
    if kind == "etd":
        c["m"] = rng.choice([12, 24, 36, 48, 60])
    elif kind == "kcl":
        c["steps"] = rng.randint(1, 5)
    elif kind != "apply":
        c["steps"] = min(rng.randint(1, 20), max(1, int(2.2e8 / (36 * np_ * nx * ny * nz))))
    if kind == "lserk":
        c["engine"] = rng.choice(["tc", "tc", "tc", "fp32", "fp32_small"])
    return c


# ------------------------------------------------------------------ meshes and inputs

# spectral radius of the upwind operator times the smallest tetrahedron height,
# the largest over the mesh kinds below, by order
_RHO_H = {1: 15.3, 2: 25.3, 3: 35.0, 4: 49.0, 5: 64.5}
_CFL_Z = 1.4  # half of LSERK4's reach along the negative real axis
_KUHN = ((0, 1, 3, 7), (0, 2, 3, 7), (0, 2, 6, 7), (0, 4, 6, 7), (0, 4, 5, 7), (0, 1, 5, 7))


def _box_mesh(nx, ny, nz, kind):
    """(vertices [n,3], tets [K,4]): six tetrahedra per cell, vertex ids of a
    tetrahedron ascending."""
    size = {"guide": (2.286, 1.016, 6.0)}.get(kind, (1.0, 1.0, 1.0))
    x, y, z = (np.linspace(0.0, s, n + 1) for s, n in zip(size, (nx, ny, nz)))
    if kind == "graded":  # geometric, 20 : 1 toward z = 0
        step = 20.0 ** (np.arange(nz) / max(nz - 1, 1))
        z = np.concatenate([[0.0], np.cumsum(step) / step.sum()])
    zz, yy, xx = np.meshgrid(z, y, x, indexing="ij")
    v = np.stack([xx, yy, zz], axis=-1).reshape(-1, 3)
    if kind == "jitter":  # interior vertices moved by up to a tenth of a cell
        rng = np.random.default_rng(2024)
        d = rng.uniform(-0.1, 0.1, (nz + 1, ny + 1, nx + 1, 3)) / np.array([nx, ny, nz])
        for ax, i in ((2, 0), (1, 1), (0, 2)):
            s = [slice(None)] * 3
            for end in (0, -1):
                s[ax] = end
                d[tuple(s) + (i,)] = 0.0
        v = v + d.reshape(-1, 3)
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    corner = lambda c: ((k + (c >> 2)) * (ny + 1) + j + ((c >> 1) & 1)) * (nx + 1) + i + (c & 1)  # noqa: E731
    tets = np.stack([np.stack([corner(c) for c in t], axis=-1) for t in _KUHN], axis=1).reshape(-1, 4)
    return np.ascontiguousarray(v), np.ascontiguousarray(tets.astype(np.int32))


def _materials(v, tets, mesh):
    """[K,8]: eps_xyz, mu_xyz, sigma, sigma_m of the mesh kinds' configurations."""
    cen = v[tets].mean(axis=1)
    m = np.zeros((tets.shape[0], 8))
    m[:, :6] = 1.0
    if mesh == "jitter":
        m[np.linalg.norm(cen - 0.5, axis=1) < 0.25, :3] = 4.0
    elif mesh == "graded":
        m[cen[:, 2] < 0.2, :3] = 2.2
        m[cen[:, 2] < 0.2, 6] = 5.0
    elif mesh == "guide":
        m[np.hypot(cen[:, 0] - 1.143, cen[:, 2] - 3.0) < 0.15, :3] = 6.0
    return m


def _ports(v, tets, mesh):
    """[K,4] absorbing ends of the guide (port 0 at z = 0, port 1 at the far end)."""
    if mesh != "guide":
        return None
    p = np.full((tets.shape[0], 4), -1, dtype=np.int32)
    for f, t in enumerate(_FACE_VERTS):
        z = v[tets[:, list(t)], 2]
        p[np.all(z < 1e-9, axis=1), f] = 0
        p[np.all(z > 6.0 - 1e-9, axis=1), f] = 1
    return p


def _step(v, tets, order):
    p = v[tets]
    e = p[:, 1:] - p[:, :1]
    det = np.abs(np.linalg.det(e))
    face = [np.linalg.norm(np.cross(p[:, t[1]] - p[:, t[0]], p[:, t[2]] - p[:, t[0]]), axis=1) for t in _FACE_VERTS]
    return _CFL_Z * float((det / np.max(face, axis=0)).min()) / _RHO_H[order]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _node_coords(v, tets, order):
    """[K,Np,3] f64 on the device."""
    ref = torch.tensor(_lattice(order), dtype=torch.float64, device=_device()) / order
    p = torch.as_tensor(v, device=_device())[torch.as_tensor(tets, device=_device()).long()]
    return p[:, None, 0] + torch.einsum("nk,eki->eni", ref, p[:, 1:] - p[:, :1])


def _fields(x, seed):
    """[K,Np,6] f64: a Gaussian pulse on one E component over a few smooth waves
    on every component, the fields of a run that is under way."""
    rng = np.random.default_rng(7919 * (seed + 1))
    lo, hi = x.amin((0, 1)).cpu().numpy(), x.amax((0, 1)).cpu().numpy()
    y = torch.zeros(*x.shape[:2], 6, dtype=torch.float64, device=x.device)
    for c in range(6):
        for _ in range(2):
            k = torch.tensor(rng.uniform(-9.0, 9.0, 3), device=x.device)
            y[:, :, c] += rng.uniform(0.05, 0.2) * torch.sin(x @ k + rng.uniform(0, 2 * np.pi))
    mid = torch.tensor(lo + rng.uniform(0.25, 0.75, 3) * (hi - lo), device=x.device)
    y[:, :, rng.integers(0, 3)] += torch.exp(-((x - mid) ** 2).sum(-1) / (2 * rng.uniform(0.05, 0.15) ** 2))
    return y


def _waveform(seed, n, scale):
    rng = np.random.default_rng(104729 * (seed + 1))
    t = np.arange(n) * rng.uniform(0.05, 0.15)
    return scale * np.sin(t + rng.uniform(0, 2 * np.pi)) * rng.uniform(0.5, 1.5)


def _polynomial(seed, h):
    """Eight coefficients of the source over one step of h (a smooth pulse)."""
    rng = np.random.default_rng(1299709 * (seed + 1))
    return np.array([rng.uniform(-1, 1) / math.factorial(q) * (0.5 / h) ** q for q in range(8)]) * 5.0


@functools.lru_cache(maxsize=2)
def _guide_terms(nx, ny, nz, order):
    """Source pattern b [n_dof] (a TE10 current sheet at z = 0) and the weights
    of two modal amplitudes [(idx, w)], from node positions."""
    v, tets = _box_mesh(nx, ny, nz, "guide")
    x = _node_coords(v, tets, order).cpu().numpy().reshape(-1, 3)
    mode = np.sin(np.pi * x[:, 0] / 2.286)
    b = np.zeros((x.shape[0], 6))
    near = x[:, 2] < 1e-9
    b[near, 1] = 50.0 * mode[near]
    fun = []
    for at in (near, x[:, 2] > 6.0 - 1e-9):
        node = np.nonzero(at)[0]
        fun.append((node * 6 + 1, mode[node] / node.size))
    return b.ravel(), fun


def _instances(c):
    """The batch: (cells, order) of every cavity, drawn once per case."""
    rng = np.random.default_rng(20250 + 31 * c["count"] + c["nx"])
    return [(int(rng.integers(c["nx"], c["nz"] + 1)), int(rng.integers(2, 6))) for _ in range(c["count"])]


def _batch_groups(c, seed):
    """Per order: (order, [cells], eps [K], dt_scale [K], y0 [K,Np,6])."""
    rng = np.random.default_rng(15485863 * (seed + 1))
    inst, out = _instances(c), []
    for order in sorted({o for _, o in inst}):
        cells = [n for n, o in inst if o == order]
        eps, dts, y0 = [], [], []
        for n in cells:
            v, tets = _box_mesh(n, n, n, "box")
            cen = v[tets].mean(axis=1)
            lo = rng.uniform(0.0, 0.6, 3)
            hi = lo + rng.uniform(0.2, 0.4, 3)
            eps.append(np.where(np.all((cen >= lo) & (cen <= hi), axis=1), rng.uniform(1, 10), 1.0))
            dts.append(np.full(tets.shape[0], _step(v, tets, order)))
            y0.append(_fields(_node_coords(v, tets, order), int(rng.integers(1 << 30))))
        out.append((order, cells, np.concatenate(eps), np.concatenate(dts), torch.cat(y0)))
    return out


# ------------------------------------------------------------------ prepare and run

_ENGINES = {"tc": nat.ENGINE_TF32X3, "fp32": nat.ENGINE_FP32, "fp32_small": nat.ENGINE_FP32_SMALL_TILES}


@functools.lru_cache(maxsize=1)
def _ctx():
    return G.GpuContext(0)  # a program has one context (and stream) per device


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    order, mesh = case["order"], case["mesh"]
    v, tets = _box_mesh(case["nx"], case["ny"], case["nz"], mesh)
    host = O.MaxwellOperator(O.Mesh(v, tets), order, 1.0, face_port=_ports(v, tets, mesh),
                             materials=_materials(v, tets, mesh))
    op = G.GpuOperator(_ctx(), host)
    op.set_engine(_ENGINES[case.get("engine", "tc")])
    y0 = _fields(_node_coords(v, tets, order), seed).reshape(-1)
    h = _step(v, tets, order)
    s = {"case": case, "op": op, "h": h}
    kind = case["kind"]
    if kind == "f64":
        s["y0"] = y0.cpu().numpy()
    elif kind in ("functionals", "kcl"):
        s["y0"] = y0.to(torch.float32).cpu().numpy()
    else:
        s["y0"] = y0.to(torch.float32).contiguous()
        s["out"] = torch.empty_like(s["y0"])
    s["src"] = 6 * (y0.numel() // 12) + 2
    if kind == "stages":
        s["g"] = _waveform(seed, 5 * case["steps"], 20.0).astype(np.float32)
    if kind == "functionals":
        b, s["fun"] = _guide_terms(case["nx"], case["ny"], case["nz"], order)
        s["b"] = b
        s["g"] = _waveform(seed, case["steps"], 1.0).astype(np.float32)
    if kind == "etd":
        s["h"] = _etd_step(case, h)
        s["coef"] = _polynomial(seed, s["h"])
    torch.cuda.synchronize()
    return s


def _etd_step(case, h):
    # a step that the m-dimensional space resolves to the tolerance below
    return h / _CFL_Z * 0.14 * case["m"]


def _prepare_batch(case, seed):
    inst = [B.Instance(n, o, None, np.zeros(3), 1.0, 0) for n, o in _instances(case)]
    want = _batch_groups(case, seed)
    for order, cells, eps, _, _ in want:
        at = 0
        for i in (i for i in inst if i.order == order):
            k = 6 * i.cells ** 3
            i.materials = O.isotropic_materials(eps[at:at + k])
            at += k
    groups = B.build_groups(inst)
    y0 = []
    for g, (_, _, _, dts, y) in zip(groups, want):
        g.dt_scale[:] = dts
        y0.append(y.reshape(-1).to(torch.float32).contiguous())
        g.y0 = y0[-1].cpu().numpy()
    torch.cuda.synchronize()
    runner = B.BatchRunner(G.GpuContext(0), groups)
    runner.load()
    runner.capture(case["steps"])
    torch.cuda.synchronize()
    return {"case": case, "runner": runner, "y0": y0, "out": [torch.empty_like(y) for y in y0]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        r = state["runner"]
        r.stream.wait_stream(torch.cuda.current_stream())
        r.load_device([y.data_ptr() for y in state["y0"]])
        r.run(case["steps"])
        r.store_device([y.data_ptr() for y in state["out"]])
        torch.cuda.current_stream().wait_stream(r.stream)
        return state["out"]
    op, h = state["op"], state["h"]
    if kind == "kcl":
        traj, _ = op.transient_kcl(state["y0"], 4.0 * h, case["steps"])
        return traj
    if kind == "f64":
        return op.transient_f64(state["y0"], h * case["steps"], 1, substeps=case["steps"])
    if kind == "functionals":
        series, y = op.transient_functionals(state["y0"], h, case["steps"], drive=("vector", state["b"]), g=state["g"],
                                             functionals=state["fun"])
        return [series, y]
    y0, out = state["y0"], state["out"]
    if kind == "apply":
        op.apply_device(y0.data_ptr(), out.data_ptr())
        return out
    op.load_device(y0.data_ptr())
    if kind == "lserk":
        op.run_lserk(h, case["steps"])
    elif kind == "stages":
        op.run_lserk_stages(h, case["steps"], drive=("point", state["src"]), g_stages=state["g"])
    else:
        op.etd_try(h, case["m"], 1e-6, coef=state["coef"], drive=("point", state["src"]))
        op.etd_commit()
    op.store_device(out.data_ptr())
    return out


# ------------------------------------------------------------------ work and tolerance


def _stage_flops(order, n_dof):
    np_, nfp = (order + 1) * (order + 2) * (order + 3) // 6, (order + 1) * (order + 2) // 2
    return n_dof * (6 * np_ + 8 * nfp)


def work(case):
    """Bytes and flops of one pass.  A stage reads and writes the state and the
    residual register (not read by the first stage, not written by the last)
    and reads 168 bytes of geometry and materials per element; loading and
    storing the resident state are 8 bytes per value each."""
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for n, o in _instances(case):
            w = work({"kind": "lserk", "order": o, "nx": n, "ny": n, "nz": n, "steps": case["steps"]})
            total = {k: total[k] + w[k] for k in total}
        return total
    order = case["order"]
    K = 6 * case["nx"] * case["ny"] * case["nz"]
    np_ = (order + 1) * (order + 2) * (order + 3) // 6
    n = 6 * np_ * K
    one = _stage_flops(order, n)
    if kind == "apply":
        return {"bytes": 8 * n + 168 * K + 16 * n, "flops": one}
    if kind == "etd":
        # ceil(m/12) sub-steps; step j of one reads the j + 1 basis vectors for
        # the projections and again for the update, and reads and writes w
        k = -(-case["m"] // 12)
        d = -(-case["m"] // k)
        vecs = k * (sum(2 * (j + 1) + 4 for j in range(d)) + d + 2)
        return {"bytes": 4 * n * vecs + k * d * 168 * K + 16 * n,
                "flops": k * (d * one + n * sum(4 * (j + 1) for j in range(d)))}
    if kind == "kcl":
        # about five attempts per frame; a stage reads its point, reads and
        # writes the solution and the error, writes the next point
        stages = 5 * 5 * case["steps"]
        return {"bytes": stages * (24 * n + 168 * K) + 4 * n * (2 + case["steps"]), "flops": stages * one}
    size = 8 if kind == "f64" else 4
    steps = case["steps"]
    return {"bytes": steps * (18 * size * n + 5 * (42 * size) * K) + 4 * size * n, "flops": 5 * steps * one}


def tolerance(case):
    # 32-bit runs differ from the f64 ones by 1e-7 to 4e-7 (every entry by less
    # than 7e-6 of the larger of its value and the field's mean square root)
    f32 = {"rel": 1.6e-6, "max": 3e-5}
    if case["kind"] == "etd":  # and the step's own tolerance
        return {"rel": 4e-6, "max": 1e-4}
    if case["kind"] == "kcl":  # step sizes follow an error norm that is rounded itself
        return {"rel": 1e-5, "max": 2e-4}
    if case["kind"] == "f64":  # the conditioning of the nodal matrices grows with the order
        return {"rel": {1: 1e-14, 2: 4e-14, 3: 5e-13, 4: 1.5e-11, 5: 3e-10}[case["order"]]}
    return f32


# ------------------------------------------------------------------ exact (f64, plain torch)

_FACE_VERTS = ((0, 1, 2), (0, 2, 3), (0, 1, 3), (1, 2, 3))


def _lattice(p):
    return [(i, j, k) for i in range(p + 1) for j in range(p + 1 - i) for k in range(p + 1 - i - j)]


def _bary(p):
    return [(p - sum(q), *q) for q in _lattice(p)]


@functools.lru_cache(maxsize=8)
def _element(p):
    """Equispaced nodal element: D [3,Np,Np], LIFT [Np,4*Nfp], face nodes [4,Nfp]."""
    pts = np.array(_lattice(p), dtype=np.float64) / p
    mono = [q for q in itertools.product(range(p + 1), repeat=3) if sum(q) <= p]
    val = lambda x, q: np.prod([x[:, a] ** q[a] for a in range(len(q))], axis=0)  # noqa: E731
    V = np.stack([val(pts, q) for q in mono], axis=1)
    C = np.linalg.inv(V)
    fact = math.factorial
    gram = lambda qs, d: np.array([[math.prod(fact(a + b) for a, b in zip(q, r)) / fact(sum(q) + sum(r) + d)  # noqa: E731
                                    for r in qs] for q in qs])
    M = C.T @ gram(mono, 3) @ C
    D = []
    for ax in range(3):
        dV = np.stack([q[ax] * val(pts, tuple(e - (a == ax) for a, e in enumerate(q))) if q[ax] else np.zeros(len(pts))
                       for q in mono], axis=1)
        D.append(dV @ C)
    bary = _bary(p)
    faces, E = [], []
    m2 = [q for q in itertools.product(range(p + 1), repeat=2) if sum(q) <= p]
    for t in _FACE_VERTS:
        off = (set(range(4)) - set(t)).pop()
        nodes = [n for n, b in enumerate(bary) if b[off] == 0]
        uv = np.array([[bary[n][t[1]], bary[n][t[2]]] for n in nodes], dtype=np.float64) / p
        C2 = np.linalg.inv(np.stack([val(uv, q) for q in m2], axis=1))
        e = np.zeros((len(bary), len(nodes)))
        e[nodes] = C2.T @ gram(m2, 2) @ C2
        faces.append(nodes)
        E.append(e)
    return np.stack(D), np.linalg.solve(M, np.concatenate(E, axis=1)), np.array(faces)


class _Exact:
    """dy = A y in f64 for one mesh and order; y is [K,Np,6]."""

    def __init__(self, v, tets, order, materials, ports=None):
        dev = _device()
        D, lift, faces = _element(order)
        t = torch.as_tensor(tets, device=dev).long()
        p = torch.as_tensor(v, device=dev)[t]
        K, nfp = t.shape[0], faces.shape[1]
        J = (p[:, 1:] - p[:, :1]).transpose(1, 2)
        self.Jinv = torch.linalg.inv(J)  # [K,k,x]
        det = torch.linalg.det(J).abs()
        self.D = torch.as_tensor(D, device=dev)
        self.lift = torch.as_tensor(lift, device=dev)
        self.faces = torch.as_tensor(faces, device=dev)
        normal, scale = [], []
        for q in _FACE_VERTS:
            n = torch.linalg.cross(p[:, q[1]] - p[:, q[0]], p[:, q[2]] - p[:, q[0]])
            area2 = torch.linalg.norm(n, dim=1, keepdim=True)
            off = p[:, (set(range(4)) - set(q)).pop()] - p[:, q[0]]
            n = n / area2 * -torch.sign((n * off).sum(1, keepdim=True))
            normal.append(n)
            scale.append(area2[:, 0] / det)
        self.n = torch.stack(normal, 1)[:, :, None, :]  # [K,4,1,3]
        self.half = 0.5 * torch.stack(scale, 1)[:, :, None, None]
        # faces with the same three vertices; a face's nodes are matched by their
        # barycentric weights on the three vertices in ascending order
        nv = int(t.max()) + 1
        key = torch.stack([(t[:, q[0]] * nv + t[:, q[1]]) * nv + t[:, q[2]] for q in _FACE_VERTS], 1).reshape(-1)
        srt, at = torch.sort(key)
        same = torch.nonzero(srt[1:] == srt[:-1])[:, 0]
        other = torch.full((4 * K,), -1, dtype=torch.long, device=dev)
        other[at[same]], other[at[same + 1]] = at[same + 1], at[same]
        bary = _bary(order)
        # face nodes in the order of their weights, and each node's place in it
        weights = [[tuple(bary[n][w] for w in q) for n in f] for f, q in zip(faces, _FACE_VERTS)]
        rank = np.array([[sorted(w).index(x) for x in w] for w in weights])
        by_rank = np.stack([f[np.argsort(r)] for f, r in zip(faces, rank)])
        node = torch.as_tensor(by_rank, device=dev)[other.clamp(min=0) % 4]  # [4K,nfp]
        own = torch.as_tensor(rank, device=dev).repeat(K, 1)
        nb = torch.gather(node, 1, own) + (other.clamp(min=0) // 4)[:, None] * len(bary)
        self.nb = nb.reshape(K, 4, nfp)
        port = torch.as_tensor(ports, device=dev) >= 0 if ports is not None else torch.zeros(K, 4, dtype=torch.bool, device=dev)
        self.port = port[:, :, None, None]
        self.wall = ((other.reshape(K, 4) < 0) & ~port)[:, :, None, None]
        m = torch.as_tensor(materials, device=dev)
        self.inv = torch.cat([1 / m[:, :3], 1 / m[:, 3:6]], 1)[:, None, :]
        self.sig = torch.cat([m[:, 6:7] / m[:, :3], m[:, 7:8] / m[:, 3:6]], 1)[:, None, :]
        self.order = order

    def __call__(self, y):
        K, Np, _ = y.shape
        cross = torch.linalg.cross
        own = y[:, self.faces]  # [K,4,nfp,6]
        nb = y.reshape(K * Np, 6)[self.nb]
        jump = torch.where(self.port, own, own - nb)
        n = self.n.expand(*own.shape[:3], 3)
        e, h = own[..., :3], own[..., 3:]
        ne, nh = (n * e).sum(-1, keepdim=True), (n * h).sum(-1, keepdim=True)
        je = torch.where(self.wall, 2 * (e - ne * n), jump[..., :3])
        jh = torch.where(self.wall, 2 * nh * n, jump[..., 3:])
        ce, ch = cross(n, je), cross(n, jh)
        flux = self.half * torch.cat([-ch + cross(n, ce), ce + cross(n, ch)], -1)
        dy = torch.matmul(self.lift, flux.reshape(K, -1, 6))
        del own, nb, jump, e, h, je, jh, ce, ch, flux
        d = 0
        for k in range(3):  # d/dx_i = sum_k Jinv[k,i] D_k
            d = d + self.Jinv[:, k, None, :, None] * torch.matmul(self.D[k], y)[:, :, None, :]  # [K,Np,3,6]
        for c in range(3):
            a, b = (c + 1) % 3, (c + 2) % 3
            dy[..., c] += d[:, :, a, 3 + b] - d[:, :, b, 3 + a]
            dy[..., 3 + c] -= d[:, :, a, b] - d[:, :, b, a]
        return self.inv * dy - self.sig * y


# Carpenter and Kennedy (1994), five stages, fourth order
_LSERK_A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
            -1275806237668 / 842570457699)
_LSERK_B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
            3134564353537 / 4481467310338, 2277821191437 / 14882151754819)


def _lserk(A, y, h, steps, add=None, g=None, after=None):
    """LSERK4; `add(k, g_value)` adds the source, g[5*steps]."""
    for s in range(steps):
        p = torch.zeros_like(y)
        for q in range(5):
            k = A(y)
            if add is not None:
                add(k, float(g[5 * s + q]))
            p = _LSERK_A[q] * p + h * k
            y = y + _LSERK_B[q] * p
        if after is not None:
            after(y)
    return y


# the adaptive scheme: Kennedy, Carpenter and Lewis (2000), RK4(3)5[2R+]C, and
# the PI controller's default settings
_KCL_A = (970286171893 / 4311952581923, 6584761158862 / 12103376702013, 2251764453980 / 15575788980749,
          26877169314380 / 34165994151039)
_KCL_B = (1153189308089 / 22510343858157, 1772645290293 / 4653164025191, -1672844663538 / 4480602732383,
          2114624349019 / 3568978502595, 5198255086312 / 14908931495163)
_KCL_BH = (1016888040809 / 7410784769900, 11231460423587 / 58533540763752, -1563879915014 / 6823010717585,
           606302364029 / 971179775848, 1097981568119 / 3980877426909)


def _kcl(A, y, dt, frames):
    rows, h, prev = [y], dt, 0.0
    for _ in range(frames):
        t = 0.0
        while t < dt * (1 - 1e-6):
            step = min(h, dt - t)
            new, err, at = y, 0.0, y
            for q in range(5):
                f = step * A(at)
                new = new + _KCL_B[q] * f
                err = err + (_KCL_BH[q] - _KCL_B[q]) * f
                if q < 4:
                    at = new + (_KCL_A[q] - _KCL_B[q]) * f
            e = float(((err / (1e-8 + 1e-4 * torch.maximum(y.abs(), new.abs()))) ** 2).mean().sqrt())
            f = 0.9 * max(e, 1e-12) ** (-0.7 / 4)
            if e <= 1.0:
                t, y = t + step, new
                if prev > 0:
                    f *= prev ** (0.4 / 4)
                h, prev = step * min(max(f, 0.2), 5.0), max(e, 1e-12)
            else:
                h = step * max(f, 0.2)
        rows.append(y)
    return torch.stack([r.reshape(-1) for r in rows])


def _etd(A, y, h, coef, src):
    """y' = A y + e_src g(t) over h by Taylor series of order 20 on short pieces."""
    pieces = max(1, math.ceil(h * _rho_of(A, y) / 2.0))
    d = h / pieces
    for s in range(pieces):
        # the derivatives of g at the piece's start
        t = s * d
        g = [sum(coef[k] * math.perm(k, q) * t ** (k - q) for k in range(q, len(coef))) for q in range(len(coef))]
        term, out = y, y.clone()
        for k in range(1, 21):
            term = A(term)
            if k <= len(g):
                term.view(-1)[src] += g[k - 1]
            out = out + term * (d ** k / math.factorial(k))
        y = out
    return y


def _rho_of(A, y):
    v = torch.randn(y.shape, dtype=torch.float64, device=y.device, generator=torch.Generator(y.device).manual_seed(1))
    r = 1.0
    for _ in range(15):
        v = A(v)
        r = float(v.norm())
        v = v / r
    return 1.1 * r


def exact(case, seed):
    kind, order, mesh = case["kind"], case["order"], case["mesh"]
    if kind == "batch":
        out = []
        for o, cells, eps, dts, y in _batch_groups(case, seed):
            at, ys = 0, []
            for n in cells:
                v, tets = _box_mesh(n, n, n, "box")
                K = tets.shape[0]
                m = np.ones((K, 8))
                m[:, :3] = eps[at:at + K, None]
                m[:, 6:] = 0.0
                A = _Exact(v, tets, o, m)
                ys.append(_lserk(A, y[at:at + K].float().double(), float(np.float32(dts[at])), case["steps"]).reshape(-1))
                at += K
            out.append(torch.cat(ys))
        return out
    v, tets = _box_mesh(case["nx"], case["ny"], case["nz"], mesh)
    A = _Exact(v, tets, order, _materials(v, tets, mesh), _ports(v, tets, mesh))
    y0 = _fields(_node_coords(v, tets, order), seed)
    y = y0 if kind == "f64" else y0.float().double()
    h = _step(v, tets, order)
    src = 6 * (y.numel() // 12) + 2
    if kind == "apply":
        return A(y).reshape(-1)
    if kind == "kcl":
        return _kcl(A, y, float(np.float32(4.0 * h)), case["steps"])
    if kind == "etd":
        h = _etd_step(case, h)
        return _etd(A, y, h, _polynomial(seed, h), src).reshape(-1)
    steps = case["steps"]
    if kind == "f64":
        return _lserk(A, y, h * steps / steps, steps).reshape(-1).cpu().numpy()
    hf = float(np.float32(h))
    if kind == "stages":
        g = _waveform(seed, 5 * steps, 20.0).astype(np.float32).astype(np.float64)

        def add(k, gv):
            k.view(-1)[src] += gv

        return _lserk(A, y, hf, steps, add, g).reshape(-1)
    if kind == "functionals":
        b, fun = _guide_terms(case["nx"], case["ny"], case["nz"], order)
        bd = torch.as_tensor(b.astype(np.float32).astype(np.float64), device=y.device).reshape(y.shape)
        g = np.repeat(_waveform(seed, steps, 1.0).astype(np.float32).astype(np.float64), 5)
        terms = [(torch.as_tensor(i, device=y.device), torch.as_tensor(w, device=y.device)) for i, w in fun]
        rows = []

        def record(z):
            rows.append([float((z.reshape(-1)[i] * w).sum()) for i, w in terms])

        record(y)
        y = _lserk(A, y, hf, steps, lambda k, gv: k.add_(bd, alpha=gv), g, record)
        return [np.array(rows), y.reshape(-1).cpu().numpy()]
    return _lserk(A, y, hf, steps).reshape(-1)
