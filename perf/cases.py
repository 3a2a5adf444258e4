"""The workloads the library's speed is judged on, through its public entry points.

listed() names them; draw() gives more of the same kinds at other sizes, odd
ones among them.  prepare() makes what a program holds before the call (the
mesh's handle and the input fields, on the GPU or in host memory as that call
takes them), run() is one pass through the public calls, work() the bytes and
operations a pass cannot do without, exact() the same results from plain
64-bit torch (element matrices assembled and systems solved to round-off).

Kinds
  frame        the interactive application's frame: host values in, one heat
               step, the instability check, host values and normals out
  steps        a run of time steps from device-resident fields: heat, wave,
               advection-diffusion and Gray-Scott, FP32 and FP64
  adjoint      loss and gradients of an inverse problem (advection-diffusion
               or Gray-Scott), checkpointed reverse sweep
  batch        a parameter sweep of Gray-Scott instances stepped together
  open         a mesh opened: handle, matrices out, first frame
"""
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fea-visualizer_gb300"))
import fea_gb300 as F  # noqa: E402
from fea_gb300 import meshgen as mg  # noqa: E402

DEV = "cuda"
GS = dict(rd_feed_rate=0.037, rd_kill_rate=0.06, rd_time_step=1.0, reaction_mode=1)


def listed():
    return [
        # the reference application's frame loop on its own icosphere.obj size
        {"name": "frame_icosphere5", "kind": "frame", "mesh": "icosphere", "n": 5},
        # a small drawn-domain sized mesh with a Dirichlet boundary: launch latency only
        {"name": "heat_cylinder_small", "kind": "steps", "eq": "heat", "mesh": "cylinder", "n": 37, "bc": 0,
         "prec": 0, "steps": 20},
        # FP64 heat over 100 steps on the level-5 icosphere
        {"name": "heat_fp64_icosphere5", "kind": "steps", "eq": "heat", "mesh": "icosphere", "n": 5, "bc": 1,
         "prec": 1, "steps": 100},
        # implicit advection-diffusion (the reference's scheme), mid-size closed mesh
        {"name": "advdiff_icosphere6", "kind": "steps", "eq": "advdiff", "mesh": "icosphere", "n": 6, "bc": 1,
         "prec": 0, "steps": 20},
        # Gray-Scott on a mid-size planar mesh of odd size
        {"name": "gray_scott_grid251", "kind": "steps", "eq": "gs", "mesh": "grid", "n": 251, "bc": 1, "prec": 0,
         "steps": 20},
        # Gray-Scott on a well-shaped closed mesh
        {"name": "gray_scott_icosphere7", "kind": "steps", "eq": "gs", "mesh": "icosphere", "n": 7, "bc": 1,
         "prec": 0, "steps": 20},
        # the flagship: Gray-Scott on the 1024 x 1024 jittered grid
        {"name": "gray_scott_grid1024", "kind": "steps", "eq": "gs", "mesh": "grid", "n": 1024, "bc": 1, "prec": 0,
         "steps": 10},
        # Newmark wave on the level-8 icosphere
        {"name": "wave_icosphere8", "kind": "steps", "eq": "wave", "mesh": "icosphere", "n": 8, "bc": 1, "prec": 0,
         "steps": 50},
        # the inverse problem of the diffusivity: FP64 adjoint on the 512 x 512 grid
        {"name": "adjoint_advdiff_fp64_grid512", "kind": "adjoint", "eq": "advdiff", "mesh": "grid", "n": 512,
         "prec": 1, "steps": 12, "ckpt": 4},
        # the inverse problem of the reaction rates: FP32 adjoint on the 512 x 512 grid
        {"name": "adjoint_gray_scott_grid512", "kind": "adjoint", "eq": "gs", "mesh": "grid", "n": 512, "prec": 0,
         "steps": 10, "ckpt": 5},
        # the parameter sweep: instances of uneven size stepped together
        {"name": "batch_64", "kind": "batch", "count": 64, "lo": 3, "hi": 6, "steps": 50},
        # a mesh opened: assembly, matrices out, first frame
        {"name": "open_grid512", "kind": "open", "mesh": "grid", "n": 512, "bc": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "steps", "steps", "steps", "steps", "adjoint", "batch", "open"])
    if kind == "frame":
        if rng.random() < 0.3:
            return {"kind": kind, "mesh": "icosphere", "n": rng.randint(3, 6)}
        return {"kind": kind, "mesh": rng.choice(["grid", "cylinder"]), "n": _log_int(rng, 16, 200)}
    if kind == "steps":
        eq = rng.choice(["heat", "heat", "advdiff", "wave", "gs", "gs", "gs"])
        mesh = rng.choice(["grid", "cylinder"]) if eq != "advdiff" else "cylinder"
        prec = rng.choice([0, 0, 0, 1])
        n = _log_int(rng, 20, 300 if prec or mesh == "cylinder" else 900)
        return {"kind": kind, "eq": eq, "mesh": mesh, "n": n, "bc": rng.randint(0, 1), "prec": prec,
                "steps": rng.randint(3, 12)}
    if kind == "adjoint":
        steps = rng.randint(4, 10)
        return {"kind": kind, "eq": rng.choice(["advdiff", "gs"]), "mesh": "grid", "n": _log_int(rng, 24, 400),
                "prec": rng.randint(0, 1), "steps": steps, "ckpt": rng.randint(1, steps)}
    if kind == "batch":
        lo = rng.randint(2, 4)
        return {"kind": kind, "count": _log_int(rng, 3, 120), "lo": lo, "hi": rng.randint(lo, 5),
                "steps": rng.randint(5, 30)}
    return {"kind": kind, "mesh": rng.choice(["grid", "cylinder"]), "n": _log_int(rng, 20, 400),
            "bc": rng.randint(0, 1)}


# ---- meshes and parameters ---------------------------------------------------


@functools.lru_cache(maxsize=4)
def _mesh(kind, n):
    if kind == "icosphere":
        return mg.icosphere(n)
    if kind == "grid":
        return mg.jittered_grid(n, seed=0)
    return mg.cylinder(n, max(3, (2 * n) // 3))


def _params(case):
    eq, prec = case.get("eq", "heat"), case.get("prec", 0)
    if eq == "heat":
        return F.default_params(equation=F.HEAT, heat_time_step=1e-3, heat_conductivity=1.0,
                                cg_tolerance=1e-10 if prec else 1e-6)
    if eq == "wave":
        return F.default_params(equation=F.WAVE, wave_time_step=2e-3, wave_c=1.0, wave_scheme=1,
                                cg_tolerance=1e-12 if prec else 1e-7)
    if eq == "advdiff":  # the reference's defaults (implicit scheme)
        return F.default_params(equation=F.ADVECTION_DIFFUSION, cg_tolerance=1e-10 if prec else 1e-6)
    if case["mesh"] == "grid":  # Du, Dv of the 1024 x 1024 workload, scaled with the cell
        s = (1023.0 / max(case["n"] - 1, 1)) ** 2
        return F.default_params(equation=F.REACTION_DIFFUSION, rd_Du=2e-5 * s, rd_Dv=1e-5 * s,
                                cg_tolerance=1e-10 if prec else 1e-5, cg_initial_guess=1, **GS)
    return F.default_params(equation=F.REACTION_DIFFUSION, rd_Du=2e-4, rd_Dv=1e-4,
                            cg_tolerance=1e-10 if prec else 1e-6, cg_initial_guess=1, **{**GS, "rd_time_step": 0.5})


def _adjoint_params(case):
    tol = 1e-12 if case["prec"] else 1e-6
    if case["eq"] == "advdiff":
        return F.default_params(equation=F.ADVECTION_DIFFUSION, advection_scheme=1, advdiff_time_step=1e-2,
                                advdiff_c=1.0, velocity_mode=1, cg_tolerance=tol)
    return F.default_params(equation=F.REACTION_DIFFUSION, rd_Du=2e-5, rd_Dv=1e-5, cg_tolerance=tol, **GS)


def _bumps(xyz, seed, n=3, width2=0.05):
    """Seeded sum of Gaussians centred on points of the mesh."""
    rng = np.random.default_rng(seed)
    p = xyz.astype(np.float64)
    out = np.zeros(len(p))
    for _ in range(n):
        c = p[rng.integers(len(p))]
        out += rng.uniform(0.3, 1.0) * np.exp(-np.sum((p - c) ** 2, axis=1) / width2)
    return out


def _fields(case, xyz, seed):
    """Node-indexed start (u, v) of a time-stepping case."""
    eq = case.get("eq", "heat")
    if eq == "gs":
        if case["mesh"] == "icosphere":
            return mg.sphere_patches(xyz, seed=seed)
        if case["mesh"] == "grid":
            return mg.gray_scott_patches(xyz, seed=seed)
        rng = np.random.default_rng(seed)
        g = np.clip(_bumps(xyz, seed, 6), 0, 1)
        noise = rng.uniform(-0.01, 0.01, (2, len(xyz)))
        return (np.clip(1 - 0.5 * g + noise[0], 0, 1).astype(np.float32),
                np.clip(0.25 * g + noise[1], 0, 1).astype(np.float32))
    u = _bumps(xyz, seed).astype(np.float32)
    if eq == "wave":  # a moving state
        return u, _bumps(xyz, seed + 7777).astype(np.float32)
    return u, np.zeros_like(u)


def _normals(xyz):
    r = np.linalg.norm(xyz, axis=1, keepdims=True)
    return np.ascontiguousarray(xyz / np.maximum(r, 1e-6), dtype=np.float32)


def _unknowns(xyz, tri, bc):
    """Vertices that carry an unknown, in order."""
    if bc == F.NEUMANN:
        return np.arange(len(xyz))
    return np.flatnonzero(mg.boundary_vertices(tri, len(xyz)) == 0)


def _adjoint_inputs(case, seed):
    """Node-indexed inputs of an inverse problem: start, target and, for
    advection-diffusion, the per-element velocity and diffusivity."""
    xyz, tri = _mesh(case["mesh"], case["n"])
    if case["eq"] == "gs":
        u, v = mg.gray_scott_patches(xyz, seed=seed)
        tu, tv = mg.gray_scott_patches(xyz, seed=seed + 1)
        return dict(u=u, v=v, tu=0.5 * (u + tu), tv=0.5 * (v + tv))
    cen = xyz[tri].mean(axis=1)
    vel = (np.stack([-(cen[:, 1] - 0.5), cen[:, 0] - 0.5, np.zeros(len(tri))], 1) * 0.5).astype(np.float32)
    D = 1e-3 * np.exp(0.5 * mg.fourier_field(cen, seed=seed, n_modes=16))
    return dict(u=_bumps(xyz, seed, 1, 0.02), t=_bumps(xyz, seed + 1, 1, 0.03), vel=vel, D=D)


def _instances(case, seed):
    rng = np.random.default_rng(17)  # the sweep's meshes and rates; the seed makes the fields
    insts, starts = [], []
    for i in range(case["count"]):
        xyz, tri = _mesh("icosphere", int(rng.integers(case["lo"], case["hi"] + 1)))
        insts.append(dict(vertices=xyz, triangles=tri, boundary_condition=F.NEUMANN, time_step=0.5, Du=2e-4,
                          Dv=1e-4, feed_rate=float(np.float32(rng.uniform(0.01, 0.06))),
                          kill_rate=float(np.float32(rng.uniform(0.045, 0.07)))))
        starts.append(mg.sphere_patches(xyz, seed=1000 * (seed % 100000) + i))
    return insts, starts


def _real(case):
    return torch.float64 if case.get("prec", 0) else torch.float32


# ---- the passes ------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "batch":
        insts, st["starts"] = _instances(case, seed)
        st["B"] = F.BatchSolver(insts, cg_tolerance=1e-6)
        st["B"].set_initial_guess(1)
        return st
    xyz, tri = _mesh(case["mesh"], case["n"])
    if kind == "open":
        st.update(xyz=xyz, tri=tri, params=_params(case), u=_bumps(xyz, seed).astype(np.float32))
    elif kind == "frame":
        st["s"] = F.CUDASolver(xyz, tri, boundary_condition=F.DIRICHLET, params=_params(case))
        st.update(u=_bumps(xyz, seed).astype(np.float32), normals=_normals(xyz))
    elif kind == "steps":
        dt = _real(case)
        idx = _unknowns(xyz, tri, case["bc"])
        u, v = _fields(case, xyz, seed)
        st["s"] = F.CUDASolver(xyz, tri, boundary_condition=case["bc"], precision=case["prec"],
                               params=_params(case))
        st["in"] = [torch.tensor(f[idx], dtype=dt, device=DEV) for f in (u, v)]
        st["out"] = [torch.zeros(len(idx), dtype=dt, device=DEV) for _ in range(2)]
    elif kind == "adjoint":
        dt = _real(case)
        x = _adjoint_inputs(case, seed)
        s = st["s"] = F.CUDASolver(xyz, tri, boundary_condition=F.NEUMANN, precision=case["prec"],
                                   params=_adjoint_params(case))
        if case["eq"] == "advdiff":
            s.set_element_fields(velocity=x["vel"])
            st["D"] = torch.tensor(x["D"], dtype=dt, device=DEV)
            st["in"] = [torch.tensor(x[k], dtype=dt, device=DEV) for k in ("u", "t")]
        else:
            st["in"] = [torch.tensor(x[k], dtype=dt, device=DEV) for k in ("u", "v", "tu", "tv")]
    torch.cuda.synchronize()  # the handles run on streams of their own
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "frame":
        s = st["s"]
        s.set_values(st["u"])
        s.advance_time(1)
        s.has_numerical_instability()
        return s.get_values(), s.smooth_normals(st["normals"], 0.25)
    if kind == "steps":
        s = st["s"]
        s.set_fields_device(st["in"][0].data_ptr(), st["in"][1].data_ptr())
        s.advance_time(case["steps"])
        s.get_fields_device(st["out"][0].data_ptr(), st["out"][1].data_ptr())
        return st["out"] if case["eq"] in ("gs", "wave") else st["out"][0]
    if kind == "adjoint":
        if case["eq"] == "advdiff":
            st["s"].set_element_diffusivity_device(st["D"])  # an optimiser's new iterate
            return st["s"].adjoint_advdiff_device(*st["in"], case["steps"], case["ckpt"])
        return st["s"].adjoint_gray_scott_device(*st["in"], case["steps"], case["ckpt"])
    if kind == "batch":
        B = st["B"]
        for i, (u, v) in enumerate(st["starts"]):
            B.set_fields(i, u, v)
        B.advance_time(case["steps"])
        out = [B.get_fields(i) for i in range(B.num_instances)]
        return np.concatenate([o[0] for o in out]), np.concatenate([o[1] for o in out])
    s = F.CUDASolver(st["xyz"], st["tri"], boundary_condition=case["bc"], params=st["params"])
    rp, col, K, _ = s.matrix(F.STIFFNESS)
    M = s.matrix(F.MASS)[2]
    s.set_values(st["u"])
    s.advance_time(1)
    out = s.get_values()
    s.close()
    return rp, col, K, M, out


def _sizes(case):
    """Unknowns and stored entries (about) of a mesh."""
    if case["mesh"] == "icosphere":
        n = 10 * 4 ** case["n"] + 2
    elif case["mesh"] == "grid":
        n = case["n"] ** 2
    else:
        n = case["n"] * max(3, (2 * case["n"]) // 3)
    return n, 7 * n


def work(case):
    """Bytes: the operator (values and columns) and the inputs read once, the
    outputs written once.  Operations: one product with the operator and one
    with the right-hand side's matrix per step and field; three such sweeps per
    gradient (forward, replay, reverse)."""
    if case["kind"] == "batch":
        rng = np.random.default_rng(17)
        n = 0
        for _ in range(case["count"]):
            n += 10 * 4 ** int(rng.integers(case["lo"], case["hi"] + 1)) + 2
            rng.uniform(0.01, 0.06), rng.uniform(0.045, 0.07)
        nnz, nf = 7 * n, 2
    else:
        n, nnz = _sizes(case)
        nf = 2 if case.get("eq") == "gs" else 1
    r = 8 if case.get("prec", 0) else 4
    steps = case.get("steps", 1) * (3 if case["kind"] == "adjoint" else 1)
    more = {"frame": 36 * n + 24 * n, "open": 36 * n + 12 * nnz,  # mesh and normals; mesh, K, M and columns
            "adjoint": 3 * n * r * nf}.get(case["kind"], 0)
    return {"bytes": nnz * (4 + r * nf) + 2 * n * r * nf + more, "flops": steps * 4 * nnz * nf}


# ---- the same in 64 bits, plain torch --------------------------------------------------


def _elements(xyz, tri, velocity=None, elem_velocity=None):
    """FP64 element matrices [T, 3, 3]: stiffness, mass, advection."""
    p = torch.tensor(xyz, dtype=torch.float64, device=DEV)[torch.tensor(tri.astype(np.int64), device=DEV)]
    e = [p[:, 2] - p[:, 1], p[:, 0] - p[:, 2], p[:, 1] - p[:, 0]]  # edge opposite each corner
    nrm = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    dbl = nrm.norm(dim=1)  # twice the area
    nrm = nrm / dbl[:, None]
    g = torch.stack([torch.linalg.cross(nrm, x) for x in e], 1) / dbl[:, None, None]  # gradients [T, 3, 3]
    K = 0.5 * dbl[:, None, None] * (g @ g.transpose(1, 2))
    M = dbl[:, None, None] / 24 * (torch.ones(3, 3, dtype=torch.float64, device=DEV)
                                   + torch.eye(3, dtype=torch.float64, device=DEV))
    Adv = None
    if velocity is not None or elem_velocity is not None:
        if elem_velocity is not None:
            w = torch.tensor(elem_velocity, dtype=torch.float64, device=DEV)
        else:
            w = torch.tensor(velocity, dtype=torch.float64, device=DEV).expand(len(tri), 3)
        t = w - (w * nrm).sum(1, keepdim=True) * nrm
        if elem_velocity is None:
            ln = t.norm(dim=1, keepdim=True)
            t = torch.where(ln > 0, t / ln.clamp_min(1e-300), t)
        Adv = (dbl / 6)[:, None, None] * (g @ t[:, :, None]).transpose(1, 2).expand(-1, 3, 3)
    return K, M, Adv


class _System:
    """Assembled FP64 matrices over the unknowns on one shared pattern."""

    def __init__(self, xyz, tri, bc, velocity=None, elem_velocity=None, D=None):
        V = len(xyz)
        onb = torch.tensor(mg.boundary_vertices(tri, V).astype(bool), device=DEV)
        keep = torch.ones(V, dtype=torch.bool, device=DEV) if bc == F.NEUMANN else ~onb
        self.nodes = torch.nonzero(keep).flatten()
        self.N = N = len(self.nodes)
        idx = torch.full((V,), -1, dtype=torch.int64, device=DEV)
        idx[self.nodes] = torch.arange(N, device=DEV)
        t = torch.tensor(tri.astype(np.int64), device=DEV)
        self.tri = idx[t]
        i = self.tri[:, :, None].expand(-1, 3, 3).reshape(-1)
        j = self.tri[:, None, :].expand(-1, 3, 3).reshape(-1)
        ok = (i >= 0) & (j >= 0)
        key, inv = torch.unique(i[ok] * N + j[ok], return_inverse=True)
        self.row, self.col = key // N, key % N
        self.rp = torch.zeros(N + 1, dtype=torch.int64, device=DEV)
        self.rp[1:] = torch.cumsum(torch.bincount(self.row, minlength=N), 0)
        self.diag = torch.nonzero(self.row == self.col).flatten()

        def total(loc, mask=None):
            w = loc.reshape(-1)[ok]
            if mask is not None:
                w = w * mask[ok]
            return torch.zeros(len(key), dtype=torch.float64, device=DEV).index_add_(0, inv, w)

        Kl, Ml, Al = _elements(xyz, tri, velocity, elem_velocity)
        self.Kl = Kl
        self.M, self.K = total(Ml), total(Kl if D is None else D[:, None, None] * Kl)
        if Al is not None:  # entries of boundary vertices do not exist, whatever the condition
            b = onb[t]
            self.Adv = total(Al, (~(b[:, :, None] | b[:, None, :])).reshape(-1).double())

    def mat(self, val):
        return torch.sparse_csr_tensor(self.rp, self.col, val, (self.N, self.N))

    def matT(self, val):
        order = torch.argsort(self.col * self.N + self.row)  # the pattern is symmetric
        return torch.sparse_csr_tensor(self.rp, self.row[order], val[order], (self.N, self.N))


def _solve(A, dinv, b, x, tol=1e-14):
    """Jacobi-PCG on columns b [N, k] (k systems on one matrix) to round-off."""
    r = b - A @ x
    z = dinv * r
    p, g = z.clone(), (r * z).sum(0)
    goal, best, since = tol * b.norm(dim=0), None, 0
    for it in range(6000):
        q = A @ p
        a = g / (p * q).sum(0).clamp_min(1e-300)
        x = x + a * p
        r = r - a * q
        z = dinv * r
        g2 = (r * z).sum(0)
        p = z + (g2 / g.clamp_min(1e-300)) * p
        g = g2
        if it % 25 == 24:
            rn = r.norm(dim=0)
            if bool((rn <= goal).all()):
                break
            worst = float((rn / goal.clamp_min(1e-300)).max())
            if best is None or worst < 0.5 * best:
                best, since = worst, 0
            else:
                since += 1
                if since > 40:
                    break
    return x


class _Op:
    def __init__(self, S, val):
        self.A, self.dinv = S.mat(val), (1 / val[S.diag])[:, None]

    def solve(self, b, x=None):
        return _solve(self.A, self.dinv, b[:, None], (torch.zeros_like(b) if x is None else x)[:, None])[:, 0]


def _exact_steps(case, S, p, u, v):
    eq = case.get("eq", "heat")
    M, K = S.mat(S.M), S.mat(S.K)
    n = case.get("steps", 1)
    if eq == "heat":
        dt = p.heat_time_step
        A = _Op(S, S.M / dt + p.heat_conductivity * S.K)
        for _ in range(n):
            u = A.solve(M @ u / dt, u)
        return u
    if eq == "advdiff":  # implicit: (M/dt + cK) x = b + Adv x, iterated to its fixed point
        dt = p.advdiff_time_step
        A, Adv = _Op(S, S.M / dt + p.advdiff_c * S.K), S.mat(S.Adv)
        for _ in range(n):
            b, x = M @ u / dt, u
            for _ in range(60):
                y = A.solve(b + Adv @ x, x)
                d = float((y - x).norm() / y.norm())
                x = y
                if d < 1e-15:
                    break
            u = x
        return u
    if eq == "wave":
        dt, c2, be, ga = p.wave_time_step, p.wave_c ** 2, p.newmark_beta, p.newmark_gamma
        a = _Op(S, S.M).solve(-c2 * (K @ u))
        A = _Op(S, S.M + be * dt * dt * c2 * S.K)
        for _ in range(n):
            ut = u + dt * v + dt * dt * (0.5 - be) * a
            vt = v + dt * (1 - ga) * a
            a = A.solve(-c2 * (K @ ut), a)
            u, v = ut + be * dt * dt * a, vt + ga * dt * a
        return u, v
    u, v = _gray_scott(S, p, p.rd_feed_rate, p.rd_kill_rate, u[:, None], v[:, None], n)
    return u[:, 0], v[:, 0]


def _gray_scott(S, p, f, k, u, v, steps):
    """Mass-weighted steps of columns (u, v) [N, c] with rates f, k."""
    M, dt = S.mat(S.M), p.rd_time_step
    Au, Av = _Op(S, S.M / dt + p.rd_Du * S.K), _Op(S, S.M / dt + p.rd_Dv * S.K)
    for _ in range(steps):
        uvv = u * v * v
        bu, bv = M @ (u / dt - uvv + f * (1 - u)), M @ (v / dt + uvv - (f + k) * v)
        u, v = _solve(Au.A, Au.dinv, bu, u), _solve(Av.A, Av.dinv, bv, v)
    return u, v


def _cuda64(a):
    return torch.tensor(np.asarray(a), device=DEV).double()


def _scatter(S, V, u):
    out = torch.zeros(V, dtype=torch.float64, device=DEV)
    out[S.nodes] = u
    return out


def _exact_adjoint(case, seed):
    xyz, tri = _mesh(case["mesh"], case["n"])
    p, x, n = _adjoint_params(case), _adjoint_inputs(case, seed), case["steps"]
    dt32 = np.float64 if case["prec"] else np.float32
    if case["eq"] == "advdiff":
        dt, c, sg = p.advdiff_time_step, p.advdiff_c, p.advection_sign
        S = _System(xyz, tri, F.NEUMANN, elem_velocity=x["vel"], D=_cuda64(x["D"].astype(dt32)))
        M, Adv, AdvT = S.mat(S.M), S.mat(S.Adv), S.matT(S.Adv)
        A = _Op(S, S.M / dt + c * S.K)
        u = [_cuda64(x["u"].astype(dt32))]
        for _ in range(n):
            u.append(A.solve(M @ u[-1] / dt + sg * (Adv @ u[-1]), u[-1]))
        d = u[-1] - _cuda64(x["t"].astype(dt32))
        lam = M @ d
        J = 0.5 * float(d @ lam)
        gD = torch.zeros(len(tri), dtype=torch.float64, device=DEV)
        mu = None
        for k in reversed(range(n)):
            mu = A.solve(lam, mu)
            gD -= c * (mu[S.tri][:, None, :] @ S.Kl @ u[k + 1][S.tri][:, :, None]).flatten()
            lam = M @ mu / dt + sg * (AdvT @ mu)
        return J, lam, gD
    dt, f, k = p.rd_time_step, p.rd_feed_rate, p.rd_kill_rate
    S = _System(xyz, tri, F.NEUMANN)
    M, K = S.mat(S.M), S.mat(S.K)
    Au, Av = _Op(S, S.M / dt + p.rd_Du * S.K), _Op(S, S.M / dt + p.rd_Dv * S.K)
    u, v, tu, tv = ([_cuda64(x[name].astype(dt32))] for name in ("u", "v", "tu", "tv"))
    for _ in range(n):
        a, b = u[-1], v[-1]
        u.append(Au.solve(M @ (a / dt - a * b * b + f * (1 - a)), a))
        v.append(Av.solve(M @ (b / dt + a * b * b - (f + k) * b), b))
    du, dv = u[-1] - tu[0], v[-1] - tv[0]
    lu, lv = M @ du, M @ dv
    J = 0.5 * float(du @ lu + dv @ lv)
    gp = np.zeros(4)
    mu = mv = None
    for s in reversed(range(n)):
        mu, mv = Au.solve(lu, mu), Av.solve(lv, mv)
        pu, pv = M @ mu, M @ mv
        a, b = u[s], v[s]
        gp += [float(pu @ (1 - a) - pv @ b), -float(pv @ b), -float(mu @ (K @ u[s + 1])), -float(mv @ (K @ v[s + 1]))]
        lu, lv = ((1 / dt - b * b - f) * pu + b * b * pv,
                  -2 * a * b * pu + (1 / dt + 2 * a * b - f - k) * pv)
    return J, lu, lv, gp


def _smooth_normals(xyz, tri, normals, values, extrusion):
    p = _cuda64(xyz) + (extrusion * values.clamp_min(0)).clamp_max(1)[:, None] * _cuda64(normals)
    t = torch.tensor(tri.astype(np.int64), device=DEV)
    q = p[t]
    n = torch.linalg.cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0])
    out = torch.zeros_like(p)
    for c in range(3):
        out.index_add_(0, t[:, c], n)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "batch":
        insts, starts = _instances(case, seed)
        out = [None] * len(insts)
        for size in sorted({len(d["vertices"]) for d in insts}):  # instances of one mesh: columns of one system
            at = [i for i, d in enumerate(insts) if len(d["vertices"]) == size]
            p = F.default_params(equation=F.REACTION_DIFFUSION, rd_time_step=0.5, rd_Du=2e-4, rd_Dv=1e-4)
            f, k = (_cuda64([insts[i][name] for i in at]) for name in ("feed_rate", "kill_rate"))
            S = _System(insts[at[0]]["vertices"], insts[at[0]]["triangles"], F.NEUMANN)
            u, v = (torch.stack([_cuda64(starts[i][c]) for i in at], 1) for c in (0, 1))
            u, v = _gray_scott(S, p, f, k, u, v, case["steps"])
            for c, i in enumerate(at):
                out[i] = u[:, c], v[:, c]
        return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])
    xyz, tri = _mesh(case["mesh"], case["n"])
    p = _params(case)
    bc = {"frame": F.DIRICHLET}.get(kind, case.get("bc"))
    vel = list(p.advdiff_velocity) if case.get("eq") == "advdiff" else None
    S = _System(xyz, tri, bc, velocity=vel)
    if kind == "steps":
        u, v = (_cuda64(f)[S.nodes] for f in _fields(case, xyz, seed))
        return _exact_steps(case, S, p, u, v)
    u = _exact_steps({"eq": "heat"}, S, p, _cuda64(_bumps(xyz, seed).astype(np.float32))[S.nodes], None)
    values = _scatter(S, len(xyz), u)
    if kind == "frame":
        return values, _smooth_normals(xyz, tri, _normals(xyz), values, 0.25)
    return None, None, S.K, S.M, values
