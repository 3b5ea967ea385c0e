"""The work that users of this framework have it do, as cases that can be timed and checked.

Most cases are one time step of a scene whose particle state lives on the GPU:
the caller hands the state in as device arrays (``wcg_upload_liquid_device``),
steps (``wcg_step``: the sub-step count, then grid build, P2G, prediction,
pressure solve, extrapolation, constraint, correction, G2P and advection) and
takes the new state back (``wcg_download_liquid_device``).  Beside them stand
the reverse mode of a sub-step through ``autograd.substep``, a batch of scenes
(``FluidBatch``) and the solve of a caller-assembled system
(``wcg_pcg_solve_csr``).

Every cell size is a power of two and the solid box spans whole cells, so that
the position of a wall against a grid corner is the same in FP32, in FP64 and
in the plain restatement below.

``exact`` restates one step in plain torch at 64 bits on a dense grid, with
the pressure solved to 1e-13; the framework stops at its default criterion of
1e-6, which is most of the difference that its results show.
"""
import math

import numpy as np
import torch

from libwetcloth_b200 import _capi, autograd, scenes
from libwetcloth_b200.solver import FluidBatch, FluidScene, make_params

DEV = "cuda"


# --------------------------------------------------------------------------
# the cases
def listed():
    return [
        # the smallest scene of the tests: launches and waits are what it costs
        step("dam16_fp64", "dam", 16, "fp64", "mic0"),
        # the 64^3 dam break in the default precision and solver
        step("dam64_fp64", "dam", 64, "fp64", "mic0"),
        # an odd size with the particle correction on (strength 0.2, the
        # reference's parser default), as interactive FP32 scenes run it
        step("dam90_correct_fp32", "dam", 90, "fp32", "mic0", correction=0.2),
        # a half-filled box at 128^3, 2 particles per cell, full precision
        step("half128_fp64", "half", 128, "fp64", "mic0"),
        # the same with the reference's default solver (multigrid-PCG)
        step("half128_mg_fp64", "half", 128, "fp64", "mg"),
        # the benchmark scene: 256^3 half box, 16.8M particles, FP32 with FP64
        # refinement
        step("half256_fp32", "half", 256, "fp32", "mic0"),
        # the largest scene with the multigrid solver
        step("half256_mg_fp32", "half", 256, "fp32", "mg"),
        # liquid onto a cloth sheet: the solid phase's transfers and the drag
        step("cloth128_fp32", "sheet", 128, "fp32", "mic0", dt=5e-4),
        # a gradient through one sub-step (forward and backward), as the
        # optimisation runs take 200 of
        {"name": "adjoint48_fp64", "kind": "adjoint", "scene": "dam", "n": 48, "precision": "fp64",
         "solver": "mic0", "ppc": 8, "dt": 1e-3, "correction": 0.0},
        # many small scenes of uneven size stepped together
        {"name": "batch12_fp32", "kind": "batch", "count": 12, "n": 28, "n_max": 56,
         "precision": "fp32", "solver": "mic0", "ppc": 8, "dt": 1e-3, "correction": 0.0},
        # a system that the caller assembled (an implicit solve of its own)
        {"name": "csr40_fp64", "kind": "csr", "n": 40, "extra": 0.02, "tol": 1e-8},
    ]


def step(name, scene, n, precision, solver, ppc=None, dt=1e-3, correction=0.0):
    return {"name": name, "kind": "step", "scene": scene, "n": n, "precision": precision,
            "solver": solver, "ppc": ppc if ppc else (2 if scene == "half" else 8), "dt": dt,
            "correction": correction}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dam", "dam", "half", "half", "half", "sheet", "adjoint", "batch", "csr"])
    precision = rng.choice(["fp64", "fp32"])
    solver = rng.choice(["mic0", "mic0", "mg"])
    if kind == "half":
        c = step("", "half", size(24, 240 if precision == "fp32" else 160), precision, solver,
                 ppc=rng.choice([2, 2, 4]))
    elif kind == "dam":
        c = step("", "dam", size(12, 128), precision, solver,
                 correction=rng.choice([0.0, 0.0, 0.2]))
    elif kind == "sheet":
        c = step("", "sheet", size(24, 144), precision, solver, dt=5e-4)
    elif kind == "adjoint":
        c = {"kind": "adjoint", "scene": "dam", "n": size(16, 72), "precision": precision,
             "solver": solver, "ppc": 8, "dt": 1e-3, "correction": 0.0}
    elif kind == "batch":
        n = size(16, 36)
        c = {"kind": "batch", "count": rng.randint(3, 16), "n": n, "n_max": n + rng.randint(4, 28),
             "precision": precision, "solver": "mic0", "ppc": 8, "dt": 1e-3, "correction": 0.0}
    else:
        c = {"kind": "csr", "n": size(8, 48), "extra": rng.choice([0.0, 0.02, 0.1]), "tol": 1e-8}
    c.pop("name", None)
    return c


# --------------------------------------------------------------------------
# inputs
def cell_size(n):
    """The largest power of two with n cells in at most one unit."""
    return 2.0 ** -math.ceil(math.log2(n))


def block(dx, lo, hi, ppc, gen):
    """Jittered particles that fill [lo, hi]: one per half-cell for 8 per
    cell, else ppc in each cell (scenes.liquid_block, on the GPU)."""
    h, per = (dx / 2, 1) if ppc == 8 else (dx, ppc)
    axes = [torch.arange(math.floor(lo[a] / h), math.ceil(hi[a] / h), device=DEV) for a in range(3)]
    axes = [ax[((ax + 0.5) * h >= lo[a]) & ((ax + 0.5) * h <= hi[a])] for a, ax in enumerate(axes)]
    z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    cells = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1).repeat_interleave(per, 0)
    jitter = torch.rand(cells.shape, generator=gen, device=DEV, dtype=torch.float64)
    return (cells + jitter) * h


def noise_velocity(x, dx, n, amplitude, sigma, gen):
    """Velocity at x and its gradient (9 values, row-major) from the curl of
    Gaussian-smoothed noise, sigma cells wide, scaled to a largest speed of
    `amplitude` (scenes.curl_noise_velocity, on the GPU)."""
    k = torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) * (2 * math.pi)
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    psi = []
    for _ in range(3):
        w = torch.randn((n, n, n), generator=gen, device=DEV, dtype=torch.float64)
        psi.append(torch.fft.ifftn(torch.fft.fftn(w) * torch.exp(-0.5 * sigma * sigma * kk)).real)

    def d(f, axis):
        return (torch.roll(f, -1, axis) - torch.roll(f, 1, axis)) / (2.0 * dx)

    vel = torch.stack([d(psi[2], 1) - d(psi[1], 2), d(psi[0], 2) - d(psi[2], 0),
                       d(psi[1], 0) - d(psi[0], 1)], -1)
    vel = (vel * (amplitude / vel.square().sum(-1).sqrt().max())).reshape(-1, 3)

    def at(p):
        p = p / dx - 0.5
        i = torch.floor(p).long()
        f = p - i
        out = torch.zeros_like(p)
        for t in range(8):
            o = [t & 1, t >> 1 & 1, t >> 2]
            w = 1.0
            for a in range(3):
                w = w * (f[:, a] if o[a] else 1 - f[:, a])
            q = [(i[:, a] + o[a]).clamp(0, n - 1) for a in range(3)]
            out += w[:, None] * vel[(q[0] * n + q[1]) * n + q[2]]
        return out

    C = torch.empty((x.shape[0], 3, 3), device=DEV, dtype=torch.float64)
    for a in range(3):
        e = torch.zeros(3, device=DEV, dtype=torch.float64)
        e[a] = 0.5 * dx
        C[:, :, a] = (at(x + e) - at(x - e)) / dx
    return at(x), C


def make(case, n, seed):
    """(SceneParams, dict of particle tensors, elasto set or None)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 1000003 + n)
    dx = cell_size(n)
    side = n * dx
    prm = scenes.SceneParams(dx=dx, box_center=(side / 2,) * 3, box_half=(side / 2,) * 3,
                             correction_strength=case["correction"])
    elasto = None
    scene = case["scene"]
    if scene == "half":
        x = block(dx, (0.0,) * 3, (side, 0.5 * side, side), case["ppc"], gen)
        v, C = noise_velocity(x, dx, n, 0.5, 4.0, gen)
    elif scene == "dam":
        x = block(dx, (0.0,) * 3, (0.4 * side, 0.8 * side, 0.4 * side), case["ppc"], gen)
        v, C = noise_velocity(x, dx, n, 0.5, 4.0, gen)
    else:  # a spinning liquid sphere that meets the sheet at y = 0.4
        c = torch.tensor([0.5, 0.5, 0.5], device=DEV, dtype=torch.float64) * side
        x = block(dx, (0.35 * side,) * 3, (0.65 * side,) * 3, case["ppc"], gen)
        middle = (torch.floor(x / (dx / 2)) + 0.5) * (dx / 2)  # of the half-cell, not the particle
        x = x[(middle - c).norm(dim=1) <= 0.15 * side].contiguous()
        r = x - c
        v = torch.stack([3.0 * r[:, 2], torch.full_like(r[:, 0], -1.0), -3.0 * r[:, 0]], 1)
        C = torch.zeros((x.shape[0], 3, 3), device=DEV, dtype=torch.float64)
        C[:, 0, 2], C[:, 2, 0] = 3.0, -3.0
        elasto = scenes.cloth_sheet((0.1 * side,) * 2, (0.9 * side,) * 2, 0.4 * side, dx,
                                    int(seed) % 100000 + 1)
    r = scenes.particle_radius(dx, case["ppc"])
    vol = 4.0 / 3.0 * math.pi * r ** 3
    full = lambda a: torch.full((x.shape[0],), a, device=DEV, dtype=torch.float64)  # noqa: E731
    parts = {"x": x.contiguous(), "v": v.contiguous(), "C": C.contiguous(),
             "m": full(prm.liquid_density * vol), "vol": full(vol), "r": full(r)}
    return prm, parts, elasto


def batch_sizes(case):
    """Grid sizes of a batch: the smallest and the largest always among them."""
    rng = np.random.default_rng(case["count"])
    return [case["n"], case["n_max"]] + [int(rng.integers(case["n"], case["n_max"] + 1))
                                         for _ in range(case["count"] - 2)]


def csr_system(case, seed):
    """A symmetric, diagonally dominant system: 7-point couplings of random
    weight on an n^3 grid and a share of long-range ones, sorted CSR rows."""
    rng = np.random.default_rng(int(seed))
    n = case["n"]
    idx = np.arange(n ** 3).reshape(n, n, n)
    i, j = [], []
    for ax in range(3):
        a = np.moveaxis(idx, ax, 0)
        i.append(a[:-1].ravel())
        j.append(a[1:].ravel())
    far = int(case["extra"] * n ** 3)
    i.append(rng.integers(0, n ** 3, far))
    j.append(rng.integers(0, n ** 3, far))
    i, j = np.concatenate(i), np.concatenate(j)
    w = np.where(np.arange(i.size) < i.size - far, -rng.uniform(0.2, 1.0, i.size),
                 -rng.uniform(0.05, 0.5, i.size))
    lo, hi = np.minimum(i, j), np.maximum(i, j)
    keep = lo != hi
    pair, first = np.unique((lo * n ** 3 + hi)[keep], return_index=True)
    w = w[keep][first]
    lo, hi = pair // n ** 3, pair % n ** 3
    diag = rng.uniform(0.002, 0.02, n ** 3)
    np.add.at(diag, lo, -w)
    np.add.at(diag, hi, -w)
    row = np.concatenate([lo, hi, np.arange(n ** 3)])
    col = np.concatenate([hi, lo, np.arange(n ** 3)])
    val = np.concatenate([w, w, diag])
    order = np.lexsort((col, row))
    rowstart = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n ** 3))])
    return (rowstart.astype(np.int32), col[order].astype(np.int32), val[order],
            rng.standard_normal(n ** 3))


# --------------------------------------------------------------------------
# the framework's calls
def open_scene(case, prm):
    prec = _capi.WCG_FP64 if case["precision"] == "fp64" else _capi.WCG_FP32_REFINE
    solver = _capi.WCG_SOLVER_MIC0 if case["solver"] == "mic0" else _capi.WCG_SOLVER_MG
    return FluidScene(params=make_params(prm, prec, solver=solver))


def holder(case, n, seed):
    prm, p, elasto = make(case, n, seed)
    out = {k: torch.empty_like(p[k]) for k in ("x", "v", "C")}
    return {"scene": open_scene(case, prm), "p": p, "out": out, "elasto": elasto}


def prepare(case, seed):
    if case["kind"] == "csr":
        return {"case": case, "system": csr_system(case, seed)}
    if case["kind"] == "batch":
        hold = [holder({**case, "scene": "dam"}, n, int(seed) * 100 + k)
                for k, n in enumerate(batch_sizes(case))]
        s = {"case": case, "hold": hold, "batch": FluidBatch([h["scene"] for h in hold])}
    elif case["kind"] == "adjoint":
        prm, p, _ = make(case, case["n"], seed)
        s = {"case": case, "scene": open_scene(case, prm), "p": p, "cot": cotangents(p, seed)}
        s["scene"].upload(*[p[k].cpu().numpy() for k in ("x", "v", "C", "m", "vol", "r")])
    else:
        s = {"case": case, **holder(case, case["n"], seed)}
    torch.cuda.synchronize()
    return s


def cotangents(p, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) + 77)
    return [torch.randn(p[k].shape, generator=gen, device=DEV, dtype=torch.float64)
            * (1.0 if k != "C" else 0.01) for k in ("x", "v", "C")]


def put(h):
    p, sc = h["p"], h["scene"]
    sc.upload_device(p["x"].shape[0], *[p[k].data_ptr() for k in ("x", "v", "C", "m", "vol", "r")])
    if h["elasto"] is not None:
        sc.upload_elasto(h["elasto"])
    sc.set_correction_count(0)


def take(h):
    sc, o = h["scene"], h["out"]
    _capi.check(sc.L.wcg_download_liquid_device(sc.h, *[o[k].data_ptr() for k in ("x", "v", "C")]))
    if h["elasto"] is None:
        return [o["x"], o["v"], o["C"]]
    return [o["x"], o["v"], o["C"], *sc.download_elasto()]


def run(state):
    case = state["case"]
    if case["kind"] == "csr":
        rs, col, val, b = state["system"]
        return _capi.pcg_solve_csr(rs, col, val, b, case["tol"], 2000)[0]
    if case["kind"] == "batch":
        for h in state["hold"]:
            put(h)
        state["batch"].step(case["dt"])
        return [t for h in state["hold"] for t in take(h)]
    if case["kind"] == "adjoint":
        p = state["p"]
        x, v, C = (p[k].detach().requires_grad_(True) for k in ("x", "v", "C"))
        out = autograd.substep(state["scene"], x, v, C.reshape(-1, 9), case["dt"],
                               correction_call=0)
        got = torch.autograd.grad(out, (x, v, C), [g.reshape(o.shape) for g, o in
                                                   zip(state["cot"], out)])
        return [*[o.detach() for o in out], *got]
    put(state)
    state["scene"].step(case["dt"])
    return take(state)


# --------------------------------------------------------------------------
# what a pass cannot do without
def particles(case, n):
    side = {"half": 0.5 * n ** 3, "dam": 0.128 * n ** 3, "sheet": 0.01414 * n ** 3}[case["scene"]]
    return side * case["ppc"]


def work(case):
    if case["kind"] == "csr":
        n = case["n"] ** 3
        nnz = n * (7 + 2 * case["extra"])
        return {"bytes": 12 * nnz + 4 * n + 16 * n, "flops": 30 * (4 * nnz + 10 * n)}
    if case["kind"] == "batch":
        np_ = sum(particles({**case, "scene": "dam"}, n) for n in batch_sizes(case))
    else:
        np_ = particles(case, case["n"])
    # state in (18 values) and out (15) per particle; weights, P2G and G2P of
    # 27 nodes on three face grids and the cell centres
    one = {"bytes": 33 * 8 * np_, "flops": 27 * (3 * 22 + 12) * np_}
    if case["kind"] == "adjoint":  # forward and reverse: cotangents in and out
        return {"bytes": one["bytes"] + 30 * 8 * np_, "flops": 3 * one["flops"]}
    if case.get("scene") == "sheet":
        nv = (0.8 * case["n"]) ** 2
        one["bytes"] += 45 * 8 * nv
    return one


def tolerance(case):
    """About four times the largest difference from `exact` that was measured:
    the solver's stopping criterion in FP64; in FP32 also the rounding of
    positions and velocities, which the ghost-fluid fraction of a surface that
    grazes a cell centre multiplies by up to 100 in single particles."""
    if case["kind"] == "csr":
        return {"rel": 1e-7}
    if case["kind"] == "adjoint":
        return {"rel": 2e-5, "max": 1e-3} if case["precision"] == "fp64" else \
            {"rel": 1e-4, "max": 4e-3}
    return {"rel": 4e-6, "max": 2e-4} if case["precision"] == "fp64" else {"rel": 6e-4, "max": 0.4}


# --------------------------------------------------------------------------
# one step in plain torch, 64 bits, on a dense grid
def bspline(d):
    d = d.abs()
    return torch.where(d < 0.5, 0.75 - d * d,
                       torch.where(d < 1.5, 0.5 * (1.5 - d) * (1.5 - d), torch.zeros_like(d)))


def inside2(a, b):
    """Part of the segment a -> b where phi < 0."""
    cut = (a < 0) != (b < 0)
    part = torch.where(a < 0, a, -b) / torch.where(cut, a - b, 1.0)
    return torch.where(cut, part, ((a < 0) & (b < 0)).to(a.dtype))


def inside4(c):
    """Part of a square where phi < 0, corner values c in cyclic order.  The
    scenes' walls lie on grid planes, so opposite corners alone never occur."""
    count = sum((q < 0).long() for q in c)
    out = torch.where(count == 4, 1.0, 0.0).to(c[0].dtype)
    for k in range(4):
        p = [c[(k + t) % 4] for t in range(4)]
        one = (count == 1) & (p[0] < 0)
        out = torch.where(one, 0.5 * inside2(p[0], p[3]) * inside2(p[0], p[1]), out)
        two = (count == 2) & (p[0] < 0) & (p[1] < 0)
        out = torch.where(two, 0.5 * (inside2(p[0], p[3]) + inside2(p[1], p[2])), out)
        three = (count == 3) & (p[0] >= 0)
        out = torch.where(three, 1 - 0.5 * (1 - inside2(p[0], p[3])) * (1 - inside2(p[0], p[1])),
                          out)
    return out


def shift(f, axis, by, fill=0):
    """g[i] = f[i + by] along an axis, `fill` outside."""
    out = torch.full_like(f, fill)
    n = f.shape[axis]
    if by > 0:
        out.narrow(axis, 0, n - by).copy_(f.narrow(axis, by, n - by))
    else:
        out.narrow(axis, -by, n + by).copy_(f.narrow(axis, 0, n + by))
    return out


class Shift(torch.autograd.Function):
    @staticmethod
    def forward(ctx, f, axis, by):
        ctx.a = (axis, by)
        return shift(f, axis, by)

    @staticmethod
    def backward(ctx, g):
        return shift(g, ctx.a[0], -ctx.a[1]), None, None


class Solve(torch.autograd.Function):
    """p of A p = b; A: diagonal and couplings to the +x, +y, +z cells."""

    @staticmethod
    def apply_a(d, off, p):
        q = d * p
        for a in range(3):
            q = q + off[a] * shift(p, a, 1) + shift(off[a] * p, a, -1)
        return q

    @staticmethod
    def cg(d, off, b):
        inv = torch.where(d > 0, 1 / d, torch.zeros_like(d))
        x, r = torch.zeros_like(b), b.clone()
        s = z = inv * r
        rho = (z * r).sum()
        goal = 1e-13 * b.abs().max()
        for it in range(6000):
            q = Solve.apply_a(d, off, s)
            al = rho / (s * q).sum()
            x = x + al * s
            r = r - al * q
            if it % 25 == 0 and r.abs().max() <= goal:
                break
            z = inv * r
            new = (z * r).sum()
            s = z + (new / rho) * s
            rho = new
        return x

    @staticmethod
    def forward(ctx, d, o0, o1, o2, b):
        p = Solve.cg(d, (o0, o1, o2), b)
        ctx.save_for_backward(d, o0, o1, o2, p)
        return p

    @staticmethod
    def backward(ctx, g):
        d, o0, o1, o2, p = ctx.saved_tensors
        lam = Solve.cg(d, (o0, o1, o2), torch.where(d > 0, g, torch.zeros_like(g)))
        return (-lam * p, *[-(lam * shift(p, a, 1) + shift(lam, a, 1) * p) for a in range(3)], lam)


class Plain:
    """One sub-step of a scene in plain torch."""

    def __init__(self, prm, p, elasto, dt):
        self.prm, self.p, self.dt, self.dx = prm, p, dt, prm.dx
        self.e = None
        x = p["x"].detach()
        allx = x
        if elasto is not None:
            t = lambda a: torch.as_tensor(a, device=DEV, dtype=torch.float64)  # noqa: E731
            self.e = {"x4": t(elasto.x4), "v4": t(elasto.v4), "B": t(elasto.B).reshape(-1, 3, 3),
                      "m": (t(elasto.m4) + t(elasto.fm4))[:, :3], "rv": t(elasto.rest_vol),
                      "rf": t(elasto.rest_vf), "fv": t(elasto.fluid_vol),
                      "sf": t(elasto.shape_factor), "o": t(elasto.orientation)}
            allx = torch.cat([x, self.e["x4"][:, :3]])
        bs = 4 * self.dx
        lo = torch.floor(allx.min(0).values / (2 * bs)) * 2 * bs
        hi = torch.ceil(allx.max(0).values / (2 * bs)) * 2 * bs
        self.org = lo - 3 * bs
        self.N = [4 * max(1, math.ceil((float(h - l) + 6 * bs) / bs)) for l, h in zip(lo, hi)]
        self.nn = self.N[0] * self.N[1] * self.N[2]

    # nodes of axis-offset o (0 or 1/2 per axis) around positions x
    def stencil(self, x, o):
        off = torch.tensor(o, device=DEV, dtype=torch.float64)
        lp = (x.detach() - self.org) / self.dx - off
        fl = torch.floor(lp)
        base = fl.long() - 1 + (lp - fl > 0.5).long()
        q = (x - self.org) / self.dx - off  # in cells, follows x
        return base, q

    def nodes(self, st):
        """The 27 nodes of a stencil: (linear index, weight, (x_n - x) / dx)."""
        base, q = st
        w = [[bspline(q[:, a] - (base[:, a] + t)) for t in range(3)] for a in range(3)]
        for k in range(3):
            for j in range(3):
                for i in range(3):
                    o = (i, j, k)
                    idx = ((base[:, 0] + i) * self.N[1] + base[:, 1] + j) * self.N[2] + base[:, 2] + k
                    d = torch.stack([base[:, a] + o[a] - q[:, a] for a in range(3)], 1)
                    yield idx, w[0][i] * w[1][j] * w[2][k], d

    def zeros(self, dtype=torch.float64):
        return torch.zeros(self.nn, device=DEV, dtype=dtype)

    def grid(self, f):
        return f.reshape(self.N)

    def activate(self, xs):
        nb = [n // 4 for n in self.N]
        on = torch.zeros(nb, device=DEV, dtype=torch.bool)
        for x in xs:
            for o in ((0, .5, .5), (.5, 0, .5), (.5, .5, 0), (0, 0, 0), (.5, .5, .5)):
                base, _ = self.stencil(x, o)
                for t in range(8):
                    b = [(base[:, a] + 2 * (t >> a & 1)) >> 2 for a in range(3)]
                    on[b[0], b[1], b[2]] = True
        f = on.to(torch.float32)[None, None]
        on = torch.nn.functional.max_pool3d(f, 3, 1, 1)[0, 0] > 0
        for a in range(3):
            on = on.repeat_interleave(4, a)
        return on

    def wall(self, pos):
        """Solid phi of the box whose inside holds the liquid."""
        c = torch.tensor(self.prm.box_center, device=DEV, dtype=torch.float64)
        h = torch.tensor(self.prm.box_half, device=DEV, dtype=torch.float64)
        d = [(pos[a] - c[a]).abs() - h[a] for a in range(3)]
        m = torch.maximum(torch.maximum(d[0], d[1]), d[2]).clamp(max=0)
        s = sum(q.clamp(min=0) ** 2 for q in d).sqrt()
        return (-(m + s - self.prm.box_radius)).clamp(max=12 * self.dx)

    def positions(self, o):
        ax = [self.org[a] + (torch.arange(self.N[a], device=DEV) + o[a]) * self.dx
              for a in range(3)]
        return torch.meshgrid(*ax, indexing="ij")

    def p2g(self):
        p, dx = self.p, self.dx
        x, v, C, m, vol = p["x"], p["v"], p["C"].reshape(-1, 3, 3), p["m"], p["vol"]
        self.mass, self.vel, self.vol = [], [], []
        for a in range(3):
            o = [0.5] * 3
            o[a] = 0.0
            mass, mom, vf = self.zeros(), self.zeros(), self.zeros()
            for idx, w, d in self.nodes(self.stencil(x, o)):
                mom = mom.index_add(0, idx, (v[:, a] + (C[:, a] * d).sum(1) * dx) * m * w)
                mass = mass.index_add(0, idx, m * w)
                vf = vf.index_add(0, idx, vol * w)
            heavy = mass > 1e-20
            self.mass.append(self.grid(mass))
            self.vel.append(self.grid(torch.where(heavy, mom / torch.where(heavy, mass, 1.0), 0.0)))
            self.vol.append(self.grid(vf))
        rad = torch.maximum(p["r"], torch.full_like(p["r"], 0.883644 * dx))
        phi = torch.full((self.nn,), 12 * dx, device=DEV, dtype=torch.float64)
        cen = self.zeros()
        for idx, w, d in self.nodes(self.stencil(x, (0.5,) * 3)):
            phi = phi.scatter_reduce(0, idx, d.square().sum(1).sqrt() * dx - rad, "amin")
            if self.e is not None:
                cen = cen.index_add(0, idx, vol * w)
        phi = self.grid(phi)
        self.phi = torch.where(self.wall(self.positions((.5, .5, .5))) < 0, -0.5 * dx, phi)
        # saturation per face; with cloth the held liquid and the solid volume join
        self.sat = [(f / dx ** 3).clamp(0, 1) for f in self.vol]
        if self.e is not None:
            self.p2g_solid(self.grid(cen))

    def p2g_solid(self, vliq):
        e, dx = self.e, self.dx
        x, dV = e["x4"][:, :3], dx ** 3
        self.E = []
        for a in range(3):
            o = [0.5] * 3
            o[a] = 0.0
            keys = ("mom", "mass", "vs", "vfe", "sf", "w", "o0", "o1", "o2")
            s = {k: self.zeros() for k in keys}
            for idx, w, d in self.nodes(self.stencil(x, o)):
                vel = e["v4"][:, a] + (e["B"][:, a] * d).sum(1) * dx
                add = {"mom": vel * e["m"][:, a], "mass": e["m"][:, a], "vs": e["rv"] * e["rf"],
                       "vfe": e["fv"], "sf": e["sf"], "w": torch.ones_like(w),
                       "o0": e["o"][:, 0], "o1": e["o"][:, 1], "o2": e["o"][:, 2]}
                for k in keys:
                    s[k].index_add_(0, idx, add[k] * w)
            s = {k: self.grid(f) for k, f in s.items()}
            some = s["mass"] > 1e-20
            ln = (s["o0"] ** 2 + s["o1"] ** 2 + s["o2"] ** 2).sqrt()
            self.E.append({
                "mass": s["mass"],
                "vel": torch.where(some, s["mom"] / torch.where(some, s["mass"], 1.0), 0.0),
                "vol": s["vs"] + s["vfe"], "psi": (s["vs"] / dV).clamp(0, 1),
                "sf": torch.where(s["w"] > 1e-20, s["sf"] / s["w"], s["sf"]),
                "o": [torch.where(ln > 1e-20, s["o%d" % q] / ln, s["o%d" % q]) for q in range(3)]})
            self.sat[a] = ((self.vol[a] + s["vfe"]) / (dV - s["vs"]).clamp(min=1e-20)).clamp(0, 1)
        vl, vs = self.zeros(), self.zeros()
        for idx, w, _ in self.nodes(self.stencil(x, (0.5,) * 3)):
            vl.index_add_(0, idx, e["fv"] * w)
            vs.index_add_(0, idx, e["rv"] * e["rf"] * w)
        vl, vs = self.grid(vl), self.grid(vs)
        psi = (vs / dV).clamp(0, 1)
        sat = ((vliq + vl) / (dV - vs).clamp(min=1e-20)).clamp(0, 1)
        cap = psi / (1 - psi) * 72.8 * math.cos(40.8 / 180 * math.pi) / 0.005
        self.pore = torch.where(1 - psi < 1e-20, 0.0, cap * (1 - sat))

    def drag(self, a):
        """getDragCoeffWithOrientation on the faces of axis a."""
        E, prm = self.E[a], self.prm
        psi, n2 = E["psi"], sum(q * q for q in E["o"])
        on = (psi != 0) & (self.sat[a] != 0) & ~(n2 < 1e-20)
        ps = torch.where(on, psi, 0.5)
        lp, di, yp = -torch.log(ps), 0.01, 1.6
        ka = ((lp - 1.476 + 2 * ps - 0.5 * ps ** 2) / (16 * ps) * di * di).clamp(min=1e-20)
        kb = ((lp - 1.476 + 2 * ps - 1.774 * ps ** 2 + 4.078 * ps ** 3) / (32 * ps) * di * di)
        kb = kb.clamp(min=1e-20)
        mu, rho = prm.drag_viscosity, prm.liquid_density
        inertial = 0.1428869017 * di ** (yp - 1) * mu ** (1 - yp)
        flow = (rho * (self.vel[a] - E["vel"]).abs()) ** yp
        den = (1 - ps) ** 1.5
        ca = (mu / ka + inertial / (den * ka.sqrt()) * flow).clamp(max=1e63)
        cb = (mu / kb + inertial / (den * kb.sqrt()) * flow).clamp(max=1e63)
        cxy, cz = ca * (1 - E["sf"]) + cb * E["sf"], ca * E["sf"] + cb * (1 - E["sf"])
        n2 = torch.where(on, n2, 1.0)
        return torch.where(on, cxy + (cz - cxy) * E["o"][a] * sum(E["o"]) / n2, 0.0)

    def step(self):
        dx, dt = self.dx, self.dt
        self.on = self.activate([self.p["x"]] + ([self.e["x4"][:, :3]] if self.e else []))
        self.p2g()
        on, phi = self.on, self.phi
        corner = self.wall(self.positions((0, 0, 0)))
        self.sphi = torch.where(on, corner, 3 * dx)
        cw = torch.where(on, corner, 0.5 * dx)
        up = lambda f, *axes: f if not axes else up(shift(f, axes[0], 1, 0.5 * dx), *axes[1:])  # noqa: E731
        weight = [(1 - inside4([cw, up(cw, b), up(cw, b, c), up(cw, c)])).clamp(0, 1)
                  for b, c in ((1, 2), (0, 2), (0, 1))]
        # prediction
        rhs, inv_c, psi_fs, vstar, qd = [], [], [], [], []
        for a in range(3):
            m, u, g = self.mass[a], self.vel[a], self.prm.gravity[a]
            r = m * g * dt
            heavy = m > 1e-20
            ic = torch.where(heavy, 1 / torch.where(heavy, m, 1.0), 1.0)
            ps = ic * m
            if self.e is not None:
                E = self.E[a]
                grad = (self.pore - shift(torch.where(on, self.pore, 0.0), a, -1)) / dx
                n2 = sum(q * q for q in E["o"])
                pc = torch.where(n2 > 0, (2 - E["sf"]) + (2 * E["sf"] - 1) * E["o"][a] *
                                 sum(E["o"]) / torch.where(n2 > 0, n2, 1.0), 0.0)
                r = r + torch.where((self.vol[a] > 0) & (weight[a] > 0),
                                    grad * self.vol[a] * dt * self.sat[a] * weight[a] * pc, 0.0)
                hdv = dt * self.drag(a) * (E["vol"] + self.vol[a])
                msh = E["mass"] + hdv
                Q = torch.where(msh > 1e-20, hdv / torch.where(msh > 1e-20, msh, 1.0), 1.0)
                Cm = m + Q * E["mass"]
                ic = torch.where(Cm > 1e-20, 1 / torch.where(Cm > 1e-20, Cm, 1.0), 1.0)
                ps = (1 - E["psi"]) * ic * m
                qd.append(Q)
            r = r + m * u
            rhs.append(r)
            inv_c.append(ic)
            psi_fs.append(ps)
            vstar.append(torch.where(heavy, r / torch.where(heavy, m, 1.0), r))
        # pressure system
        wet = on & (phi < 0)
        is_open = torch.zeros_like(wet)
        for a in range(3):
            here = on & (weight[a] > 0)
            is_open |= here | shift(here, a, 1)
        dof = wet & is_open
        diag, b, off = torch.zeros_like(phi), torch.zeros_like(phi), []
        for a in range(3):
            w = torch.where(on, weight[a], 0.0)
            t = vstar[a] * psi_fs[a] * w / dx
            t = torch.where(on, t, 0.0)
            vf = self.vol[a]
            term = inv_c[a] * vf
            if self.e is not None:
                E = self.E[a]
                term = (1 - E["psi"]) * inv_c[a] * (vf + E["vol"] * qd[a])
            term = w * dt / dx ** 2 * torch.where(on, term, 0.0)
            low, low_on = Shift.apply(phi, a, -1), shift(on, a, -1)
            both = on & low_on & (w > 0)  # the face between cell - 1 and cell
            th = torch.where(both, inside2(low, phi), 1.0).clamp(min=0.01)
            # lower side of this cell, then upper side: the face of cell + 1
            fluid_low, fluid = low < 0, phi < 0
            d_here = torch.where(both, torch.where(fluid_low, term, term / th), 0.0)
            d_low = torch.where(both, torch.where(fluid, term, term / th), 0.0)
            diag = diag + d_here + Shift.apply(d_low, a, 1)
            b = b + t - Shift.apply(t, a, 1)
            pair = dof & shift(dof, a, 1)
            off.append(torch.where(pair, -Shift.apply(torch.where(both, term, 0.0), a, 1), 0.0))
        zero = torch.zeros_like(phi)
        pr = Solve.apply(torch.where(dof, diag, zero), *off, torch.where(dof, b, zero))
        # pressure gradient, extrapolation, wall constraint
        U = []
        for a in range(3):
            low_on = shift(on, a, -1)
            ph_l = torch.where(low_on, Shift.apply(phi, a, -1), 0.0)
            p_l = torch.where(low_on, Shift.apply(pr, a, -1), 0.0)
            valid = on & (weight[a] > 0) & ((ph_l < 0) | (phi < 0))
            cut = (phi >= 0) | (ph_l >= 0)
            th = torch.where(valid & cut, inside2(ph_l, phi).clamp(min=0.01), 1.0)
            vf, r = self.vol[a], rhs[a]
            if self.e is not None:
                E = self.E[a]
                r = r + qd[a] * E["mass"] * E["vel"]
                vf = vf + E["vol"] * qd[a]
            r = r - torch.where(valid, (pr - p_l) / (dx * th) * dt * vf, 0.0)
            u = torch.where(on, r * inv_c[a], 0.0)
            for _ in range(2):
                ok = valid.to(u.dtype)
                cnt = sum(shift(ok, q, s) for q in range(3) for s in (-1, 1))
                tot = sum(Shift.apply(u * ok, q, s) for q in range(3) for s in (-1, 1))
                fill = on & ~valid & (cnt > 0)
                u = torch.where(fill, tot / cnt.clamp(min=1), u)
                valid = valid | fill
            fr = self.prm.liquid_boundary_friction
            U.append(torch.where(on, torch.where(weight[a] == 0, (1 - fr) * u, u), 0.0))
        return self.g2p(U)

    def solid(self, xw, pos):
        """Solid phi and its unit gradient, weights taken at xw."""
        dx, S = self.dx, self.sphi.reshape(-1)
        phi, g = 0.0, 0.0
        mv = (pos - xw) / dx
        for idx, w, d in self.nodes(self.stencil(xw, (0,) * 3)):
            phi = phi + S[idx] * w
            g = g + (S[idx] * w * 4 / dx)[:, None] * (d - mv)
        return phi, g / (g * g).sum(1, keepdim=True).clamp(min=1e-40).sqrt()

    def correct(self, xw):
        """correctLiquidParticles, call 0 of the seeded stream (seed 0)."""
        prm, dx, dt = self.prm, self.dx, self.dt
        x = xw.detach()
        mix = 2 ** 64 - 1

        def splitmix(z):
            z = (z + 0x9E3779B97F4A7C15) & mix
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mix
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mix
            return z ^ (z >> 31)

        sel = splitmix(splitmix(0)) % prm.correction_step
        n = x.shape[0]
        mine = torch.arange(n, device=DEV) % prm.correction_step == sel
        phi, g = self.solid(x, x)
        if prm.correction_strength == 0:
            move = mine & (phi < 0)
            # the projection moves the position; derivatives pass through
            return xw + torch.where(move[:, None], -phi[:, None] * g, 0.0).detach()
        cell = torch.floor((x - self.org) / dx).long()
        lin = (cell[:, 0] * self.N[1] + cell[:, 1]) * self.N[2] + cell[:, 2]
        order = torch.argsort(lin, stable=True)
        start = torch.zeros(self.nn + 1, device=DEV, dtype=torch.long)
        start[1:] = torch.cumsum(torch.bincount(lin, minlength=self.nn), 0)
        most = int((start[1:] - start[:-1]).max())
        rad = self.p["r"]
        x = x.clone()
        for colour in range(8):
            par = (colour & 1, colour >> 1 & 1, colour >> 2)
            here = mine & ((cell & 1) == torch.tensor(par, device=DEV)).all(1)
            ids = order[here[order]]
            rank = torch.arange(ids.numel(), device=DEV)
            first = torch.ones_like(rank, dtype=torch.bool)
            first[1:] = lin[ids][1:] != lin[ids][:-1]
            rank = rank - torch.cummax(torch.where(first, rank, 0), 0).values
            for k in range(int(rank.max()) + 1 if ids.numel() else 0):
                i = ids[rank == k]
                spring = torch.zeros((i.numel(), 3), device=DEV, dtype=torch.float64)
                for t in range(27):
                    nb = lin[i] + ((t // 9 - 1) * self.N[1] + t // 3 % 3 - 1) * self.N[2] + t % 3 - 1
                    for s in range(most):
                        at = start[nb] + s
                        ok = at < start[nb + 1]
                        j = order[torch.where(ok, at, 0)]
                        d = x[i] - x[j]
                        re = (rad[i] * rad[j]).sqrt() * prm.correction_multiplier
                        dist = d.square().sum(1).sqrt()
                        w = prm.correction_strength / dt * (1 - dist ** 2 / re ** 2).clamp(min=0) ** 3
                        ok = ok & (j != i) & (dist <= re) & (dist > 1e-4 * re)
                        f = torch.where(ok, w * re / dist.clamp(min=1e-30), 0.0)
                        spring += f[:, None] * d
                dp = spring * dt
                now = phi[i] + (g[i] * dp).sum(1)
                x[i] = x[i] + dp + torch.where((now < 0)[:, None], -now[:, None] * g[i], 0.0)
        return x

    def g2p(self, U):
        dx, dt, p = self.dx, self.dt, self.p
        xw = p["x"]
        x = self.correct(xw)
        mv = ((x - xw) / dx).detach()
        vs, Cs = [], []
        for a in range(3):
            o = [0.5] * 3
            o[a] = 0.0
            u, v, B = U[a].reshape(-1), 0.0, 0.0
            for idx, w, d in self.nodes(self.stencil(xw, o)):
                uw = u[idx] * w
                v = v + uw
                B = B + uw[:, None] * (d - mv)
            vs.append(v)
            Cs.append(B * (4 / dx * self.prm.flip_coeff))
        v, C = torch.stack(vs, 1), torch.stack(Cs, 1)
        d = v * dt
        pos = x + d
        phi, g = self.solid(xw, pos)
        now = phi + (g * d).sum(1)
        out = [torch.where((now < 0)[:, None], pos - now[:, None] * g, pos), v, C]
        if self.e is not None:
            out += self.g2p_solid()
        return out

    def g2p_solid(self):
        e, dx, prm = self.e, self.dx, self.prm
        v4, B = e["v4"].clone(), torch.zeros_like(e["B"])
        for a in range(3):
            o = [0.5] * 3
            o[a] = 0.0
            v, u = 0.0, torch.where(self.on, self.E[a]["vel"], 0.0).reshape(-1)
            for idx, w, d in self.nodes(self.stencil(e["x4"][:, :3], o)):
                v = v + u[idx] * w
                B[:, a] += (u[idx] * w * 4 / dx)[:, None] * d
            v4[:, a] = v
        v4 = v4 * prm.elasto_advect_coeff
        c1 = prm.elasto_flip_coeff + prm.elasto_flip_asym_coeff
        c2 = prm.elasto_flip_coeff - prm.elasto_flip_asym_coeff
        for j in range(3):  # in place, column by column, as the reference assigns it
            for i in range(3):
                B[:, i, j] = (c1 * B[:, i, j] + c2 * B[:, j, i]) * 0.5
        return [e["x4"] + v4 * self.dt, v4, B.reshape(-1, 9)]


def exact(case, seed):
    if case["kind"] == "csr":
        rs, col, val, b = (torch.as_tensor(a, device=DEV) for a in csr_system(case, seed))
        A = torch.sparse_csr_tensor(rs.long(), col.long(), val, (b.numel(),) * 2)
        row = torch.repeat_interleave(torch.arange(b.numel(), device=DEV), rs[1:] - rs[:-1])
        inv = 1 / val[row == col]
        x, r = torch.zeros_like(b), b.clone()
        s = z = inv * r
        rho = z @ r
        while r.abs().max() > 1e-14 * b.abs().max():
            q = A @ s
            al = rho / (s @ q)
            x, r = x + al * s, r - al * q
            z = inv * r
            new = z @ r
            s, rho = z + (new / rho) * s, new
        return x
    if case["kind"] == "batch":
        out = []
        for k, n in enumerate(batch_sizes(case)):
            prm, p, _ = make({**case, "scene": "dam"}, n, int(seed) * 100 + k)
            out += Plain(prm, p, None, case["dt"]).step()
        return out
    prm, p, elasto = make(case, case["n"], seed)
    if case["kind"] == "adjoint":
        for k in ("x", "v", "C"):
            p[k].requires_grad_(True)
        out = Plain(prm, p, None, case["dt"]).step()
        got = torch.autograd.grad(out, [p[k] for k in ("x", "v", "C")], cotangents(p, seed))
        out[2] = out[2].reshape(-1, 9)
        return [*[o.detach() for o in out], *got]
    with torch.no_grad():
        return Plain(prm, p, elasto, case["dt"]).step()
