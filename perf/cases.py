"""What a user of this framework has it do, as cases that can be timed and checked.

Each case goes through the package's public entry points, on the GPU, over the sizes that the
repository's own configurations, examples and tests use:

  march    DGSolver.run: LSRK45 steps of a wave, Maxwell or advection problem in place
  rhs      DGSolver.rhs: one right-hand side for an integrator outside the library
  grad     grad_: Dr, Ds and Dt of a block of element columns from one read
  lift     mul_(out, BernsteinLift(N), faces)
  fused    fused_apply_: Dr, Ds, Dt and the lift
  closure  one macro step of the learned closure: LSRK steps, features, network, correction
  batch    BatchSolver.run: one step of many uneven problems
  host     DGSolver.run_host: one step with the state in page-locked host memory

`exact` restates each of them with dense matrices in 64 bits.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "bernsteinbasis.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bbdg  # noqa: E402
from bbdg.batch import BatchSolver, config4_problems  # noqa: E402
from bbdg.mlp import MLP, closure_apply, closure_features  # noqa: E402

DEV = "cuda"
DT = {"f32": torch.float32, "f64": torch.float64}
NFIELDS = {"wave": 4, "maxwell": 6, "advection": 1, "advection3": 3}
HIDDEN = 512      # the closure network: nin -> 512 -> 512 -> nout
CLOSURE_STEPS = 3  # degree-5 steps per macro step of ten degree-10 steps


# ---- the cases -----------------------------------------------------------------------------
def listed():
    return [
        # the reference's own 3D wave script: degree 7 on 4^3 hexahedra in double precision,
        # ten time steps between two looks at the solution; launches and latency count
        {"name": "wave_example_f64", "kind": "march", "physics": "wave", "dtype": "f64", "N": 7,
         "n": 4, "steps": 10},
        # one right-hand side of a small low-degree Maxwell problem, called by an ODE package
        {"name": "maxwell_rhs_small_f32", "kind": "rhs", "physics": "maxwell", "dtype": "f32",
         "N": 3, "n": 4},
        # the benchmark workload: degree 9, 196,608 elements, single precision
        {"name": "wave_bench_f32", "kind": "march", "physics": "wave", "dtype": "f32", "N": 9,
         "n": 32, "steps": 1},
        # a mesh whose element count (20,250) is no multiple of four
        {"name": "wave_ragged_f32", "kind": "march", "physics": "wave", "dtype": "f32", "N": 6,
         "n": 15, "steps": 2},
        # the highest degree of the reference's published comparison
        {"name": "wave_high_degree_f32", "kind": "march", "physics": "wave", "dtype": "f32",
         "N": 15, "n": 8, "steps": 1},
        # the precision the reference's Maxwell script runs in, at a mid size
        {"name": "maxwell_f64", "kind": "march", "physics": "maxwell", "dtype": "f64", "N": 7,
         "n": 9, "steps": 1},
        # the operators one by one, as mul! calls on a block of columns (an odd number)
        {"name": "grad_f32", "kind": "grad", "dtype": "f32", "N": 9, "cols": 400_001},
        {"name": "lift_f32", "kind": "lift", "dtype": "f32", "N": 12, "cols": 150_001},
        {"name": "operators_f64", "kind": "fused", "dtype": "f64", "N": 7, "cols": 60_001},
        # a corrected degree-5 Maxwell run on 16^3 hexahedra, one macro step
        {"name": "closure_macro_step", "kind": "closure", "N": 5, "n": 16},
        # the first twelve of the 48 uneven problems the batch is benchmarked on
        {"name": "batch_12", "kind": "batch", "problems": 2, "count": 12},
        # one step with the state in host memory, copies included
        {"name": "wave_host_f32", "kind": "host", "physics": "wave", "dtype": "f32", "N": 9,
         "n": 16},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _hexes(dofs, nf, N):
    """The most hexahedra per side with nf fields of degree N in `dofs` unknowns (at least 3)."""
    return max(3, min(32, int((dofs / (6 * nf * bbdg.np3(N))) ** (1 / 3))))


def draw(rng):
    kind = rng.choice(["march", "march", "march", "rhs", "grad", "lift", "fused", "closure",
                       "batch", "host"])
    if kind in ("march", "rhs", "host"):
        physics = rng.choice(["wave", "maxwell", "wave", "maxwell", "advection", "advection3"])
        dtype = rng.choice(["f32", "f32", "f64"])
        N = rng.randint(3, 15)
        # unknowns: at most what the listed cases of that precision and kernel class hold
        most = 4e6 if dtype == "f64" else 30e6 if N <= 11 else 12e6
        c = {"kind": kind, "physics": physics, "dtype": dtype, "N": N,
             "n": _log_int(rng, 3, _hexes(most, NFIELDS[physics], N))}
        if kind == "march":
            c["steps"] = rng.choice([1, 2])
        return c
    if kind in ("grad", "lift", "fused"):
        dtype = rng.choice(["f32", "f32", "f64"])
        N = rng.randint(3, 15)
        most = (60e6 if dtype == "f32" else 8e6) / bbdg.np3(N)
        return {"kind": kind, "dtype": dtype, "N": N, "cols": _log_int(rng, 1000, int(most))}
    if kind == "closure":
        return {"kind": kind, "N": rng.randint(4, 7), "n": 2 * rng.randint(3, 7)}
    return {"kind": kind, "problems": rng.randint(10, 10_000), "count": rng.randint(3, 8)}


# ---- inputs --------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _mesh(n):
    return bbdg.uniform_tet_mesh(n)


@functools.lru_cache(maxsize=None)
def _points(N):
    """Barycentric weights (Np, 4) of the degree-N domain points on the element's vertices and
    the matrix from values at those points to Bernstein coefficients."""
    ix = _idx3(N).double() / N                                    # (Np, 4): i, j, k, l
    V = torch.ones(len(ix), len(ix), dtype=torch.float64)
    for b in range(4):
        V = V * ix[:, b:b + 1] ** _idx3(N)[:, b].double()
    V = V * torch.tensor([_multinomial(N, a) for a in _idx3(N).tolist()], dtype=torch.float64)
    return ix[:, [3, 0, 1, 2]], torch.linalg.inv(V)


def _multinomial(N, a):
    return math.factorial(N) / math.prod(math.factorial(int(x)) for x in a)


def _pulses(mesh, N, nf, seed, dtype):
    """(nf, K, Np): Bernstein coefficients of a sum of eight Gaussian pulses in each field
    (centres U[-0.8, 0.8]^3, widths U[0.1, 0.3], amplitudes N(0, 1)), interpolated at the
    domain points, as the examples start their runs."""
    W, C = (t.to(DEV) for t in _points(N))
    X = torch.as_tensor(mesh.EVX, device=DEV)
    pts = torch.einsum("pm,kmc->kpc", W, X)
    rng = np.random.default_rng(seed)
    q = torch.empty((nf, mesh.K, W.shape[0]), dtype=dtype, device=DEV)
    for m in range(nf):
        # in 64 bits: interpolation at degree 15 amplifies the rounding of the values 1e5 times
        v = torch.zeros(pts.shape[:2], dtype=torch.float64, device=DEV)
        for _ in range(8):
            c = torch.as_tensor(rng.uniform(-0.8, 0.8, 3), device=DEV)
            w, a = rng.uniform(0.1, 0.3), rng.standard_normal()
            v += a * torch.exp(-(pts - c).square().sum(-1) / w ** 2)
        q[m] = (v @ C.T).to(dtype)
    return q


def _columns(cols, rows, dtype, gen):
    return torch.rand((cols, rows), generator=gen, device=DEV, dtype=dtype) * 2 - 1


def _inputs(case, seed):
    """The numbers a case starts from, by name."""
    kind = case["kind"]
    if kind in ("march", "rhs", "host"):
        return {"q": _pulses(_mesh(case["n"]), case["N"], NFIELDS[case["physics"]], seed,
                             DT[case["dtype"]])}
    if kind in ("grad", "lift", "fused"):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        N, dt = case["N"], DT[case["dtype"]]
        d = {}
        if kind != "lift":
            d["x"] = _columns(case["cols"], bbdg.np3(N), dt, gen)
        if kind != "grad":
            d["faces"] = _columns(case["cols"], 4 * bbdg.np2(N), dt, gen)
        return d
    if kind == "closure":
        N, mesh = case["N"], _mesh(case["n"])
        q = _pulses(mesh, N, 6, seed, torch.float32)
        nin, nout = 6 * (bbdg.np3(N) + 4 * bbdg.np2(N)), 6 * bbdg.np3(N)
        rng = np.random.default_rng(seed)
        p = []
        for fan_in, fan_out in ((nin, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, nout)):
            p.append(rng.uniform(-1, 1, fan_in * fan_out) / math.sqrt(fan_in))
            p.append(rng.uniform(-1, 1, fan_out) * 0.01)
        rms = float(q.double().square().mean().sqrt())
        return {"q": q, "params": np.concatenate(p).astype(np.float32), "s_in": 1.0 / rms,
                "alpha": 1e-3 * rms}
    specs = _specs(case)
    return {"states": [_pulses(_mesh(s.n), s.N, NFIELDS[s.physics], 1000 * seed + i,
                               torch.float32) for i, s in enumerate(specs)]}


def _specs(case):
    # the first problems of the benchmark's draw; drawn cases take the smaller meshes of another
    specs = config4_problems(case["problems"], 48)
    if case["problems"] != 2:
        specs = [s for s in specs if s.n <= 14]
    return specs[:case["count"]]


def _closure_dt(mesh):
    return 10 * 0.25 * mesh.h / 11 ** 2 / CLOSURE_STEPS


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    d = _inputs(case, seed)
    if kind in ("march", "rhs", "host"):
        mesh = _mesh(case["n"])
        s["solver"] = bbdg.DGSolver(mesh, case["N"], case["physics"], DT[case["dtype"]], tau=1.0)
        s["dt"] = s["solver"].dt_cfl()
        s["q"] = d["q"]
        s["res"] = torch.zeros_like(d["q"])
        if kind == "rhs":
            s["rhs"] = torch.empty_like(d["q"])
        if kind == "host":
            s["host_in"] = d["q"].cpu().pin_memory()
            s["host_out"] = torch.empty_like(s["host_in"]).pin_memory()
    elif kind in ("grad", "lift", "fused"):
        s.update(d)
        like = d["x"] if kind != "lift" else torch.empty(
            (case["cols"], bbdg.np3(case["N"])), dtype=DT[case["dtype"]], device=DEV)
        s["out"] = [torch.empty_like(like) for _ in range({"grad": 3, "lift": 1, "fused": 4}[kind])]
    elif kind == "closure":
        N, mesh = case["N"], _mesh(case["n"])
        s.update(d)
        s["solver"] = bbdg.DGSolver(mesh, N, "maxwell", torch.float32, tau=1.0)
        s["dt"] = _closure_dt(mesh)
        s["res"] = torch.zeros_like(d["q"])
        nin, nout = 6 * (bbdg.np3(N) + 4 * bbdg.np2(N)), 6 * bbdg.np3(N)
        s["net"] = MLP((nin, HIDDEN, HIDDEN, nout), max_batch=mesh.K)
        s["net"].set_params(d["params"])
        s["X"] = torch.empty((mesh.K, nin), dtype=torch.bfloat16, device=DEV)
        s["Y"] = torch.empty((mesh.K, nout), dtype=torch.float32, device=DEV)
    else:
        s["batch"] = BatchSolver(_specs(case), torch.float32, states=d["states"])
    return s


# ---- one pass ------------------------------------------------------------------------------
# A run's result is its state q. The register res is scratch between the stages of one step:
# the next step's first stage ignores what it holds.
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "march":
        s["solver"].run(s["q"], s["res"], s["dt"], case["steps"])
        return s["q"]
    if kind == "rhs":
        return s["solver"].rhs(s["q"], out=s["rhs"])
    if kind == "grad":
        return list(bbdg.grad_(*s["out"], case["N"], s["x"]))
    if kind == "lift":
        return bbdg.mul_(s["out"][0], bbdg.BernsteinLift(case["N"]), s["faces"])
    if kind == "fused":
        return list(bbdg.fused_apply_(*s["out"], case["N"], s["x"], s["faces"]))
    if kind == "host":
        s["solver"].run_host(s["host_in"], s["host_out"], s["q"], s["res"], s["dt"], 1)
        return [s["host_out"], s["q"]]
    if kind == "closure":
        s["res"].zero_()
        s["solver"].run(s["q"], s["res"], s["dt"], CLOSURE_STEPS)
        closure_features(case["N"], 6, s["solver"].conn, s["q"], s["s_in"], X=s["X"])
        s["net"].forward(s["X"], out=s["Y"])
        closure_apply(case["N"], 6, s["alpha"], s["Y"], s["q"])
        return s["q"]
    s["batch"].run(1)
    return list(s["batch"].q)


# ---- work of one pass ----------------------------------------------------------------------
def _stage_flops(physics, N):
    """Arithmetic of one right-hand side and update per element (adds and multiplies)."""
    nf = NFIELDS[physics]
    np_, nfp, npm1 = bbdg.np3(N), bbdg.np2(N), bbdg.np3(N - 1)
    vol, nw, chains, flux = {"wave": (48, 4, 2, 16), "maxwell": (90, 6, 6, 90),
                             "advection": (9, 1, 1, 5), "advection3": (9, 1, 3, 15)}[physics]
    lift = 4 * chains * (13 * nfp + 5 * (np_ - nfp)) + np_ * (28 if physics == "wave" else 4 * nf)
    return npm1 * vol + np_ * 8 * nw + 4 * nfp * flux + lift + np_ * nf * 5


def _march_work(physics, N, K, size, stages, rhs_only=False):
    nf = NFIELDS[physics]
    rows = nf * ((2 if rhs_only else 4) * bbdg.np3(N) + 4 * bbdg.np2(N))
    return {"bytes": stages * K * (rows * size + 22 * size + 16),
            "flops": stages * K * _stage_flops(physics, N)}


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "f64" else 4
    N = case.get("N")
    if kind in ("march", "rhs", "host"):
        K = 6 * case["n"] ** 3
        w = _march_work(case["physics"], N, K, size, 5 * case.get("steps", 1) if kind != "rhs" else 1,
                        kind == "rhs")
        if kind == "host":
            w["bytes"] += 2 * NFIELDS[case["physics"]] * K * bbdg.np3(N) * size
        return w
    if kind in ("grad", "lift", "fused"):
        np_, nfp = bbdg.np3(N), bbdg.np2(N)
        grad, lift = 4 * np_, 4 * nfp + np_
        rows = {"grad": grad, "lift": lift, "fused": grad + lift}[kind]
        gflop, lflop = 6 * bbdg.np3(N - 1) + 24 * np_, 4 * (13 * nfp + 5 * (np_ - nfp)) + 4 * np_
        return {"bytes": case["cols"] * rows * size,
                "flops": case["cols"] * {"grad": gflop, "lift": lflop, "fused": gflop + lflop}[kind]}
    if kind == "closure":
        K = 6 * case["n"] ** 3
        w = _march_work("maxwell", N, K, 4, 5 * CLOSURE_STEPS)
        nout = 6 * bbdg.np3(N)
        nin = nout + 24 * bbdg.np2(N)
        weights = nin * HIDDEN + HIDDEN * HIDDEN + HIDDEN * nout
        w["bytes"] += 2 * weights + K * nout * 4 * 2
        w["flops"] += 2 * K * weights
        return w
    total = {"bytes": 0, "flops": 0}
    for s in _specs(case):
        w = _march_work(s.physics, s.N, 6 * s.n ** 3, 4, 5)
        total = {k: total[k] + w[k] for k in total}
    return total


# ---- the same in 64 bits, with dense matrices ----------------------------------------------
@functools.lru_cache(maxsize=None)
def _idx3(N):
    return torch.tensor([(i, j, k, N - i - j - k) for k in range(N + 1) for j in range(N + 1 - k)
                         for i in range(N + 1 - j - k)], dtype=torch.int64)


def _idx2(N):
    return [(a, b, N - a - b) for b in range(N + 1) for a in range(N + 1 - b)]


@functools.lru_cache(maxsize=None)
def _deriv(N):
    """Dr, Ds, Dt: (D_b x)(alpha) = sum_a alpha_a x(alpha - e_a + e_b), Dr = (D_0 - D_3) / 2."""
    ix = [tuple(a) for a in _idx3(N).tolist()]
    at = {a: m for m, a in enumerate(ix)}
    D = np.zeros((4, len(ix), len(ix)))
    for m, alpha in enumerate(ix):
        for a in range(4):
            if alpha[a] == 0:
                continue
            for b in range(4):
                g = list(alpha)
                g[a] -= 1
                g[b] += 1
                D[b, m, at[tuple(g)]] += alpha[a]
    return [torch.as_tensor((D[b] - D[3]) / 2, device=DEV) for b in range(3)]


@functools.lru_cache(maxsize=None)
def _lift(N):
    """(Np, 4 Nfp): the volume coefficients of layer d of a face are
    (-1)^d C(N, d) / (1 + d) R_{N-d+1} ... R_N L0, L0 = (N+1)^2 / 2 R_{N+1} E_{N+1}."""
    def elevate(n):  # degree n - 1 -> n
        A = {a: m for m, a in enumerate(_idx2(n))}
        E = np.zeros((len(A), len(_idx2(n - 1))))
        for c, a in enumerate(_idx2(n - 1)):
            for v in range(3):
                up = list(a)
                up[v] += 1
                E[A[tuple(up)], c] += up[v] / n
        return E
    E1 = elevate(N + 1)
    layer = (N + 1) ** 2 / 2 * E1.T @ E1
    face = [layer]                                        # layers d = 0 .. N of the stack
    for d in range(1, N + 1):
        layer = elevate(N - d + 1).T @ layer
        face.append((-1) ** d * math.comb(N, d) / (1 + d) * layer)
    # volume coefficient (i, j, k, l) sits at (first, second) of layer `third` of each face
    at2 = [{a[:2]: m for m, a in enumerate(_idx2(N - d))} for d in range(N + 1)]
    nfp = len(_idx2(N))
    L = np.zeros((len(_idx3(N)), 4 * nfp))
    for m, (i, j, k, l) in enumerate(_idx3(N).tolist()):
        for f, (a, b, d) in enumerate(((i, k, j), (j, k, l), (j, k, i), (i, j, k))):
            L[m, f * nfp:(f + 1) * nfp] = face[d][at2[d][(a, b)]]
    return torch.as_tensor(L, device=DEV)


def _face_nodes(N):
    """(4, Nfp) volume index of each face node; node (a, b, c) weighs the face's vertices."""
    at = {tuple(a): m for m, a in enumerate(_idx3(N).tolist())}
    slots = ((0, 2, 3), (1, 2, 0), (1, 2, 3), (0, 1, 3))   # barycentric places of a, b, c
    out = np.zeros((4, len(_idx2(N))), dtype=np.int64)
    for f in range(4):
        for m, abc in enumerate(_idx2(N)):
            v = [0, 0, 0, 0]
            for p, x in zip(slots[f], abc):
                v[p] = x
            out[f, m] = at[tuple(v)]
    return out


def _partner_nodes(N):
    """(4, 6, Nfp): volume index, on the partner's face, of this side's face node."""
    perms = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))
    at = {a: m for m, a in enumerate(_idx2(N))}
    fv, out = _face_nodes(N), np.zeros((4, 6, len(at)), dtype=np.int64)
    for o, p in enumerate(perms):
        for m, abc in enumerate(_idx2(N)):
            theirs = [0, 0, 0]
            for mine, x in zip(p, abc):
                theirs[mine] = x
            out[:, o, m] = fv[:, at[tuple(theirs)]]
    return out


class _Dense:
    """The right-hand side of one problem with dense matrices in 64 bits."""

    def __init__(self, mesh, N, physics, tau=1.0):
        self.physics, self.N, self.tau = physics, N, tau
        self.D, self.L = _deriv(N), _lift(N)
        t = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
        self.nbr = t(mesh.nbr)[:, :, None]
        self.vM = t(_face_nodes(N))[None]
        self.vP = t(_partner_nodes(N))[t(mesh.nbr_face), t(mesh.orient)]
        geo = t(mesh.geo)
        self.g = [geo[:, c * 3:c * 3 + 3] for c in range(3)]     # (rxJ, sxJ, txJ), y, z
        self.J = geo[:, 10][:, None]
        self.n = [geo[:, 12 + 4 * c:16 + 4 * c][:, :, None] for c in range(3)]
        self.el = torch.arange(mesh.K, device=DEV)[:, None, None]

    def outer(self, q):
        """The neighbours' values (nf, K, 4, Nfp) at this side's face nodes."""
        return torch.stack([f[self.nbr, self.vP] for f in q])

    def d(self, c, f):
        return sum(self.g[c][:, a:a + 1] * (f @ self.D[a].T) for a in range(3))

    def rhs(self, q):
        jump = self.outer(q) - torch.stack([f[self.el, self.vM] for f in q])
        nx, ny, nz = self.n
        Jf = (nx * nx + ny * ny + nz * nz).sqrt()
        cp, cu = self.tau * Jf, self.tau / Jf
        if self.physics == "wave":
            nu = nx * jump[1] + ny * jump[2] + nz * jump[3]
            B = (cu * nu - jump[0]) / 2
            flux = [(cp * jump[0] - nu) / 2, B * nx, B * ny, B * nz]
            vol = [-(self.d(0, q[1]) + self.d(1, q[2]) + self.d(2, q[3])),
                   -self.d(0, q[0]), -self.d(1, q[0]), -self.d(2, q[0])]
        elif self.physics == "maxwell":
            H, E = jump[:3], jump[3:]
            n = (nx, ny, nz)
            ndH, ndE = sum(a * b for a, b in zip(n, H)), sum(a * b for a, b in zip(n, E))
            flux, vol = [], []
            for sign, own, other, o, nd in ((-1, H, E, 3, ndH), (1, E, H, 0, ndE)):
                for c in range(3):
                    a, b = (c + 1) % 3, (c + 2) % 3
                    curl = n[a] * other[b] - n[b] * other[a]
                    flux.append((sign * curl + cp * own[c] - cu * nd * n[c]) / 2)
                    vol.append(sign * (self.d(a, q[o + b]) - self.d(b, q[o + a])))
        else:
            flux = [-(jump[m] * nx - jump[m] * Jf) / 2 for m in range(len(q))]
            vol = [-self.d(0, q[0])] + [0.0] * (len(q) - 1)
        K = q.shape[1]
        return torch.stack([(v + f.reshape(K, -1) @ self.L.T) / self.J for v, f in zip(vol, flux)])

    def march(self, q, dt, steps):
        A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238,
             -3550918686646 / 2091501179385, -1275806237668 / 842570457699)
        B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357,
             1720146321549 / 2090206949498, 3134564353537 / 4481467310338,
             2277821191437 / 14882151754819)
        res = torch.zeros_like(q)
        for _ in range(steps):
            for a, b in zip(A, B):
                res = a * res + dt * self.rhs(q)
                q = q + b * res
        return q


def exact(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    if kind in ("grad", "lift", "fused"):
        out = []
        if kind != "lift":
            out += [d["x"].double() @ D.T for D in _deriv(case["N"])]
        if kind != "grad":
            out.append(d["faces"].double() @ _lift(case["N"]).T)
        return out[0] if kind == "lift" else out
    if kind == "batch":
        out = []
        for s, q in zip(_specs(case), d["states"]):
            m = _mesh(s.n)
            out.append(_Dense(m, s.N, s.physics).march(q.double(), 0.25 * m.h / (s.N + 1) ** 2, 1))
        return out
    mesh, N = _mesh(case["n"]), case["N"]
    ref = _Dense(mesh, N, case.get("physics", "maxwell"))
    q = d["q"].double()
    if kind == "rhs":
        return ref.rhs(q)
    if kind == "closure":
        q = ref.march(q, _closure_dt(mesh), CLOSURE_STEPS)
        K = mesh.K
        X = torch.cat([q.permute(1, 0, 2).reshape(K, -1),
                       ref.outer(q).permute(1, 2, 0, 3).reshape(K, -1)], dim=1) * d["s_in"]
        sizes = (X.shape[1], HIDDEN, HIDDEN, 6 * bbdg.np3(N))
        p, at = torch.as_tensor(d["params"], device=DEV).double(), 0
        for layer, (a, b) in enumerate(zip(sizes, sizes[1:])):
            W, bias = p[at:at + a * b].reshape(b, a), p[at + a * b:at + a * b + b]
            at += a * b + b
            X = X @ W.T + bias
            if layer < 2:
                X = torch.nn.functional.gelu(X)
        return q + d["alpha"] * X.reshape(K, 6, -1).permute(1, 0, 2)
    q = ref.march(q, 0.25 * mesh.h / (N + 1) ** 2, case.get("steps", 1))
    return [q, q] if kind == "host" else q
