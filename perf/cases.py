"""Cases whose speed is measured: the calls that a user of the periodic-orbit solver makes.

Five kinds, each through the package's public entry points:

* ``orbits``: new operators come in, their orbits go out (``OrbitSolver.factor`` + ``solve_device``):
  the forward driver, one call per met draw;
* ``factor``: new operators are factored and swept once (``FactorBatch.numeric`` + ``chain``): what
  building a served (domain, month) entry, or the first monodromy of a drop-in run, costs;
* ``chain``: one chained sweep of the eight bins on factors in hand (``FactorBatch.chain``): the matvec
  of every Krylov iteration, forward and transposed, 64 and 32 bits;
* ``solve``: orbits on factors in hand (``FactorBatch.solve`` / ``solve_adjoint``): served requests,
  marginal perturbations, adjoint receptors;
* ``fct``: the limited anti-diffusive source of eight bins (``device.fct_source``): one pass of the
  deferred correction.

Domains are (nz, ny, nx); the named ones are those of the benchmark and of the serving stream.  Operators
are drawn like the benchmark's met fields: staggered winds N(0, 8 m/s) smoothed over 3 cells, exponential
(Patankar) face coefficients, K_zz log-uniform on 0.1-100 m2/s, convective exchange in 30 % of the columns,
the vertical flux closing the horizontal divergence; sinks, emissions and receptors as in the benchmark.
They are drawn on the GPU: the calls measured here take stencils and vectors that live there.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from orbit_b200 import api, device, synthetic
from orbit_b200.symbolic import Symbolic

BINS = 8
DTAU = 10800.0
RADIUS, GRAVITY = 6378137.0, 9.80665


def _case(name, kind, shape, **kw):
    c = dict(name=name, kind=kind, nz=shape[0], ny=shape[1], nx=shape[2], bits=64, sets=1, rhs=1, adjoint=False,
             periodic=False, tol=1e-8)
    c.update(kw)
    return c


def listed():
    full, large, mid, small = (15, 72, 80), (15, 54, 60), (15, 36, 40), (15, 20, 24)
    return [
        # the plain method on the small domain, tight tolerance: latency and launches count
        _case("orbit small fp64", "orbits", small, tol=1e-10),
        # the headline: 12 species of one met draw, mixed precision, factorization and solve
        _case("orbits full fp32 x12", "orbits", full, bits=32, sets=12, rhs=12),
        # the plain drop-in's factorization of one species, then its first monodromy
        _case("factor full fp64", "factor", full),
        # a served (domain, month) entry: 12 species factored together, then a refined sweep
        _case("factor large fp32 x12", "factor", large, bits=32, sets=12, rhs=12),
        # the drop-in's matvec
        _case("chain full fp64", "chain", full),
        # the drop-in adjoint's matvec on a domain with odd extents
        _case("chain adjoint odd fp64", "chain", (13, 47, 53), adjoint=True),
        # the batched matvec: 12 species in 32 bits
        _case("chain full fp32 x12", "chain", full, bits=32, sets=12, rhs=12),
        # served forward requests: 24 slots over 12 species of the smallest domain
        _case("serve small fp32 x24", "solve", small, bits=32, sets=12, rhs=24, tol=1e-6),
        # served adjoint requests: 9 receptors over 12 species of a middle domain
        _case("serve adjoint mid fp32 x9", "solve", mid, bits=32, sets=12, rhs=9, adjoint=True, tol=1e-6),
        # 64 emission perturbations on one operator
        _case("marginal full fp32 x64", "solve", full, bits=32, rhs=64, tol=1e-6),
        # 64 receptors on one operator, transposed
        _case("adjoint full fp32 x64", "solve", full, bits=32, rhs=64, adjoint=True, tol=1e-6),
        # the anti-diffusive sources of one deferred pass: 12 species, 8 bins
        _case("fct full x12", "fct", full, rhs=12),
    ]


def draw(rng):
    """One more case: domains from 10x10 columns up to the full one, 1-12 species, 1-64 right-hand sides."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("orbits", "orbits", "factor", "chain", "chain", "solve", "solve", "solve", "fct"))
    while True:
        nz, ny, nx = rng.randint(8, 17), log_int(10, 74), log_int(10, 84)
        if nz * ny * nx <= 86400 and nz * min(ny, nx) <= 1080:
            break
    bits = rng.choice((32, 32, 64))
    sets = log_int(1, 12) if bits == 32 else log_int(1, 4)
    periodic = kind != "fct" and nz * ny * nx <= 30000 and rng.random() < 0.25
    adjoint = kind in ("chain", "solve") and rng.random() < 0.5
    rhs = sets
    if kind in ("chain", "solve") and rng.random() < 0.5:
        sets, rhs = 1, log_int(2, 64 if bits == 32 else 16)
    elif kind == "solve":
        rhs = log_int(1, 2 * sets)
    elif kind == "fct":
        bits, sets, rhs = 64, 1, log_int(1, 12)
    c = _case("", kind, (nz, ny, nx), bits=bits, sets=sets, rhs=rhs, adjoint=adjoint, periodic=periodic,
              tol=rng.choice((1e-6, 1e-8)))
    del c["name"]
    return c


@functools.lru_cache(maxsize=32)
def _symbolic(nz, ny, nx, bits, batch, periodic):
    """A program keeps one analysis per domain, with the autotuner's options where it has them."""
    return Symbolic.tuned(nz, ny, nx, bits, batch, periodic=periodic)


def _sym(case):
    return _symbolic(case["nz"], case["ny"], case["nx"], case["bits"], case["sets"], case["periodic"])


# ---- inputs ----------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _smooth(f, dim, sigma=3.0):
    r = int(4 * sigma)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, dtype=f.dtype, device=f.device) / sigma) ** 2)
    k = k / k.sum()
    n = f.shape[dim]
    at = (torch.arange(n, device=f.device)[:, None] + torch.arange(-r, r + 1, device=f.device)[None]).clamp(0, n - 1)
    w = torch.zeros((n, n), dtype=f.dtype, device=f.device)
    w.scatter_add_(1, at, k.expand(n, -1).contiguous())
    return torch.movedim(torch.movedim(f, dim, -1) @ w.T, -1, dim)


def _winds(g, nz, ny, nx):
    """(8, nz, ny, nx + 1) and (8, nz, ny + 1, nx) face winds."""
    def one(shape):
        f = torch.randn(shape, generator=g, dtype=torch.float64, device=_dev()) * 8.0
        f = _smooth(_smooth(f, -1), -2)
        return f * (8.0 / f.flatten(1).std(dim=1).view(-1, 1, 1, 1))
    return one((BINS, nz, ny, nx + 1)), one((BINS, nz, ny + 1, nx))


def _geometry(ny, nx, periodic):
    dlat, dlon = 0.5, (360.0 / nx if periodic else 0.625)
    lat = 5.0 + dlat * torch.arange(ny, dtype=torch.float64, device=_dev())
    dx = RADIUS * torch.cos(lat * math.pi / 180.0) * dlon * math.pi / 180.0
    return lat, dlat, dlon, dx, RADIUS * dlat * math.pi / 180.0


def _face(u, d, K=1e3):
    """Exponential-scheme coefficients of a face: (from its low side, from its high side)."""
    pe = u * d / K
    small = pe.abs() < 1e-6
    safe = torch.where(small, torch.ones_like(pe), pe)
    b = torch.where(small, 1.0 - 0.5 * pe, safe / torch.expm1(safe)) * (K / d)  # Bernoulli function
    return (b + u) / d, b / d


def _stencils(seed, nz, ny, nx, periodic):
    """(8, 7, N) transport stencils: centre, west, east, south, north, below, above."""
    g = _gen(seed)
    _, _, _, dx, dy = _geometry(ny, nx, periodic)
    dx = dx[None, None, :, None]
    U, V = _winds(g, nz, ny, nx)
    if periodic:
        wrap = 0.5 * (U[..., 0] + U[..., -1])
        U[..., 0] = wrap
        U[..., -1] = wrap
    T = torch.zeros((BINS, 7, nz, ny, nx), dtype=torch.float64, device=_dev())
    lo, hi = _face(U, dx)
    inside = slice(None) if periodic else slice(1, None)
    T[:, 1][..., inside] -= lo[..., :nx][..., inside]
    T[:, 0][..., inside] += hi[..., :nx][..., inside]
    outside = slice(None) if periodic else slice(0, nx - 1)
    T[:, 2][..., outside] -= hi[..., 1:][..., outside]
    T[:, 0][..., outside] += lo[..., 1:][..., outside]
    if not periodic:  # open lateral edges: what leaves is lost
        T[:, 0][..., 0] += (-U[..., 0]).clamp(min=0) / dx[..., 0]
        T[:, 0][..., -1] += U[..., -1].clamp(min=0) / dx[..., 0]
    lo, hi = _face(V, torch.full_like(V, dy))
    T[:, 3][..., 1:, :] -= lo[..., 1:ny, :]
    T[:, 0][..., 1:, :] += hi[..., 1:ny, :]
    T[:, 4][..., :-1, :] -= hi[..., 1:ny, :]
    T[:, 0][..., :-1, :] += lo[..., 1:ny, :]
    T[:, 0][..., 0, :] += (-V[..., 0, :]).clamp(min=0) / dy
    T[:, 0][..., -1, :] += V[..., -1, :].clamp(min=0) / dy
    # vertical: the flux that closes the horizontal row sums, diffusion, convective exchange
    dP = (101325.0 - 6500.0) / nz
    dz = dP / (1.2 * GRAVITY)
    F = -torch.cumsum(T.sum(dim=1), dim=1)  # upward through the top of each layer, 1/s
    kz = 10.0 ** (3.0 * torch.rand((BINS, nz, ny, nx), generator=g, dtype=torch.float64, device=_dev()) - 1.0)
    amp = torch.exp(math.log(0.01) + torch.randn((BINS, 1, ny, nx), generator=g, dtype=torch.float64, device=_dev()))
    amp = amp * (torch.rand((BINS, 1, ny, nx), generator=g, dtype=torch.float64, device=_dev()) < 0.3)
    prof = torch.sin(math.pi * torch.arange(1, nz + 1, dtype=torch.float64, device=_dev()) / nz).clamp(min=0)
    mix = kz / dz ** 2 + amp * prof.view(1, nz, 1, 1) * GRAVITY / dP
    mix[:, -1] = 0.0
    up, down = F.clamp(min=0) + mix, (-F).clamp(min=0) + mix
    T[:, 0] += up
    T[:, 0][:, 1:] += down[:, :-1]
    T[:, 5][:, 1:] -= up[:, :-1]
    T[:, 6][:, :-1] -= down[:, :-1]
    return T.reshape(BINS, 7, -1)


def _sinks(seed, sets, nz, ny, nx):
    """(sets, 8, N) deposition and first-order loss."""
    g = _gen(seed)
    d = 1e-6 + 9.9e-5 * torch.rand((sets, 1, nz, ny, nx), generator=g, dtype=torch.float64, device=_dev())
    dz = (101325.0 - 6500.0) / nz / (1.2 * GRAVITY)
    vd = 0.001 + 0.019 * torch.rand((sets, 1, ny, nx), generator=g, dtype=torch.float64, device=_dev())
    d[:, :, 0] += vd / dz
    return d.expand(-1, BINS, -1, -1, -1).reshape(sets, BINS, -1).contiguous()


def _forcing(seed, case):
    """(rhs, 8, N): surface emissions; one patch's perturbation, or receptor, each on a shared operator."""
    n, nz, ny, nx = case["rhs"], case["nz"], case["ny"], case["nx"]
    g = _gen(seed)
    e = torch.zeros((n, 1, nz, ny, nx), dtype=torch.float64, device=_dev())
    if case["adjoint"] or (case["sets"] == 1 and n > 1):
        at = torch.rand((n, 3), generator=g, dtype=torch.float64, device=_dev()).tolist()
        for q in range(n):
            j, i = int(at[q][0] * (ny - 5)), int(at[q][1] * (nx - 5))
            e[q, 0, 0, j:j + 5, i:i + 5] = 1.0 / (BINS * 25) if case["adjoint"] else 1e-9 * (0.1 + at[q][2])
    else:
        e[:, 0, 0] = 1e-9 * torch.exp(1.5 * torch.randn((n, ny, nx), generator=g, dtype=torch.float64, device=_dev()))
    return e.expand(-1, BINS, -1, -1, -1).reshape(n, BINS, -1).contiguous()


def _vectors(seed, n, N):
    """(n, N) positive concentrations."""
    return torch.exp(torch.randn((n, N), generator=_gen(seed), dtype=torch.float64, device=_dev()))


def _slots(case, seed):
    """Factor set of each right-hand side: its own where there is one for each, drawn otherwise."""
    if case["rhs"] == case["sets"]:
        return list(range(case["sets"]))
    return [int(v) for v in np.random.default_rng(seed).integers(0, case["sets"], size=case["rhs"])]


def _inputs(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    T = _stencils(1000 + 10 * seed, nz, ny, nx, case["periodic"])
    return T, _sinks(1001 + 10 * seed, case["sets"], nz, ny, nx)


def _fct_met(case, seed):
    """Eight bins with terrain, and (8, n, N) end-of-bin concentrations."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    g = _gen(1000 + 10 * seed)
    lat, dlat, dlon, _, _ = _geometry(ny, nx, False)
    U, V = _winds(g, nz, ny, nx)
    ps = 101325.0 - 8000.0 * _smooth(_smooth(torch.rand((ny, nx), generator=g, dtype=torch.float64, device=_dev()), 0, 2.0), 1, 2.0)
    eta = torch.linspace(0.0, 1.0, nz + 1, dtype=torch.float64, device=_dev())
    P = 6500.0 * eta[:, None, None] + (1.0 - eta)[:, None, None] * ps[None]
    dP = P[:-1] - P[1:]
    Dz = dP / (1.2 * torch.exp(-eta[:-1] * 1.2)[:, None, None] * GRAVITY)
    c = torch.exp(_smooth(_smooth(torch.randn((BINS, case["rhs"], nz, ny, nx), generator=g, dtype=torch.float64, device=_dev()), -1, 1.0), -2, 1.0))
    return lat, dlat, dlon, U, V, dP, Dz, c.reshape(BINS, case["rhs"], -1)


def _met_devices(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    lat, dlat, dlon, U, V, dP, Dz, c = _fct_met(case, seed)
    lat, dP, Dz, U, V = (t.cpu().numpy() for t in (lat, dP, Dz, U, V))
    zero, inter = np.zeros((nz, ny, nx)), np.zeros((nz + 1, ny, nx))
    mets = []
    for t in range(BINS):
        u, ue, v, vn = U[t, :, :, :nx].copy(), U[t, :, :, nx].copy(), V[t, :, :ny].copy(), V[t, :, ny].copy()
        mets.append(device.MetDevice(synthetic.MetBin(
            nz=nz, ny=ny, nx=nx, lat=lat, lon=60.0 + dlon * np.arange(nx), dlat=dlat, dlon=dlon, dP=dP, Dz=Dz,
            u=u, v=v, u_plus=np.maximum(u, 0), u_minus=np.maximum(-u, 0), v_plus=np.maximum(v, 0),
            v_minus=np.maximum(-v, 0), u_e=ue, u_plus_e=np.maximum(ue, 0), u_minus_e=np.maximum(-ue, 0), v_n=vn,
            v_plus_n=np.maximum(vn, 0), v_minus_n=np.maximum(-vn, 0), kxxyy=zero + 1e3, kzz=zero + 1.0,
            w_plus=inter, w_minus=inter, cmfmc=inter, kmu=zero, kmv=zero)))
    return mets, c


# ---- what is measured ------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "fct":
        mets, c = _met_devices(case, seed)
        return {"kind": kind, "mets": mets, "c": c}
    T, d = _inputs(case, seed)
    s = {"kind": kind, "tol": case["tol"], "adjoint": case["adjoint"], "bits": case["bits"], "n": case["sets"],
         "T": [T[t] for t in range(BINS)], "d": [d[q, t] for q in range(case["sets"]) for t in range(BINS)]}
    sym = _sym(case)
    if kind == "orbits":
        s["solver"] = api.OrbitSolver(case["nz"], case["ny"], case["nx"], case["sets"], case["bits"], sym=sym,
                                      periodic=case["periodic"])
        s["E"] = _forcing(1002 + 10 * seed, case)
        return s
    s["fb"] = fb = device.FactorBatch(sym, case["rhs"], case["bits"], n_sets=case["sets"])
    s["T"] = [s["T"][t] for _ in range(case["sets"]) for t in range(BINS)]
    if kind in ("factor", "chain"):
        s["x"] = _vectors(1003 + 10 * seed, case["rhs"], sym.N)
    else:
        s["E"] = _forcing(1002 + 10 * seed, case)
    if kind != "factor":
        fb.map(_slots(case, seed))
        fb.numeric(s["T"], s["d"], DTAU)
    return s


def run(s):
    kind = s["kind"]
    if kind == "fct":
        return [device.fct_source(m, s["c"][t], DTAU) for t, m in enumerate(s["mets"])]
    if kind == "orbits":
        s["solver"].factor(s["T"], s["d"], s["n"], DTAU)
        return s["solver"].solve_device(s["E"], tol=s["tol"])[0]
    if kind == "factor":
        s["fb"].numeric(s["T"], s["d"], DTAU)
        return s["fb"].chain(s["x"], trans=s["adjoint"])
    if kind == "chain":
        y = s["fb"].chain(s["x"], trans=s["adjoint"], refine=False)
        return y.float() if s["bits"] == 32 else y  # a sweep on 32-bit factors has 32-bit values
    if s["adjoint"]:
        return s["fb"].solve_adjoint(s["E"], tol=s["tol"])[0]
    return s["fb"].solve(s["E"], tol=s["tol"])[0]


def work(case):
    nz, ny, nx, n, sets = case["nz"], case["ny"], case["nx"], case["rhs"], case["sets"]
    N = nz * ny * nx
    if case["kind"] == "fct":  # c in, d out, u+-, v+-, dP, Dz once a bin
        return {"bytes": 8.0 * BINS * N * (2 * n + 6), "flops": 200.0 * BINS * n * N}
    sym = _sym(case)
    vb = case["bits"] // 8
    factors = float(sets) * BINS * sym.lunz
    sweep_flops = 2.0 * n * BINS * sym.lunz
    vec = 8.0 * n * N
    if case["kind"] == "chain":
        return {"bytes": factors * vb + 2 * vec, "flops": sweep_flops}
    a, m = sym.array("n").astype(float), sym.array("m").astype(float)
    lu = float(sets) * BINS * (2.0 / 3.0) * float(((a + m) ** 3 - m ** 3).sum())
    ops = 8.0 * N * BINS * (7 + sets)
    # a solve cannot do with fewer than the forcing's sweep, one Krylov sweep and the recovery sweep
    used = min(sets, n)
    solve = {"bytes": 3 * factors * used / sets * vb + (8 + 9) * vec, "flops": 3 * sweep_flops}
    if case["kind"] == "solve":
        return solve
    if case["kind"] == "factor":
        return {"bytes": ops + 2 * factors * vb + 2 * vec, "flops": lu + sweep_flops}
    return {"bytes": ops + factors * vb + solve["bytes"], "flops": lu + solve["flops"]}


# ---- the same in 64 bits, by other means -----------------------------------

class _Bin:
    """A = I + dtau (T + diag d) of one bin on a (nz, ny, nx) box, for sets of operators."""

    def __init__(self, T, d, shape):
        nz, ny, nx = shape
        self.a = (DTAU * T).reshape(1, 7, nz, ny, nx).repeat(d.shape[0], 1, 1, 1, 1)
        self.a[:, 0] += 1.0 + DTAU * d.reshape(-1, nz, ny, nx)
        col = torch.diag_embed(self.a[:, 0].permute(0, 2, 3, 1))
        k = torch.arange(nz - 1, device=col.device)
        col[..., k + 1, k] = self.a[:, 5].permute(0, 2, 3, 1)[..., 1:]
        col[..., k, k + 1] = self.a[:, 6].permute(0, 2, 3, 1)[..., :-1]
        self.cols = torch.linalg.inv(col).reshape(-1, ny * nx, nz, nz)

    def mul(self, x, trans):
        """A x or A^T x; boundary entries are zero, wrapped ones belong to a periodic grid."""
        y = self.a[:, 0] * x
        for d, dim, by in ((1, -1, 1), (2, -1, -1), (3, -2, 1), (4, -2, -1), (5, -3, 1), (6, -3, -1)):
            y += torch.roll(self.a[:, d] * x, -by, dim) if trans else self.a[:, d] * torch.roll(x, by, dim)
        return y

    def columns(self, x, trans):
        n, nz, ny, nx = x.shape
        c = self.cols.transpose(-1, -2) if trans else self.cols
        v = x.reshape(n, nz, ny * nx)
        if c.shape[0] == 1:
            return torch.matmul(c[0], v.permute(2, 1, 0)).permute(2, 1, 0).reshape(x.shape)
        return torch.matmul(c, v.permute(0, 2, 1)[..., None])[..., 0].permute(0, 2, 1).reshape(x.shape)

    def solve(self, b, trans):
        """BiCGSTAB with the columns' inverses, restarted on the true residual."""
        dot = lambda p, q: (p * q).sum(dim=(1, 2, 3), keepdim=True)  # noqa: E731
        tiny = 1e-300
        x = torch.zeros_like(b)
        bn = dot(b, b) + tiny
        for _ in range(3):
            r = b - self.mul(x, trans)
            if float((dot(r, r) / bn).max()) < 1e-30:
                break
            r0, p, rho = r.clone(), r.clone(), dot(r, r)
            for it in range(40):
                ph = self.columns(p, trans)
                v = self.mul(ph, trans)
                open_ = dot(r, r) > 1e-32 * bn  # one that is done stays as it is
                alpha = torch.where(open_, rho / (dot(r0, v) + tiny), 0.0)
                s = r - alpha * v
                sh = self.columns(s, trans)
                t = self.mul(sh, trans)
                om = torch.where(open_, dot(t, s) / (dot(t, t) + tiny), 0.0)
                x = x + alpha * ph + om * sh
                r = s - om * t
                if it % 4 == 3 and float((dot(r, r) / bn).max()) < 1e-31:
                    break
                new = dot(r0, r)
                p = r + torch.where(open_, new * alpha / (rho * om + tiny), 0.0) * (p - om * v)
                rho = new
        return x


def _sweep(bins, x, trans, forcing=None, keep=False):
    """The chained bin solves: x -> P x (+ P dtau e), or P^T x (+ R)."""
    got = [x]
    for t in (range(BINS - 1, -1, -1) if trans else range(BINS)):
        if forcing is not None and not trans:
            x = x + DTAU * forcing[:, t]
        x = bins[t].solve(x, trans)
        if forcing is not None and trans:
            x = x + forcing[:, t]
        got.append(x)
    return got if keep else x


def _periodic(bins, e, trans):
    """The orbit: c_0 = M c_0 + s by restarted GMRES, then one sweep of it."""
    s = _sweep(bins, torch.zeros_like(e[:, 0]), trans, e)
    c = s.clone()
    n = s.shape[0]
    sn = s.reshape(n, -1).norm(dim=1) + 1e-300
    for _ in range(4):
        r = (s + _sweep(bins, c, trans) - c).reshape(n, -1)
        beta = r.norm(dim=1)
        if float((beta / sn).max()) < 2e-14:
            break
        V, H = [r / (beta[:, None] + 1e-300)], torch.zeros((n, 13, 12), dtype=s.dtype, device=s.device)
        for j in range(12):
            v = V[-1].reshape(s.shape)
            w = (v - _sweep(bins, v, trans)).reshape(n, -1)
            for _pass in range(2):
                for i, u in enumerate(V):
                    h = (u * w).sum(dim=1)
                    H[:, i, j] += h
                    w = w - h[:, None] * u
            H[:, j + 1, j] = w.norm(dim=1)
            V.append(w / (H[:, j + 1, j, None] + 1e-300))
            g = torch.zeros((n, j + 2), dtype=s.dtype, device=s.device)
            g[:, 0] = beta
            y = torch.linalg.lstsq(H[:, :j + 2, :j + 1], g[..., None]).solution
            left = (g - (H[:, :j + 2, :j + 1] @ y)[..., 0]).norm(dim=1)
            if float((left / sn).max()) < 1e-14:
                break
        c = c + sum(y[:, i] * V[i] for i in range(y.shape[1])).reshape(s.shape)
    got = _sweep(bins, c, trans, e, keep=True)
    if not trans:
        return torch.stack([c] + got[1:], dim=1).reshape(n, BINS + 1, -1)
    return torch.stack([c] + got[BINS - 1:0:-1] + [c], dim=1).reshape(n, BINS + 1, -1)


def _phi(num, den):
    """van Leer's limiter of num / den, as (r + |r|) / (1 + |r|)."""
    r = num / den
    return (r + r.abs()) / (1.0 + r.abs())


def _fct_exact(case, seed):
    """Zalesak's limited anti-diffusive source with van Leer's reconstruction, terrain weights, per bin."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    lat, dlat, dlon, U, V, dP, Dz, cs = _fct_met(case, seed)
    _, _, _, dx, dy = _geometry(ny, nx, False)
    rho = dP / (GRAVITY * Dz)
    out = []
    for t in range(BINS):
        x = cs[t].reshape(-1, nz, ny, nx) / rho
        flux, tl, th = {}, {}, {}
        for dim, W, width in ((-1, U[t][..., 1:nx], dx[:, None].expand(ny, nx - 1)),
                              (-2, V[t][..., 1:ny, :], torch.full((ny - 1, nx), dy, dtype=x.dtype, device=x.device))):
            n = x.shape[dim]
            L, H = x.narrow(dim, 0, n - 1), x.narrow(dim, 1, n - 1)
            jump = H - L
            pl, ph = torch.zeros_like(jump), torch.zeros_like(jump)
            pl.narrow(dim, 1, n - 2).copy_(_phi(jump.narrow(dim, 0, n - 2), jump.narrow(dim, 1, n - 2)))
            ph.narrow(dim, 0, n - 2).copy_(_phi(jump.narrow(dim, 1, n - 2), jump.narrow(dim, 0, n - 2)))
            flux[dim] = 0.5 * (W.clamp(min=0) * pl + (-W).clamp(min=0) * ph) * jump / width
            a, b = dP.narrow(dim, 0, n - 1), dP.narrow(dim, 1, n - 1)
            tl[dim], th[dim] = 0.5 * (a + b) / a, 0.5 * (a + b) / b
            if dim == -2:
                mid = 0.5 * (dx[:-1] + dx[1:])
                tl[dim] = tl[dim] * (mid / dx[:-1])[:, None]
                th[dim] = th[dim] * (mid / dx[1:])[:, None]
        gain, loss, top, low = torch.zeros_like(x), torch.zeros_like(x), x.clone(), x.clone()
        for dim in (-1, -2):
            n = x.shape[dim]
            into_h, into_l = th[dim] * flux[dim], -tl[dim] * flux[dim]
            for at, f in ((1, into_h), (0, into_l)):
                gain.narrow(dim, at, n - 1).add_(f.clamp(min=0))
                loss.narrow(dim, at, n - 1).add_((-f).clamp(min=0))
            L, H = x.narrow(dim, 0, n - 1), x.narrow(dim, 1, n - 1)
            for at, other in ((0, H), (1, L)):
                top.narrow(dim, at, n - 1).copy_(torch.maximum(top.narrow(dim, at, n - 1), other))
                low.narrow(dim, at, n - 1).copy_(torch.minimum(low.narrow(dim, at, n - 1), other))
        rp = torch.where(gain > 0, ((top - x) / DTAU / gain).clamp(max=1), torch.zeros_like(x))
        rm = torch.where(loss > 0, ((x - low) / DTAU / loss).clamp(max=1), torch.zeros_like(x))
        d = torch.zeros_like(x)
        for dim in (-1, -2):
            n = x.shape[dim]
            f = flux[dim]
            c = torch.where(th[dim] * f >= 0, torch.minimum(rp.narrow(dim, 1, n - 1), rm.narrow(dim, 0, n - 1)),
                            torch.minimum(rm.narrow(dim, 1, n - 1), rp.narrow(dim, 0, n - 1))).clamp(0, 1)
            d.narrow(dim, 1, n - 1).add_(th[dim] * c * f)
            d.narrow(dim, 0, n - 1).sub_(tl[dim] * c * f)
        out.append((d * rho).reshape(case["rhs"], -1))
    return out


def exact(case, seed):
    if case["kind"] == "fct":
        return _fct_exact(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    T, d = _inputs(case, seed)
    set_of = _slots(case, seed)
    if case["sets"] > 1:
        d = d[set_of]
    bins = [_Bin(T[t], d[:, t], shape) for t in range(BINS)]
    n = case["rhs"]
    if case["kind"] in ("factor", "chain"):
        x = _vectors(1003 + 10 * seed, n, math.prod(shape)).reshape(n, *shape)
        return _sweep(bins, x, case["adjoint"]).reshape(n, -1)
    e = _forcing(1002 + 10 * seed, case).reshape(n, BINS, *shape)
    return _periodic(bins, e, case["adjoint"])
