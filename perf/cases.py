"""Workloads of the interior-point numeric core, through its public entry
points: what a program that solves nonlinear programs with this package has
it do, from the single small KKT system to the batched and 3D ones.

Kinds of case:
  direction   one search direction: SparseLDL factor, inertia, solve and
              `refine` steps of refinement against the FP64 matrix (the
              mixed-precision form, precision "fp32", takes four)
  batch       the same for many independent KKT systems at once
              (BatchedSparseLDL)
  solve       a refined solve on a factorization that is kept: one right-hand
              side (directions) or several (post-optimality sensitivities)
  iteration   the numeric core of one interior-point iteration of the 2D
              SIMP model: derivatives, diagonal, factorization, direction,
              bound duals, step lengths, step
  assembly    gradient and Hessian of the 3D SIMP model into the KKT values

Models: the cart-pole transcription (N intervals) and the SIMP compliance
models (2D nx x ny, 3D nx x ny x nz).  `point` "start" is the models'
initial point (displacements and multipliers zero), "mid" an iterate in the
middle of a solve (every block of the KKT non-zero).  The diagonal carries
the barrier terms z / s of the bounded variables and the inertia
correction's shift.
"""
import functools
import math

import numpy as np
import torch

from amigo_b200 import linalg
from amigo_b200.fem import CartPoleDevice, Simp2DDevice, Simp3DDevice
from amigo_b200.ipm import InteriorPointOptimizer
from amigo_b200.problems.cartpole import (GRAV, L_POLE, M_CART, CartPole,
                                          batch_config)
from amigo_b200.problems.simp2d import E0, EMIN, PENALTY, Simp2D
from amigo_b200.problems.simp3d import Simp3D

DEV = "cuda:0"
MU = 0.1          # barrier parameter
TAU = 0.99        # fraction to the boundary
SHIFT = 1e-4      # first inertia-correction shift of the drivers
F64 = dict(dtype=torch.float64, device=DEV)


def listed():
    return [
        # one trajectory problem solved alone: a few fronts of at most 68
        # rows, a chain of short launches
        dict(name="direction_cartpole_100", kind="direction", model="cartpole",
             N=100, point="mid", precision="fp64", refine=1),
        # a coarse topology mesh, as solved while a model is set up
        dict(name="direction_simp2d_32x16", kind="direction", model="simp2d",
             nx=32, ny=16, point="start", precision="fp64", refine=1),
        # an odd mesh in the middle of a solve
        dict(name="direction_simp2d_61x27", kind="direction", model="simp2d",
             nx=61, ny=27, point="mid", precision="fp64", refine=1),
        # the benchmark's KKT
        dict(name="direction_simp2d_128x64", kind="direction", model="simp2d",
             nx=128, ny=64, point="start", precision="fp64", refine=1),
        # mixed precision: FP32 fronts, tensor-core updates, refinement
        dict(name="direction_simp3d_12x6x6_fp32", kind="direction", model="simp3d",
             nx=12, ny=6, nz=6, point="mid", precision="fp32", refine=4),
        # fronts of several thousand rows: the Schur updates' share grows
        dict(name="direction_simp3d_20x10x10", kind="direction", model="simp3d",
             nx=20, ny=10, nz=10, point="mid", precision="fp64", refine=1),
        # the batched trajectory configuration, and a small batch as the
        # serving loop sees it
        dict(name="batch_cartpole_512", kind="batch", k=512, sizes=0, nmin=50,
             nmax=400, precision="fp64", refine=1),
        dict(name="batch_cartpole_24_fp32", kind="batch", k=24, sizes=7, nmin=50,
             nmax=200, precision="fp32", refine=4),
        # refined solves on a kept factorization: a direction, sensitivities
        dict(name="solve_simp2d_128x64", kind="solve", model="simp2d", nx=128,
             ny=64, point="start", nrhs=1),
        dict(name="solve_simp3d_12x6x6_rhs8", kind="solve", model="simp3d", nx=12,
             ny=6, nz=6, point="mid", nrhs=8),
        # a whole iteration's numeric core
        dict(name="iteration_simp2d_64x32", kind="iteration", model="simp2d",
             nx=64, ny=32, point="mid"),
        # KKT assembly of the largest class of meshes
        dict(name="assembly_simp3d_24x12x12", kind="assembly", model="simp3d",
             nx=24, ny=12, nz=12, point="mid"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, model, lo, hi):
    nx = _log_int(rng, lo, hi)
    half = lambda: max(2, rng.randint(max(2, nx // 4), max(2, nx // 2)))
    c = dict(model=model, nx=nx, ny=half(), point=rng.choice(["start", "mid", "mid"]))
    if model == "simp3d":
        c["nz"] = half()
    return c


def draw(rng):
    kind = rng.choice(["direction"] * 5 + ["batch"] * 2 + ["solve"] * 2 +
                      ["iteration", "assembly"])
    prec = rng.choice(["fp64", "fp64", "fp32"])
    mix = dict(precision=prec, refine=4 if prec == "fp32" else 1)
    if kind == "batch":
        lo = rng.randint(50, 150)
        return dict(kind=kind, k=_log_int(rng, 4, 400), sizes=rng.randint(1, 999),
                    nmin=lo, nmax=rng.randint(lo + 20, 400), **mix)
    if kind == "assembly":
        model = rng.choice(["simp2d", "simp3d"])
        return dict(kind=kind, **_mesh(rng, model, 8, 128 if model == "simp2d" else 24))
    if kind == "iteration":
        return dict(kind=kind, **_mesh(rng, "simp2d", 12, 128))
    model = rng.choice(["simp2d", "simp2d", "simp3d", "cartpole"])
    mixed = kind == "direction" and prec == "fp32"
    if mixed and model == "simp2d":
        # the 2D KKT is past FP32 fronts (the drivers refactor it in FP64)
        model = "simp3d"
    if model == "cartpole":
        c = dict(model=model, N=_log_int(rng, 50, 400), point="mid")
    else:
        c = _mesh(rng, model, 8, 128 if model == "simp2d" else 16 if mixed else 20)
        if mixed:
            c["point"] = "mid"
    if kind == "solve":
        return dict(kind=kind, nrhs=rng.choice([1, 1, 2, 5, 8]), **c)
    return dict(kind=kind, **c, **mix)


# ------------------------------------------------------------------ models
@functools.lru_cache(maxsize=16)
def _build(kind, *size):
    if kind == "simp2d":
        return Simp2D(*size)
    if kind == "simp3d":
        return Simp3D(*size)
    if kind == "cartpole":
        return CartPole(N=size[0])
    return batch_config(k=size[0], seed=size[1], nmin=size[2], nmax=size[3])


def _model(c):
    if c["kind"] == "batch":
        return _build("batch", c["k"], c["sizes"], c["nmin"], c["nmax"])
    if c["model"] == "cartpole":
        return _build("cartpole", c["N"])
    if c["model"] == "simp2d":
        return _build("simp2d", c["nx"], c["ny"])
    return _build("simp3d", c["nx"], c["ny"], c["nz"])


def _is_simp(c):
    return c["kind"] != "batch" and c["model"] != "cartpole"


def _device_model(c, m):
    if c["kind"] == "batch":
        return CartPoleDevice(m, DEV, batch=True)
    if c["model"] == "cartpole":
        return CartPoleDevice(m, DEV)
    return (Simp2DDevice if c["model"] == "simp2d" else Simp3DDevice)(m, DEV)


def _point(c, m, seed):
    """The iterate x (host) of a case: primals inside their bounds."""
    r = np.random.RandomState(seed)
    if not _is_simp(c):
        x = m.x0 + np.where(m.mult, 0.1 * r.randn(m.n), 0.05 * r.randn(m.n))
        lo = np.where(m.mult, -np.inf, m.lower)
        hi = np.where(m.mult, np.inf, m.upper)
        return np.clip(x, lo + 1e-2, hi - 1e-2)
    x = np.zeros(m.n)
    rt, re = slice(m.rt0, m.rt0 + m.nnodes), slice(m.re0, m.re0 + m.nelems)
    if c["point"] == "start":
        x[re] = m.volfrac + r.uniform(-0.01, 0.01, m.nelems)
        nv = m.conn.shape[1]
        x[rt] = (np.bincount(m.conn.ravel(), np.repeat(x[re], nv), m.nnodes) /
                 np.bincount(m.conn.ravel(), minlength=m.nnodes))
        x[m.s0] = min(x[re].mean() - m.volfrac, -1e-3)
    else:
        x[:] = 0.1 * r.randn(m.n)
        x[rt] = r.uniform(0.05, 0.95, m.nnodes)
        x[re] = r.uniform(0.05, 0.95, m.nelems)
        x[m.s0] = -r.uniform(0.01, 0.1)
    return x


def _bounds(m, x, seed):
    """Slacks and bound duals of the primals (n-vectors on the host; 1 and 0
    where a bound is missing), duals within a factor two of mu / s."""
    r = np.random.RandomState(seed + 1000003)
    prim = ~np.asarray(m.mult, bool)
    out = []
    for bound, gap in ((m.lower, x - m.lower), (m.upper, m.upper - x)):
        fin = np.isfinite(bound) & prim
        s = np.where(fin, np.maximum(gap, 1e-2), 1.0)
        out += [s, np.where(fin, MU / s * r.uniform(0.5, 2.0, m.n), 0.0)]
    return out          # sl, zl, su, zu


def _diagonal(m, x, seed):
    sl, zl, su, zu = _bounds(m, x, seed)
    d = zl / sl + zu / su + SHIFT * ~np.asarray(m.mult, bool)
    if hasattr(m, "fixed"):
        d[m.fixed] = 0.0
    return d


def _rhs(n, nrhs, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn((nrhs, n) if nrhs > 1 else (n,), generator=g, **F64)


def _up(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _kkt(c, m, seed):
    """CSRMat with the KKT values of the case, assembled by the model's
    device kernels, and the model's device form."""
    x = _point(c, m, seed)
    K = linalg.CSRMat(m.n, m.n, m.rowp, m.cols, device=DEV, diag_pos=m.diag_pos)
    dm = _device_model(c, m)
    dm.hessian(_up(x), 1.0, K.vals)
    K.add_diagonal(_up(_diagonal(m, x, seed)))
    return K, dm


# ----------------------------------------------------------------- passes
def prepare(case, seed):
    c = dict(case)
    m = _model(c)
    s = dict(c=c, m=m)
    if c["kind"] == "assembly":
        x = _point(c, m, seed)
        s.update(dm=_device_model(c, m), x=_up(x), g=torch.zeros(m.n, **F64),
                 K=linalg.CSRMat(m.n, m.n, m.rowp, m.cols, device=DEV,
                                 diag_pos=m.diag_pos),
                 diag=_up(_diagonal(m, x, seed)))
        return s
    if c["kind"] == "iteration":
        return _prepare_iteration(s, seed)
    K, _ = _kkt(c, m, seed)
    nrhs = c.get("nrhs", 1)
    b = _rhs(m.n, nrhs, seed)
    s.update(K=K, b=b, x=torch.empty_like(b), r=torch.empty_like(b))
    if c["kind"] == "batch":
        s["ldl"] = linalg.BatchedSparseLDL(m.patterns(), device=DEV)
    else:
        s["ldl"] = linalg.SparseLDL(K, order=linalg.OrderingType.AMD)
    if c.get("precision", "fp64") != "fp64":
        s["ldl"].set_precision(c["precision"])
    if c["kind"] == "solve":
        s["ldl"].factor()
    return s


def _prepare_iteration(s, seed):
    m, c = s["m"], s["c"]
    x = _point(c, m, seed)
    opt = InteriorPointOptimizer(m.mult, m.lower, m.upper, device=DEV)
    v = opt.create_opt_vector(_up(x))
    prim = ~np.asarray(m.mult, bool)
    sl, zl, su, zu = _bounds(m, x, seed)
    v.duals.copy_(_up(np.concatenate([zl[prim], zu[prim]])))
    v.slacks.copy_(_up(np.concatenate([sl[prim], su[prim]])))
    K = linalg.CSRMat(m.n, m.n, m.rowp, m.cols, device=DEV, diag_pos=m.diag_pos)
    vec = lambda: torch.zeros(m.n, **F64)
    shift = np.where(prim, SHIFT, 0.0)
    shift[m.fixed] = 0.0
    s.update(opt=opt, v=v, K=K, dm=_device_model(c, m),
             ldl=linalg.SparseLDL(K, order=linalg.OrderingType.AMD),
             shift=_up(shift), g=vec(), res=vec(), diag=vec(), px=vec(), r=vec(),
             upd=opt.create_opt_vector(), new=opt.create_opt_vector(), gnew=vec())
    return s


def run(state):
    s = state
    kind = s["c"]["kind"]
    if kind == "assembly":
        s["dm"].gradient(s["x"], 1.0, s["g"])
        s["dm"].hessian(s["x"], 1.0, s["K"].vals)
        s["K"].add_diagonal(s["diag"])
        return {"gradient": s["g"], "values": s["K"].vals}
    if kind == "iteration":
        return _run_iteration(s)
    ldl, K, b, x, r = s["ldl"], s["K"], s["b"], s["x"], s["r"]
    if kind == "solve":
        x.copy_(b)
        ldl.solve_device(x)
        for xk, rk in zip(x.view(-1, x.shape[-1]), r.view(-1, x.shape[-1])):
            K.mult(xk, rk)
        torch.sub(b, r, out=r)
        ldl.solve_device(r)
        x.add_(r)
        return {"x": x}
    if kind == "batch":
        ldl.factor(K.vals)
    else:
        ldl.factor()
    inertia = np.array(ldl.get_inertia())
    x.copy_(b)
    ldl.solve_device(x)
    for _ in range(s["c"]["refine"]):
        K.mult(x, r)
        torch.sub(b, r, out=r)
        ldl.solve_device(r)
        x.add_(r)
    return {"x": x, "inertia": inertia}


def _run_iteration(s):
    opt, v, K, ldl, dm = s["opt"], s["v"], s["K"], s["ldl"], s["dm"]
    g, res, diag, px, r, upd, new = (s[k] for k in
                                     ("g", "res", "diag", "px", "r", "upd", "new"))
    dm.gradient(v.x, 1.0, g)
    dm.hessian(v.x, 1.0, K.vals)
    opt.compute_diagonal(v, diag)
    diag.add_(s["shift"])
    K.add_diagonal(diag)
    ldl.factor()
    inertia = np.array(ldl.get_inertia())
    norm = opt.compute_residual(MU, v, g, res)
    px.copy_(res)
    ldl.solve_device(px)
    K.mult(px, r)
    torch.sub(res, r, out=r)
    ldl.solve_device(r)
    px.add_(r)
    opt.compute_update(MU, v, px, upd)
    ax, ix, az, iz = opt.compute_max_step(TAU, v, upd)
    opt.apply_step_update(ax, az, v, upd, new)
    dm.gradient(new.x, 1.0, s["gnew"])
    return {"norm": norm, "inertia": inertia, "px": px, "ax": ax, "az": az,
            "first": np.array([ix, iz]), "x": new.x, "duals": new.duals,
            "slacks": new.slacks, "gradient": s["gnew"]}


# ------------------------------------------------------------------- work
@functools.lru_cache(maxsize=64)
def _front_sums(*key):
    """(factor entries, factor operations) of a KKT pattern without delays."""
    m = _build(*key)
    pats = m.patterns() if key[0] == "batch" else [(m.n, m.rowp, m.cols)]
    seen, ent, fl = {}, 0.0, 0.0
    for n, rowp, cols in pats:
        if n not in seen:
            t = linalg.analyze(n, rowp, cols)
            p = np.diff(t["node_ptr"]).astype(float)
            q = np.diff(t["contrib_ptr"]).astype(float)
            seen[n] = ((p * (p + 1) / 2 + p * q).sum(),
                       (p ** 3 / 3 + p * p * q + p * q * q).sum())
        ent += seen[n][0]
        fl += seen[n][1]
    return ent, fl


def _key(c):
    if c["kind"] == "batch":
        return ("batch", c["k"], c["sizes"], c["nmin"], c["nmax"])
    if c["model"] == "cartpole":
        return ("cartpole", c["N"])
    return (c["model"],) + tuple(c[k] for k in ("nx", "ny", "nz") if k in c)


def work(case):
    """KKT values read and factor written once, factor read once per sweep
    (two sweeps per solve), vectors once; the operations of the fronts
    without delayed pivots and of the sweeps."""
    c = dict(case)
    m = _model(c)
    if c["kind"] == "assembly":
        ne, ks, kf = m.nelems, m.ev.shape[1], m.fv.shape[1]
        return {"bytes": 8.0 * m.nnz + 4.0 * ne * (ks * ks + kf * kf) + 16.0 * m.n,
                "flops": 2.0 * ne * (ks * ks + kf * kf)}
    ent, fl = _front_sums(*_key(c))
    w = 4 if c.get("precision") == "fp32" else 8
    if c["kind"] == "solve":
        return {"bytes": 12.0 * m.nnz + 4 * w * ent + 32.0 * m.n * c["nrhs"],
                "flops": (2.0 * m.nnz + 8 * ent) * c["nrhs"]}
    solves = 1 + c.get("refine", 1)
    bytes_ = 12.0 * m.nnz * solves + w * ent * (1 + 2 * solves) + 24.0 * m.n * solves
    if c["kind"] == "iteration":
        bytes_ += 8.0 * m.nnz + 8.0 * 30 * m.n
    return {"bytes": bytes_, "flops": fl + 4 * ent * solves}


# ------------------------------------------- 64-bit values, by torch alone
def _simp_parts(m, x):
    nd, nv = m.K0.shape[0], m.A.shape[0]
    u, rt, lam = x[m.ev[:, :nd]], x[m.ev[:, nd:nd + nv]], x[m.ev[:, nd + nv:]]
    r = rt.mean(axis=1)
    span = E0 - EMIN
    return (nd, nv, rt, u @ m.K0.T, lam @ m.K0.T, lam, EMIN + r ** PENALTY * span,
            PENALTY * r ** (PENALTY - 1) * span,
            PENALTY * (PENALTY - 1) * r ** (PENALTY - 2) * span)


def _simp_values(m, x):
    nd, nv, _, Ku, Kl, lam, E, dE, d2E = _simp_parts(m, x)
    k = 2 * nd + nv
    R, L = slice(nd, nd + nv), slice(nd + nv, k)
    H = np.zeros((m.nelems, k, k))
    H[:, :nd, R] = (dE[:, None] * Kl)[:, :, None] / nv
    H[:, R, :nd] = np.transpose(H[:, :nd, R], (0, 2, 1))
    H[:, :nd, L] = E[:, None, None] * m.K0
    H[:, L, :nd] = E[:, None, None] * m.K0.T
    H[:, R, R] = (d2E * np.sum(lam * Ku, axis=1))[:, None, None] / nv ** 2
    H[:, L, R] = (dE[:, None] * Ku)[:, :, None] / nv
    H[:, R, L] = np.transpose(H[:, L, R], (0, 2, 1))
    Fb = np.zeros((2 * nv + 1, 2 * nv + 1))
    Fb[nv + 1:, :nv] = m.A
    Fb[:nv, nv + 1:] = m.A.T
    Fb[nv + 1:, nv] = Fb[nv, nv + 1:] = -1.0 / nv
    vals = np.bincount(m.epos.ravel(), H.reshape(-1), m.nnz)
    vals += np.bincount(m.fpos.ravel(), np.tile(Fb.ravel(), m.nelems), m.nnz)
    vals += np.bincount(m.vpos.ravel(), np.full(m.vpos.size, 1.0 / m.nelems), m.nnz)
    vals[m.spos] -= 1.0
    vals[m.fixed_zero_pos] = 0.0
    vals[m.fixed_diag_pos] = 1.0
    return vals


def _simp_gradient(m, x):
    nd, nv, rt, Ku, Kl, lam, E, dE, _ = _simp_parts(m, x)
    re, mu = x[m.fv[:, nv]], x[m.fv[:, nv + 1:]]
    g = m.f.copy()                          # objective f^T u
    nu = m.rt0 - m.u0
    g[m.lam0:m.lam0 + nu] -= m.f[m.u0:m.u0 + nu]
    add = lambda idx, v: np.add.at(g, idx, v)
    add(m.ev[:, :nd], E[:, None] * Kl)
    add(m.ev[:, nd:nd + nv],
        (dE * np.sum(lam * Ku, axis=1))[:, None] / nv + mu @ m.A)
    add(m.ev[:, nd + nv:], E[:, None] * Ku)
    add(m.fv[:, nv], x[m.nu0] / m.nelems - mu.sum(axis=1) / nv)
    add(m.fv[:, nv + 1:], rt @ m.A.T - re[:, None] / nv)
    g[m.nu0] += re.sum() / m.nelems - m.volfrac - x[m.s0]
    g[m.s0] -= x[m.nu0]
    g[m.fixed] = 0.0
    return g


def _cartpole_values(m, x, h, mp):
    def lagrangian(z, h, mp):
        def f(q):
            s, c = torch.sin(q[1]), torch.cos(q[1])
            den = M_CART + mp * (1.0 - c * c)
            w = q[3] * q[3]
            return torch.stack([
                q[2], q[3],
                (L_POLE * mp * s * w + q[4] + mp * GRAV * c * s) / den,
                -(L_POLE * mp * c * s * w + q[4] * c + (M_CART + mp) * GRAV * s)
                / (L_POLE * den)])
        a, b, lam = z[:5], z[5:10], z[10:]
        d = b[:4] - a[:4] - 0.5 * h * (f(a) + f(b))
        return 0.5 * h * (a[4] ** 2 + b[4] ** 2) + torch.dot(lam, d)

    H = torch.func.vmap(torch.func.hessian(lagrangian))(
        _up(x[m.iv]), _up(h), _up(mp)).cpu().numpy()
    B = np.zeros((8, 8))
    B[:4, 4:] = B[4:, :4] = np.eye(4)
    vals = np.bincount(m.ipos.ravel(), H.reshape(-1), m.nnz)
    return vals + np.bincount(m.bpos.ravel(), np.tile(B.ravel(), len(m.bpos)), m.nnz)


def _values(c, m, x, seed):
    if c["kind"] == "batch":
        v = _cartpole_values(m, x, m.h_iv, m.m_iv)
    elif c["model"] == "cartpole":
        v = _cartpole_values(m, x, np.full(m.N, m.h), np.full(m.N, m.m_pole))
    else:
        v = _simp_values(m, x)
    v[m.diag_pos] += _diagonal(m, x, seed)
    return v


def _dense_solve(rowp, cols, vals, b):
    """K x = b by a dense LU factorization with refinement (b: (nrhs, n))."""
    n = len(rowp) - 1
    rows = _up(np.repeat(np.arange(n), np.diff(rowp)))
    cl, vl = _up(cols.astype(np.int64)), _up(vals)
    A = torch.zeros((n, n), **F64)
    A[rows, cl] = vl
    lu, piv = torch.linalg.lu_factor(A)
    del A
    K = torch.sparse_csr_tensor(_up(rowp.astype(np.int64)), cl, vl, (n, n), **F64)
    x = torch.linalg.lu_solve(lu, piv, b.T.contiguous())
    for _ in range(3):
        x += torch.linalg.lu_solve(lu, piv, b.T - K @ x)
    return x.T.contiguous()


def exact(case, seed):
    c = dict(case)
    m = _model(c)
    x = _point(c, m, seed)
    if c["kind"] == "assembly":
        return {"gradient": _simp_gradient(m, x), "values": _values(c, m, x, seed)}
    vals = _values(c, m, x, seed)
    if c["kind"] == "iteration":
        return _exact_iteration(m, x, vals, seed)
    b = _rhs(m.n, c.get("nrhs", 1), seed).reshape(-1, m.n)
    if c["kind"] != "batch":
        sol = _dense_solve(m.rowp, m.cols, vals, b)
    else:
        sol = torch.cat([_dense_solve(i.rowp, i.cols, vals[z:z + i.nnz], b[:, o:o + i.n])
                         for i, o, z in zip(m.inst, m.var_off, m.nnz_off)], dim=1)
    out = {"x": sol if c.get("nrhs", 1) > 1 else sol[0]}
    return out if c["kind"] == "solve" else {**out, "inertia": None}


def _exact_iteration(m, x, vals, seed):
    sl, zl, su, zu = _bounds(m, x, seed)
    prim = ~np.asarray(m.mult, bool)
    fl, fu = np.isfinite(m.lower) & prim, np.isfinite(m.upper) & prim
    g = _simp_gradient(m, x)
    dual = g - zl + zu + np.where(fl, zl - MU / sl, 0.0) - np.where(fu, zu - MU / su, 0.0)
    res = -np.where(prim, dual, g - np.where(prim, 0.0, m.lower))
    px = _dense_solve(m.rowp, m.cols, vals, _up(res)[None])[0].cpu().numpy()
    dzl = np.where(fl, -(sl * zl - MU + zl * px) / sl, 0.0)
    dzu = np.where(fu, -(su * zu - MU - zu * px) / su, 0.0)
    ratio = lambda v, d, on: np.min(np.where(on & (d < 0), -TAU * v / np.where(d < 0, d, -1.0),
                                             1.0), initial=1.0)
    ax = min(ratio(sl, px, fl), ratio(su, -px, fu))
    az = min(ratio(zl, dzl, fl), ratio(zu, dzu, fu))
    xn = x + ax * px
    part = lambda a, b: np.concatenate([a[prim], b[prim]])
    return {"norm": float(np.linalg.norm(res)), "inertia": None, "px": px, "ax": float(ax),
            "az": float(az), "first": None, "x": xn,
            "duals": part(np.where(fl, zl + az * dzl, 0.0), np.where(fu, zu + az * dzu, 0.0)),
            "slacks": part(np.where(fl, sl + ax * px, 1.0), np.where(fu, su - ax * px, 1.0)),
            "gradient": _simp_gradient(m, xn)}
