"""Performance cases of the framework: the calls a Newton, continuation or
stability program makes, through the package's public entry points.

A case is a dict of plain values; ``prepare`` builds what such a program has in
hand (mesh, frozen pattern, library context, device buffers, state), ``run`` is
one call on it, ``exact`` is the same result in plain torch FP64.  Library
contexts belong to a mesh and are shared by the states on it, as a program
keeps one context and assembles many states with it; the factorisation that
``solve`` cases use belongs to its state.
"""
from __future__ import annotations

import functools
import math
import warnings

import numpy as np
import torch

from ve_flow_around_cylinder_fortran_gb300 import frontal as FR
from ve_flow_around_cylinder_fortran_gb300 import mesh as M
from ve_flow_around_cylinder_fortran_gb300 import newton as NW
from ve_flow_around_cylinder_fortran_gb300 import state as S
from ve_flow_around_cylinder_fortran_gb300 import vefem as V

JACOBIAN = {"residual": 0, "fd64": V.VEFEM_JAC_FD64, "exact64": V.VEFEM_JAC_EXACT64,
            "exact32": V.VEFEM_JAC_EXACT32}
# network of the learned predictor: (Wi, step) and 3 x 32 reduced coordinates in, 32 out
MLP_IN, MLP_OUT, MLP_WIDTH, MLP_HIDDEN = 98, 32, 256, 3
# solves refined to rounding level: one sweep alone leaves 1e-12 to 1e-7 in x, as its pivots fall
SOLVE_TOL = 1.0e-14


def listed():
    g = dict(model="GIESEKUS", form="SQRT", wi=0.5, ve=0.1, re=0.0)
    o = dict(model="L-PTT", form="SQRT", wi=0.5, ve=0.0, re=0.0)
    t = dict(model="L-PTT", form="T", wi=0.1, ve=0.0, re=0.0)
    return [
        # the smallest call: one residual ('MNR') of a 500-quad test mesh
        dict(name="residual-500", kind="residual", nel=500, **o),
        # a chord iteration or a predictor candidate judged on the benchmark mesh
        dict(name="residual-40000", kind="residual", nel=40000, **g),
        # the drop-in call of a Fortran host: 'NRP' on host arrays, with the outlet edges
        dict(name="host-nrp-2000", kind="host", nel=2000, **t),
        # the headline assembly: residual and forward-difference Jacobian
        dict(name="fd64-40000", kind="fd64", nel=40000, **g),
        # exact FP64 Jacobian of a PTT fluid on a mid-size mesh
        dict(name="exact64-5000", kind="exact64", nel=5000, model="e-PTT", form="T", wi=0.3,
             ve=0.05, re=0.0),
        # the precision form of the learned + mixed continuation
        dict(name="exact32-40000", kind="exact32", nel=40000, **g),
        # a batch of Weissenberg points on meshes of uneven size, FP64 residual + FP32 Jacobian
        dict(name="batched-16", kind="batched", ninst=16, lo=1000, hi=10000, **o),
        # factorise and solve a Newton correction (refined) on a small and on the benchmark mesh
        dict(name="factor-2000", kind="factor", nel=2000, **o),
        dict(name="factor-20000", kind="factor", nel=20000, **o),
        # a chord iteration's refined solve with a factorisation in hand
        dict(name="solve-20000", kind="solve", nel=20000, **o),
        # linear stability: A at 16 spanwise wavenumbers and B
        dict(name="stability-20000x16", kind="stability", nel=20000, nk=16, **dict(t, wi=0.7)),
        # online training of the predictor's network between two continuation steps
        dict(name="mlp-train-40x400", kind="mlp", rows=40, iters=400),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["residual", "host", "fd64", "exact64", "exact32", "batched", "factor",
                       "solve", "stability", "mlp"])
    if kind == "mlp":
        return dict(kind=kind, rows=size(4, 300), iters=size(50, 400))
    model, ve = rng.choice([("L-PTT", 0.0), ("L-PTT", 0.02), ("e-PTT", 0.05), ("GIESEKUS", 0.1),
                            ("GIESEKUS", 0.2)])
    c = dict(kind=kind, model=model, form="T" if kind == "stability" else rng.choice(["T", "SQRT"]),
             wi=round(rng.uniform(0.1, 1.0), 3), ve=ve, re=rng.choice([0.0, 0.0, 0.0, 1.0]))
    if kind in ("factor", "solve"):
        # Jacobians of the continuation's starting branch
        return dict(c, model="L-PTT", ve=0.0, form="SQRT", re=0.0, wi=round(rng.uniform(0.1, 0.6), 3),
                    nel=size(300, 20000))
    if kind == "batched":
        lo = size(200, 1000)
        return dict(c, ninst=rng.randint(3, 16), lo=lo, hi=lo * rng.randint(2, 8))
    if kind == "stability":
        return dict(c, nel=size(200, 20000), nk=rng.randint(1, 16))
    hi = {"host": 5000, "exact64": 20000}.get(kind, 40000)
    return dict(c, nel=size(200, hi))


# ---------------------------------------------------------------- inputs

def _phys(c, nex):
    return S.Physics(model=c["model"], form=c["form"], ReN=c["re"], WiN=c["wi"], Wi0=c["wi"],
                     BvN=0.59, VeN=c["ve"], nex=nex)


def _nex(c):
    return 0 if c["kind"] in ("batched", "stability") else 1


@functools.lru_cache(maxsize=None)
def _mesh(nel, nex):
    m = M.build_cylinder_mesh(nel, exact=False)
    return m, V.build_pattern(m.conn, m.nnodes, nex)


def _key(c):
    return tuple(sorted((k, v) for k, v in c.items() if k != "name"))


@functools.lru_cache(maxsize=None)
def _assembler(key):
    c = dict(key)
    m, (rp, ci) = _mesh(c["nel"], _nex(c))
    return V.BulkAssembler(m, _phys(c, _nex(c)), rp, ci, outlet_edges=True)


def _instances(c):
    """(quads, parameters) of a batch: sizes drawn log-uniformly, Wi uniformly."""
    rng = np.random.default_rng(c["ninst"])
    sizes = np.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]), c["ninst"]))
    wis = rng.uniform(0.1, 1.0, c["ninst"])
    return [(int(round(n)), _phys(dict(c, wi=float(w)), 0)) for n, w in zip(sizes, wis)]


@functools.lru_cache(maxsize=None)
def _batch(key):
    inst = [(_mesh(n, 0), p) for n, p in _instances(dict(key))]
    return V.BatchAssembler([m for (m, _), _ in inst], [p for _, p in inst], [p for (_, p), _ in inst])


def _jacobian_state(c, seed):
    """State, Dirichlet rows and arclength row of a Newton correction: a
    perturbed fully developed state, as at the start of a continuation."""
    m, _ = _mesh(c["nel"], 1)
    phys = _phys(c, 1)
    TL, EU = NW.initial_state(m, phys)
    TL = TL + 0.01 * (S.seeded_state(m.xyz, phys, seed)[0] - TL)
    t = np.random.default_rng(seed).standard_normal(6 * m.nnodes + 1)
    return TL, EU, t / np.linalg.norm(t)


def _x_true(c, seed):
    m, _ = _mesh(c["nel"], 1)
    return np.random.default_rng(seed + 1).standard_normal(6 * m.nnodes + 1)


def _system(c, seed):
    """AIJ values (device) of the bordered Jacobian and b = J x_true."""
    m, (rp, ci) = _mesh(c["nel"], 1)
    asm = _assembler(_key(dict(c, kind="jacobian")))
    TL, EU, t = _jacobian_state(c, seed)
    rows, values = NW.boundary_conditions(m, _phys(c, 1))
    dev = NW.DeviceAssembly(asm, rows, values, "exact64", True)
    dev.device_values = True
    _, vals = dev(TL, EU, True)
    vals[int(rp[-2]):] = torch.from_numpy(t).to(vals.device)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")       # sparse CSR support is marked beta
        A = torch.sparse_csr_tensor(torch.from_numpy(rp).cuda(), torch.from_numpy(ci.astype(np.int64)).cuda(),
                                    vals, size=(asm.N, asm.N), check_invariants=False)
    return vals, A @ torch.from_numpy(_x_true(c, seed)).cuda()


@functools.lru_cache(maxsize=None)
def _solver(nel):
    m, (rp, ci) = _mesh(nel, 1)
    return FR.FrontalLU(rp, ci, m, check_tol=SOLVE_TOL)


def _stability_base(c, seed):
    m, _ = _mesh(c["nel"], 0)
    TL, _ = S.seeded_state(m.xyz, _phys(c, 0), seed)
    base = np.zeros((10, m.nnodes))
    base[0:2], base[3:7] = TL[0:2], TL[2:6]
    return base


def _mlp_data(c, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((c["rows"], MLP_IN)).astype(np.float32)
    return X, np.tanh(X[:, :MLP_OUT] + 0.1 * rng.standard_normal((c["rows"], MLP_OUT))).astype(np.float32)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(case=c)
    if kind == "mlp":
        s["net"] = V.MLP(MLP_IN, MLP_OUT, width=MLP_WIDTH, hidden=MLP_HIDDEN, seed=seed)
        s["X"], s["Y"] = _mlp_data(c, seed)
        return s
    if kind == "batched":
        s["asm"] = _batch(_key(c))
        dev = torch.device("cuda")
        s["TL"] = [torch.from_numpy(S.seeded_state(_mesh(n, 0)[0].xyz, p, seed + 100 * i)[0]).to(dev)
                   for i, (n, p) in enumerate(_instances(c))]
        s["EU"] = [torch.zeros(1, dtype=torch.float64, device=dev) for _ in s["TL"]]
        s["b"] = [torch.zeros(n, dtype=torch.float64, device=dev) for n in s["asm"].N]
        s["vals"] = [torch.zeros(n, dtype=torch.float32, device=dev) for n in s["asm"].nnz]
        return s
    if kind in ("factor", "solve"):
        vals, s["b"] = _system(c, seed)
        if kind == "factor":
            s["lu"], s["vals"] = _solver(c["nel"]), vals
        else:
            m, (rp, ci) = _mesh(c["nel"], 1)
            s["lu"] = FR.FrontalLU(rp, ci, m, check_tol=SOLVE_TOL).factor(vals)
        return s
    asm = s["asm"] = _assembler(_key(c))
    if kind == "stability":
        nnz = len(asm.stability_pattern()[1])
        s["kws"] = np.linspace(0.0, 4.0, c["nk"])
        s["TL"] = torch.from_numpy(_stability_base(c, seed)).cuda()
        s["A"] = [torch.zeros(nnz, dtype=torch.float64, device="cuda") for _ in s["kws"]]
        s["B"] = torch.zeros(nnz, dtype=torch.float64, device="cuda")
        return s
    m, _ = _mesh(c["nel"], 1)
    TL, EU = S.seeded_state(m.xyz, _phys(c, 1), seed)
    if kind == "host":
        s["TL"], s["EU"] = TL, EU
        s["b"], s["vals"] = np.zeros(asm.N), np.zeros(asm.nnz)
        return s
    s["TL"], s["EU"] = torch.from_numpy(TL).cuda(), torch.from_numpy(EU).cuda()
    s["b"] = torch.zeros(asm.N, dtype=torch.float64, device="cuda")
    s["vals"] = None
    if kind != "residual":
        s["vals"] = torch.zeros(asm.nnz, device="cuda",
                                dtype=torch.float32 if kind == "exact32" else torch.float64)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "mlp":
        s["net"].reset_optimizer()
        loss = s["net"].train(s["X"], s["Y"], s["case"]["iters"], 1e-3)
        return {"loss": np.float32(loss), "params": s["net"].get_params()}
    if kind == "factor":
        return s["lu"].factor(s["vals"]).solve(s["b"])
    if kind == "solve":
        return s["lu"].solve(s["b"])
    if kind == "batched":
        s["asm"].assemble(s["TL"], s["EU"], V.VEFEM_RESIDUAL | V.VEFEM_JAC_EXACT32 | V.VEFEM_ZERO_FIRST,
                          s["b"], s["vals"], on_device=True)
        return {"b": s["b"], "vals": s["vals"]}
    if kind == "stability":
        s["asm"].stability_assemble(s["TL"], s["kws"], V.VEFEM_ZERO_FIRST, s["A"], s["B"], on_device=True)
        return {"A": s["A"], "B": s["B"]}
    if kind == "host":
        b, vals = s["asm"].set_equations_bulk(s["TL"], s["EU"], "NRP", s["b"], s["vals"], zero_first=True,
                                              outlet_edges=True)
        return {"b": b, "vals": vals}
    flags = V.VEFEM_RESIDUAL | V.VEFEM_ZERO_FIRST | JACOBIAN[kind]
    s["asm"].assemble(s["TL"], s["EU"], flags, s["b"], s["vals"], on_device=True)
    return {"b": s["b"], "vals": s["vals"]} if kind != "residual" else {"b": s["b"]}


# ---------------------------------------------------------------- work

def work(case):
    """Bytes: inputs (state, coordinates, connectivity) read and outputs written
    once.  Operations per element: a residual is about 14,000 (T form) or
    20,000 (SQRT); a forward difference is 56 of them; an exact Jacobian is
    the residual, its derivative by 20 interpolants at 9 points and the
    contraction with test and trial functions, about 300,000; a stability
    operator the same for its four polynomial parts, about 1,500,000."""
    c, kind = case, case["kind"]
    if kind == "mlp":
        n = MLP_IN * MLP_WIDTH + (MLP_HIDDEN - 1) * MLP_WIDTH ** 2 + MLP_WIDTH * MLP_OUT
        return {"bytes": 4.0 * (2 * n + c["rows"] * (MLP_IN + MLP_OUT)), "flops": 6.0 * n * c["rows"] * c["iters"]}
    if kind == "batched":
        nels = [_mesh(n, 0)[0].nel for n, _ in _instances(c)]
    else:
        nels = [_mesh(c["nel"], _nex(c))[0].nel]
    nel = float(sum(nels))
    nodes, nnz = 4.0 * nel, 2360.0 * nel          # Q2 meshes: ~4 nodes, ~2,360 AIJ entries per element
    inputs = nodes * 8 * (6 + 2) + nel * 36
    if kind in ("factor", "solve"):
        # LU of a column-ordered sweep: fronts grow with the channel height
        flops, entries = 0.42e12 * (nel / 20000.0) ** 2, 0.6e9 * (nel / 20000.0) ** 1.5
        if kind == "solve":
            return {"bytes": 8.0 * entries, "flops": 2.0 * entries}
        return {"bytes": 8.0 * nnz + 8.0 * entries, "flops": flops}
    res = 14000.0 if c["form"] == "T" else 20000.0
    if kind == "stability":
        return {"bytes": inputs + (c["nk"] + 1) * 6425.0 * 8 * nel, "flops": 1.5e6 * nel}
    ops = {"residual": res, "fd64": 56 * res, "host": 56 * res}.get(kind, res + 3.0e5)
    value = {"residual": 0, "exact32": 4, "batched": 4}.get(kind, 8)
    return {"bytes": inputs + nodes * 6 * 8 + nnz * value, "flops": ops * nel}


# ---------------------------------------------------------------- exact values, plain torch FP64

def _tables(points):
    """Q2 basis (value, xi, eta, xi-xi, eta-eta, xi-eta) at points [n, 2]."""
    def l3(c):
        return (np.stack([-(1 - c) * c / 2, (1 - c) * (1 + c), (1 + c) * c / 2], -1),
                np.stack([-(1 - 2 * c) / 2, -2 * c, (1 + 2 * c) / 2], -1),
                np.stack([np.ones_like(c), -2 * np.ones_like(c), np.ones_like(c)], -1))

    ij = np.array([(0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1), (1, 1)])
    (a0, a1, a2), (b0, b1, b2) = l3(points[:, 0]), l3(points[:, 1])
    i, j = ij[:, 0], ij[:, 1]
    out = (a0[:, i] * b0[:, j], a1[:, i] * b0[:, j], a0[:, i] * b1[:, j], a2[:, i] * b0[:, j],
           a0[:, i] * b2[:, j], a1[:, i] * b1[:, j])
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in out]


_P1 = np.array([1.0e-8, math.sqrt(0.6), -math.sqrt(0.6)])
_W1 = np.array([8.0, 5.0, 5.0]) / 9.0


def _geometry(xy, tab, w):
    """Per element and point: phi, gradients, second derivatives, H^2, weight."""
    phi, c, e, cc, ee, ce = tab
    J = [[torch.einsum("gn,en->eg", d, xy[..., k]) for k in range(2)] for d in (c, e)]
    det = J[0][0] * J[1][1] - J[1][0] * J[0][1]
    cx, ex, cy, ey = J[1][1] / det, -J[0][1] / det, -J[1][0] / det, J[0][0] / det
    u = [v[..., None] for v in (cx, ex, cy, ey)]
    fx, fy = u[0] * c + u[1] * e, u[2] * c + u[3] * e
    lx = u[0] ** 2 * cc + u[1] ** 2 * ee + 2 * u[0] * u[1] * ce
    ly = u[2] ** 2 * cc + u[3] ** 2 * ee + 2 * u[2] * u[3] * ce
    H2 = 1.0 / (fx ** 2 + fy ** 2).sum(-1)
    return dict(phi=phi.expand_as(fx), fx=fx, fy=fy, lap=lx + ly, H2=H2, J=J,
                WET=(w * det.abs()) if w is not None else None)


def _interpolate(x, g):
    v = torch.einsum("egn,enf->egf", g["phi"], x)
    gx = torch.einsum("egn,enf->egf", g["fx"], x)
    gy = torch.einsum("egn,enf->egf", g["fy"], x)
    return v, gx, gy, torch.einsum("egn,enf->egf", g["lap"], x)


def _mm(A, B):
    return torch.einsum("...ij,...jk->...ik", A, B)


def _sym(a, b, d):
    return torch.stack([torch.stack([a, b], -1), torch.stack([b, d], -1)], -2)


def _point(q, p, Wi):
    """Stress, constitutive residual and momentum ingredients at the points."""
    v, gx, gy, lap = q
    b, ve = p.BvN, p.VeN
    omb = 1.0 - b
    GU = torch.stack([gx[..., :2], gy[..., :2]], -2)                # GU[a][i] = d_a u_i
    div = GU[..., 0, 0] + GU[..., 1, 1]
    I = torch.eye(2, dtype=v.dtype, device=v.device)
    Gt = GU - 0.5 * div[..., None, None] * I
    Gd = Gt + Gt.mT
    T, dTx, dTy = (_sym(a[..., 3], a[..., 4], a[..., 5]) for a in (v, gx, gy))
    adv = v[..., 0, None, None] * dTx + v[..., 1, None, None] * dTy
    tr = lambda A: A[..., 0, 0] + A[..., 1, 1]  # noqa: E731
    e2 = lambda s: s[..., None, None]  # noqa: E731
    if p.form == "T":
        f1, f3 = torch.ones_like(div), torch.zeros_like(div)
        if p.model == "GIESEKUS":
            f2, f3 = f1, ve * Wi / omb * torch.ones_like(div)
        else:
            a = ve * Wi * tr(T) / omb
            f2 = 1.0 + a if p.model == "L-PTT" else torch.exp(a)
        C = (Wi * (adv - _mm(Gt.mT, T) - _mm(T, Gt)) + e2(f3) * _mm(T, T) + e2(f2) * T - omb * Gd)
        sig, dsx, dsy = T, dTx, dTy
        ddT = ddS = ddC = (T * T).sum((-1, -2))
        fT = None
    else:
        c, dcx, dcy = _mm(T, T), _mm(dTx, T) + _mm(T, dTx), _mm(dTy, T) + _mm(T, dTy)
        if p.model == "GIESEKUS":
            fT = (1 - 2 * ve) * torch.ones_like(div)
            f1, f2, f3 = 1 - ve + 0 * fT, fT, ve + 0 * fT
        else:
            a = ve * (tr(c) - 2.0)
            fT = 1.0 + a if p.model == "L-PTT" else torch.exp(a)
            f1, f2, f3 = fT, fT, torch.zeros_like(fT)
        r = omb / Wi
        sig, dsx, dsy = r * (c - I), r * dcx, r * dcy
        S11, S12, S22 = T[..., 0, 0], T[..., 0, 1], T[..., 1, 1]
        w = (-S11 * GU[..., 0, 1] + S12 * (Gt[..., 0, 0] - Gt[..., 1, 1]) + S22 * GU[..., 1, 0]) / (S11 + S22)
        W = torch.stack([torch.stack([0 * w, w], -1), torch.stack([-w, 0 * w], -1)], -2)
        inv = _sym(S22, -S12, S11) / e2(S11 * S22 - S12 * S12)
        C = Wi * (adv - _mm(T, Gt) - _mm(W, T)) + 0.5 * (e2(f3) * _mm(T, c) + e2(f2) * T - e2(f1) * inv)
        ddT = (sig * sig).sum((-1, -2)) + r * r
        ddS, ddC = (T * T).sum((-1, -2)), (c * c).sum((-1, -2))
    divT = torch.stack([dsx[..., 0, 0] + dsy[..., 0, 1], dsx[..., 0, 1] + dsy[..., 1, 1]], -1)
    conv = p.ReN * torch.einsum("...a,...ai->...i", v[..., :2], GU)
    mom = conv - (-torch.stack([gx[..., 2], gy[..., 2]], -1) + divT + b * lap[..., :2])
    return dict(C=C, P=sig + b * Gd - e2(v[..., 2]) * I, p=v[..., 2], div=div, mom=mom, conv=conv, Gd=Gd, T=T,
                dTx=dTx, dTy=dTy, ddT=ddT, ddS=ddS, ddC=ddC, f2=f2, f3=f3, fT=fT, u=v[..., :2])


def _element_residual(x, g, p, Wi):
    """Weak-form element residuals [E, 9, 6] of states x [E, 9, 6]."""
    a = _point(_interpolate(x, g), p, Wi)
    phi, fx, fy, H2, n1 = g["phi"], g["fx"], g["fy"], g["H2"], lambda s: s[..., None]
    omb, r = 1.0 - p.BvN, (1.0 - p.BvN) / Wi
    du = n1(a["u"][..., 0]) * fx + n1(a["u"][..., 1]) * fy
    ts = du.abs().sum(-1)
    ddG = (a["Gd"] ** 2).sum((-1, -2))
    Ha = torch.sqrt(r * r + 0.5 * a["ddT"]) / torch.sqrt(1 + 0.5 * ddG)
    tm = 1 / torch.sqrt((p.ReN * ts) ** 2 + (p.BvN / H2) ** 2 + (Ha / H2) ** 2)
    tic = H2 / tm
    td = H2 / torch.sqrt(0.5 * a["ddS"] + (r * r if p.form == "T" else 0.0))
    C = a["C"]
    mag = torch.sqrt(0.5 * (C * C.mT).sum((-1, -2)))
    tc = 1 / torch.sqrt((Wi * ts) ** 2 + Wi ** 2 * 0.5 * ddG + a["f2"] ** 2
                        + a["f3"] ** 2 * 0.5 * a["ddC"] + (td * mag / H2) ** 2)
    grad = torch.stack([fx, fy], -1)                                     # [E, g, n, a]
    P, mom = a["P"], a["mom"]
    t = []
    for i in range(2):
        G = torch.zeros(fx.shape + (2, 2), dtype=x.dtype, device=x.device)
        G = G + grad[..., :, None] * torch.eye(2, dtype=x.dtype, device=x.device)[i]   # column i = grad phi
        if p.form == "T":
            L = -n1(tc)[..., None, None] * G
        else:
            T = a["T"][..., None, :, :]
            m = _mm(T, G)
            w = (-T[..., 0, 0] * G[..., 0, 1] + T[..., 0, 1] * (G[..., 0, 0] - G[..., 1, 1])
                 + T[..., 1, 1] * G[..., 1, 0]) / (T[..., 0, 0] + T[..., 1, 1])
            W = torch.stack([torch.stack([0 * w, w], -1), torch.stack([-w, 0 * w], -1)], -2)
            L = n1(tc)[..., None, None] * (-m - _mm(W, T)) * r
        lsce = (L * C[..., None, :, :].mT).sum((-1, -2))
        t.append(n1(a["conv"][..., i]) * phi + n1(P[..., 0, i]) * fx + n1(P[..., 1, i]) * fy
                 + n1(tm * p.ReN * mom[..., i]) * du + n1(tic * a["div"]) * grad[..., i] + lsce)
    t.append(n1(a["div"]) * phi + n1(tm) * (fx * n1(mom[..., 0]) + fy * n1(mom[..., 1])))
    M1, M2 = n1(mom[..., 0]), n1(mom[..., 1])
    lce = n1(tc) * (Wi * du + (0.0 if a["fT"] is None else 0.5 * n1(a["fT"]) * phi))
    for (j, k), ls in (((0, 0), -fx * M1), ((0, 1), -fy * M1 - fx * M2), ((1, 1), -fy * M2)):
        gd = n1(a["dTx"][..., j, k]) * fx + n1(a["dTy"][..., j, k]) * fy
        t.append(n1(C[..., j, k]) * (phi + lce) + n1(tm) * ls * (omb if p.form == "T" else Wi) + n1(td * mag) * gd)
    return torch.einsum("egnf,eg->enf", torch.stack(t, -1), g["WET"])


def _edge_residual(x, xy, side, p, Wi):
    """Open-boundary terms of one edge per element (x, xy of those elements)."""
    pts = np.stack([[_P1, [-1.0] * 3], [[1.0] * 3, _P1], [_P1, [1.0] * 3], [[-1.0] * 3, _P1]][side], -1)
    g = _geometry(xy, _tables(np.array(pts, dtype=float)), None)
    a = _point(_interpolate(x, g), p, Wi)
    d = g["J"][side % 2]
    n = torch.stack([d[1], -d[0]], -1) * (1.0 if side < 2 else -1.0)
    w = torch.from_numpy(_W1).cuda()
    n = n * w[:, None]                       # unit normal x weight x edge length
    q = torch.einsum("ega,egai->egi", n, a["P"]) + n * a["p"][..., None]
    out = torch.zeros_like(x)
    out[..., :2] = -torch.einsum("egi,egn->eni", q, g["phi"])
    return out


class _Mesh:
    """Device tables of a mesh: element nodes, coordinates, geometry, CSR keys."""

    def __init__(self, nel, nex, rp=None, ci=None, neq=6, keys=False):
        m, (rp6, ci6) = _mesh(nel, nex)
        rp, ci = (rp6, ci6) if rp is None else (rp, ci)
        self.N, self.neq, self.mesh = len(rp) - 1, neq, m
        self.en = torch.from_numpy(m.element_nodes().astype(np.int64)).cuda()
        self.xy = torch.from_numpy(m.xyz[:2].T.copy()).cuda()
        pts = np.array([(c, e) for c in _P1 for e in _P1])
        self.tab, self.w = _tables(pts), torch.from_numpy(np.outer(_W1, _W1).ravel()).cuda()
        if keys:
            rows = torch.repeat_interleave(torch.arange(self.N, device="cuda"), torch.from_numpy(np.diff(rp)).cuda())
            self.keys = rows * self.N + torch.from_numpy(ci.astype(np.int64)).cuda()

    def rows(self, e):
        return (self.en[e][:, :, None] * self.neq + torch.arange(self.neq, device="cuda")).reshape(len(e), -1)

    def geometry(self, e):
        return _geometry(self.xy[self.en[e]], self.tab, self.w)

    def add(self, vals, rows, cols, block):
        k = (rows[:, :, None] * self.N + cols[:, None, :]).reshape(-1)
        vals.index_add_(0, torch.searchsorted(self.keys, k), block.reshape(-1))


def _exact_assembly(nel, nex, phys, TL, EU, jac, edges):
    d = _Mesh(nel, nex, keys=jac)
    X = torch.from_numpy(TL.T.copy()).cuda()                             # [nodes, 6]
    eu = torch.tensor(float(EU[0]) if nex else 1.0, dtype=torch.float64, device="cuda")
    b = torch.zeros(d.N, dtype=torch.float64, device="cuda")
    vals = torch.zeros(len(d.keys), dtype=torch.float64, device="cuda") if jac else None
    for e in torch.arange(d.en.shape[0], device="cuda").split(1000):
        g, x, rows = d.geometry(e), X[d.en[e]].reshape(len(e), 54), d.rows(e)

        def f(x, eu):
            return _element_residual(x.reshape(-1, 9, 6), g, phys, phys.WiN * eu).reshape(-1, 54)

        b.index_add_(0, rows.reshape(-1), f(x, eu).reshape(-1))
        if jac:
            basis = torch.eye(54, dtype=torch.float64, device="cuda")
            K = torch.func.vmap(lambda v: torch.func.jvp(lambda y: f(y, eu), (x,), (v.expand_as(x),))[1])(basis)
            d.add(vals, rows, rows, K.permute(1, 2, 0))
            if nex:
                col = torch.func.jvp(lambda s: f(x, s), (eu,), (torch.ones_like(eu),))[1]
                d.add(vals, rows, torch.full((len(e), 1), d.N - 1, device="cuda"), col)
    if edges:
        ed = torch.from_numpy(d.mesh.outlet_edges.astype(np.int64)).cuda()
        for side in range(4):
            e = ed[ed[:, 1] == side + 1, 0]
            if len(e):
                r = _edge_residual(X[d.en[e]], d.xy[d.en[e]], side, phys, phys.WiN * eu)
                b.index_add_(0, d.rows(e).reshape(-1), r.reshape(-1))
    return b, vals


_JK = [(0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2)]       # stress unknowns of the 3-D perturbation


def _fields3(v, gx, gy):
    """Velocity gradient GU[a][i] and symmetric stress S, dS[...][c] from ten fields."""
    z = torch.zeros_like(v[..., 0])
    GU = torch.stack([gx[..., :3], gy[..., :3], torch.zeros_like(gx[..., :3])], -2)

    def sym(f):
        full = [[None] * 3 for _ in range(3)]
        for c, (j, k) in enumerate(_JK):
            full[j][k] = full[k][j] = f[..., 4 + c]
        return torch.stack([torch.stack(r, -1) for r in full], -2)

    return GU, sym(v), torch.stack([sym(gx), sym(gy), sym(gx) * 0], -1), z


def _stability_blocks(x, g, p):
    """Element matrices (B, A(0), A(1), A(-1)) as [E, 9, 10, 9, 10]."""
    Wi, b, omb, ve = p.WiN, p.BvN, 1 - p.BvN, p.VeN
    v, gx, gy, _ = _interpolate(x, g)
    GU, Sb, dS, _ = _fields3(v, gx, gy)
    U, H2 = v[..., :3], g["H2"]
    I = torch.eye(3, dtype=x.dtype, device=x.device)
    tr = lambda A: A.diagonal(dim1=-2, dim2=-1).sum(-1)  # noqa: E731
    e2 = lambda s: s[..., None, None]  # noqa: E731
    Gt = GU - e2(tr(GU)) * I / 3
    Gdt = Gt + Gt.mT
    one, zero = torch.ones_like(H2), torch.zeros_like(H2)
    if p.model == "GIESEKUS":
        f1, f2, fT = one, ve * Wi / omb * one, one
    else:
        arg = ve * Wi * tr(Sb) / omb
        fT = 1 + arg if p.model == "L-PTT" else torch.exp(arg)
        f1, f2 = fT, zero
    CE = (Wi * (torch.einsum("...k,...ijk->...ij", U, dS) - _mm(Gt.mT, Sb) - _mm(Sb, Gt)) + e2(f2) * _mm(Sb, Sb)
          + e2(f1) * Sb - omb * Gdt)
    dd = lambda A, B: (A * B.mT).sum((-1, -2))  # noqa: E731
    ts = (U[..., 0, None] * g["fx"] + U[..., 1, None] * g["fy"]).abs().sum(-1)
    r = omb / Wi
    Ha = torch.sqrt(r * r + 0.5 * dd(Sb, Sb)) / torch.sqrt(1 + 0.5 * dd(Gdt, Gdt))
    tm = 1 / torch.sqrt((p.ReN * ts) ** 2 + (b / H2) ** 2 + (Ha / H2) ** 2)
    td = H2 / torch.sqrt(0.5 * dd(Sb, Sb) + r * r)
    mag = torch.sqrt(0.5 * dd(CE, CE))
    tc = 1 / torch.sqrt((Wi * ts) ** 2 + Wi ** 2 * 0.5 * dd(Gdt, Gdt) + f1 ** 2 + f2 ** 2 * 0.5 * dd(Sb, Sb)
                        + (td * mag / H2) ** 2)
    # unit perturbations: field f, component s (value, d/dx, d/dy, Laplacian of a velocity)
    unit = torch.zeros(4, 10, 4, 10, dtype=x.dtype, device=x.device)     # [component, f, s, field]
    for f in range(10):
        for s in range(4 if f < 3 else 3):
            unit[s, f, s, f] = 1.0
    q = [u.reshape(40, 10) for u in unit]
    u, P, lap = q[0][:, :3], q[0][:, 3], q[3][:, :3]
    dP = torch.stack([q[1][:, 3], q[2][:, 3], 0 * P], -1)
    dGU, s, ds, _ = _fields3(q[0], q[1], q[2])
    test = torch.stack([g["phi"], g["fx"], g["fy"]], -1) * g["WET"][..., None, None]
    chi = torch.stack([g["phi"], g["fx"], g["fy"], g["lap"]], -1)
    n1 = lambda t: t[..., None]  # noqa: E731  (a base scalar against the 40 unit perturbations)
    bt = lambda t: t.unsqueeze(2)  # noqa: E731
    out = []
    for K in (0.0, 1.0, -1.0):
        G, dp, dT, L = dGU.clone(), dP.clone(), ds.clone(), lap - K * K * u
        G[:, 2, 0], G[:, 2, 1], G[:, 2, 2] = -K * u[:, 0], -K * u[:, 1], K * u[:, 2]
        dp[:, 2] = -K * P
        dT[..., 2] = -K * s
        for j in (0, 1):
            dT[:, j, 2, 2] = dT[:, 2, j, 2] = K * s[:, j, 2]
        Gd = G + G.mT
        df = 0 * n1(fT) * tr(s)
        if p.model != "GIESEKUS":
            df = ve * Wi / omb * tr(s) * (n1(fT) if p.model == "e-PTT" else n1(one))
        Pt = s + b * Gd - P[:, None, None] * I
        S_, GU_ = bt(Sb), bt(GU)
        ucd = (torch.einsum("egk,qijk->egqij", U, dT) + torch.einsum("qk,egijk->egqij", u, dS)
               - _mm(GU_.mT, s) - _mm(G.mT, S_) - _mm(S_, G) - _mm(s, GU_))
        ce = (Wi * ucd + e2(n1(f2)) * (_mm(S_, s) + _mm(s, S_)) + e2(df) * S_ + e2(n1(f1)) * s - omb * Gd)
        conv = torch.einsum("egk,qki->egqi", U, G) + torch.einsum("qk,egki->egqi", u, GU)
        mom = p.ReN * conv - (-dp + torch.einsum("qjij->qi", dT.transpose(1, 2)) + b * L)
        mt = p.ReN * u + 0 * mom
        ct = Wi * s + 0 * ce
        div = tr(G) + 0 * n1(one)
        magd = dd(bt(CE), ce) / n1(2 * mag + 1e-12)
        ca = torch.zeros(mom.shape[:3] + (10, 3), dtype=x.dtype, device=x.device)
        cb = torch.zeros_like(ca)
        for i in range(3):
            ca[..., i, 0] = p.ReN * conv[..., i] - (-K if i == 2 else K) * Pt[:, i, 2]
            cb[..., i, 0] = mt[..., i]
            for c in range(2):
                up = n1(tm * p.ReN * U[..., c])
                ca[..., i, 1 + c] = (Pt[:, i, c] + up * mom[..., i] + (n1(H2 / tm) * div if i == c else 0)
                                     - n1(tc) * ce[..., c, i])
                cb[..., i, 1 + c] = up * mt[..., i] - n1(tc) * ct[..., c, i]
        ca[..., 3, 0] = div
        for c in range(2):
            ca[..., 3, 1 + c], cb[..., 3, 1 + c] = n1(tm) * mom[..., c], n1(tm) * mt[..., c]
        for e, (j, k) in enumerate(_JK):
            ca[..., 4 + e, 0], cb[..., 4 + e, 0] = ce[..., j, k], ct[..., j, k]
            for c in range(2):
                pick = lambda m: -((m[..., j] if k == c else 0 * m[..., j])  # noqa: E731
                                   + (m[..., k] if j == c and j != k else 0 * m[..., j]))
                up = n1(tc * Wi * U[..., c])
                ca[..., 4 + e, 1 + c] = (n1(tm) * omb * pick(mom) + up * ce[..., j, k]
                                         + n1(td * dS[..., j, k, c]) * magd)
                cb[..., 4 + e, 1 + c] = n1(tm) * omb * pick(mt) + up * ct[..., j, k]
        for coef, wanted in ((-cb, K == 0.0), (ca, True)):
            if wanted:
                D = coef.reshape(coef.shape[:2] + (10, 4, 10, 3))
                T1 = torch.einsum("egnk,egfsqk->egnqfs", test, D)
                out.append(torch.einsum("egnqfs,egms->enqmf", T1, chi))
    return out


def _exact_stability(c, seed):
    p = _phys(c, 0)
    asm = _assembler(_key(c))
    rp, ci = asm.stability_pattern()         # the layout of the outputs
    d = _Mesh(c["nel"], 0, rp, ci, neq=10, keys=True)
    X = torch.from_numpy(_stability_base(c, seed).T.copy()).cuda()
    M4 = [torch.zeros(len(ci), dtype=torch.float64, device="cuda") for _ in range(4)]
    for e in torch.arange(d.en.shape[0], device="cuda").split(250):
        rows = d.rows(e)
        k = torch.searchsorted(d.keys, (rows[:, :, None] * d.N + rows[:, None, :]).reshape(-1))
        for m, blk in zip(M4, _stability_blocks(X[d.en[e]], d.geometry(e), p)):
            m.index_add_(0, k, blk.reshape(-1))
    B, A0, Ap, An = M4
    A = [A0 + K * ((Ap - An) / 2) + K * K * ((Ap + An) / 2 - A0) for K in np.linspace(0.0, 4.0, c["nk"])]
    return {"A": A, "B": B}


def _exact_mlp(c, seed):
    """Adam on FP64 masters whose BF16 rounding enters the products."""
    net = V.MLP(MLP_IN, MLP_OUT, width=MLP_WIDTH, hidden=MLP_HIDDEN, seed=seed)
    flat = torch.from_numpy(net.get_params()).double().cuda()            # the seeded initial weights
    net.close()
    dims = [MLP_IN] + [MLP_WIDTH] * MLP_HIDDEN + [MLP_OUT]
    X, Y = (torch.from_numpy(a).double().cuda() for a in _mlp_data(c, seed))
    m, v, loss = torch.zeros_like(flat), torch.zeros_like(flat), 0.0
    for it in range(1, c["iters"] + 1):
        flat = flat.detach().requires_grad_(True)
        h, o = X, 0
        for i, (a, b) in enumerate(zip(dims[:-1], dims[1:])):
            W, bias = flat[o:o + a * b].reshape(b, a), flat[o + a * b:o + a * b + b]
            o += a * b + b
            W = W + (W.float().bfloat16().double() - W).detach()
            h = h @ W.T + bias
            h = torch.nn.functional.gelu(h) if i < MLP_HIDDEN else h
        loss = ((h - Y) ** 2).mean()
        g, = torch.autograd.grad(loss, flat)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        flat = flat.detach() - 1e-3 * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
    # the loss of an overfitted training set is round-off of the weights: no exact form
    return {"loss": None, "params": flat.cpu().numpy()}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "mlp":
        return _exact_mlp(c, seed)
    if kind in ("factor", "solve"):
        return torch.from_numpy(_x_true(c, seed))
    if kind == "stability":
        return _exact_stability(c, seed)
    if kind == "batched":
        got = []
        for i, (n, p) in enumerate(_instances(c)):
            TL, _ = S.seeded_state(_mesh(n, 0)[0].xyz, p, seed + 100 * i)
            got.append(_exact_assembly(n, 0, p, TL, None, True, False))
        return {"b": [b for b, _ in got], "vals": [v for _, v in got]}
    m, _ = _mesh(c["nel"], 1)
    p = _phys(c, 1)
    TL, EU = S.seeded_state(m.xyz, p, seed)
    # a forward difference is defined by its own rounding: its values have no other exact form
    b, vals = _exact_assembly(c["nel"], 1, p, TL, EU, kind in ("exact64", "exact32"), kind == "host")
    return {"b": b, "vals": vals} if kind != "residual" else {"b": b}
