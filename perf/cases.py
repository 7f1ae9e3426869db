"""Performance cases of the triangular-dislocation library: the calls that a
user of the framework makes, over the sizes they make them at.

    listed()   the named cases          draw(rng)   one more of the same ranges
    prepare()  inputs in hand           run()       one pass through the public API
    work()     bytes / flops needed     tolerance() agreement of two correct results
    exact()    the outputs in 64 bits from plain torch, by other formulas

Kinds of case:
    inf       influence fields of every triangle at every point (cad_td_inf_dev)
    sum       summed strain / displacement at the points (cad_td_sum_eval_dev)
    sum_host  the same through TD(..., Strains, Disps) with numpy arrays
    slip      system matrix and dense solve on the device (cad_assemble_dev, cad_solve_dev)
    slip_host SlipCalculator3D with numpy arrays, the system matrix returned as well
    learned   cad_slip_calculator with the learned-preconditioner GMRES, host arrays
    friction  SlipCalculator3D with frictional boundary conditions, host arrays
    batch     many independent cracks in one call (cad_slip_calculator_batched_dev)

`exact` evaluates the dislocations as line integrals along the triangle sides
(de Wit 1960; Hirth and Lothe, chapter 4) with the free-surface displacements
of Comninou and Dundurs (1975) as Nikkhoo and Walter (2015) print them, and
takes strains by complex-step differentiation.
"""
import functools
import math

import numpy as np
import torch

import cutanddisplacejulia_b200 as cad
from cutanddisplacejulia_b200 import _lib, precond, workloads

NU, G = 0.25, 1.0
LAM = 2.0 * G * NU / (1.0 - 2.0 * NU)
TOL = 1e-10   # relative residual of the iterative solves


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a quick look at a few triangles from an interactive session: launch and call latency
        dict(name="sum_host_fs_16x16", kind="sum_host", hs=0, mesh="fault", ntri=16, nobs=16, strain=1, disp=1),
        # the forward evaluation of the README: a 100-triangle fault seen from a 50 x 50 grid
        dict(name="inf_fs_100x2500", kind="inf", hs=0, mesh="fault", ntri=100, nobs=2500, strain=1, disp=1),
        # half-space strain influence between the elements of a mid-size mesh and a ragged point set
        dict(name="inf_hs_900x1111", kind="inf", hs=1, mesh="dip", ntri=900, nobs=1111, strain=1, disp=0),
        # strain around a crack on a fine grid of points, full space
        dict(name="sum_fs_2013x20000", kind="sum", hs=0, mesh="penny", ntri=2013, nobs=20000, strain=1, disp=0),
        # surface strain and displacement of a slipping fault, half space (the largest forward evaluation)
        dict(name="sum_hs_10000x10000", kind="sum", hs=1, mesh="dip", ntri=10000, nobs=10000, strain=1, disp=1),
        # the usual interactive slip solve: numpy in, slips and system matrix out
        dict(name="slip_host_fs_500", kind="slip_host", hs=0, mesh="penny", ntri=500),
        # the pressurised penny crack, FP64 assembly and LU
        dict(name="slip_fs_2013", kind="slip", hs=0, mesh="penny", ntri=2013, solver="lu64", assembly="fp64"),
        # the largest dense solve: dipping half-space crack, 30 000 unknowns, FP64 LU
        dict(name="slip_hs_10000", kind="slip", hs=1, mesh="dip", ntri=10000, solver="lu64", assembly="fp64"),
        # FP32 far field, FP32 LU and FP64 refinement on a mid-size half-space crack
        dict(name="slip_mixed_hs_3000", kind="slip", hs=1, mesh="dip", ntri=3000, solver="mixed", assembly="mixed"),
        # the same large crack by the learned-preconditioner GMRES, end to end from host arrays
        dict(name="learned_hs_10000", kind="learned", hs=1, mesh="dip", ntri=10000),
        # frictional slip of a closed crack under shear
        dict(name="friction_fs_496", kind="friction", hs=0, mesh="penny", ntri=496),
        # a population of uneven cracks in one call
        dict(name="batch_fs_64", kind="batch", hs=0, mesh="cracks", ntri=64, nmin=200, nmax=1500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["inf", "inf", "sum", "sum", "sum_host", "slip_host", "slip", "slip", "learned", "friction",
                       "batch"])
    hs = rng.randrange(2)
    mesh = "dip" if hs else rng.choice(["penny", "fault", "dip"])
    if kind in ("inf", "sum", "sum_host"):
        strain, disp = rng.choice([(1, 0), (0, 1), (1, 1)])
        if kind == "inf":       # outputs of M x N: bounded by memory a user would hold
            ntri, nobs = _log(rng, 2, 2500), _log(rng, 4, 10000)
            nobs = min(nobs, 6000000 // ntri)
        elif kind == "sum":
            ntri, nobs = _log(rng, 10, 10000), _log(rng, 100, 20000)
            nobs = min(nobs, 100000000 // ntri)
        else:
            ntri, nobs = _log(rng, 2, 500), _log(rng, 4, 2500)
        return dict(kind=kind, hs=hs, mesh=mesh, ntri=ntri, nobs=nobs, strain=strain, disp=disp)
    if kind == "slip":
        solver = rng.choice(["lu64", "lu64", "mixed", "gmres_block_jacobi"])
        assembly = "mixed" if solver == "mixed" else "fp64"
        return dict(kind=kind, hs=hs, mesh="dip" if hs else "penny", ntri=_log(rng, 40, 6000), solver=solver,
                    assembly=assembly)
    if kind == "slip_host":
        return dict(kind=kind, hs=hs, mesh="dip" if hs else "penny", ntri=_log(rng, 20, 800))
    if kind == "learned":
        return dict(kind=kind, hs=1, mesh="dip", ntri=_log(rng, 1000, 9000))
    if kind == "friction":
        return dict(kind=kind, hs=0, mesh="penny", ntri=_log(rng, 60, 900))
    return dict(kind="batch", hs=0, mesh="cracks", ntri=rng.randrange(2, 64), nmin=100, nmax=_log(rng, 200, 1500))


# ------------------------------------------------------------------ inputs
def _mesh(case, seed):
    """P1, P2, P3 of a seeded mesh of about `ntri` triangles (the number of
    triangles depends on the case alone)."""
    n = case["ntri"]
    if case["mesh"] == "penny":
        a, b = np.random.default_rng(seed + 1000).uniform(0.9, 1.1, 2)
        return workloads.ellipse_crack(seed=0, a=a, b=b, ntri=n)
    if case["mesh"] == "dip":
        rng = np.random.default_rng(seed + 1000)
        P = workloads.dipping_rect(seed=seed, ntri=max(n, 2), dip=60.0 + rng.uniform(-5, 5), top_depth=2.0)
        return P
    nz = max(1, int(round(math.sqrt(n / 4))))
    f = workloads.fault_grid(seed=seed, nx=max(1, n // (2 * nz)), nz=nz, ngrid=2)
    bow = 0.02 * np.cos(0.9 * np.array([f["P1"], f["P2"], f["P3"]])[..., 0] + seed)
    P = [p.copy() for p in (f["P1"], f["P2"], f["P3"])]
    for p, b in zip(P, bow):
        p[:, 1] += b
    return tuple(P)


def _points(case, seed):
    """Observation points about the mesh: a plane grid's worth, jittered; at the
    free surface for displacement and strain sums of large half-space cases."""
    m = case["nobs"]
    rng = np.random.default_rng(seed + 7)
    w = int(math.ceil(math.sqrt(m)))
    g = np.linspace(-4.0, 4.0, max(w, 2))
    X, Y = np.meshgrid(g, g)
    X = X.ravel()[:m] + rng.uniform(-0.01, 0.01, m)
    Y = Y.ravel()[:m] + rng.uniform(-0.01, 0.01, m)
    if case["kind"] == "sum" and case["hs"]:
        return X, Y, np.zeros(m)
    return X, Y + 0.3, rng.uniform(-1.9, -0.1, m)


def _slips(P, seed):
    mid = (P[0] + P[1] + P[2]) / 3.0
    rng = np.random.default_rng(seed + 3)
    s = np.stack([1e-3 * np.cos(0.7 * mid[:, 0] + k) * np.cos(0.9 * mid[:, 2] - k) for k in range(3)])
    return s + rng.uniform(-1e-4, 1e-4, s.shape)   # Dss, Dds, Dn


def _tractions(nrm, seed):
    """(Tn, Tss, Tds) of a seeded remote stress."""
    s = np.random.default_rng(seed + 5).uniform(-1e-3, 1e-3, 6)
    Tn, Tds, Tss = cad.CalculateNormalAndShearTractions3D(*s, nrm)
    return Tn, Tss, Tds


def _friction_loads(mid, seed):
    n = len(mid)
    k = 1.0 + 0.1 * np.random.default_rng(seed + 9).uniform(-1, 1, 3)
    r = np.hypot(mid[:, 0], mid[:, 1])
    # closed but for a patch that fluid pressure opens, sheared obliquely
    Tn = -2e-3 * k[0] + 3e-3 * np.exp(-8.0 * ((mid[:, 0] - 0.4) ** 2 + mid[:, 1] ** 2))
    return (Tn, np.full(n, 1e-3 * k[1]), np.full(n, 6e-4 * k[2])), np.full(n, 0.3), 2e-4 * r


def _cracks(case, seed):
    cracks, stresses = workloads.crack_batch(seed=0, count=case["ntri"], n_range=(case["nmin"], case["nmax"]))
    rng = np.random.default_rng(seed)
    cracks = [tuple(p * k for p in P) for P, k in zip(cracks, rng.uniform(0.9, 1.1, (len(cracks), 3)))]
    return cracks, rng.uniform(-1e-3, 1e-3, np.shape(stresses))


@functools.lru_cache(maxsize=None)
def _network():
    """A preconditioner network trained once, as a program that solves many
    cracks keeps it."""
    ts = precond.training_set(precond.training_meshes(seed=0, count=8, n_range=(500, 1200)))
    net = precond.Network(seed=0)
    net.train(ts, steps=1500)
    return net


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=np.float64).ravel(order="F"))).cuda()


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=np.float64).ravel(order="F"))).pin_memory()


def prepare(case, seed):
    kind = case["kind"]
    L, ctx = cad.load(), cad.context()
    st = dict(case=case, L=L, ctx=ctx, stream=torch.cuda.ExternalStream(L.cad_get_stream(ctx)))
    if kind == "batch":
        cracks, stresses = _cracks(case, seed)
        parts = {k: [] for k in ("P1", "P2", "P3", "nrm", "mid", "T")}
        offs = [0]
        for P, s in zip(cracks, stresses):
            nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
            Tn, Tds, Tss = cad.CalculateNormalAndShearTractions3D(*s, nrm)
            for k, a in zip(parts, (*P, nrm, mid, np.concatenate([Tn, Tss, Tds]))):
                parts[k].append(np.asfortranarray(a).ravel(order="F"))
            offs.append(offs[-1] + len(nrm))
        st.update({k: _dev(np.concatenate(v)) for k, v in parts.items()})
        st.update(offs=np.asarray(offs, dtype=np.int64), rel=np.zeros(len(cracks)),
                  D=torch.zeros(3 * offs[-1], dtype=torch.float64, device="cuda"))
        return st
    P = _mesh(case, seed)
    n = st["n"] = len(P[0])
    if kind in ("inf", "sum", "sum_host"):
        XYZ, sl = _points(case, seed), _slips(P, seed)
        m = st["m"] = len(XYZ[0])
        if kind == "sum_host":
            st.update(P=P, XYZ=XYZ, sl=sl)
            return st
        nf = n if kind == "inf" else 1
        k = 3 if kind == "inf" else 1
        st.update(P=[_dev(p) for p in P], XYZ=[_dev(a) for a in XYZ], sl=[_dev(s) for s in sl])
        st["E"] = torch.zeros(6 * k, nf, m, dtype=torch.float64, device="cuda") if case["strain"] else None
        st["U"] = torch.zeros(3 * k, nf, m, dtype=torch.float64, device="cuda") if case["disp"] else None
        return st
    nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
    if kind == "friction":
        (Tn, Tss, Tds), mu, Sf = _friction_loads(mid, seed)
        z = np.zeros(n)
        bc = cad.MixedBoundaryConditions(cad.Stresses(z, z, z, z, z, z), cad.Tractions(Tn, Tss, Tds))
        st.update(P=P, nrm=nrm, mid=mid,
                  bc=cad.MixedBoundaryConditionsFriction(bc, cad.FrictionParameters(mu, Sf)))
        return st
    T = _tractions(nrm, seed)
    if kind == "slip_host":
        st.update(P=P, nrm=nrm, mid=mid, bc=cad.Tractions(*T))
        return st
    if kind == "learned":
        st.update(net=_network(), geo=[_pinned(a) for a in (*P, mid, nrm)], T=[_pinned(t) for t in T],
                  D=[_pinned(np.zeros(n)) for _ in range(3)])
        return st
    st.update(P=[_dev(p) for p in P], nrm=_dev(nrm), mid=_dev(mid), b=_dev(np.concatenate(T)),
              x=torch.zeros(3 * n, dtype=torch.float64, device="cuda"),
              A=torch.zeros(9 * n * n, dtype=torch.float64, device="cuda"))
    return st


# --------------------------------------------------------------------- run
def _p(t):
    return None if t is None else t.data_ptr()


def run(st):
    c, L, ctx = st["case"], st["L"], st["ctx"]
    kind, hs = c["kind"], c["hs"]
    if kind in ("inf", "sum"):
        call = L.cad_td_inf_dev if kind == "inf" else L.cad_td_sum_eval_dev
        _lib.check(call(ctx, *map(_p, st["XYZ"]), st["m"], *map(_p, st["P"]), st["n"], *map(_p, st["sl"]), NU,
                        c["disp"], c["strain"], hs, _p(st["E"]), _p(st["U"])), ctx)
        return {"E": st["E"], "U": st["U"]}
    if kind == "sum_host":
        S, U = cad.TD(*st["XYZ"], *st["P"], *st["sl"], NU, G, c["disp"], c["strain"], hs, cad.Strains(), cad.Disps())
        return {"E": list(S) if c["strain"] else None, "U": list(U) if c["disp"] else None}
    if kind == "slip_host":
        D = cad.SlipCalculator3D(*st["P"], NU, G, LAM, st["mid"], st["nrm"], hs, st["bc"], None)
        return {"Dn": D[0], "Dss": D[1], "Dds": D[2], "A": D[3]}
    if kind == "friction":
        return np.concatenate(cad.SlipCalculator3D(*st["P"], NU, G, LAM, st["mid"], st["nrm"], hs, st["bc"], None))
    if kind == "learned":
        st["net"]._load()
        P1, P2, P3, mid, nrm = st["geo"]
        with _lib.solver_mode(ctx, "gmres_learned", TOL, 2000):
            _lib.check(L.cad_slip_calculator(ctx, _p(P1), _p(P2), _p(P3), st["n"], NU, G, LAM, _p(mid), _p(nrm), hs,
                                             *map(_p, st["T"]), *map(_p, st["D"]), None, None), ctx)
        return st["D"]
    if kind == "batch":
        with _lib.solver_mode(ctx, "mixed", TOL, 400), _lib.assembly_mode(ctx, "mixed"):
            _lib.check(L.cad_slip_calculator_batched_dev(ctx, len(st["rel"]), st["offs"].ctypes.data, _p(st["P1"]),
                                                         _p(st["P2"]), _p(st["P3"]), _p(st["nrm"]), _p(st["mid"]), NU,
                                                         G, LAM, hs, _p(st["T"]), _p(st["D"]),
                                                         st["rel"].ctypes.data), ctx)
        return st["D"]
    n = st["n"]
    with torch.cuda.stream(st["stream"]), _lib.solver_mode(ctx, c["solver"], TOL, 2000), \
            _lib.assembly_mode(ctx, c["assembly"]):
        _lib.check(L.cad_assemble_dev(ctx, _p(st["nrm"]), _p(st["mid"]), *map(_p, st["P"]), n, NU, G, LAM, hs,
                                      _p(st["A"]), 3 * n), ctx)
        st["x"].copy_(st["b"])
        _lib.check(L.cad_solve_dev(ctx, 3 * n, _p(st["A"]), 3 * n, _p(st["x"]), 3 * n, 1), ctx)
    return st["x"]


# -------------------------------------------------------- work, tolerances
def work(case):
    """Inputs and outputs once; per pair, what the line-integral form of the
    dislocation needs at least (three sides, three modes), and per dense solve
    (2/3) n^3 (LU) or one FP32 pass over A per iteration (GMRES)."""
    n, hs = case["ntri"], case["hs"]
    pair = 300.0 * (2 if hs else 1)
    if case["kind"] in ("inf", "sum", "sum_host"):
        m = case["nobs"]
        out = 6.0 * case["strain"] + 3.0 * case["disp"]
        nout = 3 * out * n * m if case["kind"] == "inf" else out * m
        return {"bytes": 8.0 * (12 * n + 3 * m + nout), "flops": pair * n * m}
    if case["kind"] == "batch":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"] + 1e-9)
        k = [case["ntri"] * (math.exp(p * hi) - math.exp(p * lo)) / (p * (hi - lo)) for p in (1, 2, 3)]
        return {"bytes": 8.0 * 21 * k[0], "flops": pair * k[1] + 18.0 * k[2]}
    if case["kind"] == "learned" or case.get("solver") == "gmres_block_jacobi":
        its = 54.0
        return {"bytes": 8.0 * 21 * n + its * 36.0 * n * n, "flops": pair * n * n + its * 18.0 * n * n}
    out = 8.0 * 9 * n * n if case["kind"] == "slip_host" else 0.0
    factorisations = 6.0 if case["kind"] == "friction" else 1.0
    return {"bytes": 8.0 * 21 * n + out, "flops": pair * n * n + factorisations * 18.0 * n ** 3}


def tolerance(case):
    """About four times the largest distance from exact() seen over the ranges,
    rounded up: 1.6e-11 for FP64 fields and sums, 1.1e-12 after an FP64 LU."""
    if case["kind"] == "friction":
        return {"rel": 1e-8}                 # Newton to max|Phi| <= 1e-10 max|q|
    if case["kind"] == "batch" or case.get("assembly") == "mixed":
        return {"rel": 2e-5, "max": 2e-3}    # FP32 far field of the matrix
    if case["kind"] == "learned" or case.get("solver") == "gmres_block_jacobi":
        return {"rel": 2e-9}                 # GMRES to relative residual 1e-10
    return {"rel": 1e-10}


# ------------------------------------------------------- reference in 64 bits
def _loop(x, V, nu):
    """Displacement of a unit Burgers vector along each axis on the triangle V
    (3 vertices of 3 components, each [1, n]) at x (3 components [m, 1]):
    U[j][c]."""
    U = [[0.0] * 3 for _ in range(3)]
    r = [[V[k][i] - x[i] for i in range(3)] for k in range(3)]
    R = [torch.sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]) for a in r]

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    def cross(a, b):
        return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]

    one = dot(r[0], cross(r[1], r[2]))
    two = R[0] * R[1] * R[2] + dot(r[0], r[1]) * R[2] + dot(r[0], r[2]) * R[1] + dot(r[1], r[2]) * R[0]
    # solid angle / 2, its imaginary (derivative) part from d atan(one / two)
    half = torch.complex(torch.atan2(one.real, two.real),
                         (one.imag * two.real - two.imag * one.real) / (one.real ** 2 + two.real ** 2))
    for j in range(3):
        U[j][j] = half * (-2.0 / (4.0 * math.pi))
    k1, k2 = 1.0 / (4.0 * math.pi), -1.0 / (8.0 * math.pi * (1.0 - nu))
    for k in range(3):
        A, B = k, (k + 1) % 3
        t = [V[B][i] - V[A][i] for i in range(3)]
        ln = torch.sqrt(dot(t, t))
        t = [a / ln for a in t]
        sA = dot(r[A], t)
        sB = sA + ln
        rho = [r[A][i] - sA * t[i] for i in range(3)]
        rho2 = dot(rho, rho)
        fwd = (sA + sB).real >= 0
        a, b = torch.where(fwd, sA, -sB), torch.where(fwd, sB, -sA)
        Ra, Rb = torch.where(fwd, R[A], R[B]), torch.where(fwd, R[B], R[A])

        def plus(s, Rs):   # Rs + s without cancellation
            return torch.where(s.real >= 0, Rs + s, rho2 / (Rs - s))
        pa, pb = plus(a, Ra), plus(b, Rb)
        Lg = torch.log(pb / pa)
        K = 1.0 / (Ra * pa) - 1.0 / (Rb * pb)          # int dl / R^3
        T = 1.0 / R[A] - 1.0 / R[B]                     # int s dl / R^3
        w = cross(rho, t)
        g = [rho[i] * K + t[i] * T for i in range(3)]   # gradient of int dl / R
        for j in range(3):
            e = [1.0 if i == j else 0.0 for i in range(3)]
            bt = cross(e, t)
            for c in range(3):
                U[j][c] = U[j][c] + k1 * bt[c] * Lg + k2 * (bt[c] * Lg + w[j] * g[c])
    return U


def _free_surface(x, A, B, nu):
    """Free-surface displacement of side A -> B for a unit Burgers vector along
    each axis: U[j][c] (zero for near-vertical sides, as the method drops them)."""
    S = [B[i] - A[i] for i in range(3)]
    hn = torch.sqrt(S[0] ** 2 + S[1] ** 2)
    beta = torch.acos((-S[2] / torch.sqrt(S[0] ** 2 + S[1] ** 2 + S[2] ** 2)).real)
    keep = torch.abs(1.0 / torch.tan(beta)) <= 5e3
    hs = torch.where(keep, hn.real, torch.ones_like(hn.real))
    a, b = S[0] / hs, S[1] / hs
    dX = [x[i] - A[i] for i in range(3)]
    yA = [a * dX[0] + b * dX[1], b * dX[0] - a * dX[1], -dX[2]]
    yS = [a * S[0] + b * S[1], b * S[0] - a * S[1], -S[2]]
    be = torch.where((beta * yA[0].real) >= 0, beta - math.pi, beta.expand_as(yA[0].real))
    be = torch.where(keep.expand_as(be), be, torch.ones_like(be))
    D = [[0.0] * 3 for _ in range(3)]   # D[g][d]: ADCS component d, slip g
    for sgn, P, y in ((-1.0, A, yA), (1.0, B, [yA[i] - yS[i] for i in range(3)])):
        v = _angular_free_surface(y, be, -P[2].real, nu)
        for g in range(3):
            for d in range(3):
                D[g][d] = D[g][d] + sgn * v[g][d]
    rot = [[a, b, 0.0], [b, -a, 0.0], [0.0, 0.0, -1.0]]   # symmetric: ADCS <-> EFCS
    U = [[0.0] * 3 for _ in range(3)]
    for j in range(3):
        u = [sum(rot[g][j] * D[g][d] for g in range(3)) for d in range(3)]
        for c in range(3):
            U[j][c] = keep * sum(rot[c][d] * u[d] for d in range(3)) / (4.0 * math.pi * (1.0 - nu))
    return U


def _atan(u):
    return torch.complex(torch.atan(u.real), u.imag / (1.0 + u.real ** 2))


def _angular_free_surface(y, beta, a, nu):
    """Harmonic-image displacement of an angular dislocation below a free
    surface: [slip g][component d], without 1 / (4 pi (1 - nu))."""
    y1, y2 = y[0], y[1]
    s, c = torch.sin(beta), torch.cos(beta)
    ct = c / s
    z = y[2] + a                 # depth of the point
    q = z + a                    # its distance from the image plane's origin
    r = torch.sqrt(y1 * y1 + y2 * y2 + q * q)
    z1 = y1 * c + q * s
    p, w = r + q, r - y1 * s + q * c
    F = 2.0 * _atan(-y2 / (-p / torch.tan(beta / 2.0) + y1))
    N1, N2 = 1.0 - 2.0 * nu, 2.0 * (1.0 - nu)
    h, k = r * c + q, r * s - y1
    ca, na, ma, ra = c + a / r, nu + a / r, 2.0 * nu + a / r, 1.0 + a / (r * c)
    lp, lw = torch.log(p), torch.log(w)
    r2, r3, y2s = r * r, r * r * r, y2 * y2
    b1 = [-N2 * N1 * F * ct ** 2 + N1 * y2 / p * ((N1 - a / r) * ct - y1 / p * na) + N1 * y2 * c * ct / w * ca
          + a * y2 * z * ct / r3 + y2 * z / (r * p) * (-N1 * ct + y1 / p * ma + a * y1 / r2)
          + y2 * z / (r * w) * (c / w * (h * (N1 * c - a / r) * ct + N2 * k * c) - a * q * c * ct / r2),
          N1 * ((N2 * ct ** 2 - nu) * lp - (N2 * ct ** 2 + N1) * c * lw)
          - N1 / p * (y1 * ct * (N1 - a / r) + nu * q - a + y2s / p * na) - N1 * z1 * ct / w * ca
          - a * y1 * z * ct / r3 + z / p * (-2.0 * nu + (N1 * y1 * ct - a) / r + y2s / (r * p) * ma + a * y2s / r3)
          + z / w * (c ** 2 - (N1 * z1 * ct + a * c) / r + a * q * z1 * ct / r3
                     - (y2s * c ** 2 - a * z1 * ct / r * h) / (r * w)),
          N2 * (N1 * F * ct + y2 / p * ma - y2 * c / w * ca) + y2 * z / r * (2.0 * nu / p + a / r2)
          + y2 * z * c / (r * w) * (N1 - h / w * ca - a * q / r2)]
    b2 = [N1 * ((N2 * ct ** 2 + nu) * lp - (N2 * ct ** 2 + 1.0) * c * lw)
          + N1 / p * (-N1 * y1 * ct + nu * q - a + a * y1 * ct / r + y1 * y1 / p * na)
          - N1 * ct / w * (z1 * c - a * k / (r * c)) - a * y1 * z * ct / r3
          + z / p * (2.0 * nu + (N1 * y1 * ct + a) / r - y1 * y1 / (r * p) * ma - a * y1 * y1 / r3)
          + z * ct / w * (-c * s + a * y1 * q / (r3 * c) + k / r * (N2 * c - h / w * ra)),
          N2 * N1 * F * ct ** 2 + N1 * y2 / p * (-(N1 - a / r) * ct + y1 / p * na) - N1 * y2 * ct / w * ra
          - a * y2 * z * ct / r3 + y2 * z / (r * p) * (N1 * ct - 2.0 * nu * y1 / p - a * y1 / r * (1.0 / r + 1.0 / p))
          + y2 * z * ct / (r * w) * (-N2 * c + h / w * ra + a * q / (r2 * c)),
          -N2 * N1 * ct * (lp - c * lw) - N2 * y1 / p * ma + N2 * z1 / w * ca
          + z / r * (N1 * ct - 2.0 * nu * y1 / p - a * y1 / r2)
          - z / w * (c * s + h * ct / r * (N2 * c - h / w) + a / r * (s - q * z1 / r2 - z1 * h / (r * w)))]
    b3 = [N1 * (y2 / p * (1.0 + a / r) - y2 * c / w * ca) - y2 * z / r * (a / r2 + 1.0 / p)
          + y2 * z * c / (r * w) * (h / w * ca + a * q / r2),
          N1 * (-s * lw - y1 / p * (1.0 + a / r) + z1 / w * ca) + y1 * z / r * (a / r2 + 1.0 / p)
          - z / w * (s * (c - a / r) + z1 / r * (1.0 + a * q / r2) - (y2s * c * s - a * z1 / r * h) / (r * w)),
          N2 * F + N2 * y2 * s / w * ca + y2 * z * s / (r * w) * (1.0 + h / w * ca + a * q / r2)]
    return [b1, b2, b3]


def _axes(V):
    """Unit normal, strike and dip vectors of triangles V [3][3][1, n] (real)."""
    a = torch.stack([V[1][i] - V[0][i] for i in range(3)])
    b = torch.stack([V[2][i] - V[0][i] for i in range(3)])
    vn = torch.linalg.cross(a, b, dim=0)
    vn = vn / torch.linalg.vector_norm(vn, dim=0)
    vs = torch.stack([-vn[1], vn[0], torch.zeros_like(vn[0])])
    flat = (vs == 0).all(0)
    vs = torch.where(flat, torch.stack([torch.zeros_like(vn[0]), vn[2], torch.zeros_like(vn[0])]), vs)
    vs = vs / torch.linalg.vector_norm(vs, dim=0)
    return [vn, vs, torch.linalg.cross(vn, vs, dim=0)]


def _modes(x, V, nu, hs):
    """Displacement of unit Dn, Dss, Dds slip: [mode][component], complex [m, n]."""
    parts = [(_loop(x, V, nu), _axes(V))]
    if hs:
        fs = [[0.0] * 3 for _ in range(3)]
        for k in range(3):
            u = _free_surface(x, V[k], V[(k + 1) % 3], nu)
            fs = [[fs[j][c] + u[j][c] for c in range(3)] for j in range(3)]
        parts.append((fs, _axes(V)))
        W = [[v[0], v[1], -v[2]] for v in V]
        parts.append((_loop(x, W, nu), _axes(W)))
    return [[sum(ax[m][j] * u[j][c] for u, ax in parts for j in range(3)) for c in range(3)] for m in range(3)]


def _fields(XYZ, P, hs, strain, disp, chunk=1 << 21):
    """Unit-mode strains [3][6] and displacements [3][3], by chunks of
    triangles: yields (slice, E, U)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = [torch.as_tensor(a, dtype=torch.float64, device=dev).reshape(-1, 1) for a in XYZ]
    Q = [torch.as_tensor(np.ascontiguousarray(p), dtype=torch.float64, device=dev) for p in P]
    m, n = len(X[0]), len(Q[0])
    step = max(1, chunk // max(m, 1))
    h = 1e-40
    for j in range(0, n, step):
        V = [[q[j:j + step, i].reshape(1, -1) for i in range(3)] for q in Q]
        grad, U = [], None
        for k in range(3 if strain else 1):
            x = [torch.complex(X[i], torch.full_like(X[i], h if i == k else 0.0)) for i in range(3)]
            u = _modes(x, V, NU, hs)
            grad.append([[u[a][c].imag / h for c in range(3)] for a in range(3)])
            U = [[u[a][c].real for c in range(3)] for a in range(3)] if k == 0 else U
        E = None
        if strain:
            E = [[grad[0][a][0], grad[1][a][1], grad[2][a][2], 0.5 * (grad[0][a][1] + grad[1][a][0]),
                  0.5 * (grad[0][a][2] + grad[2][a][0]), 0.5 * (grad[1][a][2] + grad[2][a][1])] for a in range(3)]
        yield slice(j, min(n, j + step)), E, U


def _system(P, nrm, mid, hs):
    """A = -[Atn; Atss; Atds] for columns [Dn, Dss, Dds] (row-major tensor)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = len(nrm)
    N = torch.as_tensor(nrm, device=dev).T.reshape(3, n, 1)
    ss, ds = (torch.as_tensor(v, device=dev).T.reshape(3, n, 1) for v in _directions(nrm))
    A = torch.empty(3 * n, 3 * n, dtype=torch.float64, device=dev)
    for cols, E, _ in _fields((mid - 1e-12 * nrm).T, P, hs, 1, 0):
        for m in range(3):
            e = E[m]
            tr = LAM * (e[0] + e[1] + e[2])
            S = [[2 * G * e[0] + tr, 2 * G * e[3], 2 * G * e[4]], [2 * G * e[3], 2 * G * e[1] + tr, 2 * G * e[5]],
                 [2 * G * e[4], 2 * G * e[5], 2 * G * e[2] + tr]]
            t = [sum(S[i][k] * N[k] for k in range(3)) for i in range(3)]
            for r, d in enumerate((N, ss, ds)):
                A[r * n:(r + 1) * n, m * n + cols.start:m * n + cols.stop] = -sum(t[i] * d[i] for i in range(3))
    return A


def _directions(nrm):
    """Strike and dip directions of element normals, as the reference has them."""
    cx, cy, cz = nrm.T
    flat = (cx == 0) & (cy == 0)
    d = np.where(flat, 1.0, np.hypot(cx, cy))
    ss = np.stack([-cy / d, cx / d, 0 * cx], 1)
    ds = np.stack([-cx / d * cz, -cy / d * cz, d], 1)
    ss[flat & (cz < 1.0)], ss[flat & (cz >= 1.0)], ds[flat] = [0, -1, 0], [0, 1, 0], [-1, 0, 0]
    return ss, ds


def _friction(A, b, mu, Sf, scl):
    """Frictional slip: the 5n complementarity problem of the reference, by a
    damped Newton method on the Fischer-Burmeister function."""
    n = len(mu)
    C = torch.linalg.inv(A * scl)
    M = torch.zeros(5 * n, 5 * n, dtype=torch.float64, device=A.device)
    eye, dmu = torch.eye(n, dtype=torch.float64, device=A.device), torch.diag(mu)
    M[:3 * n, :3 * n] = C
    M[:3 * n, :n] = C[:, :n] - C[:, n:2 * n] * mu - C[:, 2 * n:] * mu
    for k in (1, 2):
        M[k * n:(k + 1) * n, (k + 2) * n:(k + 3) * n] = eye
        M[(k + 2) * n:(k + 3) * n, :n] = 2 * dmu
        M[(k + 2) * n:(k + 3) * n, k * n:(k + 1) * n] = -eye
    q = torch.cat([C @ (b - torch.cat([0 * Sf, Sf, Sf])), 2 * Sf, 2 * Sf])
    x = torch.zeros_like(q)

    def phi(x):
        y = M @ x + q
        return torch.hypot(x, y) - x - y

    for _ in range(200):
        y, f = M @ x + q, phi(x)
        if float(f.abs().max()) <= 1e-14 * float(q.abs().max()):
            break
        h = torch.hypot(x, y)
        tie = h == 0
        h = torch.where(tie, torch.ones_like(h), h)
        da = torch.where(tie, -torch.ones_like(h) * (1 - math.sqrt(0.5)), x / h - 1.0)
        db = torch.where(tie, -torch.ones_like(h) * (1 - math.sqrt(0.5)), y / h - 1.0)
        d = torch.linalg.solve(db[:, None] * M + torch.diag(da), -f)
        t = 1.0
        while t > 1e-9 and float(phi(x + t * d).norm()) > (1.0 - 1e-4 * t) * float(f.norm()):
            t *= 0.5
        if t <= 1e-9:
            break
        x = x + t * d
    if float(phi(x).abs().max()) > 1e-11 * float(q.abs().max()):
        return None
    y = M @ x + q
    return (torch.cat([y[:n], y[n:2 * n] - x[3 * n:4 * n], y[2 * n:3 * n] - x[4 * n:]]) * scl).cpu().numpy()


def exact(case, seed):
    kind, hs = case["kind"], case["hs"]
    if kind == "batch":
        out = []
        for P, s in zip(*_cracks(case, seed)):
            nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
            Tn, Tds, Tss = cad.CalculateNormalAndShearTractions3D(*s, nrm)
            A = _system(P, nrm, mid, hs)
            out.append(torch.linalg.solve(A, torch.as_tensor(np.concatenate([Tn, Tss, Tds]), device=A.device)))
        return torch.cat(out).cpu()
    P = _mesh(case, seed)
    n = len(P[0])
    if kind in ("inf", "sum", "sum_host"):
        XYZ, sl = _points(case, seed), _slips(P, seed)
        m, total = len(XYZ[0]), kind != "inf"
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        s = torch.as_tensor(np.stack([sl[2], sl[0], sl[1]]), device=dev)   # Dn, Dss, Dds
        shape = (m,) if total else (n, m)
        E = torch.zeros(6 if total else 18, *shape, dtype=torch.float64, device=dev)
        U = torch.zeros(3 if total else 9, *shape, dtype=torch.float64, device=dev)
        for cols, e, u in _fields(XYZ, P, hs, case["strain"], case["disp"]):
            for out, f, w in ((E, e, 6), (U, u, 3)):
                for a in range(3):
                    for k in range(w if f is not None else 0):
                        if total:
                            out[k] += f[a][k] @ s[a, cols]
                        else:
                            out[w * a + k, cols] = (f[a][k] * s[a, cols]).T
        if kind == "sum":
            E, U = E.reshape(6, 1, m), U.reshape(3, 1, m)
        got = {"E": E if case["strain"] else None, "U": U if case["disp"] else None}
        if kind == "sum_host":
            got = {k: None if v is None else [t.cpu().numpy() for t in v] for k, v in got.items()}
        return got
    nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
    A = _system(P, nrm, mid, hs)
    if kind == "friction":
        T, mu, Sf = _friction_loads(mid, seed)
        side = sum(np.linalg.norm(P[k] - P[(k + 1) % 3], axis=1) for k in range(3))
        return _friction(A, *(torch.as_tensor(v, device=A.device) for v in (np.concatenate(T), mu, Sf)),
                         float(np.mean(0.5 * side)) / G)
    b = torch.as_tensor(np.concatenate(_tractions(nrm, seed)), device=A.device)
    x = torch.linalg.solve(A, b).cpu()
    if kind == "slip_host":
        return {"Dn": x[:n], "Dss": x[n:2 * n], "Dds": x[2 * n:], "A": A.cpu()}
    return [x[:n], x[n:2 * n], x[2 * n:]] if kind == "learned" else x
