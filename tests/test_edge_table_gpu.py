"""GPU tests of the device-built mesh-edge table (csrc/edges.cu) through the
half-space sums and the system matrix, shared edges against the per-side
path: side counts around the 256-side blocks and the table's powers of two,
an edge shared by many triangles, repeated triangles, and -0.0 vertices."""
import numpy as np
import pytest

from helpers import assert_parity, rel_inf_err

pytestmark = pytest.mark.gpu


def _sums(cad, P, sl, pts, shared):
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    _lib.check(L.cad_set_shared_edges(ctx, int(shared)), ctx)
    try:
        S, U = cad.TD(*pts.T, *P, *sl, 0.25, 1.0, 1, 1, 1, cad.Strains(), cad.Disps())
    finally:
        _lib.check(L.cad_set_shared_edges(ctx, 1), ctx)
    return np.stack(list(S)), np.stack(list(U))


def _strip(n):
    """n triangles of a bent strip, neighbours sharing an edge."""
    k = np.arange(n + 2)
    node = np.stack([0.3 * (k // 2), 0.4 * (k % 2) + 0.01 * np.sin(k), -0.5 - 0.2 * (k % 2) - 0.02 * np.cos(k)], 1)
    P1, P2, P3 = node[:-2].copy(), node[1:-1].copy(), node[2:].copy()
    odd = np.arange(n) % 2 == 1
    return P1, np.where(odd[:, None], P3, P2), np.where(odd[:, None], P2, P3)


@pytest.mark.parametrize("n", [2, 3, 10, 11, 21, 22, 85, 86, 171, 342])
def test_sums_over_side_counts(cad, n):
    rng = np.random.default_rng(n)
    P = _strip(n)
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    pts = np.column_stack([rng.uniform(-1, 0.2 * n, 70), rng.uniform(-1, 1, 70), rng.uniform(-2, -0.05, 70)])
    a, b = _sums(cad, P, sl, pts, True), _sums(cad, P, sl, pts, False)
    assert_parity(a[0], b[0])
    assert_parity(a[1], b[1])
    # the table is filled in no fixed order; the sums are the same every time
    c = _sums(cad, P, sl, pts, True)
    assert np.array_equal(a[0], c[0]) and np.array_equal(a[1], c[1])


def test_edge_with_many_triangles_repeats_and_negative_zero(cad):
    rng = np.random.default_rng(1)
    k = 9
    th = np.linspace(0, np.pi, k)
    A, B = np.array([0.0, 0.0, -0.5]), np.array([1.0, 0.0, -0.7])
    C = np.stack([0.5 + 0 * th, np.cos(th), -0.6 - 0.5 * np.sin(th)], 1)
    P1, P2, P3 = np.tile(A, (k, 1)), np.tile(B, (k, 1)), C
    flip = rng.random(k) < 0.5                    # the common edge run both ways
    P1, P2 = np.where(flip[:, None], P2, P1), np.where(flip[:, None], P1, P2)
    P1[0, 1] = P2[0, 1] = -0.0                    # equal to the others' 0.0
    P = [np.concatenate([p, p[:3]]) for p in (P1, P2, P3)]   # three triangles twice
    n = len(P[0])
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    pts = rng.uniform([-1, -1, -2], [2, 1, -0.05], (60, 3))
    a, b = _sums(cad, P, sl, pts, True), _sums(cad, P, sl, pts, False)
    assert_parity(a[0], b[0])
    assert_parity(a[1], b[1])
    assert rel_inf_err(a[0], b[0]) < 1e-12


def _meshes():
    from cutanddisplacejulia_b200 import workloads
    dip = workloads.dipping_rect(seed=3, ntri=240, top_depth=0.1)
    sill = workloads.ellipse_crack(seed=4, ntri=200)
    sill = tuple(p - [0.0, 0.0, 0.8] for p in sill)          # exactly horizontal
    wall = workloads.dipping_rect(seed=5, ntri=200, dip=90.0, top_depth=0.3, jitter=0.0)   # vertical sides
    both = tuple(np.concatenate([a, b - [0.0, 3.0, 0.0]]) for a, b in zip(dip, sill))
    return {"dip": dip, "sill": sill, "wall": wall, "both": both}


@pytest.mark.parametrize("name", ["dip", "sill", "wall", "both"])
def test_fields_sums_and_tractions_over_meshes(cad, oracle, name):
    from cutanddisplacejulia_b200 import _lib
    P = _meshes()[name]
    n = len(P[0])
    rng = np.random.default_rng(7)
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    sl[1, ::5] = 0.0
    pts = rng.uniform([-2, -4, -2.5], [2, 2, -0.01], (131, 3))
    # points in a triangle's plane and on its sides (NaN there)
    pts[:5] = [0.5 * (P[0][k] + P[1][k]) for k in range(5)]
    pts[5:8] = [(P[0][k] + P[1][k] + P[2][k]) / 3 for k in range(3)]
    pts[8] = P[0][4]
    L, ctx = _lib.load(), _lib.context(0)
    nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
    _, _, lam, nu, G = cad.ElasticConstantsCheck(1.0, 0.25)
    got = {}
    for shared in (1, 0):
        _lib.check(L.cad_set_shared_edges(ctx, shared), ctx)
        try:
            S, U = cad.TD(*pts.T, *P, *sl, nu, G, 1, 1, 1)
            S1, _ = cad.TD(*pts.T, *P, *sl, nu, G, 0, 1, 1)
            Ss, Us = cad.TD(*pts.T, *P, *sl, nu, G, 1, 1, 1, cad.Strains(), cad.Disps())
            Sn, _ = cad.TD(*pts.T, *P, *sl, nu, G, 0, 1, 1, cad.Strains(), cad.Disps())
            T = cad.CalculateInfluenceMatrices3D(nrm, mid, *P, nu, G, lam, None, 1, n)
        finally:
            _lib.check(L.cad_set_shared_edges(ctx, 1), ctx)
        got[shared] = [np.stack(list(v)) for v in (S, U, S1, Ss, Us, Sn, T)]
    for a, b in zip(got[1], got[0]):
        # on a side the pair is NaN or, where rounding puts the point off the
        # plane, singular: only the NaN masks agree there
        k = 9 if a.shape[1] == len(pts) else 0
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isfinite(a[:, k:]).all()
        assert_parity(a[:, k:], b[:, k:])
    So, Uo = oracle.td_inf(*pts[9:].T, *P, *sl, nu, G, 1, 1, 1)
    assert_parity(got[1][0][:, 9:], So)
    assert_parity(got[1][1][:, 9:], Uo)


@pytest.mark.parametrize("hs", [0, 1])
@pytest.mark.parametrize("k", [31, 32, 33, 100, 3001, 100000])
def test_one_patch_listed_with_many_slips(cad, oracle, hs, k):
    """k copies of two neighbours, some with their vertices turned round: their
    five edges carry up to 2 k sides, and the field is that of the two with the
    net slips.  The lists are filled in no fixed order; the sums do not show it."""
    rng = np.random.default_rng(k)
    v = np.array([[0.0, 0.0, -0.5], [1.0, 0.1, -0.6], [0.2, 0.9, -1.1], [1.1, 1.2, -1.4]])
    tri = np.array([[0, 1, 2], [1, 3, 2]])
    which = rng.integers(0, 2, k)
    turn = rng.integers(0, 3, k)
    idx = tri[which][np.arange(k)[:, None], (np.arange(3) + turn[:, None]) % 3]
    P = [v[idx[:, c]] for c in range(3)]
    sl = rng.uniform(-1e-3, 1e-3, (3, k)) * 10.0 ** rng.uniform(-3, 0, k)
    sl[:, ::7] = 0.0
    M = max(300, (5 << 20) // k + 1) if hs == 0 else 300       # full space: over edges from 5 * 2^20 pairs on
    pts = rng.uniform([-2, -2, -3], [3, 3, -0.01], (M, 3))
    import math
    net = np.array([[math.fsum(sl[m][which == t]) for t in range(2)] for m in range(3)])

    def run():
        S, U = cad.TD(*pts.T, *P, *sl, 0.25, 1.0, 1, 1, hs, cad.Strains(), cad.Disps())
        return np.stack(list(S)), np.stack(list(U))

    a = run()
    b = run()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    n = 300
    So, Uo = oracle.td_sum_eval(*pts[:n].T, *[v[tri[:, c]] for c in range(3)], *net, 0.25, 1.0, 1, 1, hs)
    # a sum of k terms in another order: k eps of the largest patch's field at most, scaled by the slips
    lost = k * 2.3e-16 * np.abs(sl).sum(1).max() / np.abs(net).max()
    assert rel_inf_err(a[0][:, :n], So) < 1e-12 + lost
    assert rel_inf_err(a[1][:, :n], Uo) < 1e-12 + lost


@pytest.mark.parametrize("strain,disp", [(1, 0), (0, 1), (1, 1)])
def test_degenerate_triangles_without_slip(cad, strain, disp):
    """Point-like and collinear triangles that carry no slip, repeats and a
    reversed triangle in a half-space mesh: they add nothing, per edge as per side."""
    from cutanddisplacejulia_b200 import _lib
    rng = np.random.default_rng(2)
    P = [np.concatenate([p, p[:5]]) for p in _strip(60)]       # repeats
    P[0][7], P[1][7] = P[1][7].copy(), P[0][7].copy()          # reversed
    P[1][20] = P[0][20]                                        # a side of no length
    P[1][31] = P[2][31] = P[0][31]                             # a point
    P[2][44] = 0.5 * (P[0][44] + P[1][44])                     # collinear
    n = len(P[0])
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    sl[:, [20, 31, 44]] = 0.0
    sl[:, 50:53] = 0.0                                         # neighbours: an edge without slip
    pts = rng.uniform([-1, -1, -2], [8, 1, -0.05], (90, 3))
    L, ctx = _lib.load(), _lib.context(0)
    got = []
    for shared in (1, 0):
        _lib.check(L.cad_set_shared_edges(ctx, shared), ctx)
        try:
            S, U = cad.TD(*pts.T, *P, *sl, 0.25, 1.0, disp, strain, 1, cad.Strains(), cad.Disps())
        finally:
            _lib.check(L.cad_set_shared_edges(ctx, 1), ctx)
        got.append([np.stack(list(f)) for f, on in ((S, strain), (U, disp)) if on])
    for a, b in zip(*got):
        assert np.isfinite(b).all() and np.isfinite(a).all()
        assert_parity(a, b)
