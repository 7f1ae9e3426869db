"""GPU tests of the full-space sums over mesh edges (segment_sum_kernel)
against the per-triangle sums: meshes with shared, repeated and unshared
sides, points on vertices, sides and inside elements, zero-slip and
degenerate triangles, and the sizes at which the edges take over."""
import ctypes

import numpy as np
import pytest

from helpers import assert_parity

pytestmark = pytest.mark.gpu


def _sums(cad, P, sl, pts, shared, strain=1, disp=1):
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    _lib.check(L.cad_set_shared_edges(ctx, int(shared)), ctx)
    try:
        S, U = cad.TD(*pts.T, *P, *sl, 0.25, 1.0, disp, strain, 0, cad.Strains(), cad.Disps())
    finally:
        _lib.check(L.cad_set_shared_edges(ctx, 1), ctx)
    return [np.stack(list(f)) for f, on in ((S, strain), (U, disp)) if on]


def _grid(n, m, z):
    """2 n m triangles over an n x m grid of squares (exact coordinates)."""
    i, j = np.meshgrid(np.arange(n), np.arange(m), indexing="ij")
    q = lambda di, dj: np.stack([(i + di).ravel(), (j + dj).ravel(), z(i + di, j + dj).ravel()], 1) * 0.25
    a, b, c, d = q(0, 0), q(1, 0), q(1, 1), q(0, 1)
    return [np.concatenate(v) for v in ((a, a), (b, c), (c, d))]


def _mesh(kind, rng):
    if kind == "flat":
        return _grid(12, 14, lambda i, j: -1.0 * np.ones(i.shape))
    if kind == "bent":
        return _grid(12, 14, lambda i, j: np.sin(0.7 * i) - 0.3 * j)
    if kind == "soup":
        return [rng.uniform([0, 0, -2], [3, 3, -1], (336, 3)) for _ in range(3)]
    P = _grid(12, 14, lambda i, j: -0.2 * i)           # repeats, a reversed triangle, a point-like one
    P = [np.concatenate([p, p[:5]]) for p in P]
    P[0][7], P[1][7] = P[1][7].copy(), P[0][7].copy()
    P[1][20] = P[0][20]
    return P


@pytest.mark.parametrize("strain,disp", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("kind", ["flat", "bent", "soup", "odd"])
def test_edges_match_triangles(cad, kind, strain, disp):
    rng = np.random.default_rng(3)
    P = _mesh(kind, rng)
    n = len(P[0])
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    sl[:, ::9] = 0.0
    if kind == "odd":
        sl[:, 20] = 0.0                                # the degenerate one adds nothing
    M = ((5 << 20) if strain else (1 << 24)) // n + 1
    pts = rng.uniform([-2, -2, -3], [5, 5, 1], (M, 3))
    # vertices, midpoints of the first sides, centroids (the degenerate one's lies on a side)
    on = np.concatenate([P[0][:50], 0.5 * (P[0] + P[1])[:50], ((P[0] + P[1] + P[2]) / 3)[21:50]])
    pts[:len(on)] = on
    a, b = _sums(cad, P, sl, pts, True, strain, disp), _sums(cad, P, sl, pts, False, strain, disp)
    far = slice(len(on), None)
    for x, y in zip(a, b):
        assert np.array_equal(np.isnan(x), np.isnan(y))
        assert_parity(x[:, far], y[:, far])
        assert_parity(x[:, 100:], y[:, 100:])
    c = _sums(cad, P, sl, pts, True, strain, disp)     # the lists are filled in no fixed order
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, c))


@pytest.mark.parametrize("n,M", [(1, 5 << 20), (2, (5 << 19) + 1), (20480, 256), (20480, 255), (85, 61681)])
def test_edges_over_sizes(cad, n, M):
    rng = np.random.default_rng(n)
    P = [p[:n].copy() for p in _grid(128, 129, lambda i, j: 0.1 * np.cos(i + 2 * j))]
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    pts = rng.uniform([-2, -2, -3], [34, 34, 1], (M, 3))
    for x, y in zip(_sums(cad, P, sl, pts, True), _sums(cad, P, sl, pts, False)):
        assert_parity(x, y)


@pytest.mark.parametrize("hs", [0, 1])
def test_no_slip_adds_nothing_anywhere(cad, hs):
    """Triangles without slip add nothing, also at points far out of range or
    without coordinates, over the edges as by the pairs; a slipping mesh gives
    NaN there."""
    from cutanddisplacejulia_b200 import _lib
    rng = np.random.default_rng(4)
    P = _mesh("bent", rng)
    P = [p - [0.0, 0.0, 8.0] for p in P]
    n = len(P[0])
    pts = rng.uniform([-2, -2, -12], [5, 5, -0.1], ((5 << 20) // n + 1, 3))
    pts[0], pts[1], pts[2] = [np.nan, 0, -1], [np.inf, 0, -1], [0, 1e160, -1e160]
    L, ctx = _lib.load(), _lib.context(0)
    for shared in (1, 0):
        _lib.check(L.cad_set_shared_edges(ctx, shared), ctx)
        try:
            S, U = cad.TD(*pts.T, *P, *np.zeros((3, n)), 0.25, 1.0, 1, 1, hs, cad.Strains(), cad.Disps())
            T, _ = cad.TD(*pts.T, *P, *np.full((3, n), 1e-3), 0.25, 1.0, 0, 1, hs, cad.Strains(), cad.Disps())
        finally:
            _lib.check(L.cad_set_shared_edges(ctx, 1), ctx)
        assert not np.stack(list(S)).any() and not np.stack(list(U)).any()
        assert np.isnan(np.stack(list(T))[:, :2]).all()


def test_sums_where_only_the_pairs_fit(cad, fresh_context):
    """A full-space sum runs over the pairs where the edges' workspaces cannot be
    had: only the arrays every sum needs are refused."""
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    rng = np.random.default_rng(11)
    P = _mesh("bent", rng)
    n = len(P[0])
    sl = rng.uniform(-1e-3, 1e-3, (3, n))
    pts = rng.uniform([-2, -2, -3], [5, 5, 1], ((5 << 20) // n + 1, 3))
    want = _sums(cad, P, sl, pts, False)
    outcome = []
    for nth in range(1, 12):
        h = ctypes.c_void_p()
        _lib.check(L.cad_init(0, ctypes.byref(h)), None)
        _lib._ctx[0] = h
        try:
            _lib.check(L.cad_fail_allocation(h, nth), h)
            try:
                got = _sums(cad, P, sl, pts, True)
            except cad.CadError as e:
                assert e.code == _lib.CAD_ERR_OOM
                outcome.append("refused")
            else:
                for x, y in zip(got, want):
                    assert_parity(x, y)
                outcome.append("pairs" if all(np.array_equal(x, y) for x, y in zip(got, want)) else "edges")
        finally:
            _lib._ctx[0] = fresh_context
            L.cad_destroy(h)
    # inputs, outputs, records; then flag, edge records, partial sums, end points, table
    assert outcome == 3 * ["refused"] + 5 * ["pairs"] + 3 * ["edges"], outcome
