"""GPU tests of the dense LU's panel path (csrc/lu.cu) at the sizes where it
changes: leaf widths and their remainders, one to several CTAs per leaf
cluster, the update kernel's rows per thread, block columns and look-ahead,
and the split panels beyond one row per leaf thread.  Factors against numpy
LAPACK's solution and the backward error of the solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(n, nrhs, seed, rows=None):
    import torch

    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.randn(n, n, generator=g, dtype=torch.float64, device="cuda")
    if rows is not None:
        A = A[rows]
    B = torch.randn(nrhs, n, generator=g, dtype=torch.float64, device="cuda")
    F, X = A.t().contiguous(), B.clone()          # column-major copies
    torch.cuda.synchronize()
    _lib.check(L.cad_solve_dev(ctx, n, F.data_ptr(), n, X.data_ptr(), n, nrhs), ctx)
    torch.cuda.synchronize()
    R = A @ X.t() - B.t()
    # backward error of a stable LU: a modest multiple of n eps |A| |x|
    scale = A.abs().sum(1).max() * X.abs().max()
    return float(R.abs().max() / scale), A, B, X


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 255, 256, 257, 288, 511, 513, 544, 769, 1025, 1537, 2049,
                               4097, 4200])
def test_lu_sizes(cad, n):
    # growth of partial pivoting on random matrices is ~ n^(2/3): 64 n eps covers it
    for nrhs in (1, 3):
        err, A, B, X = _solve(n, nrhs, 100 + n)
        assert err < 64 * n * 2.3e-16
    if n <= 600:
        x = np.linalg.solve(A.cpu().numpy(), B.cpu().numpy().T)
        cond = np.linalg.cond(A.cpu().numpy())
        assert np.abs(X.cpu().numpy().T - x).max() <= 64 * cond * n * 2.3e-16 * np.abs(x).max()


def test_lu_split_panels(cad):
    err, *_ = _solve(8600, 1, 9)      # more rows than one per leaf thread: split panels, then leaf by leaf
    assert err < 64 * 8600 * 2.3e-16


@pytest.mark.parametrize("n", [300, 1100])
def test_lu_rows_moved_across_the_matrix(cad, n):
    import torch
    rows = torch.arange(n - 1, -1, -1, device="cuda")   # every pivot far from the diagonal
    err, *_ = _solve(n, 1, 5, rows=rows)
    assert err < 64 * n * 2.3e-16


def test_lu_repeated_entries_and_singular(cad):
    n = 400
    # equal magnitudes everywhere: ties go to the first row, as LAPACK's
    H = np.where(np.random.default_rng(0).random((n, n)) < 0.5, -1.0, 1.0)
    x = cad.solve(H, np.arange(n, dtype=float))
    assert np.abs(H @ x - np.arange(n)).max() < 1e-8
    S = np.ones((n, n))
    with pytest.raises(cad.CadError):
        cad.solve(S, np.ones(n))
    # the context solves as before afterwards
    assert _solve(n, 1, 6)[0] < 64 * n * 2.3e-16


@pytest.mark.parametrize("n", [511, 513, 1100, 2100])
def test_lu_wide_blocks(cad, n):
    # the block width large systems take
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    _lib.check(L.cad_set_lu_block(ctx, 512), ctx)
    try:
        for nrhs in (1, 3):
            assert _solve(n, nrhs, 300 + n)[0] < 64 * n * 2.3e-16
    finally:
        _lib.check(L.cad_set_lu_block(ctx, 0), ctx)


@pytest.mark.parametrize("rpt", [2, 4])
def test_lu_narrow_leaves(cad, tmp_path, rpt):
    """The leaves of 16 and 8 columns (2 and 4 rows per thread: 1024 and 2048 rows
    per thread block) that the autotuner may choose, and their update kernels, at
    remainders of leaves and panels and one to nine blocks per cluster."""
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"lu_leaf_f64_n{1 << k} {rpt}\n" for k in range(15)))
    _lib.check(L.cad_set_autotune(ctx, 2, str(cache).encode()), ctx)     # read, never timed
    try:
        sizes = [7, 9, 17, 33, 255, 257, 263, 530, 1023, 1025, 1100, 2049, 2100, 4200] + ([8600] if rpt == 2 else [])
        for n in sizes:
            for nrhs in (1, 3):
                err, A, B, X = _solve(n, nrhs, 500 + n)
                assert err < 64 * n * 2.3e-16, n
            if n <= 600:
                x = np.linalg.solve(A.cpu().numpy(), B.cpu().numpy().T)
                cond = np.linalg.cond(A.cpu().numpy())
                assert np.abs(X.cpu().numpy().T - x).max() <= 64 * cond * n * 2.3e-16 * np.abs(x).max(), n
        import torch
        rows = torch.arange(1099, -1, -1, device="cuda")
        assert _solve(1100, 1, 5, rows=rows)[0] < 64 * 1100 * 2.3e-16
    finally:
        _lib.check(L.cad_set_autotune(ctx, 0, None), ctx)
