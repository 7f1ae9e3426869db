"""A device wait that runs out ends its kernel normally with an error status
that the host reads (no fault, no hang), and the context stays usable.

The waits are made to run out on purpose, with a short limit set by
cad_set_wait_limit: the one-right-hand-side solve's chain flags
(cad_wait_timeout_probe starts the chain's order counter past block 0, so every
block waits for a flag that nothing sets) and the LU leaves' pivot exchange
(cad_leaf_timeout_probe loses the pushes to each leaf's first thread block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_chain_wait_runs_out_and_the_context_survives(cad):
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    ctx = _lib.context(0)
    try:
        _lib.check(L.cad_set_wait_limit(ctx, 2000), ctx)
        for n in (640, 1000):
            rc = L.cad_wait_timeout_probe(ctx, n)
            assert rc == _lib.CAD_ERR_TIMEOUT
            assert b"wait ran out" in L.cad_last_error(ctx)
    finally:
        _lib.check(L.cad_set_wait_limit(ctx, 1 << 22), ctx)
    # the same context solves correctly afterwards
    rng = np.random.default_rng(0)
    A = rng.standard_normal((300, 300)) + 300 * np.eye(300)
    b = rng.standard_normal(300)
    x = cad.solve(A, b)
    assert np.linalg.norm(A @ x - b) <= 1e-12 * np.linalg.norm(b)


def _solves(cad, n=300):
    rng = np.random.default_rng(0)
    A = rng.standard_normal((n, n)) + n * np.eye(n)
    b = rng.standard_normal(n)
    x = cad.solve(A, b)
    assert np.linalg.norm(A @ x - b) <= 1e-12 * np.linalg.norm(b)


# two to eight thread blocks per leaf; remainders of leaves and block columns
@pytest.mark.parametrize("n", [513, 1025, 1600, 4096])
def test_leaf_wait_runs_out_and_the_context_survives(cad, n):
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    ctx = _lib.context(0)
    try:
        _lib.check(L.cad_set_wait_limit(ctx, 64), ctx)
        for _ in range(2):
            assert L.cad_leaf_timeout_probe(ctx, n) == _lib.CAD_ERR_TIMEOUT
            assert b"pivot exchange" in L.cad_last_error(ctx)
    finally:
        _lib.check(L.cad_set_wait_limit(ctx, 1 << 22), ctx)
    _solves(cad)
    _solves(cad, 1600)


def test_solve_with_the_shortest_limit(cad):
    # each wait gives up at its first poll that finds nothing: the solve ends
    # with the status or with the right answer
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    ctx = _lib.context(0)
    rng = np.random.default_rng(1)
    A = rng.standard_normal((1600, 1600)) + 1600 * np.eye(1600)
    b = rng.standard_normal(1600)
    try:
        _lib.check(L.cad_set_wait_limit(ctx, 1), ctx)
        for _ in range(3):
            try:
                x = cad.solve(A, b)
            except cad.CadError as e:
                assert e.code == _lib.CAD_ERR_TIMEOUT
            else:
                assert np.linalg.norm(A @ x - b) <= 1e-12 * np.linalg.norm(b)
    finally:
        _lib.check(L.cad_set_wait_limit(ctx, 1 << 22), ctx)
    _solves(cad, 1600)


def test_wait_limit_arguments(cad):
    from cutanddisplacejulia_b200 import _lib
    L = _lib.load()
    ctx = _lib.context(0)
    assert L.cad_set_wait_limit(ctx, 0) == _lib.CAD_ERR_ARG
    assert L.cad_wait_timeout_probe(ctx, 64) == _lib.CAD_ERR_ARG
    assert L.cad_leaf_timeout_probe(ctx, 512) == _lib.CAD_ERR_ARG
    assert L.cad_leaf_timeout_probe(ctx, 4097) == _lib.CAD_ERR_ARG
