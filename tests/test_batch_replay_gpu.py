"""GPU tests of the batched solve's plan: the first call of a plan is issued
directly, the second captured and later ones replayed, whatever the arrays;
each call's slip is that of its own inputs, bit for bit, also after a larger
batch moved the lanes' buffers and then ran out of memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hs", [0, 1])
@pytest.mark.parametrize("mode", ["grouped", "lanes", "lanes_chain"])
def test_replays_serve_other_arrays(cad, mode, hs):
    from cutanddisplacejulia_b200 import workloads
    _, _, lam, nu, G = cad.ElasticConstantsCheck(1.0, 0.25)

    def solve(count, scale, depth):
        cracks, stresses = workloads.crack_batch(seed=3, count=count, n_range=(20, 200))
        cracks = [tuple(p * scale - [0, 0, depth] for p in P) for P in cracks]
        bcs = [cad.Stresses(*[v * scale for v in s]) for s in stresses]
        out, rel = cad.SlipCalculator3D_batched(cracks, nu, G, lam, hs, bcs, tol=1e-10, mode=mode)
        assert np.all(rel <= 1e-10)
        return [np.concatenate(r) for r in out]

    states = [(1.0, 50.0), (1.1, 60.0), (0.9, 70.0)]
    alone = []
    for s in states:
        solve(3, 1.0, 50.0)          # another plan: the next call is its plan's first
        alone.append(solve(6, *s))
    assert not np.array_equal(alone[0][0], alone[1][0])
    for k in (2, 0, 1, 2, 1):        # captured, then replayed
        assert all(np.array_equal(a, b) for a, b in zip(solve(6, *states[k]), alone[k])), k


@pytest.mark.parametrize("mode", ["grouped", "lanes_chain"])
def test_plan_after_a_larger_batch_that_ran_out_of_memory(cad, fresh_context, mode):
    from cutanddisplacejulia_b200 import _lib, workloads
    L, ctx = _lib.load(), fresh_context
    _, _, lam, nu, G = cad.ElasticConstantsCheck(1.0, 0.25)

    def solve(n):
        cracks, stresses = workloads.crack_batch(seed=5, count=5, n_range=(n, n + 40))
        bcs = [cad.Stresses(*v) for v in stresses]
        out, rel = cad.SlipCalculator3D_batched(cracks, nu, G, lam, 0, bcs, tol=1e-10, mode=mode)
        assert np.all(rel <= 1e-10)
        return [np.concatenate(r) for r in out]

    want = solve(30)
    failed = 0
    try:
        for nth in range(1, 200):
            solve(30)
            solve(30)                        # captured, or replayed
            _lib.check(L.cad_fail_allocation(ctx, nth), ctx)
            try:
                solve(100 + 4 * nth)         # each larger than the one before
            except cad.CadError as e:
                assert e.code == _lib.CAD_ERR_OOM
                failed += 1
            else:
                break                        # fewer allocations than nth
            finally:
                _lib.check(L.cad_fail_allocation(ctx, 0), ctx)
            assert all(np.array_equal(a, b) for a, b in zip(solve(30), want)), nth
    finally:
        L.cad_fail_allocation(ctx, 0)
    assert failed > 5


def test_failed_call_leaves_the_slips_alone(cad, fresh_context):
    import torch

    from cutanddisplacejulia_b200 import _lib, workloads
    L, ctx = _lib.load(), fresh_context
    _lib.check(L.cad_set_solver(ctx, _lib.CAD_SOLVER_MIXED, 1e-10, 400), ctx)

    def call(count, n):
        cracks, _ = workloads.crack_batch(seed=6, count=count, n_range=(n, n + 10))
        offs = np.concatenate([[0], np.cumsum([len(P[0]) for P in cracks])]).astype(np.int64)
        args = []
        for k in range(5):
            parts = []
            for P in cracks:
                nrm, mid = cad.CreateFaceNormalAndMidPoint(*P)
                parts.append(np.asfortranarray((*P, nrm, mid)[k]).ravel(order="F"))
            args.append(torch.tensor(np.concatenate(parts), device="cuda"))
        T = torch.ones(3 * int(offs[-1]), dtype=torch.float64, device="cuda")
        D = torch.full_like(T, -7.0)
        torch.cuda.synchronize()
        rc = L.cad_slip_calculator_batched_dev(ctx, count, offs.ctypes.data, *[a.data_ptr() for a in args], 0.25, 1.0,
                                               1.0, 0, T.data_ptr(), D.data_ptr(), None)
        torch.cuda.synchronize()
        return rc, D

    rc, D = call(4, 30)
    assert rc == _lib.CAD_OK and not bool((D == -7.0).any())
    for nth in range(2, 8):          # the first is the copies' own
        _lib.check(L.cad_fail_allocation(ctx, nth), ctx)
        rc, D = call(4, 40 + 20 * nth)
        _lib.check(L.cad_fail_allocation(ctx, 0), ctx)
        assert rc == _lib.CAD_ERR_OOM and bool((D == -7.0).all()), nth
