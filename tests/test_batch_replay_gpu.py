"""GPU test of the batched solve's plan: the first call of a plan is issued
directly, the second captured and later ones replayed, whatever the arrays;
each call's slip is that of its own inputs, bit for bit."""
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
