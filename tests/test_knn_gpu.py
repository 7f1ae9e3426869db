"""GPU test of the nearest-centroid lists (one warp per element over tiles of
256): sizes around the list's length and the tiles, with many exact ties,
against sorting by (distance, index)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K = 16


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 255, 256, 257, 600])
def test_nearest_by_distance_then_index(cad, n):
    import torch
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    rng = np.random.default_rng(n)
    cen = rng.integers(0, 6, (n, 3)).astype(np.float64)   # lattice points, several times over: exact distances
    if n > 300:
        cen[40:300] = cen[40]                              # more than a list's worth at one point
    off = np.array([[3.0, 0, -6], [0, 6, 3], [-3, -6, 3]])
    P = [torch.from_numpy(np.ascontiguousarray((cen + o).T)).cuda() for o in off]
    X = torch.empty(n, 7 * K, dtype=torch.float32, device="cuda")
    nbr = torch.empty(n, K, dtype=torch.int32, device="cuda")
    h = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(L.cad_lpc_features_dev(ctx, *[p.data_ptr() for p in P], n, X.data_ptr(), nbr.data_ptr(),
                                      h.data_ptr()), ctx)
    torch.cuda.synchronize()
    d = ((cen[:, None] - cen[None]) ** 2).sum(2)
    want = np.argsort(d, axis=1, kind="stable")[:, :K]     # stable: ties to the smaller index
    want = np.concatenate([want, np.repeat(want[:, -1:], K - want.shape[1], axis=1)], axis=1)
    assert np.array_equal(nbr.cpu().numpy(), want)


@pytest.mark.parametrize("n", [5, 16, 40, 300])
def test_elements_without_coordinates_stay_in_range(cad, n):
    """Centroids that are not numbers are nobody's neighbours; the places they
    leave in the lists name the element itself."""
    import torch
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    rng = np.random.default_rng(n)
    cen = rng.uniform(-1, 1, (n, 3))
    bad = np.arange(n) % 3 == 1
    off = np.array([[0.3, 0, -0.6], [0, 0.6, 0.3], [-0.3, -0.6, 0.3]])
    V = [cen + o for o in off]
    V[1][bad, 2] = np.nan
    P = [torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for v in V]
    X = torch.empty(n, 7 * K, dtype=torch.float32, device="cuda")
    nbr = torch.empty(n, K, dtype=torch.int32, device="cuda")
    h = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(L.cad_lpc_features_dev(ctx, *[p.data_ptr() for p in P], n, X.data_ptr(), nbr.data_ptr(),
                                      h.data_ptr()), ctx)
    torch.cuda.synchronize()
    got = nbr.cpu().numpy()
    cen = (V[0] + V[1] + V[2]) / 3
    good = np.flatnonzero(~bad)
    for i in range(n):
        if bad[i]:
            assert (got[i] == i).all()
            continue
        k = min(K, len(good))
        d = ((cen[good] - cen[i]) ** 2).sum(1)
        assert set(got[i, :k]) == set(good[np.argsort(d)[:k]])
        rest = got[i, k:]
        assert np.isin(rest, [i, got[i, k - 1]]).all()
