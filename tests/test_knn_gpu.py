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
