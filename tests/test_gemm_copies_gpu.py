"""GPU tests of the FP64 product's copies: 16-byte and 8-byte ones, tiles inside
the matrices and at their edges, every DMMA shape, both tile sizes.  Integer
operands, so every sum is exact."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 3, 4])
@pytest.mark.parametrize("lda,ldb,off", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 2, 2)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 31, 15), (65, 33, 17), (64, 32, 16), (127, 200, 40),
                                   (2433, 1025, 31), (2560, 1024, 32), (2561, 1023, 49)])
def test_product_is_exact(cad, m, n, k, lda, ldb, off, prec):
    import torch
    from cutanddisplacejulia_b200 import _lib
    L, ctx = _lib.load(), _lib.context(0)
    la, lb = m + m % 2 + lda, k + k % 2 + ldb        # even, then odd with the extra row
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    draw = lambda *s: torch.randint(-8, 9, s, generator=g, device="cuda").double()
    A, B, C = draw(k * la + off), draw(n * lb + off), draw(n, m)
    want = C - B[off:].view(n, lb)[:, :k] @ A[off:].view(k, la)[:, :m]
    torch.cuda.synchronize()
    _lib.check(L.cad_gemm_sub_dev(ctx, prec, m, n, k, A[off:].data_ptr(), la, B[off:].data_ptr(), lb, C.data_ptr(),
                                  m), ctx)
    assert torch.equal(C, want)
