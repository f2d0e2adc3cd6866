"""The 32-bit product: a row's bits do not depend on what else is in the call, whichever of the fast
bodies takes it, and the result is the 64-bit one within 32 bits."""
import pytest
import torch

from test_kernels_gpu import DEV, close, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu

# both sides of a few rows' body, of its row counts, and of the two tiles
ROWS = [1, 2, 3, 5, 9, 16, 17, 33, 64, 65, 130, 300]


@pytest.mark.parametrize("N,K", [(1, 4), (70, 36), (33, 132), (960, 576), (3072, 576), (576, 1536),
                                 (2305, 260), (258, 8192), (16, 8196), (20000, 64)])
def test_a_row_of_the_product_does_not_depend_on_the_others(ops, N, K):  # noqa: F811
    a, w = rnd(700, K), rnd(N, K, seed=1)
    whole = torch.empty(700, N, device=DEV)
    ops.gemm_simt(a, w, whole)
    # K eps bounds a sum of K products; a chain here is 16 long, the slabs' sums K / 32
    close(whole, a.double() @ w.double().T, 2e-6)
    for m in ROWS:
        c = torch.empty(m, N, device=DEV)
        ops.gemm_simt(a[:m], w, c)
        assert torch.equal(c, whole[:m]), m
        ops.gemm_simt(a[700 - m:], w, c)
        assert torch.equal(c, whole[700 - m:]), m
