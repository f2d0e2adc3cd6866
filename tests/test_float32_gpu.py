"""The 32-bit path's fast product against float64."""
import pytest
import torch

from test_kernels_gpu import DEV, close, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


# rows around the few-row body's tiles (1, 2, 4, 8), its last row count and the tiles' edges; columns
# around a warp's four and a tile's 32 and 64; k around a lane's four, a slab's 32 and a warp's 128
@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16, 17, 64, 65, 130])
@pytest.mark.parametrize("N,K", [(1, 4), (5, 36), (33, 128), (70, 132), (577, 576), (2305, 260)])
def test_product(ops, M, N, K):  # noqa: F811
    a = rnd(M, K + 4)[:, :K]                          # strided rows, still 16-byte aligned
    w = rnd(N, K, seed=1)
    want = a.double() @ w.double().T
    c = torch.full((M, N + 3), 7.0, device=DEV)
    ops.gemm_simt(a, w, c[:, :N])
    # sums of at most K products with unit operands: K eps is a bound, a tenth of it is seen
    close(c[:, :N], want, 2e-6)
    assert bool((c[:, N:] == 7.0).all())
    ops.gemm_simt(a, w, c[:, :N], accumulate=True)
    close(c[:, :N], 2 * want, 2e-6)


def test_product_of_few_rows_does_not_depend_on_the_others(ops):  # noqa: F811
    a, w = rnd(16, 576), rnd(960, 576, seed=1)
    whole = torch.empty(16, 960, device=DEV)
    ops.gemm_simt(a, w, whole)
    for m in (1, 2, 5, 9):
        c = torch.empty(m, 960, device=DEV)
        ops.gemm_simt(a[:m], w, c)
        assert torch.equal(c, whole[:m])
