"""The matrix products' further bodies against float64: weights held in registers for few rows, the
float32 store through TMA, q|k|v with two CTAs on a tile."""
import pytest
import torch

from test_kernels_gpu import DEV, ToyCache, _norm_bf16, close, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(48, 768), (40, 776), (576, 1536), (33, 1544), (130, 2048), (16, 2056),
                                 # beyond one wave of tiles: the ring again
                                 (4800, 960)])
def test_held_in_registers(ops, M, N, K):  # noqa: F811
    """Around every depth of the register body and the widths where it gives way to the ring.  Sums of K
    exact products of bfloat16 in 32 bits: 1e-5 of the largest; normed rows are rounded once more."""
    w = rnd(N, K, dtype=torch.bfloat16, seed=2)
    x = rnd(M, K, dtype=torch.bfloat16, seed=4)
    before = ops.variant_counts()
    base = rnd(M, N, seed=5)
    acc = base.clone()
    ops.fused_linear_add(x, w, acc)
    after = ops.variant_counts()
    close(acc, base.double().cpu() + x.double().cpu() @ w.double().cpu().T, 1e-5)
    held = K <= (2048 if M <= 8 else 1536) and N <= 296 * 16
    assert (after["fused_registers"] > before["fused_registers"]) == held
    assert (after["stream"] > before["stream"]) == (not held)
    h, nw = rnd(M, K), rnd(K, seed=1) * 0.1 + 1
    out = torch.empty(M, N, device=DEV)
    ops.fused_norm_linear(h, nw, 1e-5, w, out)
    close(out, _norm_bf16(h, nw, 1e-5) @ w.double().cpu().T, 3e-3)


@pytest.mark.parametrize("M,N,K,bn", [(300, 200, 72, 0), (129, 68, 136, 64), (70, 1000, 1544, 128),
                                      (1000, 960, 576, 192), (2100, 2048, 264, 256), (20000, 520, 72, 256)])
def test_float32_store_through_tma(ops, M, N, K, bn):  # noqa: F811
    """Stored by the threads and through TMA: the same numbers, tails clipped, the padding beside the
    matrix untouched; with a factor as well."""
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, seed=1)
    want = x.double() @ w.double().T
    ldc = -(-N // 8) * 8 + 8
    got, took = [], []
    for bulk in (False, True):
        for alpha in (1.0, -0.7):
            old = ops.set_tc_bulk_add(bulk)
            before = ops.variant_counts()["tc_bulk_add"]
            full = torch.full((M, ldc), 7.0, device=DEV)
            ops.gemm_tc(x, w, full[:, :N], bn=bn, alpha=alpha)
            ops.set_tc_bulk_add(old)
            took.append(ops.variant_counts()["tc_bulk_add"] > before)
            close(full[:, :N], alpha * want, 1e-5)
            assert bool((full[:, N:] == 7.0).all())
            got.append(full)
    assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[3])
    assert not any(took[:2]) and (all(took[2:]) or bn in (64, 128, 192))
