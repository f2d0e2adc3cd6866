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


@pytest.mark.parametrize("M", [1, 8, 16])
def test_the_narrowest_held_product(ops, M):  # noqa: F811
    """K = 768, where held products begin, takes a held body (which starts the kernel behind late) and not
    the three-chunk one, which covers as many columns but starts it early."""
    took = {}
    for K in (760, 768, 776):
        w, x = rnd(48, K, dtype=torch.bfloat16, seed=2), rnd(M, K, dtype=torch.bfloat16, seed=4)
        base = rnd(M, 48, seed=5)
        acc, before = base.clone(), ops.variant_counts()["fused_held"]
        ops.fused_linear_add(x, w, acc)
        took[K] = ops.variant_counts()["fused_held"] - before
        close(acc, base.double().cpu() + x.double().cpu() @ w.double().cpu().T, 1e-5)
    assert took == {760: 0, 768: 1, 776: 1}


@pytest.mark.parametrize("M,N,K,bn,taken", [(300, 200, 72, 0, True), (129, 68, 136, 64, True),
                                            (70, 1000, 1544, 128, True), (1000, 960, 576, 192, True),
                                            (2100, 2048, 264, 256, True), (20000, 520, 72, 256, True),
                                            # the slabs would take the second CTA its place on the SM
                                            (4000, 1000, 1544, 128, False)])
def test_float32_store_through_tma(ops, M, N, K, bn, taken):  # noqa: F811
    """Stored by the threads and through TMA: the same numbers, tails clipped, the padding beside the
    matrix untouched; with a factor as well.  A launch of at most one tile an SM always goes through TMA."""
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, seed=1)
    want = x.double() @ w.double().T
    ldc = -(-N // 8) * 8 + 8
    got, took = [], []
    for bulk in (False, True):
        for alpha in (1.0, -0.7):
            old = ops.set_tc_bulk_add(bulk)
            try:
                before = ops.variant_counts()["tc_bulk_add"]
                full = torch.full((M, ldc), 7.0, device=DEV)
                ops.gemm_tc(x, w, full[:, :N], bn=bn, alpha=alpha)
                took.append(ops.variant_counts()["tc_bulk_add"] > before)
            finally:
                ops.set_tc_bulk_add(old)
            close(full[:, :N], alpha * want, 1e-5)
            assert bool((full[:, N:] == 7.0).all())
            got.append(full)
    assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[3])
    assert took == [False, False, taken, taken]


@pytest.mark.parametrize("pairing", [0, 1])
@pytest.mark.parametrize("nh,nkv,hd,K", [(9, 3, 64, 72), (2, 1, 128, 96), (15, 5, 64, 136), (6, 1, 128, 64)])
def test_qkv_rope_with_two_ctas_on_a_tile(ops, pairing, nh, nkv, hd, K):  # noqa: F811
    """Against the body with one CTA on a tile, which sums in the same order and rounds at the same places,
    and its queries against float64: rows of several sequences in a tile, a chunk at a cached position,
    the last tile's heads beyond the matrix, one step that may not write the cache."""
    P, lens, news = 512, [200, 70, 333], [200, 70, 150]
    j = torch.arange(hd // 2, dtype=torch.float64)
    ang = torch.arange(P, dtype=torch.float64)[:, None] / 10000.0 ** (2 * j / hd)[None, :]
    cos, sin = torch.cos(ang).float().to(DEV), torch.sin(ang).float().to(DEV)
    qpos, qseq = [], []
    for b, (n, m) in enumerate(zip(lens, news)):
        qpos += list(range(n - m, n))
        qseq += [b] * m
    T = len(qpos)
    pos_t = torch.tensor(qpos, dtype=torch.int32, device=DEV)
    seq_t = torch.tensor(qseq, dtype=torch.int32, device=DEV)
    x = rnd(T, K, dtype=torch.bfloat16)
    w = rnd((nh + 2 * nkv) * hd, K, dtype=torch.bfloat16, seed=2, scale=0.3)
    fault = ops.fault_word(DEV)
    fault.zero_()
    got = []
    for pair in (0, 1):
        cache = ToyCache(lens, nkv, hd, torch.bfloat16, seed=3)
        q = torch.zeros(T, nh * hd, device=DEV, dtype=torch.bfloat16)
        old = ops.set_tc_pair(pair)
        try:
            before = ops.variant_counts()["tc_pair"]
            ops.gemm_tc_qkv_rope(x, w, q, cos, sin, pairing, nh, nkv, hd, pos_t, seq_t, cache.seq_slot,
                                 cache.table, cache.k, cache.v, 64, True)
            assert (ops.variant_counts()["tc_pair"] > before) == bool(pair)
            kept = cache.k.clone(), cache.v.clone()
            ops.gemm_tc_qkv_rope(x + 1, w, q.clone(), cos, sin, pairing, nh, nkv, hd, pos_t, seq_t,
                                 cache.seq_slot, cache.table, cache.k, cache.v, 64, False)
        finally:
            ops.set_tc_pair(old)
        assert torch.equal(kept[0], cache.k) and torch.equal(kept[1], cache.v)
        got.append((q, *kept))
    assert fault.item() == 0
    for a, b in zip(*got):
        assert torch.equal(b, a)
    # rounded before and behind the rotation: 2^-9 of each of the two channels and of the result
    u = (x.double() @ w.double().T)[:, :nh * hd].view(T, nh, hd).cpu()
    c, s = torch.cos(ang)[qpos][:, None], torch.sin(ang)[qpos][:, None]
    even, odd = (slice(0, hd, 2), slice(1, hd, 2)) if pairing else (slice(0, hd // 2), slice(hd // 2, hd))
    turned = torch.empty_like(u)
    turned[..., even], turned[..., odd] = u[..., even] * c - u[..., odd] * s, u[..., odd] * c + u[..., even] * s
    close(got[1][0], turned.view(T, nh * hd), 3 * 2.0 ** -9)


def test_the_ring_beside_another_streams_loads(ops):  # noqa: F811
    """A ring that turns more than once (16 steps in eight stages), while products on another stream ask
    for whole tiles of weights on the same SMs: a stage may be refilled only when its reads are done."""
    w, x = rnd(2048, 8192, dtype=torch.bfloat16, seed=1), rnd(1, 8192, dtype=torch.bfloat16, seed=2)
    v, y = rnd(2176, 2048, dtype=torch.bfloat16, seed=3), rnd(1, 2048, dtype=torch.bfloat16, seed=4)
    want = torch.zeros(1, 2048, device=DEV)
    before = ops.variant_counts()
    ops.fused_linear_add(x, w, want)
    ops.fused_linear_add(y, v, torch.zeros(1, 2176, device=DEV))
    after = ops.variant_counts()
    assert after["stream"] > before["stream"] and after["fused_held"] > before["fused_held"]
    close(want, x.double().cpu() @ w.double().cpu().T, 1e-5)
    got, beside = torch.zeros(300, 2048, device=DEV), torch.zeros(1, 2176, device=DEV)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(len(got)):
        with torch.cuda.stream(other):
            for _ in range(2):
                ops.fused_linear_add(y, v, beside)
        ops.fused_linear_add(x, w, got[i:i + 1])
    torch.cuda.synchronize()
    assert bool((got == want).all())
