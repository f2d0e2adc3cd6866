"""The 32-bit path's fast kernels: the product against float64, the attention of heads of 64
against the general kernel (which has its own tests against float64)."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, ToyCache, close, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


# rows around the few-row body's tiles (1, 2, 4, 8) and its last row count; columns around a CTA's 4, 8 and 32;
# k around a lane's four and a slab's 32.  (All but the last rows go to the few-row body and the 32 x 32
# tiles; test_float32_order_gpu.py names the body of every shape, the 64 x 64 tiles among them.)
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


# how many tokens each sequence brings, and how many it has cached before them
STEPS = [([1], [0]), ([1, 1, 1], [63, 64, 700]), ([32], [0]), ([33, 8, 200], [0, 5, 64]),
         ([65, 1, 7, 40, 1], [3, 129, 60, 0, 0]), ([7, 2], [0, 1])]


@pytest.mark.parametrize("new,cached", STEPS)
@pytest.mark.parametrize("nh,nkv", [(3, 1), (2, 2)])
@pytest.mark.parametrize("window,extras", [(0, ""), (40, "sink"), (-48, "slope"), (0, "sink,slope")])
def test_attention(ops, new, cached, nh, nkv, window, extras):  # noqa: F811
    cache = ToyCache([c + n for c, n in zip(cached, new)], nkv, 64, torch.float32)
    pos = [c + i for c, n in zip(cached, new) for i in range(n)]
    seq = [b for b, n in enumerate(new) for _ in range(n)]
    as_ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    q = rnd(len(pos), nh * 64 + 4, seed=6)[:, :nh * 64]
    kw = {}
    if "sink" in extras:
        kw["sink"] = rnd(nh, seed=9)
    if "slope" in extras:
        kw["slope"] = torch.tensor([2.0 ** -(h + 1) for h in range(nh)], device=DEV)
    outs = []
    for news in (None, new):
        out = torch.full((len(pos), nh * 64 + 4), 7.0, device=DEV)
        ops.attn_simt(q, out[:, :nh * 64], cache.k, cache.v, cache.table, as_ints(pos), as_ints(seq),
                      cache.seq_slot, nh, nkv, 64, 1.3 / math.sqrt(64), window, 64, news=news, **kw)
        assert bool((out[:, nh * 64:] == 7.0).all())
        outs.append(out[:, :nh * 64])
    # two 32-bit orders of sums of a few hundred terms
    close(outs[1], outs[0], 1e-5)


def test_an_unseen_key_may_hold_anything(ops):  # noqa: F811
    """Later keys of a prompt do not reach earlier rows even where their values are infinite."""
    cache = ToyCache([80], 1, 64, torch.float32)
    blk = int(cache.table_host[cache.slots[0], 1])
    cache.v[blk, 0, 70 - 64] = float("inf")
    pos = torch.arange(80, dtype=torch.int32, device=DEV)
    seq = torch.zeros(80, dtype=torch.int32, device=DEV)
    q, outs = rnd(80, 64, seed=6), []
    for news in (None, [80]):
        out = torch.empty(80, 64, device=DEV)
        ops.attn_simt(q, out, cache.k, cache.v, cache.table, pos, seq, cache.seq_slot, 1, 1, 64,
                      0.125, 0, 64, news=news)
        outs.append(out)
    assert bool(torch.isfinite(outs[1][:70]).all())
    close(outs[1][:70], outs[0][:70], 1e-5)
    assert torch.equal(torch.isinf(outs[1][70:]), torch.isinf(outs[0][70:]))
