"""The 32-bit product and the attention of heads of 64: a row's bits do not depend on what else is in
the call, whichever of the fast bodies takes it, and the result is the 64-bit one within 32 bits."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, ToyCache, close, ops, rnd  # noqa: F401

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


# every body at remainders in rows, columns and k, with strided rows and added onto what is there
@pytest.mark.parametrize("M,N,K,body", [
    (1, 577, 260, "few"), (2, 70, 2052, "few"), (3, 3081, 36, "few"), (5, 333, 8196, "few"),
    (8, 9001, 132, "few"), (33, 577, 1540, "few"), (64, 130, 36, "few"),
    (65, 577, 576, "tile32"), (24, 20001, 36, "tile32"), (130, 333, 8196, "tile32"), (577, 2305, 260, "tile32"),
    (580, 2605, 260, "tile64"), (580, 2605, 36, "tile64"), (580, 2605, 4, "tile64"),
    (1153, 1665, 2052, "tile64")])
def test_product_bodies(ops, M, N, K, body):  # noqa: F811
    a = rnd(M, K + 4)[:, :K]
    w = rnd(N, K, seed=1)
    c = torch.full((M, N + 3), 7.0, device=DEV)
    before = ops.variant_counts()
    ops.gemm_simt(a, w, c[:, :N])
    after = ops.variant_counts()
    assert {k for k in after if after[k] != before[k]} == {"f32_" + body}
    want = a.double() @ w.double().T
    close(c[:, :N], want, 2e-6)
    assert bool((c[:, N:] == 7.0).all())
    ops.gemm_simt(a, w, c[:, :N], accumulate=True)
    close(c[:, :N], 2 * want, 2e-6)
    # 2-norm: a slab's two chains of 16, their sum and K / 128 slabs four times over, each rounding to
    # 2^-24 of a partial sum, random in sign
    plain = torch.empty(M, N, device=DEV)
    ops.gemm_simt(a, w, c[:, :N])
    ops.gemm_simt(a, w, plain, plain=True)
    off, plain_off = (float((x.double() - want).norm() / want.norm()) for x in (c[:, :N], plain))
    assert off <= 2.0 ** -24 * (16 + 4 + K / 128) ** 0.5 + 1e-8, (off, plain_off)


@pytest.mark.parametrize("M", [1, 8, 33])
def test_a_vocabulary_of_262144(ops, M):  # noqa: F811
    """More columns than four times a grid's second dimension still take the fast bodies: their bits, by
    a smaller matrix of some of the rows, which are not those of the kernel that takes every shape."""
    N, K = 262144, 96
    a, w = rnd(M, K), rnd(N, K, seed=1)
    c, part, plain = (torch.empty(M, n, device=DEV) for n in (N, 1000, 1000))
    ops.gemm_simt(a, w, c)
    ops.gemm_simt(a, w[-1000:], part)
    ops.gemm_simt(a, w[-1000:], plain, plain=True)
    assert torch.equal(c[:, -1000:], part) and not torch.equal(part, plain)
    close(c[:, :1000], a.double() @ w[:1000].double().T, 2e-6)


@pytest.mark.parametrize("M", [3, 70])
def test_the_plain_product_can_be_chosen(ops, M):  # noqa: F811
    """With the plain kernels forced, float32 rows that a fast body would take go to the kernel that
    takes every shape as well: the bits of the same numbers in rows that no fast body takes."""
    from cretif_b200.parts.linear import force_plain_kernels, linear
    a, w = rnd(M, 576), rnd(200, 576, seed=1)
    odd = torch.empty(200, 577, device=DEV)[:, :576]
    odd.copy_(w)
    want = linear(a, odd)
    fast = linear(a, w)
    force_plain_kernels(True)
    try:
        plain = linear(a, w)
    finally:
        force_plain_kernels(False)
    assert torch.equal(plain, want) and not torch.equal(fast, want)
    close(fast, want, 2e-6)


def _attend(ops, cache, new, cached, qs, nh, nkv, window, kw, use=None):  # noqa: F811
    """Rows of the sequences ``use`` (all by default) in one step; a sequence's queries are
    qs[b][cached .. cached + new - 1]."""
    use = list(range(len(new))) if use is None else use
    as_ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos = [cached[b] + i for b in use for i in range(new[b])]
    seq = [i for i, b in enumerate(use) for _ in range(new[b])]
    q = torch.cat([qs[b][cached[b]:cached[b] + new[b]] for b in use])
    out = torch.empty_like(q)
    ops.attn_simt(q, out, cache.k, cache.v, cache.table, as_ints(pos), as_ints(seq),
                  cache.seq_slot[use].contiguous(), nh, nkv, 64, 0.17, window, 64,
                  news=[new[b] for b in use], **kw)
    return list(out.split([new[b] for b in use]))


@pytest.mark.parametrize("nh,nkv", [(3, 1), (2, 2)])
@pytest.mark.parametrize("window,extras", [(0, ""), (40, "sink"), (-48, "slope"), (0, "sink,slope")])
def test_a_token_of_the_attention_does_not_depend_on_the_step(ops, nh, nkv, window, extras):  # noqa: F811
    """Prompts in one step, each alone, in cuts, token by token, and single tokens beside a prompt."""
    lens = [200, 37, 5, 130]
    cache = ToyCache(lens, nkv, 64, torch.float32)
    qs = [rnd(n, nh * 64, seed=20 + b, scale=3.0) for b, n in enumerate(lens)]
    kw = {}
    if "sink" in extras:
        kw["sink"] = rnd(nh, seed=9)
    if "slope" in extras:
        kw["slope"] = torch.tensor([2.0 ** -(h + 1) for h in range(nh)], device=DEV)
    none = [0] * len(lens)
    whole = _attend(ops, cache, lens, none, qs, nh, nkv, window, kw)
    for b, n in enumerate(lens):
        alone = _attend(ops, cache, lens, none, qs, nh, nkv, window, kw, use=[b])[0]
        assert torch.equal(alone, whole[b])
    for cut in (1, 8, 33, 64):
        first = [min(n, cut) for n in lens]
        rest = [n - f for n, f in zip(lens, first)]
        left = [b for b, r in enumerate(rest) if r]
        for part, at, use in ((first, none, None), (rest, first, left)):
            got = _attend(ops, cache, part, at, qs, nh, nkv, window, kw, use=use)
            for g, b in zip(got, use or range(len(lens))):
                assert torch.equal(g, whole[b][at[b]:at[b] + part[b]]), (cut, b)
    for i in range(0, lens[1], 3):                # one token each, and single ones beside a prompt
        at = [min(i * 5, n - 1) for n in lens]
        ones = _attend(ops, cache, [1] * 4, at, qs, nh, nkv, window, kw)
        for b in range(4):
            assert torch.equal(ones[b][0], whole[b][at[b]])
        mixed = _attend(ops, cache, [lens[0], 1, 1, 1], [0] + at[1:], qs, nh, nkv, window, kw)
        assert torch.equal(mixed[0], whole[0])
        for b in (1, 2, 3):
            assert torch.equal(mixed[b][0], whole[b][at[b]])


@pytest.mark.parametrize("new,cached", [([1, 1], [2047, 2100]), ([1], [9000]), ([300], [0]),
                                        ([40, 1], [5000, 63]), ([2500], [0])])
@pytest.mark.parametrize("sharp", [1.0, 8.0, 1e4])
def test_attention_against_64_bits(ops, new, cached, sharp):  # noqa: F811
    """Contexts past the tiles whose sums the decode body keeps (2,048 keys).  A score is a sum of 64
    products: 2^-24 sqrt(64) of its terms, at most 6e-7 of the largest score, and so much may every
    probability be off; the sums add a few units of the last place."""
    nh, nkv = 3, 1
    lens = [c + n for c, n in zip(cached, new)]
    cache = ToyCache(lens, nkv, 64, torch.float32)
    qs = [rnd(n, nh * 64, seed=30 + b, scale=sharp) for b, n in enumerate(lens)]
    got = torch.cat(_attend(ops, cache, new, cached, qs, nh, nkv, 0, {}))
    want, most = [], 0.0
    for b, n in enumerate(lens):
        blocks = cache.table_host[cache.slots[b], :-(-n // 64)]
        k, v = (x[torch.as_tensor(blocks).long()].permute(1, 0, 2, 3).reshape(64 * len(blocks), 64)[:n]
                .double() for x in (cache.k, cache.v))
        q = qs[b][cached[b]:].double().view(new[b], nh, 64)
        s = torch.einsum("thd,kd->thk", q, k) * 0.17
        ahead = torch.arange(n, device=DEV)[None] > torch.arange(cached[b], n, device=DEV)[:, None]
        s = s.masked_fill(ahead[:, None], -math.inf)
        most = max(most, float((torch.einsum("thd,kd->thk", q.abs(), k.abs()) * 0.17).max()))
        want.append(torch.einsum("thk,kd->thd", torch.softmax(s, -1), v).reshape(new[b], -1))
    want = torch.cat(want)
    off = float((got.double() - want).norm() / want.norm())
    assert off <= 1e-6 + 8 * 2.0 ** -24 * most, off


def test_scores_without_bounds(ops):  # noqa: F811
    """Scores of 1e30 and minus infinity: the largest key's value, and no number where one is none."""
    cache = ToyCache([100, 100, 100], 1, 64, torch.float32)
    as_ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    row = lambda b, i: (int(cache.table_host[cache.slots[b], i // 64]), 0, i % 64)  # noqa: E731
    q = torch.zeros(3, 64, device=DEV)
    q[:, 0] = 1e15
    for b in range(3):
        for i in range(100):
            cache.k[row(b, i)][0] = -1e15
    cache.k[row(0, 70)][0] = 1e15                  # one key far above the others
    cache.k[row(1, 3)][0] = -math.inf              # ... one that is seen and weighs nothing
    cache.k[row(2, 5)][0] = math.nan
    outs = []
    for new in ([1, 1, 1], None):
        out = torch.empty(3, 64, device=DEV)
        if new:
            ops.attn_simt(q, out, cache.k, cache.v, cache.table, as_ints([99] * 3), as_ints([0, 1, 2]),
                          cache.seq_slot, 1, 1, 64, 1.0, 0, 64, news=new)
        else:                                      # the prompt body: eight rows of each
            wide = q.repeat_interleave(8, 0)
            pos = [92 + i for _ in range(3) for i in range(8)]
            full = torch.empty(24, 64, device=DEV)
            ops.attn_simt(wide, full, cache.k, cache.v, cache.table, as_ints(pos),
                          as_ints([i // 8 for i in range(24)]), cache.seq_slot, 1, 1, 64, 1.0, 0, 64,
                          news=[8, 8, 8])
            out = full[7::8]
        outs.append(out)
        close(out[0], cache.v[row(0, 70)], 1e-6)
        others = torch.stack([cache.v[row(1, i)] for i in range(100) if i != 3]).double().mean(0)
        close(out[1], others, 2e-6)
        assert bool(torch.isnan(out[2]).all())
    assert torch.equal(outs[0][:2], outs[1][:2])


def test_logits_of_small_steps_do_not_depend_on_the_cut(tmp_path):
    """A whole float32 model with heads of 64: a prompt alone, beside others, in two cuts and token by token
    gives the same bits, as long as its steps bring fewer than 64 tokens (from there on the norms sum a
    row in another order)."""
    from cretif_b200.engine import Engine
    from cretif_b200.weights.random_model import write_random_model
    config = {"architectures": ["LlamaForCausalLM"], "hidden_size": 192, "num_hidden_layers": 2,
              "num_attention_heads": 3, "num_key_value_heads": 1, "intermediate_size": 320,
              "vocab_size": 500, "rope_theta": 10000.0, "rms_norm_eps": 1e-5,
              "tie_word_embeddings": True, "max_position_embeddings": 256}
    write_random_model(str(tmp_path), config, seed=4)
    engine = Engine(str(tmp_path), dtype="float32", max_tokens=1024, step_graphs=False)
    gen = torch.Generator().manual_seed(3)
    texts = [torch.randint(500, (n,), generator=gen).tolist() for n in (31, 5, 20)]

    def logits(cuts):
        """Logits [sum of the first text's tokens] of a list of steps, each {text: tokens it brings}."""
        slots, at, rows = {}, {}, []
        for step in cuts:
            for b in step:
                if b not in slots:
                    slots[b], at[b] = engine.alloc_slot(), 0
            entries = [(slots[b], texts[b][at[b]:at[b] + n]) for b, n in step.items()]
            out, first = engine.step(entries, "all"), 0
            for b, n in step.items():
                if b == 0:
                    rows.append(out[first:first + n])
                first += n
                at[b] += n
        for s in slots.values():
            engine.free_slot(s)
        return torch.cat(rows)
    alone = logits([{0: 31}])
    for cuts in ([{1: 5, 0: 31, 2: 20}], [{0: 13, 2: 20}, {0: 18}], [{0: 30, 1: 5}, {2: 20, 0: 1}],
                 [{2: 20}] + [{0: 1}] * 31, [{1: 1, 0: 1} for _ in range(5)] + [{0: 26}]):
        assert torch.equal(logits(cuts), alone), cuts
