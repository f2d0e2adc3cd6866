"""The delta rules in chunks of 32 tokens against the token-by-token formula in 64 bits, at the
edges of a chunk, beside the kernels that walk token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [(1, 31, 32, 33, 0, 95), (200,), (64, 2, 129)]


def _gated(prep, state, lens, slots, H, G, d, e):
    """[T, H e] read-outs and the new states, in float64."""
    P, M = prep.double(), state.double().clone()
    out, at = [], 0
    for n, slot in zip(lens, slots):
        S = M[slot].view(H, d, e)
        for t in range(at, at + n):
            q = P[t, :G * d].view(G, d).repeat_interleave(H // G, 0)
            k = P[t, G * d:2 * G * d].view(G, d).repeat_interleave(H // G, 0)
            v = P[t, 2 * G * d:2 * G * d + H * e].view(H, e)
            beta, g = P[t, -2 * H:-H], P[t, -H:]
            S.mul_(g[:, None, None])
            u = beta[:, None] * (v - torch.einsum("hde,hd->he", S, k))
            S.add_(torch.einsum("hd,he->hde", k, u))
            out.append(torch.einsum("hde,hd->he", S, q).reshape(-1))
        at += n
    return torch.stack(out), M


def _general(proj, prep, state, lens, slots, H, d, e):
    P, Q, M = proj.double(), prep.double(), state.double().clone()
    out, at = [], 0
    for n, slot in zip(lens, slots):
        S = M[slot].view(H, d, e)
        for t in range(at, at + n):
            r, k = P[t, :H * d].view(H, d), P[t, H * d:2 * H * d].view(H, d)
            v = P[t, 2 * H * d:2 * H * d + H * e].view(H, e)
            u, nb, w = (Q[t, i * H * d:(i + 1) * H * d].view(H, d) for i in range(3))
            x = torch.einsum("hde,hd->he", S, u)
            S.mul_(w[..., None]).add_(torch.einsum("hd,he->hde", nb, x)
                                      + torch.einsum("hd,he->hde", k, v))
            out.append(torch.einsum("hde,hd->he", S, r).reshape(-1))
        at += n
    return torch.stack(out), M


def _off(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("general,H,G,d,e", [(False, 4, 2, 64, 16), (False, 2, 2, 128, 48),
                                             (False, 40, 8, 64, 128), (True, 2, 2, 64, 48),
                                             (True, 3, 3, 128, 16), (True, 40, 40, 64, 64)])
def test_chunks_against_the_formula(general, H, G, d, e, lens):
    """Both ways are 32-bit sums of the same terms: the chunks' result may be no further from the
    64-bit one than 1e-6 (16 times 2^-24), and than four times the walk's.  Some decays are 0 or
    tiny (a quotient of cumulated decays would not survive them)."""
    from cretif_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    T, B = sum(lens), len(lens)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def unit(x, heads, width):
        x = x.view(T, heads, width)
        return (x / x.norm(dim=2, keepdim=True)).reshape(T, heads * width)
    decays = torch.rand(T, H * d if general else H, generator=gen, device="cuda") * 0.5 + 0.5
    decays[5::7] = 0.999
    decays[11::23] = 1e-30
    decays[17::29] = 0.0
    slots = list(range(B, 0, -1))
    state = torch.randn(B + 2, H * d * e, generator=gen, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    seq_slot = torch.tensor(slots, **i32)
    gate, norm_w = rand(T, H * e), torch.ones(e, device="cuda")
    if general:
        key = unit(rand(T, H * d), H, d)
        proj = torch.cat([rand(T, H * d), key, rand(T, H * e)], 1)
        prep = torch.cat([key, -torch.rand(T, H * d, generator=gen, device="cuda") * key, decays], 1)
        want, want_state = _general(proj, prep, state, lens, slots, H, d, e)
    else:
        beta = torch.rand(T, H, generator=gen, device="cuda")
        prep = torch.cat([unit(rand(T, G * d), G, d), unit(rand(T, G * d), G, d), rand(T, H * e),
                          beta, decays], 1)
        prep = torch.nn.functional.pad(prep, (0, -prep.shape[1] % 4))[:, :prep.shape[1]]
        want, want_state = _gated(prep, state, lens, slots, H, G, d, e)
    # the gate and the norm after the recurrence are the same kernel on both ways
    w64 = want.view(T, H, e)
    w64 = (w64 / torch.sqrt((w64 * w64).mean(2, keepdim=True) + 1e-5)).reshape(T, H * e)
    w64 = w64 * (torch.sigmoid(gate.double()) if general else
                 gate.double() * torch.sigmoid(gate.double()))
    off = {}
    for longest in (0, 1 << 20):
        mine, out = state.clone(), torch.empty(T, H * e, device="cuda")
        if general:
            ops.general_delta_recurrence(proj, prep, gate, mine, cu, seq_slot, B, H, d, e, norm_w,
                                         1e-5, out, per_head_weight=False, longest=longest)
        else:
            ops.delta_recurrence(prep, gate, mine, cu, seq_slot, B, H, G, d, e, norm_w, 1e-5, out,
                                 longest=longest)
        off[longest] = _off(out, w64), _off(mine, want_state)
        assert torch.equal(mine[0], state[0]) and torch.equal(mine[B + 1], state[B + 1])
    for chunks, walk in zip(off[1 << 20], off[0]):
        assert chunks <= 1e-6 and chunks <= 4 * walk, off
    frozen, out = state.clone(), torch.empty(T, H * e, device="cuda")
    if not general:
        ops.delta_recurrence(prep, gate, frozen, cu, seq_slot, B, H, G, d, e, norm_w, 1e-5, out,
                             write_state=False, longest=1 << 20)
        assert torch.equal(frozen, state) and _off(out, w64) <= 1e-6


def test_small_or_odd_sizes_walk():
    from cretif_b200.csrc import ops
    state = torch.zeros(2, 2 * 64 * 16, device="cuda")
    prep = torch.zeros(70, 2 * 128, device="cuda")
    room = ops._delta_chunk_room
    assert room(70, 70, 2, 64, 16, False, state, (prep,)) is not None
    assert room(ops.DELTA_CHUNKS_FROM - 1, 70, 2, 64, 16, False, state, (prep,)) is None
    assert room(70, 70 * 129, 2, 64, 16, False, state, (prep,)) is None
    assert room(70, 70 * 128, 2, 64, 16, False, state, (prep,)) is not None
    assert room(70, 70, 2, 64, 24, False, state, (prep,)) is None
    assert room(70, 70, 2, 96, 16, False, state, (prep,)) is None
    assert room(70, 70, 2, 64, 16, False, state, (prep[:, 1:],)) is None
    assert room(70, 70, 2, 64, 16, False, state, (torch.zeros(70, 257, device="cuda"),)) is None
    assert room(70, 70, 2, 64, 16, False, state[:, 2:], (prep,)) is None


@pytest.mark.parametrize("general,H,G,d,e", [(False, 16, 8, 128, 32), (True, 9, 9, 64, 64)])
@pytest.mark.parametrize("lens", [(70,) + (1,) * 40, (1,) * 20 + (100, 0, 7, 33) + (3,) * 30])
def test_mixed_steps(general, H, G, d, e, lens):
    """Single tokens beside a prompt are walked, the others go in chunks: the read-outs and states of
    either are, to the bit, those of the whole step walked and of the whole step in chunks."""
    from cretif_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(7)
    T, B = sum(lens), len(lens)
    short = [n < ops.DELTA_WALK_BELOW for n in lens]
    assert ops._delta_short(lens, H) == sum(n for n, s in zip(lens, short) if s)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    decays = torch.rand(T, H * d if general else H, generator=gen, device="cuda")
    start, gate, norm_w = rand(B, H * d * e), rand(T, H * e), torch.ones(e, device="cuda")
    key = rand(T, G * d)
    key = (key.view(T, G, d) / key.view(T, G, d).norm(dim=2, keepdim=True)).reshape(T, G * d)
    if general:
        proj = torch.cat([rand(T, H * d), key, rand(T, H * e)], 1)
        prep = torch.cat([key, -torch.rand(T, H * d, generator=gen, device="cuda") * key, decays], 1)
    else:
        prep = torch.cat([rand(T, G * d), key, rand(T, H * e), decays, decays], 1)
    at = torch.tensor([0] + list(lens)).cumsum(0).tolist()

    cu = torch.tensor(at, dtype=torch.int32, device="cuda")
    slots = torch.arange(B, dtype=torch.int32, device="cuda")

    def step(**kw):
        state, out = start.clone(), torch.empty(T, H * e, device="cuda")
        if general:
            ops.general_delta_recurrence(proj, prep, gate, state, cu, slots, B, H, d, e, norm_w, 1e-5,
                                         out, per_head_weight=False, **kw)
        else:
            ops.delta_recurrence(prep, gate, state, cu, slots, B, H, G, d, e, norm_w, 1e-5, out, **kw)
        return out, state
    walked, chunked = step(longest=1), step(longest=max(lens))
    out, state = step(longest=max(lens), news=lens)
    for b in range(B):
        want = walked if short[b] else chunked
        assert torch.equal(out[at[b]:at[b + 1]], want[0][at[b]:at[b + 1]]), b
        assert torch.equal(state[b], want[1][b]), b
    assert not torch.equal(out, walked[0]) and not torch.equal(out, chunked[0])


@pytest.mark.parametrize("general,H,G,d,e", [(False, 4, 2, 64, 48), (True, 3, 3, 128, 32)])
def test_the_workspace_has_a_bound(monkeypatch, general, H, G, d, e):
    """A step beyond it goes span by span (spans that end inside a chunk, inside a sequence and between
    two), and one that may not write its state between spans, or finds no memory, is walked."""
    from cretif_b200.csrc import ops
    row = int(ops.lib().cretif_delta_chunk_row(16, 128, 128, 1))
    room = ops._delta_chunk_room(2048, 1 << 20, 16, 128, 128, True, torch.empty(1, 4, device="cuda"), ())
    assert 4 * room.numel() <= ops.DELTA_CHUNKS_BYTES and room.numel() >= 2048 * row
    del room
    gen = torch.Generator(device="cuda").manual_seed(9)
    lens = (200, 0, 65, 2, 130)
    T, B = sum(lens), len(lens)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def unit(x, heads):
        x = x.view(T, heads, d)
        return (x / x.norm(dim=2, keepdim=True)).reshape(T, heads * d)
    decays = torch.rand(T, H * d if general else H, generator=gen, device="cuda") * 0.5 + 0.5
    start, gate, norm_w = rand(B, H * d * e), rand(T, H * e), torch.ones(e, device="cuda")
    slots = list(range(B))
    if general:
        key = unit(rand(T, H * d), H)
        proj = torch.cat([rand(T, H * d), key, rand(T, H * e)], 1)
        prep = torch.cat([key, -torch.rand(T, H * d, generator=gen, device="cuda") * key, decays], 1)
        want, want_state = _general(proj, prep, start, lens, slots, H, d, e)
    else:
        prep = torch.cat([unit(rand(T, G * d), G), unit(rand(T, G * d), G), rand(T, H * e),
                          torch.rand(T, H, generator=gen, device="cuda"), decays], 1)
        want, want_state = _gated(prep, start, lens, slots, H, G, d, e)
    w64 = want.view(T, H, e)
    w64 = (w64 / torch.sqrt((w64 * w64).mean(2, keepdim=True) + 1e-5)).reshape(T, H * e)
    w64 = w64 * (torch.sigmoid(gate.double()) if general else
                 gate.double() * torch.sigmoid(gate.double()))
    cu = torch.tensor([0] + list(lens)).cumsum(0).int().cuda()
    seq_slot = torch.tensor(slots, dtype=torch.int32, device="cuda")

    def step(longest, write_state=True):
        state, out = start.clone(), torch.empty(T, H * e, device="cuda")
        if general:
            ops.general_delta_recurrence(proj, prep, gate, state, cu, seq_slot, B, H, d, e, norm_w, 1e-5,
                                         out, per_head_weight=False, longest=longest,
                                         write_state=write_state)
        else:
            ops.delta_recurrence(prep, gate, state, cu, seq_slot, B, H, G, d, e, norm_w, 1e-5, out,
                                 longest=longest, write_state=write_state)
        return out, state
    whole, walked = step(200), step(1)
    row = int(ops.lib().cretif_delta_chunk_row(H, d, e, int(general)))
    for tokens in (32, 96, 100, 265, T - 1):
        monkeypatch.setattr(ops, "DELTA_CHUNKS_BYTES", 4 * row * tokens)
        before = ops.launch_count()
        out, state = step(200)
        assert ops.launch_count() - before == 2 * -(-T // (tokens // 32 * 32)) + 1, tokens
        # (the bounds of test_chunks_against_the_formula)
        assert _off(out, w64) <= 1e-6 and _off(state, want_state) <= 1e-6, tokens
        out, state = step(200, write_state=False)
        assert torch.equal(out, walked[0]) and torch.equal(state, start)
    monkeypatch.setattr(ops, "DELTA_CHUNKS_BYTES", 4 * row * 31)
    assert all(torch.equal(a, b) for a, b in zip(step(200), walked))
    monkeypatch.setattr(ops, "DELTA_CHUNKS_BYTES", 4 * row * T)
    assert all(torch.equal(a, b) for a, b in zip(step(200), whole))
    empty = torch.empty

    def full(*args, **kw):
        if args and args[0] == T * row:
            raise torch.OutOfMemoryError("no room")
        return empty(*args, **kw)
    monkeypatch.setattr(torch, "empty", full)
    assert all(torch.equal(a, b) for a, b in zip(step(200), walked))


@pytest.mark.parametrize("general,H,d,e,lens,chunks", [
    (False, 9, 64, 64, (96,) * 20, True), (False, 9, 64, 64, (96,) * 28, False),
    (True, 9, 64, 64, (96,) * 28, True), (False, 9, 64, 64, (64,) + (48,) * 32, False),
    (False, 9, 64, 64, (64,) + (1,) * 63, True), (False, 16, 128, 32, (64,) * 8, True),
    (False, 16, 128, 32, (64,) * 16, False), (True, 32, 128, 64, (64,) * 64, False),
    (False, 32, 128, 64, (64,) * 64, True), (True, 32, 128, 128, (64,) * 64, True)])
def test_which_steps_go_in_chunks(general, H, d, e, lens, chunks):
    """By the heads that the chunks keep in flight: the walk is as fast or faster beyond."""
    from cretif_b200.csrc import ops
    state, row = torch.zeros(1, 4, device="cuda"), torch.zeros(1, 4, device="cuda")
    short = ops._delta_short(lens, H)
    room = ops._delta_chunk_room(max(lens), sum(lens), H, d, e, general, state, (row,), True,
                                 ops._delta_in_chunks(lens, short))
    assert (room is not None) == chunks


@pytest.mark.parametrize("general,H,G", [(False, 16, 4), (True, 16, 16)])
@pytest.mark.parametrize("lens,slices", [((70, 0, 33, 96, 1, 40), 32), ((200, 95), 16)])
def test_slices_of_columns(general, H, G, lens, slices):
    """Heads of 128 x 128 in both widths of a slice (32 columns from two CTAs an SM on), a short last
    chunk and an empty sequence among them."""
    from cretif_b200.csrc import ops
    before = ops.variant_counts()
    test_chunks_against_the_formula(general, H, G, 128, 128, lens)
    after = ops.variant_counts()
    assert {k for k in after if k.startswith("delta_slices") and after[k] != before[k]} \
        == {"delta_slices%d" % slices}


@pytest.mark.parametrize("general,H,G,d,e", [(False, 8, 4, 128, 64), (False, 9, 9, 64, 64),
                                             (True, 8, 8, 128, 64)])
@pytest.mark.parametrize("T", [64, 300])
def test_chunks_are_as_exact_as_the_walk(general, H, G, d, e, T):
    """Both round the same terms to 32 bits; the 2-norms are over 20,000 numbers and more, so that two
    orders of like exactness differ by a few parts in a hundred."""
    from cretif_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(2)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device="cuda")

    def unit(x, heads):
        x = x.view(T, heads, d)
        return (x / x.norm(dim=2, keepdim=True)).reshape(T, heads * d)
    decays = torch.exp(-0.2 * uniform(T, H * d if general else H))
    start, gate, norm_w = torch.zeros(1, H * d * e, device="cuda"), rand(T, H * e), torch.ones(e, device="cuda")
    if general:
        key = unit(rand(T, H * d), H)
        proj = torch.cat([rand(T, H * d), key, rand(T, H * e)], 1)
        prep = torch.cat([key, -uniform(T, H * d) * key, decays], 1)
        want, want_state = _general(proj, prep, start, [T], [0], H, d, e)
    else:
        prep = torch.cat([unit(rand(T, G * d), G), unit(rand(T, G * d), G), rand(T, H * e), uniform(T, H),
                          decays], 1)
        prep = torch.nn.functional.pad(prep, (0, -prep.shape[1] % 4))[:, :prep.shape[1]]
        want, want_state = _gated(prep, start, [T], [0], H, G, d, e)
    w64 = want.view(T, H, e)
    w64 = (w64 / torch.sqrt((w64 * w64).mean(2, keepdim=True) + 1e-5)).reshape(T, H * e)
    w64 = w64 * (torch.sigmoid(gate.double()) if general else
                 gate.double() * torch.sigmoid(gate.double()))
    cu = torch.tensor([0, T], dtype=torch.int32, device="cuda")
    slot = torch.zeros(1, dtype=torch.int32, device="cuda")
    off = {}
    for longest in (1, T):
        state, out = start.clone(), torch.empty(T, H * e, device="cuda")
        if general:
            ops.general_delta_recurrence(proj, prep, gate, state, cu, slot, 1, H, d, e, norm_w, 1e-5, out,
                                         per_head_weight=False, longest=longest)
        else:
            ops.delta_recurrence(prep, gate, state, cu, slot, 1, H, G, d, e, norm_w, 1e-5, out,
                                 longest=longest)
        off[longest] = _off(out, w64), _off(state, want_state)
    for chunks, walk in zip(off[T], off[1]):
        assert chunks <= 1.25 * walk, off
