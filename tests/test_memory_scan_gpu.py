"""The matrix memory's chunks scanned against chunks walked: the same sums of the same terms in
another order, over lengths at the edges of a chunk and beyond the scan's 64 chunks at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,e,lens", [(2, 64, 64, (64 * 66 + 5, 1, 64, 63)), (3, 20, 48, (65, 700)),
                                        (1, 256, 80, (129, 128)), (9, 128, 128, (40, 24, 200))])
@pytest.mark.parametrize("write_state", [True, False])
def test_scan_and_walk(H, d, e, lens, write_state):
    """Read-outs are normed, so they are compared by their 2-norm (both forms sum in 32 bits:
    2^-24 times the square root of the terms, a thousand at most, and the norm's gain); states by
    theirs."""
    from cretif_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(4)
    T, B, width = sum(lens), len(lens), -(-(2 * H * (d + e) + 2 * H) // 4) * 4
    proj = torch.randn(T, width, generator=gen, device="cuda")
    proj[:, -2 * H:] *= 3.0
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    seq = torch.repeat_interleave(torch.arange(B, **i32), torch.tensor(lens, device="cuda")).int()
    slots = torch.arange(B, 0, -1, **i32)
    bias, norm_w = torch.zeros(H, device="cuda"), torch.ones(H * e, device="cuda")
    start = torch.randn(B + 2, -(-(H * (d * (e + 1) + 1)) // 4) * 4, generator=gen, device="cuda")
    outs, states = [], []
    for form in ("walk", "chunk"):
        state, out = start.clone(), torch.empty(T, H * e, device="cuda")
        kept, ops.memory_scans = ops.memory_scans, lambda *_: True
        try:
            ops.matrix_memory(proj, bias, bias, 12.0, d ** -0.5, state, cu, slots, seq, B, H, d, e,
                              norm_w, 1e-6, out, write_state=write_state, form=form)
        finally:
            ops.memory_scans = kept
        outs.append(out.double())
        states.append(state.double())
        assert torch.equal(state[0], start[0]) and torch.equal(state[B + 1], start[B + 1])
    assert bool(torch.isfinite(outs[0]).all())
    assert (outs[0] - outs[1]).norm() <= 1e-4 * outs[0].norm()
    assert (states[0] - states[1]).norm() <= 2e-6 * states[0].norm()


def test_a_step_beyond_the_workspace_walks(monkeypatch):
    """The scan's workspace has a bound, and a step that finds no memory for it still runs: by the
    bits of the walk."""
    from cretif_b200.csrc import ops
    H, d, e, T = 2, 64, 64, 700
    room = ops._memory_scan_room(T, 1, H, d, e, "cuda")
    assert room is not None and 4 * room.numel() <= ops.MEMORY_SCAN_BYTES
    assert ops._memory_scan_room(1 << 20, 1, 16, 128, 128, "cuda") is None     # 17 GB
    gen = torch.Generator(device="cuda").manual_seed(5)
    proj = torch.randn(T, 2 * H * (d + e) + 2 * H, generator=gen, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    zero = torch.zeros(H, device="cuda")

    def run(form):
        state, out = torch.zeros(1, H * (d * (e + 1) + 1) + 2, device="cuda"), \
            torch.empty(T, H * e, device="cuda")
        ops.matrix_memory(proj, zero, zero, 12.0, 0.1, state, torch.tensor([0, T], **i32),
                          torch.zeros(1, **i32), torch.zeros(T, **i32), 1, H, d, e,
                          torch.ones(H * e, device="cuda"), 1e-6, out, form=form)
        return out, state
    walked = run("walk")
    assert not torch.equal(run("auto")[0], walked[0])          # (scanned)
    monkeypatch.setattr(ops, "MEMORY_SCAN_BYTES", 4 * room.numel() - 4)
    assert all(torch.equal(a, b) for a, b in zip(run("auto"), walked))
    monkeypatch.undo()
    empty = torch.empty

    def full(*args, **kw):
        if args and args[0] == room.numel():
            raise torch.OutOfMemoryError("no room")
        return empty(*args, **kw)
    monkeypatch.setattr(torch, "empty", full)
    assert all(torch.equal(a, b) for a, b in zip(run("auto"), walked))


@pytest.mark.parametrize("H,d,e,lens", [(2, 64, 64, (600,)), (1, 128, 48, (320, 300)), (3, 20, 32, (777,))])
@pytest.mark.parametrize("strong", [False, True])
def test_scan_and_walk_against_64_bits(H, d, e, lens, strong):
    """Both forms beside the recurrence written out in 64 bits: the scan may be no further from it than
    the walk by more than half (each is one draw of the same rounding), and neither than 1e-5 of the
    read-outs' 2-norm: 2^-24 times the square root of some hundred terms, normed up where a read-out is a
    small difference of large ones."""
    import plain_gibipel as plain
    from cretif_b200.csrc import ops
    from test_gibipel_gpu import _gates
    gen = torch.Generator().manual_seed(12)
    T, B, cap, qs = sum(lens), len(lens), 10.0, d ** -0.5
    assert ops.memory_scans(T, B, H)
    parts, want = [], []
    for n in lens:
        q, k, v = (torch.randn(n, H * x, generator=gen) for x in (d, d, e))
        gate = torch.randn(n, H * e, generator=gen)
        zi, zf = _gates(gen, n, H, strong)
        parts.append(torch.cat([q, k, v, gate, zi, zf], 1))
        li = cap * torch.tanh(zi.double() / cap)
        lf = plain.log_sigmoid(cap * torch.tanh(zf.double() / cap))
        o = plain.memory(q.double().reshape(n, H, d) * qs, k.double().reshape(n, H, d),
                         v.double().reshape(n, H, e), li, lf)
        want.append(plain.unit(o, 1e-5).reshape(n, H * e) * torch.sigmoid(gate.double()))
    proj, want = torch.cat(parts), torch.cat(want)
    proj = torch.nn.functional.pad(proj, (0, -proj.shape[1] % 4)).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = torch.tensor([0] + list(lens)).cumsum(0).int().cuda()
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).int().cuda()
    zero, off = torch.zeros(H, device="cuda"), {}
    for form in ("walk", "chunk", "token"):
        state = torch.zeros(B, -(-(H * (d * (e + 1) + 1)) // 4) * 4, device="cuda")
        out = torch.empty(T, H * e, device="cuda")
        ops.matrix_memory(proj, zero, zero, cap, qs, state, cu, torch.arange(B, **i32), seq, B, H, d, e,
                          torch.ones(H * e, device="cuda"), 1e-5, out, form=form)
        off[form] = float((out.cpu().double() - want).norm() / want.norm())
    print(off)
    assert off["chunk"] <= 1.5 * max(off["walk"], off["token"]) and max(off.values()) <= 1e-5, off


@pytest.mark.parametrize("d", [364, 368, 372])
def test_the_widest_heads_in_chunks(d):
    """Heads whose chunk fills the shared memory that the kernels take are not refused: chunks beside token
    by token (read-outs by their 2-norm, as above)."""
    from cretif_b200.csrc import ops
    H, e, T = 1, 16, 300
    gen = torch.Generator(device="cuda").manual_seed(6)
    proj = torch.randn(T, -(-(2 * H * (d + e) + 2 * H) // 4) * 4, generator=gen, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    zero, got = torch.zeros(H, device="cuda"), []
    for form in ("chunk", "walk", "token"):
        state = torch.zeros(1, -(-(H * (d * (e + 1) + 1)) // 4) * 4, device="cuda")
        out = torch.empty(T, H * e, device="cuda")
        ops.matrix_memory(proj, zero, zero, 12.0, d ** -0.5, state, torch.tensor([0, T], **i32),
                          torch.zeros(1, **i32), torch.zeros(T, **i32), 1, H, d, e,
                          torch.ones(H * e, device="cuda"), 1e-6, out, form=form)
        got.append((out, state))
    for out, state in got[:2]:
        assert (out - got[2][0]).norm() <= 1e-4 * out.norm()
        assert (state - got[2][1]).norm() <= 2e-6 * state.norm()
