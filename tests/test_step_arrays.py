"""What the decode attention reads ahead of the kernels launched before it comes from the host."""
import types

import pytest
import torch


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 32), (16, 1, 64), (32, 1, 128), (11, 1, 64)])
def test_decode_attention_gets_the_steps_own_arrays(monkeypatch, nh, nkv, hd):
    """The kernel asks for positions, sequences, slots and the block table before it waits for the kernel
    before it: arrays that a kernel of the same step makes (a copy per group of heads) may still be on
    their way then."""
    from cretif_b200.csrc import ops
    from cretif_b200.parts.attention import run_attention
    seen = []

    def attn_decode(q, out, kc, vc, table, tok_pos, tok_seq, seq_slot, *rest, **more):
        seen.append((table, tok_pos, tok_seq, seq_slot, q.shape[0]))
    monkeypatch.setattr(ops, "attn_decode", attn_decode)
    monkeypatch.setattr(ops, "decode_plan", lambda *a, **k: (1, True))
    B = 3
    arrays = {k: torch.arange(B, dtype=torch.int32) for k in ("tok_pos", "tok_seq", "seq_slot")}
    ctx = types.SimpleNamespace(T=B, B=B, is_decode=True, max_context=64, fault=None, extras={}, **arrays)
    cache = torch.zeros(4, nkv, 64, hd, dtype=torch.bfloat16)
    kv = types.SimpleNamespace(k=cache, v=cache, table=torch.zeros(B, 1, dtype=torch.int32), block_tokens=64)
    q = torch.zeros(B, nh * hd, dtype=torch.bfloat16)
    run_attention(q, torch.empty_like(q), ctx, kv, nh, nkv, hd, 1.0, 0, torch.bfloat16)
    assert seen
    for table, pos, seq, slot, items in seen:
        assert table is kv.table and slot is ctx.seq_slot
        assert pos is ctx.tok_pos and seq is ctx.tok_seq
        assert items % B == 0
