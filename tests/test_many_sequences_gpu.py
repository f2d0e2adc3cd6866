"""Steps of more sequences than a grid's second and third dimension take (65,535)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

B = 65537
I32 = dict(dtype=torch.int32, device="cuda")


def _rand(*shape, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=gen, device="cuda")


def test_mamba_chunks():
    """A token a sequence, by chunks and token by token: the same 32-bit terms, sums of at most
    four of them, then a norm."""
    from cretif_b200.csrc import ops
    H, G, N, e, taps = 1, 1, 4, 16, 2
    C = H * e + 2 * G * N
    proj = _rand(B, -(-(H * e + C + H) // 4) * 4)
    conv_w, conv_b = _rand(taps, C, seed=1), _rand(C, seed=2)
    start = _rand(B, H * N * e + C * (taps - 1), seed=3)
    every = torch.arange(B, **I32)
    cu = torch.arange(B + 1, **I32)
    got = []
    for form in ("chunk", "token"):
        state, out = start.clone(), torch.empty(B, H * e, device="cuda")
        ops.state_space(proj, conv_w, conv_b, torch.zeros(H, device="cuda"),
                        torch.zeros(H, device="cuda"), torch.ones(H, device="cuda"), state, H * N * e,
                        cu, every, every, B, H, G, N, e, 1, torch.ones(H * e, device="cuda"), 1e-5,
                        out, save_inputs=True, form=form)
        got.append((out, state))
    for a, b in zip(*got):
        assert (a - b).norm() <= 1e-6 * b.norm()


def test_delta_chunks():
    """A token a sequence, through the chunk kernels and token by token, the gated rule."""
    from cretif_b200.csrc import ops
    H, d, e = 1, 64, 16
    prep = _rand(B, 148)[:, :2 * d + e + 2]
    prep[:, -2:] = torch.sigmoid(prep[:, -2:])
    start, gate = _rand(B, d * e, seed=3), _rand(B, e, seed=4)
    every = torch.arange(B, **I32)
    cu = torch.arange(B + 1, **I32)
    got = []
    for longest in (1 << 20, 1):
        state, out = start.clone(), torch.empty(B, e, device="cuda")
        ops.delta_recurrence(prep, gate, state, cu, every, B, H, 1, d, e, torch.ones(e, device="cuda"),
                             1e-5, out, longest=longest)
        got.append((out, state))
    for a, b in zip(*got):
        assert (a - b).norm() <= 1e-6 * b.norm()


def test_matrix_memory_chunks(monkeypatch):
    """A token a sequence, in chunks although a scan is asked for, and token by token.  A read-out is normed
    and a small one is normed up with its rounding: 1e-4 of the 2-norm."""
    from cretif_b200.csrc import ops
    monkeypatch.setattr(ops, "memory_scans", lambda *_: True)
    H, d, e = 1, 4, 16
    proj = _rand(B, 2 * H * (d + e) + 4)
    start = _rand(B, H * d * (e + 1) + 4, seed=3).abs()
    every = torch.arange(B, **I32)
    cu = torch.arange(B + 1, **I32)
    zero = torch.zeros(H, device="cuda")
    got = []
    for form in ("chunk", "token"):
        state, out = start.clone(), torch.empty(B, H * e, device="cuda")
        ops.matrix_memory(proj, zero, zero, 10.0, 0.5, state, cu, every, every, B, H, d, e,
                          torch.ones(H * e, device="cuda"), 1e-5, out, form=form)
        got.append((out, state))
    for (a, b), bound in zip(zip(*got), (1e-4, 1e-6)):
        assert (a - b).norm() <= bound * b.norm()
