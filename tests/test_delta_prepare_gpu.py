"""The gated delta rule's preparation of prompts, eight tokens a warp, against the formula in 64 bits:
sequences that begin inside a group of eight, shorter than the taps, and that go on from saved
inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,d,e", [(2, 1, 64, 48), (3, 3, 128, 128), (4, 2, 20, 260)])
@pytest.mark.parametrize("lens", [(1, 2, 3, 300, 4, 11), (257,), (248, 9)])
def test_prompt_rows(H, G, d, e, lens):
    """Three roundings a tap and the exponential's two units: 1e-6 of the result's 2-norm."""
    from cretif_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(6)
    T, B, C = sum(lens), len(lens), 2 * G * d + H * e
    ld = -(-(C + H * e + 2 * H) // 4) * 4

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    proj, conv_w, a_log, dt_bias = rand(T, ld), rand(C, 4) * 0.5, rand(H), rand(H)
    saved = rand(B + 1, C * 3)
    i32 = dict(dtype=torch.int32, device="cuda")
    slots = torch.arange(B, 0, -1, **i32)
    starts = torch.tensor([7 * i for i in range(B)], **i32)
    seq = torch.repeat_interleave(torch.arange(B, **i32), torch.tensor(lens, device="cuda")).int()
    pos = torch.cat([torch.arange(n, **i32) + 7 * i for i, n in enumerate(lens)])
    ldo = -(-(C + 2 * H) // 4) * 4
    prep = torch.empty(T, ldo, device="cuda")[:, :C + 2 * H]
    ops.delta_prepare(proj, prep, conv_w, saved, a_log, dt_bias, pos, seq, slots, starts, H, G, d,
                      e, 1e-6)
    P, at, want = proj.double(), 0, []
    for i, n in enumerate(lens):
        before = saved[int(slots[i])].double().view(C, 3).T
        x = torch.cat([before, P[at:at + n, :C]])
        conv = sum(x[k:k + n] * conv_w[:, k].double() for k in range(4))
        conv = conv * torch.sigmoid(conv)
        heads = conv[:, :2 * G * d].view(n, 2 * G, d)
        heads = heads / torch.sqrt((heads * heads).sum(2, keepdim=True) + 1e-6)
        heads[:, :G] *= d ** -0.5
        beta = torch.sigmoid(P[at:at + n, C + H * e:C + H * e + H])
        g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(
            P[at:at + n, C + H * e + H:C + H * e + 2 * H] + dt_bias.double()))
        want.append(torch.cat([heads.reshape(n, -1), conv[:, 2 * G * d:], beta, g], 1))
        at += n
    want = torch.cat(want)
    for a, b in ((0, 2 * G * d), (2 * G * d, C), (C, C + H), (C + H, C + 2 * H)):
        off = (prep[:, a:b].double() - want[:, a:b]).norm() / want[:, a:b].norm()
        assert off <= 1e-6, (a, float(off))


@pytest.mark.parametrize("H,G,d,e", [(2, 1, 96, 72), (1, 1, 68, 260), (5, 5, 128, 128)])
@pytest.mark.parametrize("lens", [(1, 2, 3, 300, 4, 11), (257,), (248, 9)])
def test_prompt_rows_of_wide_heads(H, G, d, e, lens):
    """The sizes that go eight tokens a warp, odd ones among them; see above."""
    from cretif_b200.csrc import ops
    before = ops.variant_counts()["delta_prepare_rows"]
    test_prompt_rows(H, G, d, e, lens)
    assert ops.variant_counts()["delta_prepare_rows"] == before + 1


@pytest.mark.parametrize("H,G,d,e", [(4, 4, 64, 64), (2, 1, 64, 128), (2, 1, 128, 64)])
def test_narrow_heads_keep_a_warp_a_token(H, G, d, e):
    """Heads of 64 leave half of the lanes idle that take eight tokens in turn."""
    from cretif_b200.csrc import ops
    before = ops.variant_counts()["delta_prepare_rows"]
    test_prompt_rows(H, G, d, e, (260,))
    assert ops.variant_counts()["delta_prepare_rows"] == before
