"""As test_dependent_launch_gpu, at the layer sizes of the benchmark: products of 576, 768, 960, 1,536,
2,048 and 8,192 columns, whose bodies (weights held in registers, streamed through a ring) hold back the
kernels behind them by different amounts, and groups of heads on one cached latent."""
import pytest
import torch

import bench

pytestmark = pytest.mark.gpu

MIXED = {"rigozen": (bench.design_configs, "rigozen mixed"),
         "losorax": (bench.losorax_configs, "losorax mixed routed"),
         "virorax": (bench.virorax_configs, "virorax mixed, a span twice"),
         "mipurax": (bench.mipurax_configs, "mipurax mixed routed"),
         "gibipel": (bench.gibipel_configs, "gibipel routed"),
         "pudorax": (bench.pudorax_configs, "pudorax mixed looped")}
# layers without a fixed-size kernel between the latent's: the longest chain of early starts
LATENT = (bench.design_configs, "rigozen latent_attention")


def _config(model):
    name, size = model.rsplit("-", 1)
    if name == "llama":                    # width-feed-forward-heads-kv of a SmolLM2 size, two layers
        from cretif_b200.config import preset
        return {**preset("smollm2-" + size), "num_hidden_layers": 2, "vocab_size": 512}
    z = dict(bench.DESIGN_SIZES[size], vocab=512, experts=8, top=2)
    make, which = LATENT if name == "latent" else MIXED[name]
    configs = make(z, 4)
    return configs[which]


def _replay(engine, vocab, rows):
    gen = torch.Generator().manual_seed(rows)
    slots = [engine.alloc_slot() for _ in range(rows)]
    news = [1500 if rows == 1 else 100 + 37 * (b % 5) for b in range(rows)]
    prompts = [torch.randint(vocab, (n,), generator=gen).tolist() for n in news]
    out = [engine.step(list(zip(slots, prompts)))]
    for _ in range(40):
        fed = torch.randint(vocab, (rows, 1), generator=gen).tolist()
        out.append(engine.step(list(zip(slots, fed))))
    for s in slots:
        engine.free_slot(s)
    return torch.cat(out)


@pytest.mark.parametrize("model", ["llama-135m", "llama-360m", "llama-1.7b", "latent-m"]
                         + [f"{name}-{size}" for name in MIXED for size in "sm"])
def test_same_bits_with_and_without(tmp_path, model):
    """The same kernels on the same operands, so the same bits, whatever starts early: launched one by
    one and replayed, 1 to 16 rows a step, forty steps (a kernel that reads ahead of what it needs shows
    in replays, where nothing keeps the launches apart)."""
    from cretif_b200.csrc import ops
    from cretif_b200.engine import Engine
    from cretif_b200.weights.random_model import write_random_model
    cfg = _config(model)
    vocab = cfg.get("vocab", 512)
    write_random_model(str(tmp_path), cfg, seed=4)
    got = {}
    for on, graphs in ((False, True), (True, False), (True, True)):
        was = ops.set_dependent_launch(on)
        try:
            engine = Engine(str(tmp_path), dtype="bfloat16", max_tokens=16 * 384, max_slots=16,
                            step_graphs=graphs)
            got[on, graphs] = {rows: _replay(engine, vocab, rows) for rows in (1, 2, 3, 8, 9, 16)}
            del engine
        finally:
            ops.set_dependent_launch(was)
    for rows, want in got[False, True].items():
        assert bool(torch.isfinite(want).all())
        for how in ((True, False), (True, True)):
            off = (got[how][rows] != want).any(dim=1).nonzero().flatten().tolist()
            assert not off, (model, rows, "replayed" if how[1] else "one by one", off)
