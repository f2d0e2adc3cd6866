"""Steps whose kernels start as programmatic dependents of one another give the bits of steps
whose kernels start one after the other: every architecture's tiny models, a ragged prompt step and
decode steps, launched one by one and from a captured graph."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

DESIGNS = ["rigozen", "losorax", "virorax", "mipurax", "gibipel", "pudorax"]


def _logits(folder, dtype, vocab, graphs):
    from cretif_b200.engine import Engine
    engine = Engine(folder, dtype=dtype, max_tokens=1024, step_graphs=graphs)
    gen = torch.Generator().manual_seed(2)
    slots = [engine.alloc_slot() for _ in range(3)]
    prompts = [torch.randint(vocab, (n,), generator=gen).tolist() for n in (5, 70, 18)]
    out = [engine.step(list(zip(slots, prompts)))]
    for _ in range(40):                    # past blocks, windows and pooled entries
        fed = torch.randint(vocab, (3, 1), generator=gen).tolist()
        out.append(engine.step(list(zip(slots, fed))))
    return torch.cat(out)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("design", DESIGNS)
def test_same_bits_with_and_without(tmp_path, design, dtype):
    from cretif_b200.csrc import ops
    from cretif_b200.weights.random_model import write_random_model
    configs = importlib.import_module(design + "_tiny").CONFIGS
    for name in sorted(configs)[:2]:
        folder = str(tmp_path / name)
        write_random_model(folder, configs[name], seed=9)
        got = []
        for on, graphs in ((False, False), (True, False), (True, True)):
            was = ops.set_dependent_launch(on)
            try:
                got.append(_logits(folder, dtype, configs[name]["vocab"], graphs))
            finally:
                ops.set_dependent_launch(was)
        assert bool(torch.isfinite(got[0]).all())
        assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2]), (design, name)
