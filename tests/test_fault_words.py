"""One status word a device, under every name of it."""
import torch


def test_a_device_has_one_word_under_all_its_names(monkeypatch):
    """An engine made for "cuda" looks at the word that kernels launched on tensors of "cuda:0" write."""
    from cretif_b200.csrc import ops
    monkeypatch.setattr(ops, "_FAULT", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    monkeypatch.setattr(torch, "zeros", lambda *a, **k: object())
    words = {n: ops.fault_word(n) for n in ("cuda", "cuda:0", "cuda:1", torch.device("cuda", 1), "cpu")}
    assert words["cuda"] is words["cuda:1"] is words[torch.device("cuda", 1)]
    assert len({id(w) for w in words.values()}) == 3
