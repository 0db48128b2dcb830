"""Prefill with a layer issued per call against the same launches issued one by one: the same kernels, so the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,lengths", [("qwen2.5-0.5b", [2]), ("qwen2.5-0.5b", [301, 7, 129]), ("qwen3-4b", [64, 333]), ("qwen3-30b-a3b", [5, 200])])
def test_native_layers_issue_what_the_ops_do(kernels, monkeypatch, preset, lengths):
    from slime_b200 import ops
    from slime_b200.engine.engine import Engine
    from slime_b200.engine.server_args import ServerArgs
    from slime_b200.models.config import get_preset
    from slime_b200.ops import _lib

    monkeypatch.setattr(ops, "BATCH_INVARIANT", True)  # no sums over K slices, which come in any order
    cfg = get_preset(preset)
    cfg.num_layers, cfg.vocab_size = 2, 1024
    if cfg.num_experts:
        cfg.num_experts = 16
    e = Engine(cfg, ServerArgs(page_size=64, context_length=512, max_running_requests=4, disable_radix_cache=True), device="cuda", num_pages=24)
    e.weights.init_random(3)
    assert e.runner._native_layers
    g = torch.Generator().manual_seed(sum(lengths))
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in lengths]
    got = []
    for native in (True, False):
        e.runner._native_layers = native
        reqs = [e.open_stream(f"{native}{i}") for i in range(len(prompts))]
        logits = e.feed([(r, t, list(range(len(t)))) for r, t in zip(reqs, prompts)])
        slots = torch.tensor([s for r, t in zip(reqs, prompts) for s in e._slots(r, 0, len(t))], device="cuda")
        got.append([logits] + [c.index_select(0, slots) for c in (*e.runner.kv.k, *e.runner.kv.v)])
        for r in reqs:
            e.close_stream(r)
    _lib.check_status("cuda")
    for a, b in zip(*got):
        assert torch.equal(a, b)
