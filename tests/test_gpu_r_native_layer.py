"""Prefill with a layer issued per call against the same launches issued one by one: the same kernels, so the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(preset):
    from slime_b200.engine.engine import Engine
    from slime_b200.engine.server_args import ServerArgs
    from slime_b200.models.config import get_preset

    cfg = get_preset(preset)
    cfg.num_layers, cfg.vocab_size = 2, 1024
    if cfg.num_experts:
        cfg.num_experts = 16
    e = Engine(cfg, ServerArgs(page_size=64, context_length=512, max_running_requests=4, disable_radix_cache=True), device="cuda", num_pages=24)
    e.weights.init_random(3)
    assert e.runner._native_layers
    return e


def _both_ways(e, lengths):
    """Logits of all rows and the written cache slots, by native layers and by ops."""
    from slime_b200.ops import _lib

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
    return got


@pytest.mark.parametrize("preset,lengths", [("qwen2.5-0.5b", [2]), ("qwen2.5-0.5b", [301, 7, 129]), ("qwen3-4b", [64, 333]), ("qwen3-30b-a3b", [5, 200])])
def test_native_layers_issue_what_the_ops_do(kernels, monkeypatch, preset, lengths):
    from slime_b200 import ops

    monkeypatch.setattr(ops, "BATCH_INVARIANT", True)  # no sums over K slices, which come in any order
    for a, b in zip(*_both_ways(_engine(preset), lengths)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("preset,lengths", [("qwen2.5-0.5b", [2]), ("qwen2.5-0.5b", [301]), ("qwen3-4b", [64, 33]), ("qwen3-30b-a3b", [5, 20])])
def test_native_layers_with_slices_of_k(kernels, preset, lengths):
    """The plans that short prompts run by default: projections whose K slices are added up, in arrival order, in a buffer that earlier layers have
    used. fp32 sums in another order flip roundings to bf16 (2^-9 each) at the five places of each of two layers."""
    from slime_b200 import ops
    from slime_b200.ops import _lib

    e = _engine(preset)
    w, T, sms = e.runner.w, sum(lengths), _lib.sm_count("cuda")
    plans = [ops.gemm_plan(T, *L["o"].shape, True, sms) for L in w.layers] + [ops.gemm_plan(T, *L["down"].shape, True, sms) for L in w.layers if "down" in L]
    assert any(width == 0 and slices > 1 for width, _, slices in plans)
    for _ in range(3):
        for a, b in zip(*_both_ways(e, lengths)):
            assert float((a.float() - b.float()).norm()) <= 10**0.5 * 2**-9 * float(b.float().norm())
