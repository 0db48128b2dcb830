"""Host side of ``csrc/prefill_layer.cu``: the layers of a prefill over fresh prompts, each issued by one call.

Covers what launch-bound prompts run: softmax attention with a full rotary table, bf16 projections on one GPU, dense or mixture
MLPs (the mixture part goes through ``ModelRunner``). The same kernels with the same plans in the same order as
``ModelRunner.prefill`` otherwise issues; every buffer is allocated per call."""

from __future__ import annotations

import ctypes

import torch

from slime_b200 import ops
from slime_b200.ops import _checks, _lib, attention

_I, _F, _P = ctypes.c_int, ctypes.c_float, ctypes.c_void_p
_POINTERS = ("x", "res", "ln1", "qkv_w", "qkv_b", "q_norm", "k_norm", "o_w", "ln2", "gate_up", "down", "positions", "slots", "seg", "rope",
             "k_cache", "v_cache", "normed", "h1", "h2", "qkv", "ctx", "gu", "act", "proj", "lse", "rstd", "status")  # fmt: skip


class Layer(ctypes.Structure):
    _fields_ = [(n, _I) for n in ("bytes", "T", "H", "Hq", "Hkv", "D", "F", "nseg", "max_q_tiles", "x_f32", "num_sms")]
    _fields_ += [("eps", _F), ("scale", _F), ("plan", _I * 12), ("reserved", _I)]
    _fields_ += [(n, _P) for n in _POINTERS]


def covers(runner) -> bool:
    """Whether this runner's layers are of the kind above (its weights keep their buffers)."""
    w, cfg = runner.w, runner.cfg
    if runner.layered or runner.device.type != "cuda" or w.tp != 1 or runner.tp_group is not None or runner._composed_attention:
        return False
    if cfg.head_dim not in (64, 128) or cfg.hidden_size % 8 or runner._proj_dtype != torch.float32 or ops.library_mode() or w.hq % w.hkv:
        return False

    def plain(L):
        mats = [L.get("qkv"), L.get("o")] + ([L.get("gate_up"), L.get("down")] if "gate_up" in L else [])
        return (L["kind"] == "attention" and not any(L.get(k) is not None for k in ("gate", "sinks", "post_attn_ln", "post_mlp_ln"))
                and all(isinstance(m, torch.Tensor) and m.dtype == torch.bfloat16 and m.is_contiguous() and m.shape[-1] % 8 == 0 for m in mats)
                and L["ln1"].dtype == L["ln2"].dtype == torch.bfloat16)  # fmt: skip

    return all(plain(L) for L in w.layers)


def usable(runner, x, positions, slots, fresh: bool) -> bool:
    """Whether this pass is one: rows of fresh prompts, plain positions, a cache of contiguous slabs, no index checks asked for."""
    i32 = lambda t: t.dim() == 1 and t.dtype == torch.int32 and t.is_contiguous()  # noqa: E731
    return (fresh and x.shape[0] > 0 and x.dtype == torch.bfloat16 and x.is_contiguous() and i32(positions) and i32(slots) and not _checks.enabled()
            and all(k.is_contiguous() for k in (*runner.kv.k, *runner.kv.v)))  # fmt: skip


def prefill_layers(runner, x, positions, slots, cu_q):
    """All layers over packed fresh prompts: embeddings ``x`` [T, H] bf16 -> ``(x, residual)`` as the final norm takes them."""
    w, cfg, kv, dev = runner.w, runner.cfg, runner.kv, x.device
    T, H, hq, hkv, D = x.shape[0], x.shape[1], w.hq, w.hkv, cfg.head_dim
    row, ffn = (hq + 2 * hkv) * D, max((L["down"].shape[1] for L in w.layers if "down" in L), default=0)
    bf16 = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=dev)  # noqa: E731
    f32 = lambda *s: torch.empty(s, dtype=torch.float32, device=dev)  # noqa: E731
    seg = attention.segments_from_cu_seqlens(cu_q)
    held = dict(normed=bf16(T, H), h1=bf16(T, H), h2=bf16(T, H), qkv=bf16(T, row), ctx=bf16(T, hq * D), gu=bf16(T, 2 * ffn), act=bf16(T, ffn),
                proj=f32(T, H), lse=f32(hq, T), rstd=f32(T), seg=seg, positions=positions, slots=slots, rope=runner.rope,
                status=_lib.status_word(dev))  # fmt: skip
    sms = _lib.sm_count(dev)
    p = Layer(bytes=ctypes.sizeof(Layer), T=T, H=H, Hq=hq, Hkv=hkv, D=D, nseg=seg.shape[0], max_q_tiles=attention.query_tiles(T, seg.shape[0]),
              num_sms=sms, eps=cfg.norm_epsilon, scale=runner.scale, **{k: t.data_ptr() for k, t in held.items()})  # fmt: skip
    fn, stream, ptr = _lib.lib().sb_prefill_layer, _lib.stream(), _lib.ptr
    res = None
    for li, L in enumerate(w.layers):
        dense = "gate_up" in L
        p.F = L["down"].shape[1] if dense else 0
        shapes = [(row, H, False), (H, hq * D, True)] + ([(2 * p.F, H, False), (H, p.F, True)] if dense else [])
        for i, (N, K, out32) in enumerate(shapes):
            p.plan[3 * i : 3 * i + 3] = ops.gemm_plan(T, N, K, out32, sms)
        p.x, p.res, p.x_f32 = x.data_ptr(), ptr(res), int(x.dtype == torch.float32)
        p.ln1, p.ln2, p.qkv_w, p.o_w = L["ln1"].data_ptr(), L["ln2"].data_ptr(), L["qkv"].data_ptr(), L["o"].data_ptr()
        p.qkv_b, p.q_norm, p.k_norm = ptr(L["qkv_bias"]), ptr(L["q_norm"]), ptr(L["k_norm"])
        p.gate_up, p.down = (L["gate_up"].data_ptr(), L["down"].data_ptr()) if dense else (None, None)
        n = runner.kv_of[li]
        p.k_cache, p.v_cache = kv.k[n].data_ptr(), kv.v[n].data_ptr()
        _lib.check(fn(ctypes.addressof(p), stream), "sb_prefill_layer", launches=9 if dense else 6)
        res = held["h2"]
        x = held["proj"] if dense else runner._moe(L, held["normed"])
    return x, res
