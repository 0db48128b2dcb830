"""The sm_100a flash-attention kernels (forward, dK/dV pass, dQ pass) against fp32 PyTorch."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, seg, scale):
    from slime_b200.ops.attention import _reference_segments

    return _reference_segments(q.float(), k.float(), v.float(), seg, scale)


def _close(got, want, what, atol, rtol):
    err = (got.float() - want.float()).abs()
    bound = atol + rtol * want.float().abs()
    bad = err > bound
    assert not bad.any(), f"{what}: {int(bad.sum())} of {bad.numel()} elements off, worst {float(err.max()):.4g} (ref scale {float(want.abs().max()):.3g})"


CASES = [
    # lens, Hq, Hkv, D
    ([1, 127, 128, 129, 300], 14, 2, 64),
    ([1, 127, 128, 129, 300], 8, 2, 128),
    ([4097], 4, 1, 128),
    ([515, 64, 2000], 14, 2, 64),
    ([96, 257], 32, 8, 128),
]


@pytest.mark.parametrize("lens,Hq,Hkv,D", CASES)
def test_flash_forward_backward_match_fp32(kernels, lens, Hq, Hkv, D):
    from slime_b200.ops import _lib, attention

    torch.manual_seed(sum(lens) + Hq)
    T = sum(lens)
    pad = (-T) % 128
    Tp = T + pad
    dev = "cuda"
    # one packed qkv buffer, as the trainer has it (q / k / v are strided views)
    qkv = (torch.randn(Tp, (Hq + 2 * Hkv) * D, device=dev) * 0.8).to(torch.bfloat16)
    x3 = qkv.view(Tp, Hq + 2 * Hkv, D)
    q, k, v = x3[:, :Hq], x3[:, Hq : Hq + Hkv], x3[:, Hq + Hkv :]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)) + ([Tp] if pad else []), dtype=torch.int32, device=dev)
    seg = attention.segments_from_cu_seqlens(cu)
    scale = 1.0 / math.sqrt(D)
    out, lse = attention.flash_fwd(q, k, v, seg, scale)
    torch.cuda.synchronize()
    _lib.check_status(dev)
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = _ref(qf, kf, vf, seg.cpu(), scale)
    _close(out, ref, "out", 2e-2, 2e-2)
    # lse against the reference, valid rows only
    for (qo, ql, ko, kl) in seg.tolist():
        s = torch.einsum("thd,shd->hts", qf[qo : qo + ql].detach(), kf[ko : ko + kl].detach().repeat_interleave(Hq // Hkv, 1)) * scale
        m = torch.ones(ql, kl, dtype=torch.bool, device=dev).tril(diagonal=kl - ql)
        want = torch.logsumexp(s.masked_fill(~m, float("-inf")), -1)
        _close(lse[:, qo : qo + ql], want, "lse", 2e-2, 1e-2)
    d_o = (torch.randn(Tp, Hq, D, device=dev) * 0.5).to(torch.bfloat16)
    ref.backward(d_o.float())
    dqkv = torch.zeros_like(qkv)
    d3 = dqkv.view(Tp, Hq + 2 * Hkv, D)
    attention.flash_bwd(q, k, v, out, d_o, lse, seg, scale, dq=d3[:, :Hq], dk=d3[:, Hq : Hq + Hkv], dv=d3[:, Hq + Hkv :])
    torch.cuda.synchronize()
    _lib.check_status(dev)
    # gradients are sums over up to thousands of bf16-rounded products: absolute floor scaled by the tensor's size
    for name, got, want in (("dq", d3[:, :Hq], qf.grad), ("dk", d3[:, Hq : Hq + Hkv], kf.grad), ("dv", d3[:, Hq + Hkv :], vf.grad)):
        _close(got, want, name, 3e-2 * float(want.abs().max()) + 1e-3, 3e-2)


def test_flash_extend_segments_and_autograd(kernels):
    """Queries over a longer key range (prefill over a cached prefix; a context-parallel chunk over gathered keys),
    through the autograd wrapper."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(3)
    Hq, Hkv, D = 8, 2, 128
    q_lens, k_lens = [5, 130, 64], [200, 130, 1000]
    dev = "cuda"
    q = (torch.randn(sum(q_lens), Hq, D, device=dev) * 0.7).to(torch.bfloat16).requires_grad_()
    k = (torch.randn(sum(k_lens), Hkv, D, device=dev) * 0.7).to(torch.bfloat16).requires_grad_()
    v = (torch.randn(sum(k_lens), Hkv, D, device=dev) * 0.7).to(torch.bfloat16).requires_grad_()
    cu_q = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=dev)
    cu_k = torch.tensor([0] + list(torch.tensor(k_lens).cumsum(0)), dtype=torch.int32, device=dev)
    out = attention.extend_attention(q, k, v, cu_q, cu_k)
    w = torch.randn_like(out)
    (out.float() * w.float()).sum().backward()
    torch.cuda.synchronize()
    _lib.check_status(dev)
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = _ref(qf, kf, vf, attention.segments_extend(cu_q, cu_k).cpu(), 1.0 / math.sqrt(D))
    (ref * w.float()).sum().backward()
    _close(out, ref, "out", 2e-2, 2e-2)
    for name, got, want in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        _close(got, want, name, 3e-2 * float(want.abs().max()) + 1e-3, 3e-2)


def test_rope_attention_node_matches_reference(kernels):
    """The trainer's fused node (qk-norm + RoPE + attention) on CUDA against the same node on CPU in fp32."""
    from slime_b200 import ops

    torch.manual_seed(5)
    Hq, Hkv, D, lens = 8, 2, 128, [70, 186]
    T = sum(lens)
    qkv = (torch.randn(T, (Hq + 2 * Hkv) * D) * 0.5)
    cu = torch.tensor([0, 70, 256], dtype=torch.int32)
    pos = torch.cat([torch.arange(n) for n in lens]).to(torch.int32)
    table = ops.rope_cos_sin(512, D, 1e4)
    qw, kw = 1 + 0.1 * torch.randn(D), 1 + 0.1 * torch.randn(D)
    w = torch.randn(T, Hq * D)

    def run(dev, dt):
        x = qkv.to(dev, dt).requires_grad_()
        a, b = qw.to(dev, dt).requires_grad_(), kw.to(dev, dt).requires_grad_()
        y = ops.rope_attention(x, pos.to(dev), table.to(dev), cu.to(dev), 186, Hq, Hkv, D, a, b, 1e-6)
        (y.float() * w.to(dev)).sum().backward()
        return y.detach().float().cpu(), x.grad.float().cpu(), a.grad.float().cpu(), b.grad.float().cpu()

    got = run("cuda", torch.bfloat16)
    want = run("cpu", torch.float32)
    for name, g, r in zip(("out", "dqkv", "dq_norm_w", "dk_norm_w"), got, want):
        _close(g, r, name, 4e-2 * float(r.abs().max()) + 1e-3, 4e-2)


@pytest.mark.parametrize("lens,Hq,Hkv,D", [
    ([1 + 37 * i % 191 for i in range(70)], 14, 2, 64),  # more segments than one step of the table's search, query heads of a key tile split 7 ways
    ([63, 64, 65, 191, 192, 193], 6, 2, 128),  # edges of the streamed blocks, parts of one and two heads
    ([7201], 16, 8, 64),  # enough key tiles for the machine: one CTA for all heads of a group
])  # fmt: skip
def test_flash_backward_splits_and_tables(kernels, lens, Hq, Hkv, D):
    """The launch shapes of the backward: every split of a group's query heads gives the same sums, and long tables are searched right.
    Bounds: P and dS are rounded to bf16 (2^-9 each) and the outputs once more, on sums whose terms have random signs."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(len(lens))
    T = sum(lens)
    q, d_o = ((torch.randn(T, Hq, D, device="cuda") * 0.8).to(torch.bfloat16) for _ in range(2))
    k, v = ((torch.randn(T, Hkv, D, device="cuda") * 0.8).to(torch.bfloat16) for _ in range(2))
    seg = attention.segments_from_cu_seqlens(torch.tensor([0] + lens, device="cuda").cumsum(0))
    out, lse = attention.flash_fwd(q, k, v, seg, D**-0.5)
    got = attention.flash_bwd(q, k, v, out, d_o, lse, seg, D**-0.5)
    again = attention.flash_bwd(q, k, v, out, d_o, lse, seg, D**-0.5)
    _lib.check_status("cuda")
    at, want = 0, [torch.zeros_like(x, dtype=torch.float32) for x in (q, k, v)]
    for n in lens:
        for h in range(Hkv):
            g = slice(h * Hq // Hkv, (h + 1) * Hq // Hkv)
            qs, ks, vs, ds = q[at : at + n, g].double(), k[at : at + n, h].double(), v[at : at + n, h].double(), d_o[at : at + n, g].double()
            p = torch.einsum("igd,jd->gij", qs, ks) * D**-0.5
            p = p.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), -math.inf).softmax(-1)
            dp = torch.einsum("igd,jd->gij", ds, vs)
            s = p * (dp - (p * dp).sum(-1, keepdim=True)) * D**-0.5
            want[0][at : at + n, g] = torch.einsum("gij,jd->igd", s, ks).float()
            want[1][at : at + n, h] = torch.einsum("gij,igd->jd", s, qs).float()
            want[2][at : at + n, h] = torch.einsum("gij,igd->jd", p, ds).float()
        at += n
    for name, a, b, w in zip(("dq", "dk", "dv"), got, again, want):
        assert torch.equal(a, b), f"{name} is not the same twice"
        rel = float((a.float() - w).norm() / w.norm())
        assert rel < 3 * 2**-8, f"{name}: {rel}"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("pairs", [
    [(255, 255), (256, 256), (257, 257), (384, 384), (1, 1)],  # one tile, two whole tiles, a third one alone
    [(1, 1000), (130, 257), (300, 301), (200, 900), (129, 129)],  # behind a context of any length
])  # fmt: skip
def test_flash_forward_pairs_of_tiles(kernels, pairs, D):
    """Query tiles in pairs: the second one empty, ragged or with more key tiles than the first. Large scores make the running maximum rise.
    Bounds: probabilities are rounded to bf16 (2^-9) and so is the output."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(D)
    Hq, Hkv = 6, 2
    Tq, Tk = sum(a for a, _ in pairs), sum(b for _, b in pairs)
    q = (torch.randn(Tq, Hq, D, device="cuda") * 4).to(torch.bfloat16)
    k, v = (torch.randn(Tk, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    cu = lambda i: torch.tensor([0] + [p[i] for p in pairs], device="cuda").cumsum(0)  # noqa: E731
    seg = attention.segments_extend(cu(0), cu(1))
    out, lse = attention.flash_fwd(q, k, v, seg, D**-0.5)
    _lib.check_status("cuda")
    want = _ref(q, k, v, seg.cpu(), D**-0.5)
    assert float((out.float() - want).norm() / want.norm()) < 2 * 2**-8
    for qo, ql, ko, kl in seg.tolist():
        s = torch.einsum("thd,shd->hts", q[qo : qo + ql].double(), k[ko : ko + kl].double().repeat_interleave(Hq // Hkv, 1)) * D**-0.5
        s = s.masked_fill(~torch.ones(ql, kl, dtype=torch.bool, device="cuda").tril(kl - ql), -math.inf)
        assert float((lse[:, qo : qo + ql] - s.logsumexp(-1)).abs().max()) < 1e-4 * max(1.0, float(s.amax()))


@pytest.mark.parametrize("parts", [2, 3, 4, 7])
@pytest.mark.parametrize("lens,Hkv,D", [([1 + 37 * i % 191 for i in range(70)], 2, 64), ([7, 63, 64, 65, 127, 129, 193], 1, 128), ([300], 8, 128)])
def test_flash_backward_in_any_number_of_parts(kernels, monkeypatch, parts, lens, Hkv, D):
    """dK and dV as sums of fp32 parts against one part: sums in another order, one rounding to bf16 (2^-8); dQ has no parts. Rows outside
    every segment stay as they are."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(parts)
    T, Hq = sum(lens) + 3, 7 * Hkv
    q, d_o = (torch.randn(T, Hq, D, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(T, Hkv, D, device="cuda").bfloat16() for _ in range(2))
    seg = attention.segments_from_cu_seqlens(torch.tensor([0] + lens, device="cuda").cumsum(0))
    out, lse = attention.flash_fwd(q, k, v, seg, D**-0.5, zero_uncovered=True)
    got = []
    for p in (1, parts):
        monkeypatch.setattr(attention, "_key_parts", lambda *a: p)
        grads = [torch.full_like(t, 5.0) for t in (q, k, v)]
        got.append(attention.flash_bwd(q, k, v, out, d_o, lse, seg, D**-0.5, *grads))
    _lib.check_status("cuda")
    assert torch.equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1:], got[1][1:]):
        assert (b[-3:] == 5).all()
        torch.testing.assert_close(a, b, rtol=2**-7, atol=2.0**-16 * float(a[:-3].abs().max()))


@pytest.mark.parametrize("Hq,Hkv,D", [(14, 2, 64), (8, 2, 128), (2, 1, 128)])
@pytest.mark.parametrize("q_len,k_len", [(1, 1), (1, 700), (128, 128), (129, 129), (300, 301), (397, 397), (640, 640), (260, 2000)])
def test_flash_forward_one_tile_per_cta(kernels, Hq, Hkv, D, q_len, k_len):
    """Few tiles have a CTA each, many go in pairs: a segment's rows have the same bits alone (one tile a CTA) and in front of enough others
    (pairs). Large scores make the running maximum rise."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(q_len + k_len)
    more = 148 // Hq * 128 + 256  # rows: more tiles than SMs
    q = (torch.randn(q_len + more, Hq, D, device="cuda") * 4).to(torch.bfloat16)
    k, v = (torch.randn(k_len + more, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    one = torch.tensor([[0, q_len, 0, k_len]], dtype=torch.int32, device="cuda")
    both = torch.cat([one, torch.tensor([[q_len, more, k_len, more]], dtype=torch.int32, device="cuda")])
    alone, lse = attention.flash_fwd(q[:q_len], k[:k_len], v[:k_len], one, D**-0.5)
    among, lse_among = attention.flash_fwd(q, k, v, both, D**-0.5)
    _lib.check_status("cuda")
    assert torch.equal(alone, among[:q_len]) and torch.equal(lse, lse_among[:, :q_len])
    want = _ref(q[:q_len], k[:k_len], v[:k_len], one.cpu(), D**-0.5)
    assert float((alone.float() - want).norm() / want.norm()) < 2 * 2**-8


@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("lens", [[129], [300, 40, 1], [500] * 40])
def test_flash_attention_takes_any_factor(kernels, scale, lens):
    """Zero (the mean of the visible values) and negative factors, masked tiles included, with their gradients."""
    from slime_b200.ops import _lib, attention

    torch.manual_seed(len(lens))
    seg = attention.segments_from_cu_seqlens(torch.tensor([0] + lens, device="cuda").cumsum(0))
    ins = [torch.randn(sum(lens), h, 64, device="cuda").bfloat16() for h in (4, 2, 2)]
    g = torch.randn(sum(lens), 4, 64, device="cuda").bfloat16()
    res = []
    for fn, cast in ((attention.segment_attention, lambda t: t), (lambda *a: _ref(*a[:3], a[3].cpu(), a[4]), lambda t: t.float())):
        xs = [cast(t).clone().requires_grad_() for t in ins]
        y = fn(*xs, seg, scale)
        y.backward(g.to(y.dtype))
        res.append([y.detach().float()] + [x.grad.float() for x in xs])
    _lib.check_status("cuda")
    for a, b in zip(*res):
        assert float((a - b).norm()) <= 3 * 2**-8 * float(b.norm())
