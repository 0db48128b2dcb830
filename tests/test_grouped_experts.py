"""Grouped expert MLP: the padded-layout path against the per-expert loop (CPU), and against fp32 math on a GPU."""

import pytest
import torch

from slime_b200.ops import grouped


def _loop_reference(x, counts, w1, w2):
    outs, s = [], 0
    for e, n in enumerate(counts):
        xe = x[s : s + n].float()
        h = xe @ w1[e].float().t()
        g, u = h.chunk(2, dim=-1)
        outs.append((torch.nn.functional.silu(g) * u) @ w2[e].float().t())
        s += n
    return torch.cat(outs)


def test_padded_layout_and_stacked_view():
    lay = grouped.PaddedLayout([3, 0, 130, 128], "cpu")
    assert lay.padded == [128, 0, 256, 128] and lay.rows == 261 and lay.rows_padded == 512
    assert lay.tile_expert.tolist() == [0, 2, 2, 3] and lay.dest[:4].tolist() == [0, 1, 2, 128]
    x = torch.arange(261.0)[:, None].repeat(1, 2)
    assert torch.equal(lay.unpad(lay.pad(x)), x) and lay.pad(x)[3:128].abs().sum() == 0
    flat = torch.randn(3 * 4 * 5)
    views = [flat[i * 20 : (i + 1) * 20].view(4, 5) for i in range(3)]
    st = grouped.stacked_view(views)
    assert st is not None and st.data_ptr() == flat.data_ptr() and torch.equal(st[2], views[2])
    assert grouped.stacked_view([views[0], views[2]]) is None
    assert grouped.stacked_view([torch.randn(4, 5), torch.randn(4, 5).t().contiguous().t()]) is None
    # neighbours in memory, each with a storage of its own
    import numpy as np

    whole = np.arange(40, dtype=np.float32)
    apart = [torch.from_numpy(whole[i * 20 : (i + 1) * 20]).view(4, 5) for i in range(2)]
    assert apart[1].data_ptr() == apart[0].data_ptr() + 80 and grouped.stacked_view(apart) is None


def test_grouped_experts_module_matches_loop_on_cpu():
    from slime_b200.models.config import get_preset
    from slime_b200.models.moe import GroupedExperts
    from slime_b200.parallel import state as mpu

    if not mpu.model_parallel_is_initialized():
        mpu.initialize_model_parallel()
    cfg = get_preset("tiny-moe")
    torch.manual_seed(0)
    m = GroupedExperts(cfg, torch.float32, "cpu", 4)
    counts = [5, 0, 9, 2]
    x = torch.randn(sum(counts), cfg.hidden_size, requires_grad=True)
    y = m(x, counts)
    y.pow(2).sum().backward()
    gx, gw = x.grad.clone(), [p.grad.clone() for p in m.parameters()]
    x.grad = None
    for p in m.parameters():
        p.grad = None
    m.use_grouped_gemm = False
    y2 = m(x, counts)
    y2.pow(2).sum().backward()
    torch.testing.assert_close(y, y2, rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(gx, x.grad, rtol=1e-4, atol=1e-5)
    for a, p in zip(gw, m.parameters()):
        torch.testing.assert_close(a, p.grad if p.grad is not None else torch.zeros_like(p), rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[300, 0, 77, 129, 1, 128], [4096, 1000, 2, 3000]])
def test_grouped_gemm_gpu_matches_fp32(kernels, counts):
    from slime_b200 import ops

    torch.manual_seed(len(counts))
    E, H, F = len(counts), 512, 384
    dev = "cuda"
    flat1 = (torch.randn(E * 2 * F * H, device=dev) * 0.05).to(torch.bfloat16)  # adjacent experts: the no-copy path
    w1 = [flat1[e * 2 * F * H : (e + 1) * 2 * F * H].view(2 * F, H).requires_grad_() for e in range(E)]
    w2 = [(torch.randn(H, F, device=dev) * 0.05).to(torch.bfloat16).requires_grad_() for _ in range(E)]  # stacked by copy
    x = torch.randn(sum(counts), H, device=dev).to(torch.bfloat16).requires_grad_()
    lay = grouped.PaddedLayout(counts, dev)
    assert grouped.stacked_view([w.detach() for w in w1]) is not None
    h = grouped.grouped_linear(lay.pad(x), lay, w1)
    y = lay.unpad(grouped.grouped_linear(ops.swiglu(h), lay, w2))
    ref = _loop_reference(x.detach(), counts, [w.detach() for w in w1], [w.detach() for w in w2])
    assert (y.float() - ref).abs().max() <= 0.03 * ref.abs().max() + 1e-3
    gy = torch.randn_like(y)
    y.backward(gy)
    xr = x.detach().float().requires_grad_()
    w1r = [w.detach().float().requires_grad_() for w in w1]
    w2r = [w.detach().float().requires_grad_() for w in w2]
    outs, s = [], 0
    for e, n in enumerate(counts):
        hh = xr[s : s + n] @ w1r[e].t()
        g, u = hh.chunk(2, dim=-1)
        outs.append((torch.nn.functional.silu(g) * u) @ w2r[e].t())
        s += n
    torch.cat(outs).backward(gy.float())

    def close(a, b, what):
        assert (a.float() - b).abs().max() <= 0.04 * b.abs().max() + 1e-3, what

    close(x.grad, xr.grad, "dx")
    for e in range(E):
        close(w1[e].grad if w1[e].grad is not None else torch.zeros_like(w1[e]), w1r[e].grad if w1r[e].grad is not None else torch.zeros_like(w1r[e]), f"dw1[{e}]")
        close(w2[e].grad if w2[e].grad is not None else torch.zeros_like(w2[e]), w2r[e].grad if w2r[e].grad is not None else torch.zeros_like(w2r[e]), f"dw2[{e}]")


def _moe_reference(x, idx, probs, w13, w2):
    out = torch.zeros(x.shape[0], x.shape[1])
    for t in range(x.shape[0]):
        for j in range(idx.shape[1]):
            e = int(idx[t, j])
            h = x[t].float() @ w13[e].float().t()
            g, u = h.chunk(2)
            out[t] += float(probs[t, j]) * ((torch.nn.functional.silu(g) * u) @ w2[e].float().t())
    return out


def test_device_layout_moe_matches_per_token_reference():
    from slime_b200 import ops

    torch.manual_seed(1)
    T, k, E, H, F = 37, 2, 5, 16, 24
    x = torch.randn(T, H)
    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)])
    idx[:, 0] = torch.where(idx[:, 0] == 3, torch.tensor(0), idx[:, 0])  # expert 3 gets fewer tokens
    probs = torch.rand(T, k)
    w13, w2 = torch.randn(E, 2 * F, H) * 0.2, torch.randn(E, H, F) * 0.2
    lay = grouped.DeviceLayout(idx, E)
    assert lay.rows_padded % 128 == 0 and lay.rows_padded >= T * k
    act = ops.swiglu(grouped.grouped_gemm(lay.pad(x), w13, lay))
    y = lay.combine(grouped.grouped_gemm(act, w2, lay), probs, T)
    torch.testing.assert_close(y, _moe_reference(x, idx, probs, w13, w2), rtol=1e-4, atol=1e-5)


def test_moe_engine_decodes_consistently_on_cpu():
    """tiny-moe through the engine: decode log-probs equal teacher-forced ones (prefill and decode share the MoE path)."""
    import numpy as np

    from slime_b200.engine.engine import Engine
    from slime_b200.engine.server_args import ServerArgs
    from slime_b200.models.config import get_preset

    e = Engine(get_preset("tiny-moe"), ServerArgs(page_size=4, max_running_requests=4, context_length=64, disable_cuda_graph=True),
               device="cpu", num_pages=64)
    e.weights.init_random(0)
    r = e.generate([[1, 2, 3, 4, 5]], [dict(max_new_tokens=6, ignore_eos=True)])[0]
    rq = e.generate([r.input_ids + r.output_ids], [dict(max_new_tokens=0)], logprob_start_len=0)[0]
    assert np.abs(np.array(rq.input_logprobs[5:]) - np.array(r.output_logprobs)).max() < 1e-4


def _perm_case(device, dtype):
    torch.manual_seed(4)
    T, k, H, R = 33, 3, 64, 150
    x = torch.randn(T, H, device=device).to(dtype)
    dest = torch.randperm(R, device=device)[: T * k].to(torch.int32)
    dest[5] = -1  # a dropped route
    w = torch.rand(T, k, device=device)
    return x, dest, w, T, k, H, R


def test_route_permutation_ops_and_gradients_cpu():
    x, dest, w, T, k, H, R = _perm_case("cpu", torch.float32)
    x.requires_grad_()
    w.requires_grad_()
    rows = grouped.permute_tokens(x, dest, k, R)
    assert torch.equal(rows[dest[7].long()], x[7 // k].detach()) and rows.abs().sum(1).ne(0).sum() == T * k - 1
    y = grouped.combine_routes(rows * 2.0, dest, w, k)
    d = dest.view(T, k).long()
    ok = (d >= 0).float()
    want = (2.0 * x.detach()[:, None, :] * (w.detach() * ok)[:, :, None]).sum(1)
    torch.testing.assert_close(y, want, rtol=1e-5, atol=1e-6)
    gy = torch.randn_like(y)
    y.backward(gy)
    # d/dx sum_j 2 w_j x = 2 * sum_j w_j * gy ; d/dw_j = <2 x, gy>
    torch.testing.assert_close(x.grad, 2.0 * (w.detach() * ok).sum(1, keepdim=True) * gy, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(w.grad, ok * (2.0 * x.detach() * gy).sum(-1, keepdim=True), rtol=1e-5, atol=1e-5)


@pytest.mark.gpu
def test_route_permutation_kernels_match_cpu_reference_and_are_deterministic(kernels):
    x, dest, w, T, k, H, R = _perm_case("cuda", torch.bfloat16)
    rows = grouped.scatter_rows(x, dest, k, R)
    assert torch.equal(rows.cpu(), grouped.scatter_rows(x.cpu(), dest.cpu(), k, R))
    y = grouped.gather_sum(rows, dest, w, k)
    ref = grouped.gather_sum(rows.cpu(), dest.cpu(), w.cpu(), k)
    assert (y.cpu().float() - ref.float()).abs().max() <= 2e-2 * ref.float().abs().max()
    assert torch.equal(grouped.gather_sum(rows, dest, w, k), y)  # same bits every time
    y2 = grouped.gather_sum(rows, dest, w, k, round_each=True)
    ref2 = grouped.gather_sum(rows.cpu(), dest.cpu(), w.cpu(), k, round_each=True)
    assert (y2.cpu().float() - ref2.float()).abs().max() <= 2e-2 * ref2.float().abs().max()
    dy = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    dw = grouped.route_weight_grad(rows, dest, dy, k)
    torch.testing.assert_close(dw.cpu(), grouped.route_weight_grad(rows.cpu(), dest.cpu(), dy.cpu(), k), rtol=2e-3, atol=2e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("E,k", [(128, 8), (8, 2), (160, 6), (512, 32)])
def test_route_topk_kernel_matches_torch(kernels, E, k):
    torch.manual_seed(E)
    T = 301
    logits = torch.randn(T, E, device="cuda") * 3
    bias = torch.randn(E, device="cuda") * 0.5
    cases = [dict(), dict(pre_softmax=True), dict(renorm=False), dict(score="sigmoid", bias=bias, scale=2.5),
             dict(score="sigmoid", renorm=False)]
    for kw in cases:
        w, idx = grouped.route_topk(logits, k, **kw)
        kw_cpu = {a: (b.cpu() if torch.is_tensor(b) else b) for a, b in kw.items()}
        w_ref, idx_ref = grouped.route_topk(logits.cpu(), k, **kw_cpu)
        assert torch.equal(idx.cpu(), idx_ref), kw  # random logits: no ties, the order of the picks is the same
        torch.testing.assert_close(w.cpu(), w_ref, rtol=1e-4, atol=1e-6)


@pytest.mark.gpu
def test_moe_engine_decode_in_cuda_graphs_matches_eager_launches(kernels):
    """The MoE decode step is captured like the dense one (its layout is built on the device with static shapes): the
    replayed step draws the same tokens, log-probs and expert choices as eager launches of the same kernels."""
    from slime_b200.engine.engine import Engine
    from slime_b200.engine.server_args import ServerArgs
    from slime_b200.models.config import get_preset

    prompts = [[(5 * i + 3 * j) % 500 for j in range(6 + i)] for i in range(4)]
    got = []
    for graphs in (False, True):
        e = Engine(get_preset("tiny-moe"), ServerArgs(page_size=16, max_running_requests=4, context_length=128,
                                                      disable_cuda_graph=not graphs, enable_return_routed_experts=True),
                   device="cuda", num_pages=64)  # fmt: skip
        e.weights.init_random(0, std=0.2)
        reqs = e.generate(prompts, dict(max_new_tokens=10, temperature=0, ignore_eos=True), return_routed_experts=True)
        assert bool(e.runner.graphs) == graphs
        for r in reqs:
            routed = torch.cat(r.routed_experts)
            assert routed.shape == (len(r.input_ids) + len(r.output_ids) - 1, 2, 2)
        got.append(([r.output_ids for r in reqs], [r.output_logprobs for r in reqs], [torch.cat(r.routed_experts) for r in reqs]))
        e.shutdown()
    assert got[0][0] == got[1][0]
    assert max(abs(a - b) for x, y in zip(got[0][1], got[1][1]) for a, b in zip(x, y)) < 1e-3
    assert all(torch.equal(a, b) for a, b in zip(got[0][2], got[1][2]))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(512, 768), (264, 904), (1536, 128)])
@pytest.mark.parametrize("counts", [[300, 0, 77, 129, 1, 128, 64, 65], [0, 0, 5], [4000, 1]])
def test_weight_gradients_of_all_experts_in_one_launch(kernels, rows, cols, counts):
    """Adjacent main_grads: the one launch against a GEMM per expert, on what was there before; other experts' rows stay out of it.
    Sums of the same products in the same order: they differ by the roundings of the added fp32 parts alone."""
    from slime_b200 import ops
    from slime_b200.ops import _lib

    torch.manual_seed(sum(counts))
    lay = grouped.PaddedLayout(counts, "cuda")
    x, dy = (lay.pad(torch.randn(sum(counts), n, device="cuda").bfloat16()) for n in (cols, rows))
    flat = torch.randn(len(counts), rows, cols, device="cuda")
    want = flat.clone()
    for e, n in enumerate(counts):
        s = lay.padded_starts[e]
        if n:
            ops.gemm(dy[s : s + n], x[s : s + n], a_mn=True, b_mn=True, out=want[e], accumulate=True, bn=128, splitk=1)
    before = flat.clone()
    assert grouped._add_weight_grads(dy, x, lay, [flat[e] for e in range(len(counts))])
    _lib.check_status("cuda")
    torch.testing.assert_close(flat, want, rtol=2**-22, atol=2**-22)
    for e, n in enumerate(counts):
        assert n or torch.equal(flat[e], before[e])
    assert not grouped._add_weight_grads(dy, x, lay, [flat[e].clone() for e in range(len(counts))])  # not adjacent


@pytest.mark.gpu
@pytest.mark.parametrize("T,k,E,H", [(1, 1, 1, 8), (37, 2, 5, 136), (1000, 8, 128, 2048), (300, 3, 7, 1032)])
def test_rows_of_routes_on_gpu_match_the_definition(kernels, T, k, E, H):
    """Layout, placing and combining with their gradients against the CPU's; bf16 rows hold the same values, so the sums over k routes
    differ from fp32 ones by one rounding to bf16 (2^-8 of the value) and the dot products by the order of H fp32 products."""
    torch.manual_seed(T + H)
    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)])
    x, dy = torch.randn(T, H).bfloat16(), torch.randn(T, H).bfloat16()
    w = torch.rand(T, k)
    res = []
    for dev in ("cpu", "cuda"):
        lay = grouped.RoutedLayout(idx.to(dev), E)
        xd, wd = (t.detach().clone().to(dev).requires_grad_() for t in (x, w))
        rows = grouped.place_rows(xd, lay)
        y = grouped.combine_rows(rows * 2, lay, wd)
        y.backward(dy.to(dev))
        res.append([lay.slot_dest, lay.row_slot, lay.tile_expert, lay.expert_rows, rows.detach(), y.detach(), xd.grad, wd.grad])
        assert lay.counts == torch.bincount(idx.reshape(-1), minlength=E).tolist()
    for a, b in zip(res[0][:5], res[1][:5]):
        assert torch.equal(a, b.cpu())
    for a, b, tol in zip(res[0][5:], res[1][5:], (2**-7, 2**-6, 2e-5)):
        torch.testing.assert_close(b.cpu().float(), a.float(), rtol=tol, atol=tol * (H**0.5 if tol < 1e-3 else 1))
    with pytest.raises(IndexError):
        grouped.RoutedLayout(torch.full((4, 1), E, device="cuda"), E)


@pytest.mark.gpu
@pytest.mark.parametrize("T,k,E,fp8", [(1, 1, 4, False), (12, 8, 128, False), (12, 8, 128, True), (300, 2, 3, False), (9, 2, 8, True)])
def test_rows_behind_the_last_expert_are_left_out(kernels, T, k, E, fp8):
    """The engine's expert MLP over the used rows only, on buffers full of NaN, against zero padding and all rows: the same bits."""
    from slime_b200 import ops
    from slime_b200.engine import model_runner, quant

    torch.manual_seed(T + E)
    H, F = 256, 384
    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).cuda()
    x, probs = torch.randn(T, H, device="cuda").bfloat16(), torch.rand(T, k, device="cuda")
    w13, w2 = ((torch.randn(E, n, m, device="cuda") * 0.1).bfloat16() for n, m in ((2 * F, H), (H, F)))
    if fp8:
        w13, w2 = (quant.Fp8Weight(*w.shape, device="cuda") for w in (w13, w2))
        for w in (w13, w2):
            w.fill_random_(0.1)
    lay = grouped.DeviceLayout(idx, E)
    counts = torch.bincount(idx.reshape(-1), minlength=E)
    assert int(lay.rows_used) == int(((counts + 127) // 128 * 128).sum())
    lin = model_runner._grouped_linear
    want = lay.combine(lin(ops.swiglu(lin(lay.pad(x), w13, lay)), w2, lay), probs, T)
    junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 16, 1 << 18, 1 << 20, 1 << 22, 1 << 23, 1 << 24, 1 << 24)]
    del junk  # what the next buffers are made of
    used = lay.rows_used
    got = lay.combine(lin(ops.swiglu_used(lin(lay.place(x), w13, lay, used), used), w2, lay, used), probs, T)
    assert torch.equal(got, want)
