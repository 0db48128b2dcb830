"""tcgen05 GEMM (K-major operands) against an fp32 PyTorch reference."""

import pytest
import torch

from slime_b200 import ops

pytestmark = pytest.mark.gpu


def _ref(a, b, bias=None):
    out = a.float() @ b.float().t()
    return out + bias.float() if bias is not None else out


def _check(out, ref, tol=2e-2, K=None):
    """Per element: |out - ref| <= atol + rtol |ref|. A bf16 result carries one rounding of relative size 2^-9, a fp32
    result only the accumulation-order error; the absolute floor covers elements that cancel to ~0 (their error scales
    with sqrt(K) times the size of one product), so a wrong tile edge of small magnitude cannot hide behind the
    tensor's largest entry. ``tol`` keeps the old global bound as a second, coarser net."""
    err = (out.float() - ref).abs()
    K = K if K is not None else 1024
    rtol, atol = (1e-2, 2e-3 * K**0.5) if out.dtype == torch.bfloat16 else (2e-3, 5e-4 * K**0.5)
    bad = err > atol + rtol * ref.abs()
    assert not bad.any(), f"{int(bad.sum())} of {bad.numel()} elements off; worst {float(err.max()):.4g} at |ref| {float(ref.abs()[err.argmax() // ref.shape[1], err.argmax() % ref.shape[1]]):.4g}"
    assert err.max().item() / (ref.abs().max().item() + 1e-6) < tol


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 256, 128), (128, 256, 512), (384, 896, 896), (1000, 1152, 896),
                                   (77, 200, 72), (4096, 4864, 896), (130, 151936 // 16, 896)])  # fmt: skip
@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_nt_bf16(kernels, M, N, K, bn):
    from slime_b200.ops import _lib

    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = ops.gemm(a, b, bn=bn)
    torch.cuda.synchronize()
    _lib.check_status("cuda")
    _check(out, _ref(a, b), K=K)


def test_gemm_fp32_out_bias_accumulate(kernels):
    from slime_b200.ops import _lib

    torch.manual_seed(0)
    M, N, K = 300, 512, 256
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    out = ops.gemm(a, b, bias=bias, out_dtype=torch.float32)
    _check(out, _ref(a, b, bias), 5e-3, K=K)
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    ops.gemm(a, b, out=acc, accumulate=True)
    _check(acc, _ref(a, b) + 1.0, 5e-3, K=K)
    # strided output rows (a column block of a wider buffer)
    wide = torch.zeros(M, N + 64, device="cuda", dtype=torch.bfloat16)
    ops.gemm(a, b, out=wide[:, :N])
    _check(wide[:, :N], _ref(a, b), K=K)
    assert wide[:, N:].abs().max().item() == 0
    torch.cuda.synchronize()
    _lib.check_status("cuda")


def test_gemm_matches_cublas_closely(kernels):
    """Same bf16 inputs, fp32 accumulate: results should agree with cuBLAS to bf16 rounding."""

    torch.manual_seed(1)
    a = torch.randn(2048, 1024, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(1536, 1024, device="cuda", dtype=torch.bfloat16)
    ours = ops.gemm(a, b, out_dtype=torch.float32)
    ref = _ref(a, b)
    assert (ours - ref).abs().max().item() < 1e-2 * ref.abs().max().item()


def test_fp32_output_of_any_width(kernels):
    """Few rows and a long K ask for split-K, whose sums need rows of whole 16-byte pieces; other widths take one pass."""
    for N in (33, 90, 130, 64):
        a, b = torch.randn(7, 4096, device="cuda").bfloat16(), torch.randn(N, 4096, device="cuda").bfloat16()
        got = ops.gemm(a, b, out_dtype=torch.float32)
        torch.testing.assert_close(got, a.float() @ b.float().t(), atol=2e-2, rtol=2e-3)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (136, 136, 72), (520, 904, 320), (9728, 896, 1096)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("width", [256, 224, 192, 160, 128])
def test_pairs_of_sms(kernels, M, N, K, a_mn, b_mn, width):
    """Every width and layout of the two-SM kernel: the same sums in the same order as the one-SM kernel, bit for bit; where the last
    wave is cut along K, fp32 partial sums of the same products (half an ulp of the running sum for each of at most 74 parts)."""
    from slime_b200.ops import _lib

    torch.manual_seed(M + N + K)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device="cuda", dtype=torch.bfloat16)
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda", dtype=torch.bfloat16)
    sms = _lib.sm_count("cuda")
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    for dt in (torch.bfloat16, torch.float32):
        got = ops._gemm_pair(a, b, a_mn, b_mn, bias, None, dt, False, width, False, M, N, K, sms)
        assert torch.equal(got, ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, out_dtype=dt, bn=256, splitk=1))
    one = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, bn=256, splitk=1)
    for split in (False, True):
        acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
        ops._gemm_pair(a, b, a_mn, b_mn, None, acc, None, True, width, split, M, N, K, sms)
        torch.testing.assert_close(acc, one + 1.0, rtol=1e-5, atol=75 * 2.0**-24 * 4 * K**0.5)
    _lib.check_status("cuda")


@pytest.mark.parametrize("out,inp", [(9728, 896), (2560, 4096), (64, 128)])
def test_products_over_nothing(kernels, out, inp):
    """No rows: a linear layer gives none, its input's gradient has none, its weights' gradients gain nothing, whatever the width."""
    x = torch.empty(0, inp, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    for held in (True, False):
        w = torch.randn(out, inp, device="cuda").bfloat16().requires_grad_()
        b = torch.randn(out, device="cuda").bfloat16().requires_grad_()
        if held:
            w.main_grad = torch.ones(out, inp, device="cuda")
        y = ops.linear(x, w, b)
        y.backward(torch.empty_like(y))
        assert y.shape == (0, out) and x.grad.shape == x.shape and (b.grad == 0).all()
        assert (w.main_grad == 1).all() if held else (w.grad == 0).all()
    a, c = torch.empty(0, 16384, device="cuda", dtype=torch.bfloat16), torch.randn(16384, 896, device="cuda").bfloat16()
    assert ops.gemm(a, c, b_mn=True).shape == (0, 896)  # the gradient of no rows behind a head
    empty, bias = torch.empty(5, 0, device="cuda", dtype=torch.bfloat16), torch.randn(7, device="cuda").bfloat16()
    assert torch.equal(ops.gemm(empty, empty.new_empty(7, 0), bias=bias), bias.expand(5, 7))


@pytest.mark.parametrize("M,N,K", [(9728, 896, 15800), (2560, 4096, 9198), (264, 24904, 1096), (9472, 512, 72)])
def test_weight_gradients_are_the_same_on_every_run(kernels, M, N, K):
    """Outputs of more than a wave of tiles, added to: the ranges of a cut tile are summed in one order. Against 64 bits: each of K / 16 steps
    of a sum of at most 4 sqrt(K) may lose an ulp, 2^-23 of it."""
    torch.manual_seed(K)
    dy, x = (torch.randn(K, n, device="cuda").bfloat16() for n in (M, N))
    start = torch.randn(M, N, device="cuda")
    runs = [ops.gemm(dy, x, a_mn=True, b_mn=True, out=start.clone(), accumulate=True) for _ in range(8)]
    assert all(torch.equal(runs[0], r) for r in runs[1:])
    for cut in (False, True):  # whatever the plan is
        runs = [ops._gemm_pair(dy, x, True, True, None, start.clone(), None, True, 256, cut, M, N, K, 148) for _ in range(8)]
        assert all(torch.equal(runs[0], r) for r in runs[1:])
        torch.testing.assert_close((runs[0] - start).double(), dy.double().t() @ x.double(), rtol=1e-5, atol=K / 16 * 2.0**-23 * 4 * K**0.5 + 2e-6)


@pytest.mark.parametrize("M,N,K", [(265, 896, 151936), (1, 8, 16384), (130, 900, 20000), (257, 4, 16390)])
def test_few_rows_over_a_long_sum_are_the_same_on_every_run(kernels, M, N, K):
    """A bf16 output whose sums are cut along K, written through any row view: one order, one rounding."""
    torch.manual_seed(M)
    a, b = torch.randn(M, -(-K // 8) * 8, device="cuda").bfloat16()[:, :K], (torch.randn(K, N + (-N) % 8, device="cuda") * 0.02).bfloat16()[:, :N]
    bias = torch.randn(N, device="cuda").bfloat16()
    wide = torch.zeros(M, N + 4, device="cuda", dtype=torch.bfloat16)
    runs = [ops.gemm(a, b, b_mn=True, bias=bias) for _ in range(8)]
    assert all(torch.equal(runs[0], r) for r in runs[1:])
    ops.gemm(a, b, b_mn=True, bias=bias, out=wide[:, :N])
    assert torch.equal(wide[:, :N], runs[0]) and (wide[:, N:] == 0).all()
    torch.testing.assert_close(runs[0].double(), a.double() @ b.double() + bias.double(), rtol=2**-8, atol=1e-3)
