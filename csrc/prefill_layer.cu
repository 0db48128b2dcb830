// One transformer layer of a prefill as one call from the host: the launches of norm, projections, rotation with the cache write,
// attention and MLP in order, on buffers the caller has set aside. No kernels of its own.
//
// A prompt of 300 tokens keeps the GPU busy for 75 us a layer (Qwen2.5-0.5B); issuing the same ten launches one by one from Python
// took 330 us.
#include "common.cuh"

extern "C" {
int sb_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, float*, int, int, float, cudaStream_t);
int sb_rmsnorm_fwd_f32x(const float*, const void*, const void*, void*, void*, float*, int, int, float, cudaStream_t);
int sb_gemm_pair(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, int, float*, int, const int*,
                 const int*, int*, int, cudaStream_t);
int sb_gemm_bf16_splitk(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, int, int*, int,
                        cudaStream_t);
int sb_rope_kv_write(void*, const int*, const float*, const void*, const void*, const int*, void*, void*, int, int, int, int, int, float,
                     cudaStream_t);
int sb_flash_fwd(const void*, const void*, const void*, void*, float*, const int*, int, int, int, int, int, int, int, int, int, int, int, int,
                 float, int*, cudaStream_t);
int sb_swiglu_fwd(const void*, void*, long, int, const int*, cudaStream_t);
}

namespace sb {

// Filled by slime_b200/engine/native_layer.py::Layer, which has the same fields in the same order.
struct PrefillLayer {
  int bytes;  // sizeof(PrefillLayer) as the caller sees it
  int T, H, Hq, Hkv, D, F;  // F = 0: the layer's MLP is not of this kind; the call ends with its normed input
  int nseg, max_q_tiles, x_f32, num_sms;
  float eps, scale;
  int plan[4][3];  // qkv, output, gate and up, down: width on pairs of SMs or 0, width on one SM, slices of K
  int reserved;
  const void *x, *res, *ln1, *qkv_w, *qkv_b, *q_norm, *k_norm, *o_w, *ln2, *gate_up, *down;
  const int *positions, *slots, *seg;
  const float* rope;
  void *k_cache, *v_cache;
  void *normed, *h1, *h2, *qkv, *ctx, *gu, *act;  // bf16: [T, H] x 3, [T, (Hq + 2 Hkv) D], [T, Hq D], [T, 2 F], [T, F]
  float *proj, *lse, *rstd;                       // [T, H], [Hq, T], [T]
  int* status;
};

static int project(const PrefillLayer& p, int which, const void* a, const void* w, void* out, const void* bias, int N, int K, bool f32,
                   cudaStream_t s) {
  const int* plan = p.plan[which];
  if (plan[0] > 0)
    return sb_gemm_pair(a, w, out, bias, p.T, N, K, K, K, N, 0, 0, f32, 0, plan[0], 0, nullptr, 1, nullptr, nullptr, p.status, p.num_sms, s);
  if (plan[2] > 1)  // the slices are added up in the output
    if (cudaError_t e = cudaMemsetAsync(out, 0, static_cast<size_t>(p.T) * N * 4, s); e != cudaSuccess) return (int)e;
  return sb_gemm_bf16_splitk(a, w, out, bias, p.T, N, K, K, K, N, 0, 0, f32, 0, plan[1], plan[2], p.status, p.num_sms, s);
}

}  // namespace sb

// x [T, H] (bf16, or the fp32 sum of a projection) and the residual stream in front of it (null: x is the stream) -> `proj`, the MLP's
// sum in fp32, and the stream in front of that in h2. F = 0: `normed` and h2.
extern "C" int sb_prefill_layer(const void* layer, cudaStream_t s) {
  const sb::PrefillLayer& p = *static_cast<const sb::PrefillLayer*>(layer);
  if (p.bytes != static_cast<int>(sizeof(sb::PrefillLayer))) {
    sb::set_last_error("sb_prefill_layer: the caller's struct has another size");
    return (int)cudaErrorInvalidValue;
  }
  const int row = (p.Hq + 2 * p.Hkv) * p.D, q = p.Hq * p.D;
  const bool sum = p.res != nullptr || p.x_f32 != 0;
  const void* stream1 = sum ? p.h1 : p.x;
  int rc = p.x_f32 ? sb_rmsnorm_fwd_f32x(static_cast<const float*>(p.x), p.res, p.ln1, p.normed, p.h1, p.rstd, p.T, p.H, p.eps, s)
                   : sb_rmsnorm_fwd(p.x, p.res, p.ln1, p.normed, sum ? p.h1 : nullptr, p.rstd, p.T, p.H, p.eps, s);
  if (rc == 0) rc = sb::project(p, 0, p.normed, p.qkv_w, p.qkv, p.qkv_b, row, p.H, false, s);
  if (rc == 0)
    rc = sb_rope_kv_write(p.qkv, p.positions, p.rope, p.q_norm, p.k_norm, p.slots, p.k_cache, p.v_cache, p.T, p.Hq, p.Hkv, p.D, row, p.eps, s);
  const __nv_bfloat16* qkv = static_cast<const __nv_bfloat16*>(p.qkv);
  if (rc == 0)
    rc = sb_flash_fwd(qkv, qkv + q, qkv + q + p.Hkv * p.D, p.ctx, p.lse, p.seg, p.nseg, p.max_q_tiles, p.T, p.T, p.Hq, p.Hkv, p.D, row, row, row,
                      q, p.T, p.scale, p.status, s);
  if (rc == 0) rc = sb::project(p, 1, p.ctx, p.o_w, p.proj, nullptr, p.H, q, true, s);
  if (rc == 0) rc = sb_rmsnorm_fwd_f32x(p.proj, stream1, p.ln2, p.normed, p.h2, p.rstd, p.T, p.H, p.eps, s);
  if (rc != 0 || p.F == 0) return rc;
  rc = sb::project(p, 2, p.normed, p.gate_up, p.gu, nullptr, 2 * p.F, p.H, false, s);
  if (rc == 0) rc = sb_swiglu_fwd(p.gu, p.act, p.T, p.F, nullptr, s);
  if (rc == 0) rc = sb::project(p, 3, p.act, p.down, p.proj, nullptr, p.H, p.F, true, s);
  return rc;
}
