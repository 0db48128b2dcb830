// Varlen causal flash attention, backward, on the 5th-gen tensor cores (sm_100a). Same segment table as the forward
// (flash_fwd_sm100.cu): seg[s] = { q_off, q_len, k_off, k_len }, query i sees keys j <= (k_len - q_len) + i.
//
// Launches, no atomics, fixed summation order (bitwise reproducible):
//
//   delta    D_i = sum_d dO[i, d] * O[i, d]                                   D / 8 lanes per (token, head)
//   dkv      one CTA per (128-key tile, kv head, part of the query heads of the group): K, V stay in shared memory; the query
//            blocks (64 rows) of those heads that can see the tile stream through a ring:
//                S^T  = K Q^T          dP^T = V dO^T                (M 128 keys, N 64 queries, K D)     -> TMEM
//                P^T  = 2^(S^T c - lse),   dS^T = P^T (dP^T - D)             TMEM -> registers -> TMEM (bf16, in place)
//                dV  += P^T dO         dK  += dS^T Q                (M 128 keys, N D, K 64)   accumulated in TMEM
//   sum      with several parts: dK, dV = sum of the parts' fp32 results, in part order
//   dq       one CTA per (128-query tile, query head): Q, dO stay in shared memory, key blocks (64) stream:
//                S = Q K^T, dP = dO V^T (M 128, N 64, K D);  dS = P (dP - D);  dQ += dS K  (M 128, N D, K 64)
//   (the factor `scale` of dS is applied to the fp32 accumulators of dK and dQ)
//
// The score products are recomputed in both passes (7 tile products instead of 5); in exchange every output tile has
// one owner, so nothing is accumulated through global memory. A Q / dO (or K / V) block is loaded once by TMA and used
// twice: K-major as the B operand of the score products and MN-major as the B operand of the gradient products.
// CTA = 10 warps: TMA producer, MMA issuer, two groups of four element-wise warps that take the blocks in turn.
//
// What bounds it: the chain score product -> exponentials -> gradient product of a block. With all eight warps on the same
// block, P and dS going through one shared-memory buffer, a 128 x 64 block took 3900 cycles where its products need about 1300 and
// its exponentials 512. So (1) the two groups own one score buffer each, and while one waits for its products the other
// computes; (2) P and dS go back to TMEM over the scores they came from and are the A operand there, which saves their
// way through shared memory, its fence and the second read of 16 KB per product; (3) blocks that no mask touches skip the comparisons,
// the products of two columns are one instruction, the statistics of 64 queries are staged once per warp; (4) the longest tiles start first
// (few query tiles see the last keys, few key tiles are seen by the first queries), and a dkv launch with too few CTAs for the
// machine splits the query heads of a group. Measured,
// all launches, before -> after: 8011 + 1187 tokens, 32 / 8 heads of 128: 3821 -> 2244 us; 19 sequences of 384 to 1284 tokens, 14 / 2 heads
// of 64: 581 -> 360 us; six sequences, 8239 tokens, 32 / 4 heads of 128: 1159 -> 718 us. What is left is the chain of one block: two in
// flight hide a good part of it, a third score buffer does not fit beside dK and dV of 128 columns each.
// All mbarrier waits are bounded; on expiry the CTA records a status word, drains and frees its TMEM.
#include "common.cuh"

#include <type_traits>

namespace sb {

constexpr int FB_T = 128;        // stationary tile rows (keys in dkv, queries in dq) = TMEM lanes
constexpr int FB_S = 64;         // streamed block rows
constexpr int FB_THREADS = 320;  // TMA warp, MMA warp, 8 element-wise warps
constexpr int FB_STAGES = 4;     // of the streamed operands (dkv at D = 128: 64 KB stationary + 4 x 32 KB)

template <int D>
struct FbSmem {
  static constexpr int NCH = D / 64;
  static constexpr int TILE_BYTES = FB_T * 128 * NCH;  // stationary operand, [NCH][128 rows][128 B]
  static constexpr int BLK_BYTES = FB_S * 128 * NCH;   // streamed operand, [NCH][64 rows][128 B]
  static constexpr int STAT_BYTES = 8 * 2 * FB_S * 4;  // per element-wise warp: -lse (log2 domain) and -D of 64 queries
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = 2 * TILE_BYTES + 2 * FB_STAGES * BLK_BYTES + STAT_BYTES + BAR_BYTES + 1024;
  // block `it` uses buffer b = it & 1: scores @64 b, dP @128 + 64 b (P and dS over their first 32 columns); accumulators @256, @256 + D
  static constexpr int TMEM_COLS = 512;
};

__device__ __forceinline__ float fb_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void fb_named_barrier(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// -------------------------------------------------------------------------------------------------- delta
// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; D / 8 lanes with one 16-byte vector of each per (t, h).
template <int D>
__global__ void __launch_bounds__(256)
flash_bwd_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, float* __restrict__ delta, int T,
                       int H, int o_stride, int do_stride, int delta_stride) {
  constexpr int LANES = D / 8;
  pdl_wait();
  pdl_launch_dependents();
  const long g = (static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x) / LANES;
  const int l = threadIdx.x % LANES;
  const bool in = g < static_cast<long>(T) * H;
  const int t = static_cast<int>(g / H), h = static_cast<int>(g % H);
  float acc = 0.f;
  if (in) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + static_cast<size_t>(t) * o_stride + h * D + l * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(d_o + static_cast<size_t>(t) * do_stride + h * D + l * 8);
    const uint32_t ua[4] = {a.x, a.y, a.z, a.w}, ub[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(ua[i]), y = unpack_bf16x2(ub[i]);
      acc += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int m = LANES / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (in && l == 0) delta[static_cast<size_t>(h) * delta_stride + t] = acc;
}

// Shared skeleton of the two passes. PASS_DQ = false: stationary = (K, V) tile, streamed = (Q, dO) blocks, outputs
// dK and dV. PASS_DQ = true: stationary = (Q, dO) tile, streamed = (K, V) blocks, output dQ.
//   tmA0 / tmA1: tensor maps of the two stationary operands (box 128 rows), tmB0 / tmB1: of the streamed ones (box 64).
//   score product 0:  A0 x B0^T  (K Q^T   or  Q K^T)      score product 1:  A1 x B1^T  (V dO^T  or  dO V^T)
//   dkv: acc0 (dV) += P^T  x B1 (dO),  acc1 (dK) += dS^T x B0 (Q)          dq: acc0 (dQ) += dS x B0 (K)
// Grid (x): heads fastest, so that the CTAs that run at one time share the streamed operands in L2, then tiles, longest first.
// parts > 1 (dkv): CTA `part` takes the query heads [part * G / parts, (part + 1) * G / parts) of the group and leaves fp32 sums in
// part_out [parts][2 (dV, dK)][Tk][Hkv * D].
template <int D, bool PASS_DQ>
__global__ void __launch_bounds__(FB_THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
                 const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
                 const float* __restrict__ lse, const float* __restrict__ delta, __nv_bfloat16* __restrict__ out0,
                 __nv_bfloat16* __restrict__ out1, float* __restrict__ part_out, const int* __restrict__ seg, int nseg, int Hq, int Hkv,
                 int Tk, int parts, int tiles, int out0_stride, int out1_stride, int stat_stride, float scale, int* status) {
  using S = FbSmem<D>;
  constexpr int NCH = S::NCH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA0 = smem;
  uint8_t* sA1 = sA0 + S::TILE_BYTES;
  uint8_t* sB0 = sA1 + S::TILE_BYTES;                 // [FB_STAGES]
  uint8_t* sB1 = sB0 + FB_STAGES * S::BLK_BYTES;      // [FB_STAGES]
  float* sStat = reinterpret_cast<float*>(sB1 + FB_STAGES * S::BLK_BYTES);
  uint64_t* a_full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStat) + S::STAT_BYTES);
  uint64_t* b_full = a_full + 1;              // [FB_STAGES]
  uint64_t* b_empty = b_full + FB_STAGES;     // [FB_STAGES]
  uint64_t* sc_full = b_empty + FB_STAGES;    // [2] both score products of a block are in TMEM
  uint64_t* pds_full = sc_full + 2;           // [2] element-wise warps -> MMA: P / dS are in TMEM (4 arrivals)
  uint64_t* acc_full = pds_full + 2;          // every product has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* work = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = Hq / Hkv;
  const int per_tile = PASS_DQ ? Hq : Hkv * parts;
  const int hx = blockIdx.x % per_tile;
  const int hy = PASS_DQ ? hx : hx % Hkv;  // query head (dq) or kv head (dkv)
  const int part = PASS_DQ ? 0 : hx / Hkv;
  const int head_lo = part * G / parts, head_hi = (part + 1) * G / parts;

  if (threadIdx.x == 0) {
    mbar_init(a_full, 1);
    for (int s = 0; s < FB_STAGES; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sc_full[b], 1);
      mbar_init(&pds_full[b], 4);
    }
    mbar_init(acc_full, 1);
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA0);
    tma_prefetch_desc(&tmA1);
    tma_prefetch_desc(&tmB0);
    tma_prefetch_desc(&tmB1);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, S::TMEM_COLS);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_launch_dependents();
  if (warp == 0) {
    // dq tiles are numbered from the last one down (the last queries see the most keys); dkv tiles as they are
    const int t = blockIdx.x / per_tile;
    int tile;
    const int found = segment_of_tile(seg, nseg, PASS_DQ ? 1 : 3, FB_T, PASS_DQ ? tiles - 1 - t : t, tile);
    if (lane == 0) {
      work[0] = found;
      work[1] = tile;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int sidx = work[0];
  if (sidx >= 0) {
    const int q_off = seg[4 * sidx], q_len = seg[4 * sidx + 1], k_off = seg[4 * sidx + 2], k_len = seg[4 * sidx + 3];
    const int shift = k_len - q_len;
    const int t0 = work[1] * FB_T;  // first row of the stationary tile inside the segment
    // streamed blocks [blk_lo, blk_hi) per query head; heads: dkv loops over its heads of the group, dq has one
    int blk_lo, blk_hi, n_heads;
    if (PASS_DQ) {
      blk_lo = 0;
      blk_hi = (min(k_len, shift + t0 + FB_T) + FB_S - 1) / FB_S;
      n_heads = 1;
    } else {
      blk_lo = max(0, t0 - shift) / FB_S;
      blk_hi = (q_len + FB_S - 1) / FB_S;
      n_heads = head_hi - head_lo;
    }
    const int per_head = max(blk_hi - blk_lo, 0);
    const int n_it = per_head * n_heads;
    const int a_col = hy * D;                            // column of the stationary operand's head
    const int a_row = (PASS_DQ ? q_off : k_off) + t0;
    const int b_row0 = PASS_DQ ? k_off : q_off;

    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0) {
        mbar_arrive_expect_tx(a_full, 2 * S::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          tma_load_2d(sA0 + c * (FB_T * 128), &tmA0, a_full, a_col + c * 64, a_row);
          tma_load_2d(sA1 + c * (FB_T * 128), &tmA1, a_full, a_col + c * 64, a_row);
        }
        for (int it = 0; it < n_it; ++it) {
          const int st = it % FB_STAGES;
          if (!mbar_wait(&b_empty[st], ((it / FB_STAGES) & 1) ^ 1, cta_abort, status, ERR_WAIT_EMPTY)) break;
          const int hd = head_lo + it / per_head, blk = blk_lo + it % per_head;
          const int b_col = (PASS_DQ ? hy / G : hy * G + hd) * D;
          mbar_arrive_expect_tx(&b_full[st], 2 * S::BLK_BYTES);
#pragma unroll
          for (int c = 0; c < NCH; ++c) {
            tma_load_2d(sB0 + st * S::BLK_BYTES + c * (FB_S * 128), &tmB0, &b_full[st], b_col + c * 64, b_row0 + blk * FB_S);
            tma_load_2d(sB1 + st * S::BLK_BYTES + c * (FB_S * 128), &tmB1, &b_full[st], b_col + c * 64, b_row0 + blk * FB_S);
          }
        }
        // the stationary tile must have landed before this CTA's shared memory is given back
        if (n_it == 0) mbar_wait(a_full, 0, cta_abort, status, ERR_WAIT_FULL);
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (lane == 0 && n_it > 0) {
        constexpr uint32_t idesc_sc = make_idesc(FB_T, FB_S, 1, 1, 0, 0);  // scores: both operands K-major
        constexpr uint32_t idesc_g = make_idesc(FB_T, D, 1, 1, 0, 1);      // gradients: A in TMEM, B (streamed block) MN-major
        const uint32_t a0 = smem_u32(sA0), a1 = smem_u32(sA1);
        auto issue_scores = [&](int it) {
          const uint32_t b0 = smem_u32(sB0 + (it % FB_STAGES) * S::BLK_BYTES), b1 = smem_u32(sB1 + (it % FB_STAGES) * S::BLK_BYTES);
          const uint32_t buf = (it & 1) * FB_S;
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t oa = (k >> 2) * (FB_T * 128) + (k & 3) * 32, ob = (k >> 2) * (FB_S * 128) + (k & 3) * 32;
            umma_f16(tmem_base + buf, make_smem_desc(a0 + oa, 16, 1024, UMMA_SWIZZLE_128B),
                     make_smem_desc(b0 + ob, 16, 1024, UMMA_SWIZZLE_128B), idesc_sc, k != 0 ? 1u : 0u);
          }
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t oa = (k >> 2) * (FB_T * 128) + (k & 3) * 32, ob = (k >> 2) * (FB_S * 128) + (k & 3) * 32;
            umma_f16(tmem_base + 128 + buf, make_smem_desc(a1 + oa, 16, 1024, UMMA_SWIZZLE_128B),
                     make_smem_desc(b1 + ob, 16, 1024, UMMA_SWIZZLE_128B), idesc_sc, k != 0 ? 1u : 0u);
          }
          umma_commit(&sc_full[it & 1]);
        };
        bool ok = mbar_wait(a_full, 0, cta_abort, status, ERR_WAIT_FULL);
        for (int it = 0; it < min(2, n_it) && ok; ++it) {
          ok = mbar_wait(&b_full[it], 0, cta_abort, status, ERR_WAIT_FULL);
          if (ok) {
            tc_fence_after();
            issue_scores(it);
          }
        }
        for (int it = 0; it < n_it && ok; ++it) {
          ok = mbar_wait(&pds_full[it & 1], (it >> 1) & 1, cta_abort, status, ERR_WAIT_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
          const uint32_t b0 = smem_u32(sB0 + (it % FB_STAGES) * S::BLK_BYTES), b1 = smem_u32(sB1 + (it % FB_STAGES) * S::BLK_BYTES);
          const uint32_t p_t = tmem_base + (it & 1) * FB_S, ds_t = tmem_base + 128 + (it & 1) * FB_S;
#pragma unroll
          for (int k = 0; k < FB_S / 16; ++k) {
            // A: 16 values = 8 TMEM columns; B: streamed block read MN-major, 16 rows = 2048 B, 64-wide chunks of the head dim
            // FB_S * 128 B apart
            if (!PASS_DQ)
              umma_f16_ts(tmem_base + 256, p_t + k * 8, make_smem_desc(b1 + k * 2048, FB_S * 128, 1024, UMMA_SWIZZLE_128B), idesc_g,
                          (it != 0 || k != 0) ? 1u : 0u);
            umma_f16_ts(tmem_base + 256 + (PASS_DQ ? 0 : D), ds_t + k * 8, make_smem_desc(b0 + k * 2048, FB_S * 128, 1024, UMMA_SWIZZLE_128B),
                        idesc_g, (it != 0 || k != 0) ? 1u : 0u);
          }
          umma_commit(&b_empty[it % FB_STAGES]);
          if (it + 1 == n_it) umma_commit(acc_full);
          if (it + 2 < n_it) {
            // the scores of block it + 2 replace P and dS of block it: products of one CTA run in the order they are issued in
            ok = mbar_wait(&b_full[(it + 2) % FB_STAGES], ((it + 2) / FB_STAGES) & 1, cta_abort, status, ERR_WAIT_FULL);
            if (!ok) break;
            tc_fence_after();
            issue_scores(it + 2);
          }
        }
      }
    } else {
      // ------------------------------------------------------------------ element-wise warps
      const int quarter = warp & 3, grp = (warp - 2) >> 2;
      const int row = quarter * 32 + lane;  // TMEM lane: key (dkv) or query (dq) inside the tile
      const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const float c_log2 = scale * 1.4426950408889634f;
      const uint64_t c2 = f2_pack(c_log2, c_log2);
      const int ti = t0 + row;  // index inside the segment of this thread's key / query
      float* w_lse = sStat + (warp - 2) * 2 * FB_S;  // this warp's copy of the block's statistics
      float* w_del = w_lse + FB_S;
      uint64_t my_lse2 = 0, my_delta = 0;
      if (PASS_DQ) {
        const bool v = ti < q_len;
        const size_t at = static_cast<size_t>(hy) * stat_stride + q_off + ti;
        const float l = v ? -lse[at] * 1.4426950408889634f : -INFINITY, d = v ? -delta[at] : 0.f;
        my_lse2 = f2_pack(l, l);
        my_delta = f2_pack(d, d);
      }
      bool ok = true;
      for (int it = grp; it < n_it; it += 2) {
        const int hd = head_lo + it / per_head, blk = blk_lo + it % per_head;
        const int c0 = blk * FB_S;  // first streamed index (query in dkv, key in dq)
        if (!PASS_DQ) {
          const size_t at = static_cast<size_t>(hy * G + hd) * stat_stride + q_off + c0;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int i = lane + 32 * u;
            const bool v = c0 + i < q_len;
            w_lse[i] = v ? -lse[at + i] * 1.4426950408889634f : -INFINITY;
            w_del[i] = v ? -delta[at + i] : 0.f;
          }
          __syncwarp();
        }
        ok = mbar_wait(&sc_full[grp], (it >> 1) & 1, cta_abort, status, ERR_WAIT_TMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        // visible columns [cmin, cmax]. dkv: key ti (row) is seen by query c0 + c iff ti <= shift + c0 + c, c0 + c < q_len.
        //                               dq:  query ti sees key c0 + c iff c0 + c <= shift + ti, c0 + c < k_len.
        bool masked;  // the same for the whole tile
        int cmin, cmax;
        if (PASS_DQ) {
          masked = c0 + FB_S - 1 > min(shift + t0, k_len - 1) || t0 + FB_T > q_len;
          cmin = 0;
          cmax = min(shift + ti, k_len - 1) - c0;
        } else {
          masked = t0 + FB_T - 1 > shift + c0 || c0 + FB_S > q_len || t0 + FB_T > k_len;
          cmin = ti < k_len ? ti - shift - c0 : FB_S;
          cmax = q_len - 1 - c0;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t rs[32], rd[32], pk[16], dk[16];
          tmem_ld_32x32(lane_addr + grp * FB_S + half * 32, rs);
          tmem_ld_32x32(lane_addr + 128 + grp * FB_S + half * 32, rd);
          tmem_ld_wait();
          auto pairs = [&](auto use_mask) {
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              uint64_t l[2] = {my_lse2, my_lse2}, d[2] = {my_delta, my_delta};
              if (!PASS_DQ) {
                const float4 a = *reinterpret_cast<const float4*>(w_lse + half * 32 + c), b = *reinterpret_cast<const float4*>(w_del + half * 32 + c);
                l[0] = f2_pack(a.x, a.y);
                l[1] = f2_pack(a.z, a.w);
                d[0] = f2_pack(b.x, b.y);
                d[1] = f2_pack(b.z, b.w);
              }
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int i = c + 2 * u;
                float p0, p1, s0, s1;
                f2_unpack(f2_fma(f2_pack(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), c2, l[u]), p0, p1);
                p0 = fb_exp2(p0);
                p1 = fb_exp2(p1);
                if (decltype(use_mask)::value) {
                  if (half * 32 + i < cmin || half * 32 + i > cmax) p0 = 0.f;
                  if (half * 32 + i + 1 < cmin || half * 32 + i + 1 > cmax) p1 = 0.f;
                }
                f2_unpack(f2_mul(f2_pack(p0, p1), f2_add(f2_pack(__uint_as_float(rd[i]), __uint_as_float(rd[i + 1])), d[u])), s0, s1);
                if (decltype(use_mask)::value) {  // what lies outside may hold anything
                  if (p0 == 0.f) s0 = 0.f;
                  if (p1 == 0.f) s1 = 0.f;
                }
                pk[i >> 1] = pack_bf16x2(p0, p1);
                dk[i >> 1] = pack_bf16x2(s0, s1);
              }
            }
          };
          if (masked) pairs(std::true_type{});
          else pairs(std::false_type{});
          // in place: the packed 32 columns of a half take 16, of which the ones already read are free
          if (!PASS_DQ) tmem_st_32x16(lane_addr + grp * FB_S + half * 16, pk);
          tmem_st_32x16(lane_addr + 128 + grp * FB_S + half * 16, dk);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pds_full[grp]);
      }
      // ---- epilogue: accumulators -> bf16 -> staged through the streamed operands' buffers -> coalesced rows
      if (ok && n_it > 0) {
        ok = mbar_wait(acc_full, 0, cta_abort, status, ERR_WAIT_TMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
        constexpr int CH = D / 8;  // 16-byte chunks per output row
        constexpr int HALF_COLS = D / 2;
        const int n_acc = PASS_DQ ? 1 : 2;
        const int rows_valid = min(FB_T, (PASS_DQ ? q_len : k_len) - t0);
        const int out_row0 = (PASS_DQ ? q_off : k_off) + t0;
        for (int a = 0; a < n_acc; ++a) {
          uint8_t* stage = (a == 0) ? sB1 : sB0;  // FB_STAGES * BLK_BYTES >= 128 rows * D * 2 bytes
          const float f = PASS_DQ || a == 1 ? scale : 1.f;
#pragma unroll
          for (int c4 = 0; c4 < HALF_COLS / 32; ++c4) {
            uint32_t r[32];
            const int col = grp * HALF_COLS + c4 * 32;
            if (n_it > 0) {
              tmem_ld_32x32(lane_addr + 256 + a * D + col, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0;
            }
            if (!PASS_DQ && parts > 1) {
              if (row < rows_valid) {
                float4* dst = reinterpret_cast<float4*>(part_out + ((static_cast<size_t>(part) * 2 + a) * Tk + out_row0 + row) * (Hkv * D) + hy * D + col);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  dst[i] = make_float4(__uint_as_float(r[4 * i]) * f, __uint_as_float(r[4 * i + 1]) * f, __uint_as_float(r[4 * i + 2]) * f,
                                       __uint_as_float(r[4 * i + 3]) * f);
              }
              continue;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * i]) * f, __uint_as_float(r[8 * i + 1]) * f);
              v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * f, __uint_as_float(r[8 * i + 3]) * f);
              v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * f, __uint_as_float(r[8 * i + 5]) * f);
              v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * f, __uint_as_float(r[8 * i + 7]) * f);
              const int ch = col / 8 + i;
              *reinterpret_cast<uint4*>(stage + row * (D * 2) + ((ch ^ (row & (CH - 1))) << 4)) = v;
            }
          }
        }
        if (PASS_DQ || parts == 1) {
          fb_named_barrier(1, 256);
          const int t = threadIdx.x - 64;  // 0..255
          for (int a = 0; a < n_acc; ++a) {
            const uint8_t* stage = (a == 0) ? sB1 : sB0;
            __nv_bfloat16* dst = (a == 0) ? out0 : out1;
            const int stride = (a == 0) ? out0_stride : out1_stride;
            for (int idx = t; idx < rows_valid * CH; idx += 256) {
              const int rr = idx / CH, ch = idx % CH;
              const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * (D * 2) + ((ch ^ (rr & (CH - 1))) << 4));
              *reinterpret_cast<uint4*>(dst + static_cast<size_t>(out_row0 + rr) * stride + hy * D + ch * 8) = v;
            }
          }
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*cta_abort) {
    const unsigned long long t_a = globaltimer_ns();
    while (globaltimer_ns() - t_a < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem_base, S::TMEM_COLS);
}

// dV, dK = sum over the parts, in part order, of the rows inside a segment: CTA (tile, 0: dV, 1: dK, eight rows of the tile), one 8-column
// vector per thread and step. Parts are taken where there are few tiles, so a tile has many CTAs here (one took 50 us for 128 rows of 1024
// columns in four parts).
constexpr int FB_SUM_ROWS = 8;
__global__ void __launch_bounds__(256)
flash_bwd_sum_kernel(const float* __restrict__ part_out, __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ dk, const int* __restrict__ seg,
                     int nseg, int parts, int Tk, int width, int dv_stride, int dk_stride) {
  __shared__ int work[2];
  pdl_wait();
  pdl_launch_dependents();
  if (threadIdx.x < 32) {
    int tile;
    const int found = segment_of_tile(seg, nseg, 3, FB_T, blockIdx.x, tile);
    if (threadIdx.x == 0) {
      work[0] = found;
      work[1] = tile;
    }
  }
  __syncthreads();
  if (work[0] < 0) return;
  const int t0 = work[1] * FB_T + blockIdx.z * FB_SUM_ROWS, rows = min(FB_SUM_ROWS, seg[4 * work[0] + 3] - t0), row0 = seg[4 * work[0] + 2] + t0;
  const int a = blockIdx.y, vecs = width / 8;
  __nv_bfloat16* dst = a == 0 ? dv : dk;
  const int stride = a == 0 ? dv_stride : dk_stride;
  for (int i = threadIdx.x; i < rows * vecs; i += 256) {
    const int r = row0 + i / vecs, c = (i % vecs) * 8;
    float s[8] = {};
#pragma unroll 4
    for (int p = 0; p < parts; ++p) {
      const float4* src = reinterpret_cast<const float4*>(part_out + ((static_cast<size_t>(p) * 2 + a) * Tk + r) * width + c);
      const float4 x = src[0], y = src[1];
      s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w;
      s[4] += y.x; s[5] += y.y; s[6] += y.z; s[7] += y.w;
    }
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * stride + c) =
        make_uint4(pack_bf16x2(s[0], s[1]), pack_bf16x2(s[2], s[3]), pack_bf16x2(s[4], s[5]), pack_bf16x2(s[6], s[7]));
  }
}

template <int D>
static int launch_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                            float* delta, void* dq, void* dk, void* dv, float* part_out, int parts, const int* seg, int nseg,
                            int max_q_tiles, int max_k_tiles, int Tq, int Tk, int Hq, int Hkv, int q_stride, int k_stride,
                            int v_stride, int o_stride, int do_stride, int dq_stride, int dk_stride, int dv_stride,
                            int stat_stride, float scale, int* status, cudaStream_t s) {
  using S = FbSmem<D>;
  using bf16 = __nv_bfloat16;
  auto map = [&](const void* p, int rows, int heads, int stride, int box_rows) {
    return make_tmap_2d(p, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, size_t(heads) * D, size_t(stride) * 2, box_rows, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  };
  {
    const long threads = static_cast<long>(Tq) * Hq * (D / 8);
    cudaError_t e = launch_pdl(flash_bwd_delta_kernel<D>, dim3(static_cast<unsigned>((threads + 255) / 256)), dim3(256), 0, s, (const bf16*)o,
                               (const bf16*)d_o, delta, Tq, Hq, o_stride, do_stride, stat_stride);
    if (e != cudaSuccess) return (int)e;
  }
  {
    auto kern = flash_bwd_kernel<D, false>;
    if (cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), S::TOTAL); e != cudaSuccess) return (int)e;
    cudaError_t e = launch_pdl(kern, dim3(static_cast<unsigned>(max_k_tiles) * Hkv * parts), dim3(FB_THREADS), S::TOTAL, s,
                               map(k, Tk, Hkv, k_stride, FB_T), map(v, Tk, Hkv, v_stride, FB_T), map(q, Tq, Hq, q_stride, FB_S),
                               map(d_o, Tq, Hq, do_stride, FB_S), lse, (const float*)delta, (bf16*)dv, (bf16*)dk, part_out, seg, nseg, Hq,
                               Hkv, Tk, parts, max_k_tiles, dv_stride, dk_stride, stat_stride, scale, status);
    if (e != cudaSuccess) return (int)e;
    if (parts > 1) {
      e = launch_pdl(flash_bwd_sum_kernel, dim3(max_k_tiles, 2, FB_T / FB_SUM_ROWS), dim3(256), 0, s, (const float*)part_out, (bf16*)dv, (bf16*)dk, seg, nseg, parts,
                     Tk, Hkv * D, dv_stride, dk_stride);
      if (e != cudaSuccess) return (int)e;
    }
  }
  {
    auto kern = flash_bwd_kernel<D, true>;
    if (cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), S::TOTAL); e != cudaSuccess) return (int)e;
    cudaError_t e = launch_pdl(kern, dim3(static_cast<unsigned>(max_q_tiles) * Hq), dim3(FB_THREADS), S::TOTAL, s,
                               map(q, Tq, Hq, q_stride, FB_T), map(d_o, Tq, Hq, do_stride, FB_T), map(k, Tk, Hkv, k_stride, FB_S),
                               map(v, Tk, Hkv, v_stride, FB_S), lse, (const float*)delta, (bf16*)dq, (bf16*)nullptr, (float*)nullptr, seg,
                               nseg, Hq, Hkv, Tk, 1, max_q_tiles, dq_stride, 0, stat_stride, scale, status);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

}  // namespace sb

// Gradients of sb_flash_fwd. q / k / v / o / d_o as in the forward (o, d_o: [Tq, Hq * D] with their pitches); lse: the
// forward's [Hq, stat_stride]; delta: scratch of the same shape; dq: [Tq, Hq, D] (pitch dq_stride), dk / dv: [Tk, Hkv, D].
// Rows of dq / dk / dv outside every segment are left untouched. max_q_tiles / max_k_tiles: upper bounds of the number of
// 128-row tiles over all segments on the query and on the key side. parts (1 .. Hq / Hkv): CTAs that share the query heads of a key tile;
// above 1, part_out is scratch of parts * 2 * Tk * Hkv * D floats, 16-byte aligned.
extern "C" int sb_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                            float* delta, void* dq, void* dk, void* dv, float* part_out, int parts, const int* seg, int nseg,
                            int max_q_tiles, int max_k_tiles, int Tq, int Tk, int Hq, int Hkv, int D, int q_stride, int k_stride,
                            int v_stride, int o_stride, int do_stride, int dq_stride, int dk_stride, int dv_stride, int stat_stride,
                            float scale, int* status, cudaStream_t s) {
  if (nseg <= 0 || Tq <= 0 || Tk <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv != 0 || parts < 1 || parts > Hq / Hkv || (parts > 1 && part_out == nullptr)) return (int)cudaErrorInvalidValue;
  try {
    if (D == 64)
      return sb::launch_flash_bwd<64>(q, k, v, o, d_o, lse, delta, dq, dk, dv, part_out, parts, seg, nseg, max_q_tiles, max_k_tiles, Tq, Tk,
                                      Hq, Hkv, q_stride, k_stride, v_stride, o_stride, do_stride, dq_stride, dk_stride, dv_stride,
                                      stat_stride, scale, status, s);
    if (D == 128)
      return sb::launch_flash_bwd<128>(q, k, v, o, d_o, lse, delta, dq, dk, dv, part_out, parts, seg, nseg, max_q_tiles, max_k_tiles, Tq, Tk,
                                       Hq, Hkv, q_stride, k_stride, v_stride, o_stride, do_stride, dq_stride, dk_stride, dv_stride,
                                       stat_stride, scale, status, s);
  } catch (const std::exception& e) {
    sb::set_last_error(e.what());
    return (int)cudaErrorInvalidValue;
  }
  return -1;
}
