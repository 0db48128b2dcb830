// Varlen causal flash attention, forward, on the 5th-gen tensor cores (sm_100a). Training, prefill and
// context-parallel attention all go through this kernel: the work is described by a table of SEGMENTS
//
//     seg[s] = { q_off, q_len, k_off, k_len }        rows [q_off, q_off + q_len) of Q attend rows [k_off, k_off + k_len)
//                                                    of K / V, causally aligned at the end: query i sees keys
//                                                    j <= (k_len - q_len) + i   (k_len >= q_len)
//
// so a packed training batch is one segment per sequence with q_off = k_off, a prefill over a cached prefix has
// k_len > q_len, and a context-parallel rank passes its local query chunk against a prefix of the gathered keys.
// GQA: query head h uses kv head h / (Hq / Hkv).
//
// One CTA = 256 query rows of one head, as two tiles of 128. 10 warps: warp 0 issues TMA loads (Q once, K / V tiles of 128 keys
// through a 2-stage ring that both tiles read), warp 1 owns TMEM and issues tcgen05.mma, and each query tile g has a softmax group of
// four warps: thread r owns query row r (= TMEM lane r). Where the machine is not filled by that, one CTA = 128 rows: one tile and one
// softmax group, the scores of the next key tile computed beside the softmax of this one (see launch_flash_fwd_tiles).
//
//   S_g  = Q_g K_j^T          M 128, N 128, K D        TMEM
//   P_g  = 2^(S_g*c - m)      TMEM -> registers -> bf16 over the scores it came from (the A operand of the next product)
//   O_g += P_g V_j            M 128, N D,  K 128       accumulated in TMEM over all tiles of the row
//
// What bounds it: the chain scores -> softmax -> product of a tile. With one tile per CTA the tensor cores stood still during the
// softmax and the softmax during the products; with two, group 0's softmax runs beside the products of tile 1 and the other way
// round, K and V are read from L2 half as often, and P does not pass through shared memory. Measured, before -> after:
// 8011 + 1187 tokens, 32 / 8 heads of 128: 901 -> 520 us (1034 TFLOP/s); 19 sequences of 384 to 1284 tokens, 14 / 2 heads of 64:
// 167 -> 101 us; 4096 tokens, 32 / 8 heads of 128: 267 -> 154 us.
// CTAs are ordered heads first and last query rows (most keys) first.
// The running maximum m is only raised when a tile exceeds it by more than 2^8 (decided per warp): otherwise the stale
// maximum keeps being used, p stays below 256 and O needs no correction; when it is raised the owning thread rescales
// its O row in TMEM (tcgen05.ld / st) before the next product is issued. Scores live in the log2 domain.
// out = O / l as bf16, lse = ln(sum exp(s * scale)) per row (fp32), both written only for rows inside the segment.
// Every mbarrier wait is bounded: on expiry the CTA records a status word, drains and returns with its TMEM freed.
#include "common.cuh"

namespace sb {

constexpr int FA_BM = 128;       // query rows of one tile; a CTA has one or two
constexpr int FA_BN = 128;       // keys per tile
constexpr int FA_KV_STAGES = 2;

template <int D, int TILES>
struct FaSmem {
  static constexpr int THREADS = 64 + 128 * TILES;    // TMA warp, MMA warp, four softmax warps a tile
  static constexpr int NCH = D / 64;                  // 128-byte chunks of the head dim
  static constexpr int Q_BYTES = FA_BM * 128 * NCH;   // one query tile, [NCH][128 rows][128 B]; its output is staged here at the end
  static constexpr int KV_BYTES = FA_BN * 128 * NCH;  // one K or V tile
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = TILES * Q_BYTES + 2 * FA_KV_STAGES * KV_BYTES + BAR_BYTES + 1024;  // +1024: alignment
  // S_0 @0, S_1 @128 (P over the first 64 columns of its S), O_0 @256, O_1 @256 + D. One tile: S_b holds the scores of key tiles j % 2 = b.
  static constexpr int TMEM_COLS = 512;
};

__device__ __forceinline__ float fa_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void fa_named_barrier(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

template <int D, int TILES>
__global__ void __launch_bounds__(FaSmem<D, TILES>::THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, __nv_bfloat16* __restrict__ out, float* __restrict__ lse,
                 const int* __restrict__ seg, int nseg, int Hq, int Hkv, int tiles, int out_stride, int lse_stride, float scale,
                 int* status) {
  using S = FaSmem<D, TILES>;
  constexpr int NCH = S::NCH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                  // [TILES]
  uint8_t* sK = sQ + TILES * S::Q_BYTES;
  uint8_t* sV = sK + FA_KV_STAGES * S::KV_BYTES;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sV + FA_KV_STAGES * S::KV_BYTES);
  uint64_t* k_full = q_full + 1;
  uint64_t* k_empty = k_full + FA_KV_STAGES;
  uint64_t* v_full = k_empty + FA_KV_STAGES;
  uint64_t* v_empty = v_full + FA_KV_STAGES;
  uint64_t* s_full = v_empty + FA_KV_STAGES;  // [2 score buffers] scores are in TMEM, and every product issued before them has finished
  uint64_t* p_full = s_full + 2;              // [groups] P is in TMEM (4 arrivals)
  uint64_t* o_full = p_full + 2;              // [groups] the group's last product has finished (one tile: each product)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* work = reinterpret_cast<int*>(tmem_slot + 2);  // [0] segment or -1, [1] number of the TILES tiles in the segment

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x % Hq;
  const int kvh = h / (Hq / Hkv);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < FA_KV_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(&s_full[g], 1);
      mbar_init(&p_full[g], 4);  // one arrival per softmax warp of the group
      mbar_init(&o_full[g], 1);
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, S::TMEM_COLS);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_launch_dependents();
  if (warp == 0) {
    int pair;
    const int found = segment_of_tile(seg, nseg, 1, TILES * FA_BM, tiles - 1 - static_cast<int>(blockIdx.x / Hq), pair);
    if (lane == 0) {
      work[0] = found;
      work[1] = pair;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int sidx = work[0];
  if (sidx >= 0) {
    const int q_off = seg[4 * sidx], q_len = seg[4 * sidx + 1], k_off = seg[4 * sidx + 2], k_len = seg[4 * sidx + 3];
    const int q0 = work[1] * TILES * FA_BM;      // first query row of this CTA inside the segment
    const int shift = k_len - q_len;             // query i sees keys j <= shift + i
    // key tiles of the query tiles (none for a second tile that lies past the segment)
    auto key_tiles = [&](int g) {
      const int r0 = q0 + g * FA_BM;
      return r0 < q_len ? (max(min(k_len, shift + r0 + FA_BM), 0) + FA_BN - 1) / FA_BN : 0;
    };
    const int n_of[2] = {key_tiles(0), TILES == 2 ? key_tiles(1) : 0};
    const int n_kv = max(n_of[0], n_of[1]);

    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0 && n_kv > 0) {
        mbar_arrive_expect_tx(q_full, TILES * S::Q_BYTES);
#pragma unroll
        for (int g = 0; g < TILES; ++g)
#pragma unroll
          for (int c = 0; c < NCH; ++c)
            tma_load_2d(sQ + g * S::Q_BYTES + c * (FA_BM * 128), &tmQ, q_full, h * D + c * 64, q_off + q0 + g * FA_BM);
        for (int j = 0; j < n_kv; ++j) {
          const int st = j % FA_KV_STAGES;
          const uint32_t par = (j / FA_KV_STAGES) & 1;
          if (!mbar_wait(&k_empty[st], par ^ 1, cta_abort, status, ERR_WAIT_EMPTY)) break;
          mbar_arrive_expect_tx(&k_full[st], S::KV_BYTES);
#pragma unroll
          for (int c = 0; c < NCH; ++c)
            tma_load_2d(sK + st * S::KV_BYTES + c * (FA_BN * 128), &tmK, &k_full[st], kvh * D + c * 64, k_off + j * FA_BN);
          if (!mbar_wait(&v_empty[st], par ^ 1, cta_abort, status, ERR_WAIT_EMPTY)) break;
          mbar_arrive_expect_tx(&v_full[st], S::KV_BYTES);
#pragma unroll
          for (int c = 0; c < NCH; ++c)
            tma_load_2d(sV + st * S::KV_BYTES + c * (FA_BN * 128), &tmV, &v_full[st], kvh * D + c * 64, k_off + j * FA_BN);
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (lane == 0 && n_kv > 0) {
        constexpr uint32_t idesc_s = make_idesc(FA_BM, FA_BN, 1, 1, 0, 0);
        constexpr uint32_t idesc_o = make_idesc(FA_BM, D, 1, 1, 0, 1);  // A = P in TMEM, B = V read MN-major
        auto issue_s = [&](int g, int j) {
          const int buf = TILES == 2 ? g : j & 1;
          const uint32_t q_addr = smem_u32(sQ + g * S::Q_BYTES), k_addr = smem_u32(sK + (j % FA_KV_STAGES) * S::KV_BYTES);
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t off = (k >> 2) * (FA_BM * 128) + (k & 3) * 32;
            umma_f16(tmem_base + buf * FA_BN, make_smem_desc(q_addr + off, 16, 1024, UMMA_SWIZZLE_128B),
                     make_smem_desc(k_addr + off, 16, 1024, UMMA_SWIZZLE_128B), idesc_s, k != 0 ? 1u : 0u);
          }
          umma_commit(&s_full[buf]);
        };
        // P of the key tile in score buffer `buf` times V
        auto issue_o = [&](int g, int buf, int j) {
          const uint32_t v_addr = smem_u32(sV + (j % FA_KV_STAGES) * S::KV_BYTES);
#pragma unroll
          for (int k = 0; k < FA_BN / 16; ++k) {
            // A: 16 keys = 8 TMEM columns; B = V tile [128 keys, D]: MN-major, 16 keys = 2048 B, 64-wide chunks of the head dim
            // FA_BN * 128 B apart
            umma_f16_ts(tmem_base + 2 * FA_BN + g * D, tmem_base + buf * FA_BN + k * 8,
                        make_smem_desc(v_addr + k * 2048, FA_BN * 128, 1024, UMMA_SWIZZLE_128B), idesc_o, (j != 0 || k != 0) ? 1u : 0u);
          }
        };
        bool ok = mbar_wait(q_full, 0, cta_abort, status, ERR_WAIT_FULL) &&
                  mbar_wait(&k_full[0], 0, cta_abort, status, ERR_WAIT_FULL);
        if (ok) {
          tc_fence_after();
          for (int g = 0; g < TILES; ++g)
            if (n_of[g] > 0) issue_s(g, 0);
          umma_commit(&k_empty[0]);
        }
        for (int j = 0; j < n_kv && ok; ++j) {
          auto next_scores = [&](int g) {
            ok = mbar_wait(&k_full[(j + 1) % FA_KV_STAGES], ((j + 1) / FA_KV_STAGES) & 1, cta_abort, status, ERR_WAIT_FULL);
            if (!ok) return;
            tc_fence_after();
            issue_s(g, j + 1);
          };
          if constexpr (TILES == 1) {
            // the next scores go to the other buffer, whose P the product of tile j - 1 reads: products of one CTA run in the order they are
            // issued in
            if (j + 1 < n_kv) {
              next_scores(0);
              if (!ok) break;
              umma_commit(&k_empty[(j + 1) % FA_KV_STAGES]);
            }
            ok = mbar_wait(&v_full[j % FA_KV_STAGES], (j / FA_KV_STAGES) & 1, cta_abort, status, ERR_WAIT_FULL) &&
                 mbar_wait(&p_full[0], j & 1, cta_abort, status, ERR_WAIT_TMEM_EMPTY);
            if (!ok) break;
            tc_fence_after();
            issue_o(0, j & 1, j);
            umma_commit(&v_empty[j % FA_KV_STAGES]);
            umma_commit(&o_full[0]);
            continue;
          }
          ok = mbar_wait(&v_full[j % FA_KV_STAGES], (j / FA_KV_STAGES) & 1, cta_abort, status, ERR_WAIT_FULL);
          for (int g = 0; g < TILES && ok; ++g) {
            if (j >= n_of[g]) continue;
            ok = mbar_wait(&p_full[g], j & 1, cta_abort, status, ERR_WAIT_TMEM_EMPTY);
            if (!ok) break;
            tc_fence_after();
            issue_o(g, g, j);
            if (j + 1 == n_of[g]) umma_commit(&o_full[g]);
            if (j + 1 < n_of[g]) {  // the next scores replace P: products run in order
              next_scores(g);
              if (!ok) break;
            }
          }
          if (!ok) break;
          umma_commit(&v_empty[j % FA_KV_STAGES]);
          if (j + 1 < n_kv) umma_commit(&k_empty[(j + 1) % FA_KV_STAGES]);
        }
      }
    } else {
      // ------------------------------------------------------------------ softmax + epilogue
      const int quarter = warp & 3, g = TILES == 2 ? (warp - 2) >> 2 : 0;
      const int row = quarter * 32 + lane;  // query row inside the tile = TMEM lane
      const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t o_addr = lane_addr + 2 * FA_BN + g * D;
      const float c_log2 = scale * 1.4426950408889634f;
      const uint64_t c2 = f2_pack(c_log2, c_log2);
      const int r0 = q0 + g * FA_BM;
      const int qi = r0 + row;
      const int my_limit = shift + qi;  // last key this row may see
      const int n_my = n_of[g];
      float m_run = -INFINITY, l_run = 0.f;
      bool ok = true;
      for (int j = 0; j < n_my; ++j) {
        const int buf = TILES == 2 ? g : j & 1;
        const uint32_t s_addr = lane_addr + buf * FA_BN;
        ok = mbar_wait(&s_full[buf], (TILES == 2 ? j : j >> 1) & 1, cta_abort, status, ERR_WAIT_TMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const int key0 = j * FA_BN;
        // a tile needs masking when it reaches past the diagonal of this tile's first row or past the last key
        const bool masked = (key0 + FA_BN - 1 > shift + r0) || (key0 + FA_BN > k_len);
        const int lim = min(my_limit, k_len - 1) - key0;  // columns <= lim are visible to this row
        uint32_t r[4][32];  // the fourth quarter is read again below instead of being held (168 registers per thread are to be had)
        auto load = [&](int c4) {
          tmem_ld_32x32(s_addr + c4 * 32, r[c4]);
        };
        auto hide = [&](int c4) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c4 * 32 + i > lim) r[c4][i] = 0xff800000u;  // -infinity
        };
        load(3);
        load(0);
        tmem_ld_wait();
        load(1);
        load(2);
        float mx4[4];
        auto row_max = [&](int c4) {
          if (masked) hide(c4);
          mx4[c4] = __uint_as_float(r[c4][0]);
#pragma unroll
          for (int i = 1; i < 32; ++i) mx4[c4] = fmaxf(mx4[c4], __uint_as_float(r[c4][i]));
        };
        row_max(3);
        row_max(0);
        tmem_ld_wait();
        row_max(1);
        row_max(2);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * c_log2;  // scale > 0: the maximum commutes with the scaling
        const float m_new = fmaxf(m_run, mx);
        bool seen = TILES == 2 || j == 0;  // one tile: every product's end is waited for, in turn (a phase that is left out could be mistaken)
        if (j == 0) {
          m_run = (m_new == -INFINITY) ? 0.f : m_new;
        } else if (__any_sync(0xffffffffu, qi < q_len && m_new > m_run + 8.f)) {  // (rows behind the segment have no say)
          // O may be corrected once the product of the tile before is done; with two tiles it is, since the scores just read came after it
          if constexpr (TILES == 1) {
            ok = __all_sync(0xffffffffu, mbar_wait(&o_full[0], (j - 1) & 1, cta_abort, status, ERR_WAIT_TMEM_FULL));
            if (!ok) break;
            tc_fence_after();
            seen = true;
          }
          const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
          const float f = fa_exp2(m_run - m_use);  // <= 1
          l_run *= f;
#pragma unroll 1
          for (int c4 = 0; c4 < D / 32; ++c4) {
            uint32_t o[32];
            tmem_ld_32x32(o_addr + c4 * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st_32x32(o_addr + c4 * 32, o);
          }
          m_run = m_use;
        }
        // ---- p = 2^(s*c - m), packed to bf16; the row sum uses the unrounded values
        const uint64_t nm = f2_pack(-m_run, -m_run);
        uint64_t sum[2] = {0, 0};
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
          if (c4 == 1) load(3);  // (P takes the columns of the first two quarters only)
          if (c4 == 3) {
            tmem_ld_wait();
            if (masked) hide(3);
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0, p1;
            f2_unpack(f2_fma(f2_pack(__uint_as_float(r[c4][i]), __uint_as_float(r[c4][i + 1])), c2, nm), p0, p1);
            p0 = fa_exp2(p0);
            p1 = fa_exp2(p1);
            sum[(i >> 1) & 1] = f2_add(sum[(i >> 1) & 1], f2_pack(p0, p1));
            pk[i >> 1] = pack_bf16x2(p0, p1);
          }
          tmem_st_32x16(s_addr + c4 * 16, pk);
        }
        if (!seen) {  // (with the exponentials behind, this does not wait any more)
          ok = __all_sync(0xffffffffu, mbar_wait(&o_full[0], (j - 1) & 1, cta_abort, status, ERR_WAIT_TMEM_FULL));
          if (!ok) break;
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g]);
        float a, b;
        f2_unpack(f2_add(sum[0], sum[1]), a, b);
        l_run += a + b;
      }
      // ---- epilogue: O / l -> bf16 -> staged through shared memory (the group's Q tile) -> coalesced rows of `out`
      if (ok && n_my > 0) {
        ok = mbar_wait(&o_full[g], TILES == 2 ? 0 : (n_my - 1) & 1, cta_abort, status, ERR_WAIT_TMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok && r0 < q_len) {
        tc_fence_after();
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        constexpr int CH = D / 8;  // 16-byte chunks per output row
        uint8_t* stage = sQ + g * S::Q_BYTES;
        uint8_t* orow = stage + row * (D * 2);
#pragma unroll
        for (int c4 = 0; c4 < D / 32; ++c4) {
          uint32_t r[32];
          if (n_my > 0) {
            tmem_ld_32x32(o_addr + c4 * 32, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = 0;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(r[8 * i]) * inv, __uint_as_float(r[8 * i + 1]) * inv);
            v.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]) * inv, __uint_as_float(r[8 * i + 3]) * inv);
            v.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]) * inv, __uint_as_float(r[8 * i + 5]) * inv);
            v.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]) * inv, __uint_as_float(r[8 * i + 7]) * inv);
            const int ch = c4 * 4 + i;
            *reinterpret_cast<uint4*>(orow + ((ch ^ (row & (CH - 1))) << 4)) = v;
          }
        }
        if (qi < q_len && lse != nullptr)
          lse[static_cast<size_t>(h) * lse_stride + q_off + qi] = (m_run + log2f(fmaxf(l_run, 1e-38f))) * 0.6931471805599453f;
        if (g == 0) fa_named_barrier(1, 128);
        else fa_named_barrier(2, 128);
        const int t = (threadIdx.x - 64) & 127;
        const int rows_valid = min(FA_BM, q_len - r0);
        for (int idx = t; idx < rows_valid * CH; idx += 128) {
          const int rr = idx / CH, ch = idx % CH;
          const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * (D * 2) + ((ch ^ (rr & (CH - 1))) << 4));
          *reinterpret_cast<uint4*>(out + static_cast<size_t>(q_off + r0 + rr) * out_stride + h * D + ch * 8) = v;
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*cta_abort) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);  // let copies in flight land
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem_base, S::TMEM_COLS);
}

template <int D, int TILES>
static int launch_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* seg, int nseg,
                            int max_q_tiles, int Tq, int Tk, int Hq, int Hkv, int q_stride, int k_stride, int v_stride,
                            int out_stride, int lse_stride, float scale, int* status, cudaStream_t s) {
  using S = FaSmem<D, TILES>;
  const CUtensorMap tq = make_tmap_2d(q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tq, size_t(Hq) * D, size_t(q_stride) * 2, FA_BM, 64,
                                      CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap tk = make_tmap_2d(k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tk, size_t(Hkv) * D, size_t(k_stride) * 2, FA_BN, 64,
                                      CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap tv = make_tmap_2d(v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tk, size_t(Hkv) * D, size_t(v_stride) * 2, FA_BN, 64,
                                      CU_TENSOR_MAP_SWIZZLE_128B);
  auto kern = flash_fwd_kernel<D, TILES>;
  if (cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), S::TOTAL); e != cudaSuccess) return (int)e;
  return (int)launch_pdl(kern, dim3(static_cast<unsigned>(max_q_tiles) * Hq), dim3(S::THREADS), S::TOTAL, s, tq, tk, tv,
                         reinterpret_cast<__nv_bfloat16*>(out), lse, seg, nseg, Hq, Hkv, max_q_tiles, out_stride, lse_stride, scale, status);
}

// One tile a CTA where the CTAs of single tiles are no more than the SMs: two tiles a CTA would leave half of them idle, and a CTA of one tile
// ends earlier (two tiles -> one, us: 397 rows, 14 heads of 64 12.5 -> 9.6, 32 heads of 128 14.3 -> 10.7; 300
// rows behind 3000 59 -> 40; 1000 rows behind 8000, 14 heads of 64, 112 CTAs 138 -> 92). A row's
// arithmetic is the same in both, and so are its bits.
static int launch_flash_fwd_tiles(int D, const void* q, const void* k, const void* v, void* out, float* lse, const int* seg, int nseg,
                                  int max_q_tiles, int Tq, int Tk, int Hq, int Hkv, int q_stride, int k_stride, int v_stride,
                                  int out_stride, int lse_stride, float scale, int* status, cudaStream_t s) {
  int dev = 0, sms = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return (int)e;
  if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); e != cudaSuccess) return (int)e;
  const int held = nseg < Tq ? nseg : Tq;  // segments that can have rows
  const int singles = (Tq - held) / FA_BM + held;  // tiles there can be at most
  const bool one = static_cast<long>(singles) * Hq <= sms;
  auto run = [&](auto launch) {
    return launch(q, k, v, out, lse, seg, nseg, one ? singles : max_q_tiles, Tq, Tk, Hq, Hkv, q_stride, k_stride, v_stride, out_stride,
                  lse_stride, scale, status, s);
  };
  if (D == 64) return one ? run(launch_flash_fwd<64, 1>) : run(launch_flash_fwd<64, 2>);
  return one ? run(launch_flash_fwd<128, 1>) : run(launch_flash_fwd<128, 2>);
}

}  // namespace sb

// q: [Tq, Hq, D] bf16 with row pitch q_stride (elements; the head dim is contiguous), k / v: [Tk, Hkv, D] with pitches
// k_stride / v_stride; out: [Tq, Hq * D] with pitch out_stride; lse: [Hq, lse_stride] fp32 or null. seg: device table of
// nseg x 4 ints (see the top of this file). max_q_tiles: an upper bound of the total number of 256-row pairs of query tiles over
// all segments (CTAs beyond the real count exit at once). Base pointers 16-byte aligned, pitches multiples of 8.
// Returns 0, a cudaError_t value, or -1 when the head dim is not 64 or 128.
extern "C" int sb_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* seg, int nseg,
                            int max_q_tiles, int Tq, int Tk, int Hq, int Hkv, int D, int q_stride, int k_stride, int v_stride,
                            int out_stride, int lse_stride, float scale, int* status, cudaStream_t s) {
  if (nseg <= 0 || max_q_tiles <= 0 || Tq <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv != 0) return (int)cudaErrorInvalidValue;
  try {
    if (D == 64 || D == 128)
      return sb::launch_flash_fwd_tiles(D, q, k, v, out, lse, seg, nseg, max_q_tiles, Tq, Tk, Hq, Hkv, q_stride, k_stride, v_stride, out_stride,
                                        lse_stride, scale, status, s);
  } catch (const std::exception& e) {
    sb::set_last_error(e.what());
    return (int)cudaErrorInvalidValue;
  }
  return -1;
}
