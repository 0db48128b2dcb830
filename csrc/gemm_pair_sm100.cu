// bf16 GEMM on pairs of SMs (tcgen05.mma.cta_group::2): 256 x bn tiles, bn = 128 .. 256.
//
//   C[M,N] (+)= op(A) * op(B)  (+ bias[N]),   fp32 accumulate, bf16 or fp32 output,
//
// with the operand layouts of gemm_sm100.cu (K-major or MN-major on either side). The two CTAs of a cluster each hold 128 rows of A
// and bn / 2 rows of B; the tensor cores of both read both halves of B, so that a stage is 32 KB of shared memory for 128 x 256 outputs
// per SM instead of 48 KB: a third less traffic from L2 and a third fewer operand reads, which is what bounds the one-SM kernel.
//
// Work: full waves of tiles first, one tile per pair and wave. Where the caller asks for it (outputs that are added to, and outputs of
// less than a wave over a long K), the tiles of the last, partial wave are cut along K into as many slices as there are pairs for each: a weight
// gradient of 9728 x 896 is 152 tiles on 74 pairs and took three waves for work of 2.05. A slice leaves its fp32 sums in a workspace,
// and a second launch adds a tile's slices up in K order, so that the result is the same on every run. (Reduce-adds into
// the output itself would save that launch, but they come in any order.)
//
// Grouped (weight gradients of experts): C is a stack of matrices, C[e] += A[rows of e]^T * B[rows of e], K = the rows of e.
//
// Bound by the tensor cores (and, in long runs, by the power limit). One SM per tile -> pairs, us: 9198 x 19456 x 2560 630 -> 573
// (1598 TFLOP/s), 15800 x 9728 x 896 217 -> 193; weight gradients 9728 x 896 x 15800 302 -> 211 (258 with
// the last wave uncut), 2560 x 4096 x 9198 170 -> 133 (152). What is left below the peak is the last wave of outputs that are not added
// to, and K below 1000.
//
// CTA = 6 warps as in gemm_sm100.cu: TMA producer, MMA issuer (leader CTA only), four epilogue warps.
#include "common.cuh"

namespace sb {

constexpr int GP_BK = 64;
constexpr int GP_STAGES = 6;
constexpr int GP_THREADS = 192;
constexpr int GP_A_BYTES = 128 * GP_BK * 2;
constexpr int GP_B_BYTES = 128 * GP_BK * 2;  // bn / 2 <= 128 rows
constexpr int GP_STAGE = GP_A_BYTES + GP_B_BYTES;
constexpr int GP_EPI_BUF = 32 * 128;
constexpr int GP_EPI = 4 * 2 * GP_EPI_BUF;
constexpr int GP_SMEM = GP_STAGES * GP_STAGE + GP_EPI + (2 * GP_STAGES + 4) * 8 + 16 + 1024;
constexpr int GP_PANEL = 16;  // row tiles of a panel: as many rows as in gemm_sm100.cu

// One piece of work: a tile and a range of k-blocks.
struct PairItem {
  int m0, n0, z, kb0, kb1;  // kb absolute: rows of the group included
  int part;                 // of a cut tile: where its sums go in the workspace; -1: a whole tile
};

// How the tiles behind the last full wave are cut: each of the `left` tiles into `slices` ranges of K, one a pair.
struct PairCut {
  int full, left, slices, pairs;
};
constexpr int GP_CUT_KB = 8;  // k-blocks of a slice at least: below, its way through the workspace takes longer than its products
inline PairCut cut_last_wave(long long tiles, int num_kb, int num_sms, bool cut) {
  PairCut c;
  c.pairs = num_sms / 2;
  c.full = static_cast<int>(tiles);
  c.left = 0;
  c.slices = 1;
  const int rest = static_cast<int>(tiles % c.pairs);
  if (cut && rest > 0) {
    const int slices = c.pairs / rest < num_kb / GP_CUT_KB ? c.pairs / rest : num_kb / GP_CUT_KB;
    if (slices > 1) {
      c.full -= rest;
      c.left = rest;
      c.slices = slices;
    }
  }
  const long long most = c.full > c.left * c.slices ? c.full : c.left * c.slices;
  if (most < c.pairs) c.pairs = static_cast<int>(most);
  return c;
}

struct PairShape {
  int M, N, K, bn;
  int groups;              // 1: plain
  const int* group_start;  // first row of A and B of group e (a multiple of 64)
  const int* group_rows;   // rows of group e; what follows them up to the next multiple of 64 is zero in A or B
  PairCut cut;
};

__device__ __forceinline__ void place_tile(const PairShape& s, int tiles_m, int tiles_n, int t, PairItem& it) {
  const int per = tiles_m * tiles_n;
  it.z = t / per;
  t -= it.z * per;
  const int per_panel = GP_PANEL * tiles_n;
  const int panel = t / per_panel, r = t - panel * per_panel;
  const int pm = min(GP_PANEL, tiles_m - panel * GP_PANEL);
  it.m0 = (panel * GP_PANEL + r % pm) * 256;
  it.n0 = (r / pm) * s.bn;
}

// The sequence of a pair's pieces; every role walks the same one.
struct PairWalk {
  int tiles_m, tiles_n, num_kb, tile, pair, pairs;
  bool slice;  // one is still to come
  __device__ PairWalk(const PairShape& s, int pair_, int pairs_) {
    tiles_m = (s.M + 255) / 256;
    tiles_n = (s.N + s.bn - 1) / s.bn;
    num_kb = (s.K + GP_BK - 1) / GP_BK;
    pair = pair_;
    pairs = pairs_;
    tile = pair;
    slice = pair < s.cut.left * s.cut.slices;
  }
  __device__ __forceinline__ bool next(const PairShape& s, PairItem& it) {
    while (tile < s.cut.full) {
      place_tile(s, tiles_m, tiles_n, tile, it);
      tile += pairs;
      it.part = -1;
      it.kb0 = 0;
      it.kb1 = num_kb;
      if (s.group_rows != nullptr) {
        it.kb1 = (__ldg(s.group_rows + it.z) + GP_BK - 1) / GP_BK;
        if (it.kb1 <= 0) continue;
      }
      return true;
    }
    if (!slice) return false;
    slice = false;
    const int t = pair / s.cut.slices, i = pair - t * s.cut.slices;
    place_tile(s, tiles_m, tiles_n, s.cut.full + t, it);
    it.part = pair;
    it.kb0 = num_kb * i / s.cut.slices;
    it.kb1 = num_kb * (i + 1) / s.cut.slices;
    return true;
  }
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// Address of `p` (this CTA's shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Load into this CTA's shared memory; the bytes are counted by the barrier at `bar`, which may be the other CTA's.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               :
               : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the MMAs issued so far have retired.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

template <bool A_MN, bool B_MN, bool OUT_F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                 const __grid_constant__ CUtensorMap tmAux /* bf16: boxes of 32 columns; fp32: the workspace of cut tiles */,
                 const __nv_bfloat16* __restrict__ bias, const __grid_constant__ PairShape s, int add_out, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + GP_STAGES * GP_A_BYTES;
  uint8_t* sC = smem + GP_STAGES * GP_STAGE;
  uint64_t* full = reinterpret_cast<uint64_t*>(sC + GP_EPI);
  uint64_t* empty = full + GP_STAGES;
  uint64_t* tfull = empty + GP_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int i = 0; i < GP_STAGES; ++i) {
      mbar_init(&full[i], 1);   // leader's: its producer announces the bytes of both CTAs
      mbar_init(&empty[i], 1);  // either CTA's: the leader's commit
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 8);  // leader's: the epilogue warps of both CTAs
    }
    *cta_abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the other CTA's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();

  PairWalk walk(s, pair, pairs);
  PairItem it;
  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (each CTA loads its own halves)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const int half = s.bn / 2;
      const int b_boxes = B_MN ? (half + 63) / 64 : 1;
      const uint32_t bytes = 2 * (GP_A_BYTES + (B_MN ? b_boxes * 8192 : half * GP_BK * 2));
      while (ok && walk.next(s, it)) {
        const int k_base = s.group_start != nullptr ? __ldg(s.group_start + it.z) : 0;
        const int m = it.m0 + static_cast<int>(rank) * 128, n = it.n0 + static_cast<int>(rank) * half;
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, cta_abort, status, ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], bytes);
          const uint32_t bar = map_to_rank(&full[stage], 0);
          uint8_t* a_dst = sA + stage * GP_A_BYTES;
          uint8_t* b_dst = sB + stage * GP_B_BYTES;
          const int k = k_base + kb * GP_BK;
          if constexpr (!A_MN) {
            tma_load_2d_pair(a_dst, &tmA, bar, k, m);
          } else {
            tma_load_2d_pair(a_dst, &tmA, bar, m, k);
            tma_load_2d_pair(a_dst + 8192, &tmA, bar, m + 64, k);
          }
          if constexpr (!B_MN) {
            tma_load_2d_pair(b_dst, &tmB, bar, k, n);
          } else {
            for (int j = 0; j < b_boxes; ++j) tma_load_2d_pair(b_dst + j * 8192, &tmB, bar, n + j * 64, k);
          }
          if (++stage == GP_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer: the leader's, for both SMs
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = make_idesc(256, s.bn, 1, 1, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      while (ok && walk.next(s, it)) {
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, cta_abort, status, ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          if (!mbar_wait(&full[stage], phase, cta_abort, status, ERR_WAIT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(sA + stage * GP_A_BYTES);
          const uint32_t b_addr = smem_u32(sB + stage * GP_B_BYTES);
#pragma unroll
          for (int k = 0; k < GP_BK / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(a_addr + k * 2048, 8192, 1024, UMMA_SWIZZLE_128B)
                                     : make_smem_desc(a_addr + k * 32, 16, 1024, UMMA_SWIZZLE_128B);
            const uint64_t db = B_MN ? make_smem_desc(b_addr + k * 2048, 8192, 1024, UMMA_SWIZZLE_128B)
                                     : make_smem_desc(b_addr + k * 32, 16, 1024, UMMA_SWIZZLE_128B);
            umma_f16_pair(d_tmem, da, db, idesc, (kb != it.kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty[stage]);
          if (++stage == GP_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(&tfull[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue: 128 rows of the tile per CTA
    const int q = warp & 3;
    int acc = 0, buf = 0;
    uint32_t acc_phase = 0;
    uint8_t* stage_buf = sC + q * 2 * GP_EPI_BUF;
    constexpr int BOX = OUT_F32 ? 32 : 64;
    while (walk.next(s, it)) {
      bool ok = mbar_wait(&tfull[acc], acc_phase, cta_abort, status, ERR_WAIT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * 256;
      const int row0 = it.m0 + static_cast<int>(rank) * 128 + q * 32;
      const __nv_bfloat16* b_row = it.kb0 == 0 ? bias : nullptr;
#pragma unroll 1
      for (int c = 0; c < s.bn; c += BOX) {
        const int col0 = it.n0 + c;
        if (row0 >= s.M || col0 >= s.N) break;  // warp-uniform: each pass through a buffer commits one bulk group
        uint8_t* dst = stage_buf + buf * GP_EPI_BUF;
        if (lane == 0) bulk_wait_group_read<1>();
        __syncwarp();
        if constexpr (OUT_F32) {
          uint8_t* my_row = dst + lane * 128;
          const int sw = lane & 7;
          uint32_t r[32];
          tmem_ld_32x32(t_row + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 o = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                   __uint_as_float(r[4 * j + 3]));
            if (b_row != nullptr) {
              const int cc = col0 + 4 * j;
              if (cc + 0 < s.N) o.x += __bfloat162float(b_row[cc + 0]);
              if (cc + 1 < s.N) o.y += __bfloat162float(b_row[cc + 1]);
              if (cc + 2 < s.N) o.z += __bfloat162float(b_row[cc + 2]);
              if (cc + 3 < s.N) o.w += __bfloat162float(b_row[cc + 3]);
            }
            *reinterpret_cast<float4*>(my_row + ((j ^ sw) << 4)) = o;
          }
        } else {
          // 64 columns to a box; the last box of a width that is an odd multiple of 32 has 32 (rows of 64 bytes, 64B swizzle)
          const bool narrow = c + 64 > s.bn;
          uint8_t* my_row = dst + lane * (narrow ? 64 : 128);
          const int sw = narrow ? (lane >> 1) & 3 : lane & 7;
          const int halves = narrow ? 1 : 2;
#pragma unroll 2
          for (int half = 0; half < halves; ++half) {
            uint32_t r[32];
            tmem_ld_32x32(t_row + c + half * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * j + i]);
              if (b_row != nullptr) {
                const int cc = col0 + half * 32 + 8 * j;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                  if (cc + i < s.N) v[i] += __bfloat162float(b_row[cc + i]);
              }
              *reinterpret_cast<uint4*>(my_row + (((half * 4 + j) ^ sw) << 4)) =
                  make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
            }
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          const CUtensorMap* map = !OUT_F32 && c + 64 > s.bn ? &tmAux : &tmC;
          if (OUT_F32 && it.part >= 0)
            tma_store_3d(&tmAux, dst, c, row0 - it.m0, it.part);
          else if (add_out)
            tma_reduce_add_3d(map, dst, col0, row0, it.z);
          else
            tma_store_3d(map, dst, col0, row0, it.z);
          bulk_commit_group();
        }
        buf ^= 1;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_at(map_to_rank(&tempty[acc], 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (lane == 0) bulk_wait_group_read<0>();
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort) {  // copies in flight get a bounded time to land before the shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncwarp();
  cluster_sync_all();  // neither CTA's shared memory or TMEM goes while the other may use it
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

// Cut tiles: C (+)= sum of a tile's slices, in K order. Four rows of a tile a block, four slices' loads in flight a thread.
// Bound by L2: 72 slices of 256 KB are written and read in about 10 us (2560 x 4096 x 9198, 12 tiles in 6 slices: 152 us uncut, 133 cut).
constexpr int GP_SUM_ROWS = 4;
template <bool OUT_F32>
__global__ void __launch_bounds__(256)
gemm_pair_sum_kernel(const float* __restrict__ parts, void* __restrict__ Cv, const __grid_constant__ PairShape s, int ldc, int add_out) {
  const int tiles_m = (s.M + 255) / 256, tiles_n = (s.N + s.bn - 1) / s.bn, slices = s.cut.slices;
  constexpr int BLOCKS = 256 / GP_SUM_ROWS;
  const int t = blockIdx.x / BLOCKS, r0 = blockIdx.x % BLOCKS * GP_SUM_ROWS;
  const int vecs = s.bn / 4;
  const int r = r0 + threadIdx.x / vecs, c = threadIdx.x % vecs * 4;
  PairItem it;
  place_tile(s, tiles_m, tiles_n, s.cut.full + t, it);
  const int row = it.m0 + r, col = it.n0 + c;
  pdl_wait();
  pdl_launch_dependents();
  if (static_cast<int>(threadIdx.x) >= GP_SUM_ROWS * vecs || row >= s.M || col >= s.N) return;
  const size_t pitch = static_cast<size_t>(256) * s.bn;
  const float* src = parts + t * slices * pitch + static_cast<size_t>(r) * s.bn + c;
  float4 acc = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
  for (int i = 1; i < slices; ++i) {
    const float4 v = *reinterpret_cast<const float4*>(src + i * pitch);
    acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
  }
  const float out[4] = {acc.x, acc.y, acc.z, acc.w};
  const size_t at = static_cast<size_t>(row) * ldc + col;
  if constexpr (OUT_F32) {
    float* dst = static_cast<float*>(Cv) + at;
    if (col + 4 <= s.N) {
      const float4 old = add_out ? *reinterpret_cast<const float4*>(dst) : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(dst) = make_float4(old.x + out[0], old.y + out[1], old.z + out[2], old.w + out[3]);
    } else {
      for (int i = 0; col + i < s.N; ++i) dst[i] = (add_out ? dst[i] : 0.f) + out[i];
    }
  } else {
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(Cv) + at;
    if (col + 4 <= s.N)
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(out[0], out[1]), pack_bf16x2(out[2], out[3]));
    else
      for (int i = 0; col + i < s.N; ++i) dst[i] = __float2bfloat16(out[i]);
  }
}

static CUtensorMap pair_out_map(void* C, bool f32, int N, int M, int groups, int ldc, int box_cols) {
  CUtensorMap m;
  const int es = f32 ? 4 : 2;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M), static_cast<cuuint64_t>(groups)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ldc) * es, static_cast<cuuint64_t>(ldc) * es * M};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(box_cols), 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = get_encode_tiled()(&m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, C, dims, strides, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols * es == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled (output) failed: " + std::to_string(int(r)));
  return m;
}

// OUT_F32: what the kernel writes, in C or in `parts`; c_f32: what C is.
template <bool A_MN, bool B_MN, bool OUT_F32>
static cudaError_t launch_pair(const void* A, const void* B, void* C, const void* bias, const PairShape& s, int rows_k, int lda, int ldb, int ldc,
                               bool c_f32, int add, float* parts, int* status, cudaStream_t stream) {
  const PairCut& cut = s.cut;
  CUtensorMap tmA = A_MN ? make_tmap_2d(A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows_k, s.M, size_t(lda) * 2, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)
                         : make_tmap_2d(A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s.M, s.K, size_t(lda) * 2, 128, GP_BK, CU_TENSOR_MAP_SWIZZLE_128B);
  CUtensorMap tmB = B_MN ? make_tmap_2d(B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows_k, s.N, size_t(ldb) * 2, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)
                         : make_tmap_2d(B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s.N, s.K, size_t(ldb) * 2, s.bn / 2, GP_BK, CU_TENSOR_MAP_SWIZZLE_128B);
  CUtensorMap tmAux;
  if (cut.left > 0)
    tmAux = pair_out_map(parts, true, s.bn, 256, cut.left * cut.slices, s.bn, 32);
  else
    tmAux = pair_out_map(C, OUT_F32, s.N, s.M, s.groups, ldc, 32);
  CUtensorMap tmC = OUT_F32 == c_f32 ? pair_out_map(C, OUT_F32, s.N, s.M, s.groups, ldc, OUT_F32 ? 32 : 64) : tmAux;
  auto kern = gemm_pair_kernel<A_MN, B_MN, OUT_F32>;
  if (cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), GP_SMEM); e != cudaSuccess) {
    set_last_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    return e;
  }
  cudaError_t le = launch_pdl(kern, dim3(2 * cut.pairs), dim3(GP_THREADS), GP_SMEM, stream, tmA, tmB, tmC, tmAux,
                              reinterpret_cast<const __nv_bfloat16*>(bias), s, add, status);
  if (le == cudaSuccess && cut.left > 0)
    le = launch_pdl(c_f32 ? gemm_pair_sum_kernel<true> : gemm_pair_sum_kernel<false>, dim3(cut.left * (256 / GP_SUM_ROWS)), dim3(256), 0, stream,
                    static_cast<const float*>(parts), C, s, ldc, add);
  if (le != cudaSuccess) set_last_error(std::string("gemm_pair launch: ") + cudaGetErrorString(le));
  return le;
}

}  // namespace sb

// Operands as sb_gemm_bf16. `bn`: tile width, a multiple of 32 from 128 to 256. `add` = 1: C (fp32) is added to. `split_last` = 1: the tiles
// behind the last full wave of num_sms / 2 are cut along K where there are pairs and k-blocks for it; `parts` is then scratch of num_sms / 2 *
// 256 * bn floats, 16-byte aligned. (A bf16 C: only with fewer tiles than a wave, and at least 16 k-blocks.) `groups` > 1 (a_mn and b_mn
// only, fp32 C): C is [groups, M, N] and group e sums over the rows
// group_start[e] .. + group_rows[e] of A and B, which hold K rows in all; group_start are multiples of 64 and the rows behind a group's
// last, up to a multiple of 64, are zero. C's base and pitch are multiples of 16 bytes (8 where a bf16 C is cut).
extern "C" int sb_gemm_pair(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb, int ldc, int a_mn,
                            int b_mn, int out_f32, int add, int bn, int split_last, float* parts, int groups, const int* group_start,
                            const int* group_rows, int* status, int num_sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || groups <= 0) return 0;
  const bool grouped = group_start != nullptr;
  if (bn < 128 || bn > 256 || bn % 32 || (a_mn && !b_mn) || (add && !out_f32) || (split_last && grouped) || (groups > 1 && !grouped) ||
      (grouped && (!a_mn || !b_mn || !out_f32 || group_rows == nullptr || bias != nullptr)) || num_sms < 2) {
    sb::set_last_error("sb_gemm_pair: shape or layout not supported");
    return (int)cudaErrorInvalidValue;
  }
  const long long tiles = static_cast<long long>((M + 255) / 256) * ((N + bn - 1) / bn) * groups;
  const sb::PairCut cut = sb::cut_last_wave(tiles, (K + sb::GP_BK - 1) / sb::GP_BK, num_sms, split_last != 0);
  const int align = cut.left > 0 && !out_f32 ? 8 : 16;
  if (reinterpret_cast<uintptr_t>(C) % align || (size_t(ldc) * (out_f32 ? 4 : 2)) % align ||
      (cut.left > 0 && (parts == nullptr || (reinterpret_cast<uintptr_t>(parts) & 15) || (!out_f32 && cut.full > 0)))) {
    sb::set_last_error("sb_gemm_pair: alignment, or a cut without its workspace, or of a bf16 output of more than a wave");
    return (int)cudaErrorInvalidValue;
  }
  const sb::PairShape s{M, N, K, bn, groups, group_start, group_rows, cut};
  const bool f32 = out_f32 || cut.left > 0;
  try {
#define SB_CASE(AM, BM_, OF)                   \
  if ((a_mn != 0) == AM && (b_mn != 0) == BM_ && f32 == OF) \
    return (int)sb::launch_pair<AM, BM_, OF>(A, B, C, bias, s, K, lda, ldb, ldc, out_f32 != 0, add, parts, status, stream);
    SB_CASE(false, false, false)
    SB_CASE(false, false, true)
    SB_CASE(false, true, false)
    SB_CASE(false, true, true)
    SB_CASE(true, true, false)
    SB_CASE(true, true, true)
#undef SB_CASE
  } catch (const std::exception& e) {
    sb::set_last_error(e.what());
  }
  return (int)cudaErrorInvalidValue;
}
