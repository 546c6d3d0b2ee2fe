// The int8 GEMM of the W8A8 layers: Y[M,N] = int32(A[M,K] B[N,K]^T) * a_scale[m] * w_scale[n] (+ bias[n]) (+ low[m,n]), with
// the low-rank branch low = L[M,32] U[N,32]^T (16-bit operands, fp32 sums) computed beside it by the same tensor cores.
//
// Two launch forms of one kernel, picked by `plan` from the sizes:
//   pair (CG = 2)  persistent; the two CTAs of a cluster run 256 x tile_n tiles with cta_group::2 MMAs.  Each loads its 128
//                  rows of A and half of the B rows, so a stage moves a quarter less through L2 than two single-CTA tiles of
//                  the same area: at int8 rates (8192 multiply-adds per SM and clock) L2 -> SM bandwidth is what bounds
//                  128 x 256 tiles (393 MB in 24 us for 2048 x 4096 x 4096).  With pairs the tensor pipe is busy 52 % of a
//                  cold launch, L2 32 %: the rest is the pipeline's ramp per tile and the last wave.
//   single (CG = 1) one 128 x tile_n tile per CTA, its K range split over the CTAs of a cluster when the tiles alone leave
//                  SMs idle: int32 partial sums are exact, so they meet in distributed shared memory in any order.  For few
//                  tokens the layer is bound by streaming the weights, which takes as many SMs as possible.
// tile_n is a run-time multiple of 32: the plan takes the one whose waves waste least (4096 channels x 2048 tokens are 1.73
// waves of 256-wide pair tiles but 2.8 of 160-wide ones: 512 against 480 columns per SM).
//
// Warps (352 threads): 0 and 10 TMA producers of the activations and of the weights, 1 MMA issuer (the pair leader's), 2-9
// epilogue (tensor-memory lane quarter = warp % 4, columns by halves).  The int32 accumulators are double-buffered so that the epilogue of a tile overlaps the next one; the
// fp32 sums of the low-rank branch have a buffer of their own, computed by one more stage per tile (its operands are one
// 128-byte row per token / channel, loaded like a K block).  Every wait is bounded.
#include "common.cuh"
#include "sm100.cuh"

namespace xqt_b200 {

using namespace sm100;

int make_tile_map_ld(CUtensorMap* map, const void* base, CUtensorMapDataType dtype, int esize, long long rows, long long cols,
                     long long ld, int box_rows);

namespace gs {
constexpr int kBM = 128, kRowBytes = 128, kEpiWarps = 8, kWeightWarp = 2 + kEpiWarps, kThreads = (kWeightWarp + 1) * 32, kMaxStages = 8;
constexpr int kABytes = kBM * kRowBytes;
constexpr int kSmemBudget = 220 * 1024;
constexpr int kMaxSplit = 4, kReduceBytes = 72 * 1024;
enum Status : unsigned int { kTimeout = 16 };
constexpr int kBarFull = 0, kBarEmpty = kMaxStages, kBarTileFull = 2 * kMaxStages, kBarTileEmpty = kBarTileFull + 2;
constexpr int kBarLowEmpty = kBarTileEmpty + 2, kBarCount = kBarLowEmpty + 1;
}  // namespace gs

struct ScaledParams {
  int m, n, mtiles, ntiles, kblocks, stages, tile_n, split;
  int a_rows;               // rows of an A box: 128, or for a single row tile no more than the tokens there are
  int wide;                 // 1: rows are 32-byte aligned multiples of 16 columns
  const float* row_scale;
  const float* col_scale;
  const float* bias;
  const float* addend;      // [M, N] fp32 or null
  void* out;
  unsigned int* status;
};

template <typename T> __device__ __forceinline__ uint32_t gs_pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t gs_pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t gs_pack2<__half>(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// 16 finished columns of one row
template <typename T>
__device__ __forceinline__ void gs_store16(const ScaledParams& p, int row, int col, const float (&v)[16]) {
  T* dst = reinterpret_cast<T*>(p.out) + (size_t)row * p.n + col;
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = gs_pack2<T>(v[2 * j], v[2 * j + 1]);
  if (p.wide) {
    stg256(dst, o);
  } else {                                   // N is a multiple of 8
    *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
    if (col + 8 < p.n) *reinterpret_cast<uint4*>(dst + 8) = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

// QUADS: column scales and bias lie on 16 bytes.  A caller's slices may not: then one load per column (a form of its own: a test
// in the epilogue cost the smallest layers 2 %).
template <int CG, typename T, bool LOW, bool QUADS>
__global__ void __launch_bounds__(gs::kThreads, 1)
gemm_scaled_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_l,
                   const __grid_constant__ CUtensorMap tm_u, const __grid_constant__ ScaledParams p) {
  using namespace gs;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bars[kBarCount];
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile unsigned int s_abort;

  constexpr uint32_t kTmemCols = 512;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ns = p.stages, tile_n = p.tile_n, half_rows = CG == 2 ? tile_n / 2 : tile_n;     // B rows of this CTA
  const int stage_bytes = kABytes + half_rows * kRowBytes;
  const uint32_t rank = CG == 2 || p.split > 1 ? cluster_ctarank() : 0u;
  const bool leader = CG == 1 || rank == 0;
  const int units = CG == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x / p.split, unit = CG == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x / p.split;
  const int total_tiles = p.mtiles * p.ntiles;
  // K blocks of this CTA (all but the single form with a split: all of them), and whether it has the low-rank stage
  const int kb0 = CG == 1 ? (int)rank * p.kblocks / p.split : 0, kb1 = CG == 1 ? ((int)rank + 1) * p.kblocks / p.split : p.kblocks;
  const bool low_here = LOW && (CG == 2 || rank == 0);
  const int steps = kb1 - kb0 + (low_here ? 1 : 0);
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  const uint32_t ring_s = smem_addr(ring), bar0 = smem_addr(&bars[0]);
  auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };

  if (threadIdx.x == 0) {
    s_abort = 0u;
    for (int s = 0; s < ns; ++s) {
      mbar_init(bar(kBarFull + s), 2);
      mbar_init(bar(kBarEmpty + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(kBarTileFull + b), 1);
      mbar_init(bar(kBarTileEmpty + b), CG * kEpiWarps);
    }
    mbar_init(bar(kBarLowEmpty), CG * kEpiWarps);
    fence_barrier_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
  }
  if (warp == 1) {
    tmem_alloc_cg<CG>(smem_addr(&s_tmem_base), kTmemCols);
    tmem_relinquish_cg<CG>();
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2 || p.split > 1) {              // the other CTAs' barriers exist, and they run
    cluster_arrive_release();
    cluster_wait_acquire();
  }
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  grid_dependency_wait();                    // the activations are the kernel's before this one
  grid_launch_dependents();

  auto guarded_wait = [&](uint32_t b, uint32_t parity) {
    if (s_abort == 0u && !mbar_wait(b, parity)) {
      s_abort = 1u;
      atomicExch(p.status, (unsigned int)kTimeout);
    }
  };
  auto guarded_spin = [&](uint32_t b, uint32_t parity) {
    if (s_abort == 0u && !mbar_spin(b, parity)) {
      s_abort = 1u;
      atomicExch(p.status, (unsigned int)kTimeout);
    }
  };

  if (warp == 0 || warp == kWeightWarp) {
    // ---------------------------------------------------------------- TMA producers: warp 0 the activations, the other the weights
    if (elect_one()) {
      const bool weights = warp != 0;
      const CUtensorMap* tm = weights ? &tm_b : &tm_a;
      const CUtensorMap* tm_low = weights ? &tm_u : &tm_l;
      const uint32_t dst0 = ring_s + (weights ? kABytes : 0), bytes = (uint32_t)(CG * (weights ? half_rows : p.a_rows) * kRowBytes);
      int s = 0;
      uint32_t phase = 1;                    // a fresh barrier passes the wait for its preceding phase
      bool free = false;                     // the current stage was already seen free
      const uint32_t full0 = CG == 2 ? cluster_map(bar(kBarFull), 0) : bar(kBarFull);
      for (int tile = unit; tile < total_tiles; tile += units) {
        const int row = weights ? (tile / p.mtiles) * tile_n + (CG == 2 ? (int)rank * half_rows : 0)
                                : (tile % p.mtiles) * (kBM * CG) + (CG == 2 ? (int)rank * kBM : 0);
        for (int kb = 0; kb < steps; ++kb) {
          if (!free) guarded_spin(bar(kBarEmpty + s), phase);
          int sn = s + 1;
          uint32_t pn = phase;
          if (sn == ns) { sn = 0; pn ^= 1; }
          const bool next = mbar_test_wait(bar(kBarEmpty + sn), pn);
          const uint32_t st = dst0 + (uint32_t)(s * stage_bytes), full = full0 + 8u * (uint32_t)s;
          if (leader) mbar_expect_tx(bar(kBarFull + s), bytes);
          if (!LOW || kb < kb1 - kb0) tma_load_2d_cg<CG>(st, tm, (kb0 + kb) * kRowBytes, row, full);
          else tma_load_2d_cg<CG>(st, tm_low, 0, row, full);
          s = sn;
          phase = pn;
          free = next;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (leader && elect_one()) {
      const uint32_t idesc = umma_idesc(kAccS32, kFmtS8, kFmtS8, kBM * CG, (uint32_t)tile_n);
      const uint32_t fmt = sizeof(T) == 2 && __is_same(T, __half) ? kFmtF16 : kFmtBF16;
      const uint32_t idesc_low = umma_idesc(kAccF32, fmt, fmt, kBM * CG, (uint32_t)tile_n);
      int s = 0;
      uint32_t phase = 0, local = 0;
      bool ready = false;                    // the current stage's barrier has already been seen complete
      for (int tile = unit; tile < total_tiles; tile += units, ++local) {
        const uint32_t buf = local & 1, d_tmem = tmem_base + buf * (uint32_t)tile_n;
        guarded_spin(bar(kBarTileEmpty + buf), ((local >> 1) & 1) ^ 1);
        tc_fence_after();
        for (int kb = 0; kb < steps; ++kb) {
          if (!ready) guarded_spin(bar(kBarFull + s), phase);
          tc_fence_after();
          // the next stage's barrier is asked before this stage's MMAs are issued and the answer read after: a test takes
          // about 200 cycles, as long as the MMAs of a 96-column stage
          int sn = s + 1;
          uint32_t pn = phase;
          if (sn == ns) { sn = 0; pn ^= 1; }
          const bool next = mbar_test_wait(bar(kBarFull + sn), pn);
          const uint64_t adesc = umma_desc_sw128(ring_s + (uint32_t)(s * stage_bytes)), bdesc = umma_desc_sw128(ring_s + (uint32_t)(s * stage_bytes) + kABytes);
          if (!LOW || kb < kb1 - kb0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) umma_ss_cg<CG, kMmaI8>(d_tmem, adesc + 2 * q, bdesc + 2 * q, idesc, kb != 0 || q != 0 ? 1u : 0u);
          } else {                           // 32 of the row's 64 16-bit elements are the branch's
            guarded_spin(bar(kBarLowEmpty), (local & 1) ^ 1);
            tc_fence_after();
            umma_ss_cg<CG, kMmaF16>(tmem_base + 2 * (uint32_t)tile_n, adesc, bdesc, idesc_low, 0u);
            umma_ss_cg<CG, kMmaF16>(tmem_base + 2 * (uint32_t)tile_n, adesc + 2, bdesc + 2, idesc_low, 1u);
          }
          umma_commit_cg<CG>(bar(kBarEmpty + s));
          s = sn;
          phase = pn;
          ready = next;
        }
        umma_commit_cg<CG>(bar(kBarTileFull + buf));
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue warps
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const uint32_t empty0 = CG == 2 ? cluster_map(bar(kBarTileEmpty), 0) : 0u, low_empty = CG == 2 ? cluster_map(bar(kBarLowEmpty), 0) : 0u;
    const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int c0 = part * (tile_n / 2), c1 = c0 + tile_n / 2;
    uint32_t local = 0;
    // the single form with a split: partial sums of the other CTAs of the cluster, [split - 1][128 rows][tile_n + 4]
    // int32 (rows 16 bytes apart modulo the banks: a warp stores 32 rows at once)
    const int gstride = tile_n + 4;
    int* gather = reinterpret_cast<int*>(ring + ns * stage_bytes);
    for (int tile = unit; tile < total_tiles; tile += units, ++local) {
      const uint32_t buf = local & 1;
      const int row = (tile % p.mtiles) * (kBM * CG) + (CG == 2 ? (int)rank * kBM : 0) + quarter * 32 + lane, n0 = (tile / p.mtiles) * tile_n;
      const float rs = row < p.m ? __ldg(p.row_scale + row) : 0.f;
      // scale and bias of a 16-column chunk are asked for one chunk ahead (the first one before the tile is complete): read
      // where they are used, their L2 latency was most of the epilogue's time
      float cs[16], add[16];
      auto fetch = [&](int col) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = col + 4 * j < p.n;
          if constexpr (!QUADS) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              cs[4 * j + e] = in ? __ldg(p.col_scale + col + 4 * j + e) : 0.f;
              add[4 * j + e] = in && p.bias != nullptr ? __ldg(p.bias + col + 4 * j + e) : 0.f;
            }
          } else {
            const float4 v = in ? __ldg(reinterpret_cast<const float4*>(p.col_scale + col) + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            cs[4 * j] = v.x; cs[4 * j + 1] = v.y; cs[4 * j + 2] = v.z; cs[4 * j + 3] = v.w;
            const float4 b = in && p.bias != nullptr ? __ldg(reinterpret_cast<const float4*>(p.bias + col) + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            add[4 * j] = b.x; add[4 * j + 1] = b.y; add[4 * j + 2] = b.z; add[4 * j + 3] = b.w;
          }
        }
      };
      fetch(n0 + c0);
      guarded_wait(bar(kBarTileFull + buf), (local >> 1) & 1);
      tc_fence_after();
      if (CG == 1 && p.split > 1 && rank != 0) {
        const uint32_t to = cluster_map(smem_addr(gather + ((int)(rank - 1) * kBM + quarter * 32 + lane) * gstride), 0);
        for (int c = c0; c < c1; c += 16) {
          uint32_t r[16];
          tmem_ld_32x16(tlane + buf * (uint32_t)tile_n + (uint32_t)c, r);
          tmem_wait_ld_dep(r);
          if (row < p.m) {
#pragma unroll
            for (int j = 0; j < 4; ++j) st_cluster_b128(to + (uint32_t)(c + 4 * j) * 4, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          }
        }
        continue;                            // one tile per CTA in this form
      }
      if (CG == 1 && p.split > 1) {          // rank 0: wait for the others' partial sums (all threads of the cluster meet here)
        cluster_arrive_release();
        cluster_wait_acquire();
      }
#pragma unroll 1
      for (int c = c0; c < c1; c += 16) {
        uint32_t r[16], lo[16];
        tmem_ld_32x16(tlane + buf * (uint32_t)tile_n + (uint32_t)c, r);
        if constexpr (LOW) tmem_ld_32x16(tlane + 2 * (uint32_t)tile_n + (uint32_t)c, lo);
        const int col = n0 + c;
        float scale[16], shift[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) { scale[j] = rs * cs[j]; shift[j] = add[j]; }
        if (c + 16 < c1) fetch(col + 16);
        tmem_wait_ld_dep(r);
        if constexpr (LOW) tmem_wait_ld_dep(lo);
        if (row < p.m && col < p.n) {
          if (CG == 1 && p.split > 1) {
            for (int q = 0; q + 1 < p.split; ++q) {
              const int4* src = reinterpret_cast<const int4*>(gather + (q * kBM + quarter * 32 + lane) * gstride + c);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int4 v = src[j];
                r[4 * j] += (uint32_t)v.x; r[4 * j + 1] += (uint32_t)v.y; r[4 * j + 2] += (uint32_t)v.z; r[4 * j + 3] += (uint32_t)v.w;
              }
            }
          }
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            v[j] = (float)(int)r[j] * scale[j] + shift[j];
            if constexpr (LOW) v[j] += __uint_as_float(lo[j]);
          }
          if (p.addend != nullptr) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (col + 4 * j < p.n) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(p.addend + (size_t)row * p.n + col) + j);
                v[4 * j] += a.x; v[4 * j + 1] += a.y; v[4 * j + 2] += a.z; v[4 * j + 3] += a.w;
              }
            }
          }
          gs_store16<T>(p, row, col, v);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) {
          mbar_arrive_cluster(empty0 + 8u * buf);
          if (LOW) mbar_arrive_cluster(low_empty);
        } else {
          mbar_arrive(bar(kBarTileEmpty + buf));
          if (LOW) mbar_arrive(bar(kBarLowEmpty));
        }
      }
    }
  }
  // The single form with a split: everybody meets rank 0's epilogue warps at one cluster barrier (partial sums delivered).
  const bool met = CG == 1 && p.split > 1 && rank == 0 && warp >= 2 && warp < kWeightWarp;
  __syncwarp();
  if (CG == 1 && p.split > 1 && !met) {
    cluster_arrive_release();
    cluster_wait_acquire();
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) {                             // no CTA of a pair leaves while the other's MMAs or arrivals still reach it
    cluster_arrive_release();
    cluster_wait_acquire();
  }
  if (warp == 1) tmem_dealloc_cg<CG>(tmem_base, kTmemCols);
}

// ----------------------------------------------------------------------------------------- host

namespace {

struct ScaledPlan {
  int cg, tile_n, split;
};

// Estimated SM clocks of a form; the constants were fitted to sweeps of tile_n and split on a B200.
ScaledPlan scaled_plan(int m, int n, int k, bool low) {
  const int sms = sm_count(), kblocks = ceil_div(k, gs::kRowBytes), widest = low ? 160 : 256;
  ScaledPlan best{1, 32, 1};
  double best_cost = 1e30;
  for (int cg = 1; cg <= 2; ++cg) {
    const int mtiles = ceil_div(m, 128 * cg), units = cg == 2 ? sms / 2 : sms;
    for (int tile_n = 32; tile_n <= widest; tile_n += 32) {
      const int tiles = mtiles * ceil_div(n, tile_n);
      for (int split = 1; split <= (cg == 1 ? gs::kMaxSplit : 1); split *= 2) {
        if (split > 1 && (tiles * split > sms || split > kblocks || (split - 1) * gs::kBM * (tile_n + 4) * 4 > gs::kReduceBytes)) continue;
        const int waves = split > 1 ? 1 : ceil_div(tiles, units);
        // clocks per 128-byte K block: what L2 delivers to an SM (74 and 64 bytes a clock), the MMAs (8192 multiply-adds a
        // clock, no fewer than 60 clocks each), the producers' and the issuer's barrier round trips
        const double a_rows = cg == 1 && m < 128 ? m : 128;
        double per_kb = (a_rows + tile_n / cg) * gs::kRowBytes / (cg == 1 ? 74.0 : 64.0);
        if (per_kb < 2.1 * tile_n) per_kb = 2.1 * tile_n;
        if (per_kb < 310) per_kb = 310;
        const double cost = waves * (ceil_div(kblocks + (low ? 1 : 0), split) * per_kb + 250) + tile_n * 10 + (split > 1 ? 500 + (16 + 0.3 * a_rows) * tile_n * (split - 1) : 0);
        if (cost < best_cost) {
          best_cost = cost;
          best = ScaledPlan{cg, tile_n, split};
        }
      }
    }
  }
  return best;
}

template <int CG, typename T, bool LOW, bool QUADS>
int launch_scaled(const void* a, const void* b, const void* low_a, const void* low_b, ScaledParams p, int k, cudaStream_t stream) {
  using namespace gs;
  CUtensorMap tm_a, tm_b, tm_l, tm_u;
  const int b_rows = CG == 2 ? p.tile_n / 2 : p.tile_n;
  XQT_CUDA((cudaError_t)make_tile_map_ld(&tm_a, a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.m, k, k, p.a_rows));
  XQT_CUDA((cudaError_t)make_tile_map_ld(&tm_b, b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.n, k, k, b_rows));
  tm_l = tm_a;
  tm_u = tm_b;
  if (LOW) {
    const CUtensorMapDataType dt = __is_same(T, __half) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    XQT_CUDA((cudaError_t)make_tile_map_ld(&tm_l, low_a, dt, 2, p.m, 64, 64, p.a_rows));
    XQT_CUDA((cudaError_t)make_tile_map_ld(&tm_u, low_b, dt, 2, p.n, 64, 64, b_rows));
  }
  const int stage_bytes = kABytes + b_rows * kRowBytes;
  const int reduce = (p.split - 1) * kBM * (p.tile_n + 4) * 4;
  int stages = (kSmemBudget - 1024 - reduce) / stage_bytes;
  p.stages = stages > kMaxStages ? kMaxStages : stages;
  const size_t smem = (size_t)p.stages * stage_bytes + reduce + 1024;
  constexpr auto kern = gemm_scaled_kernel<CG, T, LOW, QUADS>;
  XQT_SMEM_OPT_IN(kern, kSmemBudget);
  const int tiles = p.mtiles * p.ntiles;
  int grid, cluster;
  if (CG == 2) {
    const int pairs = resident_pairs<kern>(kThreads, kSmemBudget);
    grid = 2 * (tiles < pairs ? tiles : pairs);
    cluster = 2;
  } else if (p.split > 1) {
    grid = tiles * p.split;
    cluster = p.split;
  } else {
    grid = tiles < sm_count() ? tiles : sm_count();
    cluster = 1;
  }
  return launch_pdl_cluster(kern, dim3((unsigned)grid), dim3(kThreads), cluster, smem, stream, tm_a, tm_b, tm_l, tm_u, p);
}

}  // namespace

// int8 A [M,K] x int8 B [N,K]^T, out = acc * row_scale[m] * col_scale[n] (+ bias[n]) (+ addend[m,n], fp32)
// (+ low_a [M,64] low_b [N,64]^T over their first 32 columns, in the output dtype)
int gemm_scaled_launch(const void* a, const void* b, const float* row_scale, const float* col_scale, const float* bias, const float* addend,
                       const void* low_a, const void* low_b, void* out, int m, int n, int k, int out_dtype, unsigned int* status,
                       cudaStream_t stream) {
  XQT_REQUIRE(m > 0 && n > 0 && k > 0 && k % 16 == 0 && n % 8 == 0 && ((uintptr_t)addend & 15) == 0);
  XQT_REQUIRE(out_dtype == XQT_B200_BF16 || out_dtype == XQT_B200_FP16);
  XQT_REQUIRE(a != nullptr && b != nullptr && row_scale != nullptr && col_scale != nullptr && out != nullptr && status != nullptr);
  XQT_REQUIRE(((uintptr_t)out & 15) == 0 && ((uintptr_t)row_scale & 3) == 0 && ((uintptr_t)col_scale & 3) == 0 && ((uintptr_t)bias & 3) == 0);
  XQT_REQUIRE((low_a != nullptr) == (low_b != nullptr));
  const bool low = low_a != nullptr;
  ScaledPlan plan = scaled_plan(m, n, k, low);
  ScaledParams p{};
  p.m = m; p.n = n; p.mtiles = ceil_div(m, gs::kBM * plan.cg); p.ntiles = ceil_div(n, plan.tile_n); p.kblocks = ceil_div(k, gs::kRowBytes);
  p.tile_n = plan.tile_n; p.split = plan.split;
  // rows past the last token are not fetched (a box past the matrix costs the copy engine as much as one inside); what the
  // tile holds there reaches only sums that are not stored
  p.a_rows = plan.cg == 1 && m < gs::kBM ? (m + 7) / 8 * 8 : gs::kBM;
  const bool quads = ((uintptr_t)col_scale & 15) == 0 && ((uintptr_t)bias & 15) == 0;
  p.wide = n % 16 == 0 && ((uintptr_t)out & 31) == 0;
  p.row_scale = row_scale; p.col_scale = col_scale; p.bias = bias; p.addend = addend; p.out = out; p.status = status;
#define XQT_GSQ(CG, T, LOW) (quads ? launch_scaled<CG, T, LOW, true>(a, b, low_a, low_b, p, k, stream) : launch_scaled<CG, T, LOW, false>(a, b, low_a, low_b, p, k, stream))
#define XQT_GS(T) (plan.cg == 2 ? (low ? XQT_GSQ(2, T, true) : XQT_GSQ(2, T, false)) : (low ? XQT_GSQ(1, T, true) : XQT_GSQ(1, T, false)))
  return out_dtype == XQT_B200_BF16 ? XQT_GS(__nv_bfloat16) : XQT_GS(__half);
#undef XQT_GS
#undef XQT_GSQ
}

}  // namespace xqt_b200
