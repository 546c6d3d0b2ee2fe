// Fused W4A16 GEMM on CTA pairs, for more tokens than one 128-row block:
//   Y[M,N] = X[M,K] * dequant(W)[N,K]^T (+ bias) (+ residual), weights read from the canonical xqt_int4_nk_v1 bytes.
//
// A pair (cluster of two CTAs, cta_group::2) owns a tile of tile_n channels x MB * 256 tokens.  Each CTA brings in and
// holds MB blocks of 128 token rows and converts HALF of the tile's weight rows; the tensor cores of both read both
// halves.  So a weight is converted once per 512 tokens (MB = 2) and a stage moves MB * 16 KiB of activations per SM
// for MB * 128 x tile_n products.  What bounded the single-CTA form at M = 512 was the conversion (about 930 clocks per
// 64-K stage of 128 channels, against 512 for the MMAs of its 256 tokens, and every weight converted twice).
//
// Now (fp16, cold weights): 28672 x 4096 at M = 512 159 -> 112 us, at M = 256 89 -> 87; 4096 x 14336 at M = 512 109 -> 75.
// A 64-K stage takes 900 clocks + 1.25 per column and block: what is left is the conversion (leaving its arithmetic out
// saves 7 %, its parameter loads 7 %), the tensor rate under the power cap, and the last wave.
//
// tile_n is a run-time multiple of 32 and K may be split: the plan takes the pair with the cheapest waves (28672 channels
// at 512 tokens are 1.51 waves of 256-wide tiles on 74 pairs, but 1.73 of 224-wide ones).  A split writes fp32 partial sums [split][M][N]
// which a second kernel, on all SMs, adds in split order (bit-reproducible); letting the last CTA of a tile add them
// took 128 threads of one SM 14 us for 512 KiB.
//
// GLU form (the gate/up projections of a SwiGLU block, rows [gate; up] of one weight): the first CTA converts gate rows, the
// second the up rows of the same channels, so a token's gate and up sums meet in one tile and the epilogue writes
// h = silu(gate) * up in fp16, the operand of the down projection.  The separate form moved [M, 2 inter] through memory
// twice and h once more (SwiGLU kernel, conversion to fp16): about 30 of 219 us at 512 tokens of a 4096 x 14336 block.
//
// Warps (864 threads): 0 activation producer, 1 MMA issuer (the leader's), 2 packed-weight producer, 3-10 epilogue,
// 11-26 conversion, four groups of four warps on the stages it = g (mod 4), one weight row per thread: converting a stage
// is a chain of waits (two barrier tests, shared loads, the proxy fence), so four stages are in conversion at a time.
// Arithmetic as gemm_w4a16_fused.cu: (code - zero) exact in fp16, times the scale rounded once, fp32 accumulation.
#include "common.cuh"
#include "sm100.cuh"
#include "w4a16_dequant.cuh"

namespace xqt_b200 {

using namespace sm100;

int make_tile_map(CUtensorMap* map, const void* base, CUtensorMapDataType dtype, int esize, long long rows,
                  long long cols, int box_rows);
int make_byte_map(CUtensorMap* map, const void* base, long long rows, long long row_bytes, int box_bytes, int box_rows);

namespace w4p {
constexpr int kBM = 128, kBK = 64;
constexpr int kRawWarp = 2, kFirstEpiWarp = 3, kEpiWarps = 8, kFirstDqWarp = kFirstEpiWarp + kEpiWarps;
constexpr int kDqGroups = 4, kDqGroupWarps = 4;
constexpr int kThreads = (kFirstDqWarp + kDqGroups * kDqGroupWarps) * 32;   // 864
constexpr int kMinRaw = 2 * kDqGroups, kMaxRaw = 16;
constexpr int kMaxStages = 5;
constexpr int kABlockBytes = kBM * 128;
constexpr int kSmemBudget = 226 * 1024;
enum Status : unsigned int { kTimeout = 48 };
constexpr int kBarFull = 0, kBarEmpty = kBarFull + kMaxStages;
constexpr int kBarRawFull = kBarEmpty + kMaxStages, kBarRawEmpty = kBarRawFull + kMaxRaw;
constexpr int kBarTileFull = kBarRawEmpty + kMaxRaw, kBarTileEmpty = kBarTileFull + 2, kBarCount = kBarTileEmpty + 2;

// Depths of the two rings: five stages, fewer where they do not fit beside kMinRaw packed-weight slots; the rest of the
// memory deepens that ring.
struct Rings {
  int stages, raws;
};
constexpr Rings rings(int mb, int tile_n) {
  const int stage_bytes = mb * kABlockBytes + tile_n / 2 * 128, raw_bytes = tile_n / 2 * (kBK / 2), budget = kSmemBudget - 1024;
  const int stages = (budget - kMinRaw * raw_bytes) / stage_bytes < kMaxStages ? (budget - kMinRaw * raw_bytes) / stage_bytes : kMaxStages;
  const int raws = (budget - stages * stage_bytes) / raw_bytes;
  return {stages, raws < kMaxRaw ? raws : kMaxRaw};
}
// A parity test tells a barrier's phase from the one before it and no further.  The conversion groups look ahead by
// kDqGroups steps, so at step `it` the phase before the one they test has to be known complete:
//   Empty(it + 4): its slot's use at it + 4 - 2 * stages; Empty(it - stages) is known and MMAs complete in order, so
//     stages >= 4 will do.
//   RawFull(it + 4): its slot's use at it + 4 - raws.  Loads complete in any order.  Known are the group's own steps (it,
//     it - 4, ..: raws == 8) and all steps up to it - stages (their conversions were waited for by MMAs that are complete:
//     raws >= stages + 4).  Six slots beside five stages, as 160-column tiles had, are neither: a load overtaken by the
//     next group's could have been taken for complete.
constexpr bool look_ahead_is_sound() {
  for (int mb = 1; mb <= 2; ++mb)
    for (int tile_n = 64; tile_n <= 256; tile_n += 32) {
      const Rings r = rings(mb, tile_n);
      if (r.stages < kDqGroups || (r.raws != 2 * kDqGroups && r.raws < r.stages + kDqGroups)) return false;
    }
  return true;
}
static_assert(look_ahead_is_sound(), "a ring is too shallow for the conversion groups' look-ahead tests");
}  // namespace w4p

struct W4PairParams {
  int m, n, group_shift, groups;      // group_shift: 64-K steps per quantisation group, as a shift
  int mchunks, ntiles, splits, kblocks, stages, raw_bufs, tile_n, bufs;
  int param_dtype, nibble_signed, out_f32;
  const void* scales;
  const void* zeros;
  const float* bias;
  const void* residual;
  void* out;
  float* partials;                    // [splits][M][N] fp32 (splits > 1)
  unsigned int* status;
  int inter;                          // GLU: gate rows (= up rows); out is then h, fp16 [M, inter]
};

constexpr unsigned int kHiddenRange = 256;   // status bit: a value beyond fp16's range was clamped (as the activations' conversion sets it)

// silu(gate) * up of eight channels as the separate kernels compute it (the sums rounded to T, the product in fp32 rounded
// to T), then as an fp16 operand
template <typename T>
__device__ __forceinline__ void w4p_gate8(const float (&g)[8], const float (&u)[8], __half* dst, unsigned int* status) {
  float v[8];
  bool clipped = false;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float x = to_float<T>(from_float<T>(g[e]));
    v[e] = to_float<T>(from_float<T>(x / (1.0f + expf(-x)) * to_float<T>(from_float<T>(u[e]))));
    if constexpr (!__is_same(T, __half)) {
      clipped |= fabsf(v[e]) > 65504.f;                        // false for NaN
      v[e] = v[e] != v[e] ? v[e] : fminf(fmaxf(v[e], -65504.f), 65504.f);
    }
  }
  w4f_store8<__half>(dst, v);
  if (clipped) atomicOr(status, kHiddenRange);
}

// 8 columns of one row: bias, residual, rounding, store
template <typename T>
__device__ __forceinline__ void w4p_finish8(const float* bias, const void* residual, void* out, int out_f32, int n, int row, int col, float (&v)[8]) {
  if (bias != nullptr) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] += __ldg(bias + col + e);
  }
  if (residual != nullptr) {
    float rv[8];
    w4f_load8<T>(reinterpret_cast<const T*>(residual) + (size_t)row * n + col, rv);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] += rv[e];
  }
  if (out_f32) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + (size_t)row * n + col);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    w4f_store8<T>(reinterpret_cast<T*>(out) + (size_t)row * n + col, v);
  }
}

// tile -> token chunk, first channel, K blocks of the split; the tiles of one weight range are adjacent
struct W4PTile {
  int mc, n0, sp, kb0, kbn;
};
__device__ __forceinline__ W4PTile w4p_tile(const W4PairParams& p, int tile) {
  W4PTile t;
  t.mc = tile % p.mchunks;
  const int rest = tile / p.mchunks;
  t.sp = rest % p.splits;
  t.n0 = rest / p.splits * p.tile_n;
  t.kb0 = t.sp * p.kblocks / p.splits;
  t.kbn = (t.sp + 1) * p.kblocks / p.splits - t.kb0;
  return t;
}

// first weight row a CTA of the pair converts
template <bool GLU>
__device__ __forceinline__ int w4p_row0(const W4PairParams& p, int n0, int rank) {
  return GLU ? n0 / 2 + rank * p.inter : n0 + rank * (p.tile_n / 2);
}

template <int MB, typename T, bool GLU>
__global__ void __launch_bounds__(w4p::kThreads, 1)
gemm_w4a16_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ W4PairParams p) {
  using namespace w4p;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) unsigned long long bars[kBarCount];
  __shared__ uint32_t s_tmem_base;
  __shared__ volatile unsigned int s_abort;

  constexpr int kABytes = MB * kABlockBytes;
  constexpr uint32_t kTmemCols = 512;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ns = p.stages, nr = p.raw_bufs, half_rows = p.tile_n / 2, stage_bytes = kABytes + half_rows * 128, raw_bytes = half_rows * (kBK / 2);
  const uint32_t rank = cluster_ctarank();
  const int unit = blockIdx.x >> 1, units = gridDim.x >> 1, total_tiles = p.mchunks * p.ntiles * p.splits;
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  unsigned char* raw_base = tiles + (size_t)ns * stage_bytes;
  const uint32_t tiles_s = smem_addr(tiles), bar0 = smem_addr(&bars[0]);
  auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };

  if (threadIdx.x == 0) {
    s_abort = 0u;
    for (int s = 0; s < ns; ++s) {
      mbar_init(bar(kBarFull + s), 1 + 2 * kDqGroupWarps);   // the activations' bytes and both CTAs' converted weights
      mbar_init(bar(kBarEmpty + s), 1);
    }
    for (int r = 0; r < nr; ++r) {
      mbar_init(bar(kBarRawFull + r), 1);
      mbar_init(bar(kBarRawEmpty + r), kDqGroupWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(kBarTileFull + b), 1);
      mbar_init(bar(kBarTileEmpty + b), 2 * kEpiWarps);
    }
    fence_barrier_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc_cg<2>(smem_addr(&s_tmem_base), kTmemCols);
    tmem_relinquish_cg<2>();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();                  // the other CTA's barriers exist, and it runs
  cluster_wait_acquire();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem_base;
  grid_dependency_wait();                    // the activations may be the kernel's before this one
  grid_launch_dependents();

  // Every wait is bounded: when one runs out the CTA stops waiting anywhere, reports and drains out.
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

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer of the activation blocks
    if (elect_one()) {
      W4FRing ring(0, ns);
      const uint32_t full0 = cluster_map(bar(kBarFull), 0);
      for (int tile = unit; tile < total_tiles; tile += units) {
        const W4PTile t = w4p_tile(p, tile);
        for (int kb = 0; kb < t.kbn; ++kb, ring.advance(1)) {
          const int s = ring.slot;
          guarded_spin(bar(kBarEmpty + s), ring.phase ^ 1);
          if (rank == 0) mbar_expect_tx(bar(kBarFull + s), 2 * kABytes);
          const uint32_t st = tiles_s + (uint32_t)(s * stage_bytes), full = full0 + 8u * (uint32_t)s;
#pragma unroll
          for (int mb = 0; mb < MB; ++mb)    // block mb of the pair is 256 rows, this CTA's half of it; rows past M are zeros
            tma_load_2d_cg<2>(st + mb * kABlockBytes, &tm_a, (t.kb0 + kb) * kBK, ((t.mc * MB + mb) * 2 + (int)rank) * kBM, full);
        }
      }
    }
  } else if (warp == kRawWarp) {
    // ---------------------------------------------------------------- TMA producer of the packed weights (this CTA's half)
    if (elect_one()) {
      const uint32_t raw_s = smem_addr(raw_base);
      W4FRing ring(0, nr);
      for (int tile = unit; tile < total_tiles; tile += units) {
        const W4PTile t = w4p_tile(p, tile);
        for (int kb = 0; kb < t.kbn; ++kb, ring.advance(1)) {
          const int r = ring.slot;
          guarded_spin(bar(kBarRawEmpty + r), ring.phase ^ 1);
          mbar_expect_tx(bar(kBarRawFull + r), raw_bytes);
          tma_load_2d(raw_s + (uint32_t)(r * raw_bytes), &tm_w, (t.kb0 + kb) * (kBK / 2), w4p_row0<GLU>(p, t.n0, (int)rank), bar(kBarRawFull + r));
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc(kAccF32, kFmtF16, kFmtF16, 2 * kBM, (uint32_t)p.tile_n);
      uint32_t buf = 0, buf_phase = 1;
      W4FRing cur(0, ns), nxt(1, ns);
      bool ready = false;                    // the current stage's barrier has already been seen complete
      for (int tile = unit; tile < total_tiles; tile += units) {
        const W4PTile t = w4p_tile(p, tile);
        guarded_spin(bar(kBarTileEmpty + buf), buf_phase);
        tc_fence_after();
        const uint32_t d0 = tmem_base + buf * (uint32_t)(MB * p.tile_n);
        for (int kb = 0; kb < t.kbn; ++kb, cur.advance(1), nxt.advance(1)) {
          const int s = cur.slot;
          if (!ready) guarded_spin(bar(kBarFull + s), cur.phase);
          tc_fence_after();
          // the next stage's barrier is asked before this stage's MMAs are issued and the answer read after
          const bool next = mbar_test_wait(bar(kBarFull + nxt.slot), nxt.phase);
          const uint32_t a_addr = tiles_s + (uint32_t)(s * stage_bytes);
          const uint64_t bdesc = umma_desc_sw128(a_addr + kABytes);
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            const uint64_t adesc = umma_desc_sw128(a_addr + mb * kABlockBytes);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              umma_ss_cg<2, kMmaF16>(d0 + (uint32_t)(mb * p.tile_n), adesc + 2 * q, bdesc + 2 * q, idesc, kb != 0 || q != 0 ? 1u : 0u);
          }
          umma_commit_cg<2>(bar(kBarEmpty + s));
          ready = next;
        }
        umma_commit_cg<2>(bar(kBarTileFull + buf));
        if (++buf == (uint32_t)p.bufs) { buf = 0; buf_phase ^= 1u; }
      }
    }
  } else if (warp < kFirstDqWarp) {
    // ---------------------------------------------------------------- epilogue warps: a lane is a token row
    const int quarter = warp & 3, part = (warp - kFirstEpiWarp) >> 2;
    const uint32_t empty0 = cluster_map(bar(kBarTileEmpty), 0);
    const int cols = MB * p.tile_n / 2;      // columns of a warp: one token block (MB = 2) or half of the only one
    uint32_t buf = 0, buf_phase = 0;
    for (int tile = unit; tile < total_tiles; tile += units) {
      const W4PTile t = w4p_tile(p, tile);
      guarded_wait(bar(kBarTileFull + buf), buf_phase);
      tc_fence_after();
      const int block = MB == 2 ? part : 0, cbase = MB == 2 ? 0 : part * cols;
      const int row = ((t.mc * MB + block) * 2 + (int)rank) * kBM + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + buf * (uint32_t)(MB * p.tile_n) + (uint32_t)(part * cols) + ((uint32_t)(quarter * 32) << 16);
      if constexpr (GLU) {
        // chunks of 16 channels: all of them for the warp's token block (MB = 2), every other one of the only block
        const uint32_t gaddr = tmem_base + buf * (uint32_t)(MB * p.tile_n) + (uint32_t)(block * p.tile_n) + ((uint32_t)(quarter * 32) << 16);
        const int j0 = t.n0 / 2;
        __half* h = reinterpret_cast<__half*>(p.out) + (size_t)row * p.inter + j0;
#pragma unroll 1
        for (int c = MB == 2 ? 0 : part * 16; c < half_rows; c += MB == 2 ? 16 : 32) {
          uint32_t rg[16], ru[16];
          tmem_ld_32x16(gaddr + (uint32_t)c, rg);
          tmem_ld_32x16(gaddr + (uint32_t)(half_rows + c), ru);
          tmem_wait_ld_dep(rg);
          tmem_wait_ld_dep(ru);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (row < p.m && j0 + c + 8 * j < p.inter) {           // inter is a multiple of 8
              float g[8], u[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) { g[e] = __uint_as_float(rg[8 * j + e]); u[e] = __uint_as_float(ru[8 * j + e]); }
              w4p_gate8<T>(g, u, h + c + 8 * j, p.status);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(empty0 + 8u * buf);
        if (++buf == (uint32_t)p.bufs) { buf = 0; buf_phase ^= 1u; }
        continue;
      }
      float* part_row = p.partials + ((size_t)t.sp * p.m + row) * p.n;
#pragma unroll 1
      for (int c = 0; c < cols; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(taddr + (uint32_t)c, r);
        tmem_wait_ld_dep(r);
        if (row < p.m) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int col = t.n0 + cbase + c + 8 * j;
            if (col < p.n) {
              float v[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * j + e]);
              if (p.splits > 1) {
                float4* dst = reinterpret_cast<float4*>(part_row + col);
                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                dst[1] = make_float4(v[4], v[5], v[6], v[7]);
              } else {
                w4p_finish8<T>(p.bias, p.residual, p.out, p.out_f32, p.n, row, col, v);
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(empty0 + 8u * buf);
      if (++buf == (uint32_t)p.bufs) { buf = 0; buf_phase ^= 1u; }
    }
  } else {
    // ---------------------------------------------------------------- conversion warps
    const int dt = threadIdx.x - kFirstDqWarp * 32;
    const int grp = dt >> 7, row = dt & 127;             // group of four warps; the thread's weight row
    const bool active = row < half_rows;
    const uint32_t ready0 = cluster_map(bar(kBarFull), 0);
    const float zbase = 1024.f + (p.nibble_signed ? 8.f : 0.f);
    const uint32_t flip = p.nibble_signed ? 0x88888888u : 0u;               // two's complement -> code + 8
    uint32_t it_base = 0;                                // the CTA's steps before this tile
    W4FRing st_cur(grp, ns), st_nxt(grp + kDqGroups, ns), raw_cur(grp, nr), raw_nxt(grp + kDqGroups, nr);
    bool ahead_raw = false, ahead_free = false;          // this group's next stage was already seen ready
    for (int tile = unit; tile < total_tiles; tile += units) {
      const W4PTile t = w4p_tile(p, tile);
      const int wrow = w4p_row0<GLU>(p, t.n0, (int)rank) + row;
      const size_t prow = (size_t)(wrow < p.n ? wrow : p.n - 1) * p.groups;
      uint32_t nsc = 0u, nzp = 0u;                       // this group's next parameters, as raw bits (see the header of the single form)
      bool have_next = false;
      auto fetch_params = [&](int kb, uint32_t& sc, uint32_t& zp) {
        const int g = (t.kb0 + kb) >> p.group_shift;
        sc = load_param_bits(p.scales, p.param_dtype, prow + g);
        zp = p.zeros != nullptr ? load_param_bits(p.zeros, p.param_dtype, prow + g) : 0u;
      };
      for (int kb = (grp - (int)(it_base % kDqGroups)) & (kDqGroups - 1); kb < t.kbn; kb += kDqGroups,
               st_cur.advance(kDqGroups), st_nxt.advance(kDqGroups), raw_cur.advance(kDqGroups), raw_nxt.advance(kDqGroups)) {
        const int s = st_cur.slot, r = raw_cur.slot;
        uint32_t scb = nsc, zpb = nzp;
        if (!have_next) fetch_params(kb, scb, zpb);
        have_next = kb + kDqGroups < t.kbn;
        if (have_next) fetch_params(kb + kDqGroups, nsc, nzp);
        if (!ahead_raw) guarded_wait(bar(kBarRawFull + r), raw_cur.phase);
        uint4 raw[2];
        if (active) {
          const uint4* src = reinterpret_cast<const uint4*>(raw_base + (size_t)r * raw_bytes + row * (kBK / 2));
          raw[0] = src[0];
          raw[1] = src[1];
        }
        const float scale = param_from_bits(scb, p.param_dtype), zero = zbase + (p.zeros != nullptr ? param_from_bits(zpb, p.param_dtype) : 0.f);
        const __half2 off2 = __float2half2_rn(zero), scale2 = __float2half2_rn(scale);
        const bool exact = __low2float(scale2) == scale;     // a scale fp16 cannot hold is multiplied in fp32: one rounding either way
        if (!ahead_free) guarded_wait(bar(kBarEmpty + s), st_cur.phase ^ 1);
        if (active) {
          unsigned char* brow = tiles + (size_t)s * stage_bytes + kABytes + row * 128;
          const uint32_t words[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
#pragma unroll
          for (int j = 0; j < 8; ++j)                    // 16-byte chunk j of the 128-byte row, K order
            *reinterpret_cast<uint4*>(brow + ((j ^ (row & 7)) << 4)) =
                exact ? w4f_dequant_word(words[j] ^ flip, off2, scale2) : w4f_dequant_word_f32(words[j] ^ flip, zero, scale);
        }
        fence_proxy_async();                             // make the generic-proxy stores visible to the tensor cores' reads
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cluster(ready0 + 8u * (uint32_t)s);
          mbar_arrive(bar(kBarRawEmpty + r));            // the packed bytes were consumed by the conversion above
        }
        ahead_raw = mbar_test_wait(bar(kBarRawFull + raw_nxt.slot), raw_nxt.phase);
        ahead_free = mbar_test_wait(bar(kBarEmpty + st_nxt.slot), st_nxt.phase ^ 1);
      }
      it_base += (uint32_t)t.kbn;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();                  // no CTA of a pair leaves while the other's MMAs or arrivals still reach it
  cluster_wait_acquire();
  if (warp == 1) tmem_dealloc_cg<2>(tmem_base, kTmemCols);
}

// partial sums of a K split, added in split order: 8 columns per thread, [splits][M][N] is read once (from L2)
template <typename T>
__global__ void __launch_bounds__(256) w4p_reduce_kernel(const float* __restrict__ partials, const float* __restrict__ bias, const void* __restrict__ residual,
                                                         void* __restrict__ out, int m, int n, int splits, int out_f32) {
  grid_dependency_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, per_row = (size_t)n / 8;
  if (i >= (size_t)m * per_row) return;
  const int row = (int)(i / per_row), col = (int)(i % per_row) * 8;
  const size_t plane = (size_t)m * n;
  const float* src = partials + (size_t)row * n + col;
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = 0.f;
#pragma unroll 4
  for (int sp = 0; sp < splits; ++sp) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(src + sp * plane)), b = __ldcg(reinterpret_cast<const float4*>(src + sp * plane) + 1);
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
  }
  w4p_finish8<T>(bias, residual, out, out_f32, n, row, col, v);
}

// ----------------------------------------------------------------------------------------- host

namespace {

struct PairPlan {
  int mb, tile_n, splits;
  double cost;
};

// Estimated SM clocks of the forms; the constants were fitted to sweeps on a B200.
PairPlan pair_plan(int m, int n, int k, int max_splits = 8) {
  const int units = sm_count() / 2, kblocks = k / w4p::kBK;
  PairPlan best{1, 64, 1, 1e30};
  for (int mb = 1; mb <= 2; ++mb) {
    const int mchunks = ceil_div(m, 256 * mb);
    for (int tile_n = 64; tile_n <= 256; tile_n += 32) {
      const int tiles = mchunks * ceil_div(n, tile_n);
      for (int splits = 1; splits <= max_splits; ++splits) {
        if (splits > 1 && kblocks < splits * 8) break;
        // clocks per 64-K block: the conversion's chain of barriers and the MMAs behind it
        const double per_kb = 900 + 1.25 * mb * tile_n;
        const int waves = ceil_div(tiles * splits, units);
        const double epilogue = mb * tile_n * (splits > 1 ? 16.0 : 10.0);
        double cost = waves * (ceil_div(kblocks, splits) * per_kb + 1500) + epilogue * (2 * mb * tile_n <= 512 ? 1 : waves);
        if (splits > 1) cost += 4500 + (double)splits * m * n * 4 / 4500.0;
        if (cost < best.cost) best = PairPlan{mb, tile_n, splits, cost};
      }
    }
  }
  return best;
}

template <int MB, typename T, bool GLU>
int launch_pair(const void* x, const void* qw, W4PairParams p, int k, cudaStream_t stream) {
  using namespace w4p;
  CUtensorMap tm_a, tm_w;
  XQT_CUDA((cudaError_t)make_tile_map(&tm_a, x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.m, k, kBM));
  XQT_CUDA((cudaError_t)make_byte_map(&tm_w, qw, p.n, k / 2, kBK / 2, p.tile_n / 2));
  const Rings ring = rings(MB, p.tile_n);
  p.stages = ring.stages;
  p.raw_bufs = ring.raws;
  const int stage_bytes = MB * kABlockBytes + p.tile_n / 2 * 128, raw_bytes = p.tile_n / 2 * (kBK / 2);
  const size_t smem_bytes = (size_t)p.stages * stage_bytes + (size_t)p.raw_bufs * raw_bytes + 1024;
  constexpr auto kern = gemm_w4a16_pair_kernel<MB, T, GLU>;
  XQT_SMEM_OPT_IN(kern, kSmemBudget);
  const int tiles = p.mchunks * p.ntiles * p.splits, pairs = resident_pairs<kern>(kThreads, kSmemBudget);
  const int rc = launch_pdl_cluster(kern, dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs))), dim3(kThreads), 2, smem_bytes, stream, tm_a, tm_w, p);
  if (rc != 0 || p.splits == 1) return rc;
  const size_t threads = (size_t)p.m * (p.n / 8);
  return launch_pdl(w4p_reduce_kernel<T>, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, stream, (const float*)p.partials, p.bias, p.residual, p.out,
                    p.m, p.n, p.splits, p.out_f32);
}

}  // namespace

// fp32 partial sums of the form this size takes
size_t w4a16_gemm_pair_scratch_bytes(int m, int n, int k) {
  const PairPlan plan = pair_plan(m, n, k);
  return plan.splits > 1 ? (size_t)plan.splits * m * n * sizeof(float) : 0;
}

// x: fp16 [M, K]; checks are the caller's (w4a16_gemm_fused_launch)
int w4a16_gemm_pair_launch(const void* x, const void* qw, const void* scales, const void* zeros, const float* bias, const void* residual,
                           void* out, int m, int n, int k, int group_size, int nibble_signed, int act_dtype, int param_dtype, int out_f32,
                           float* partials, unsigned int* status, cudaStream_t stream) {
  const PairPlan plan = pair_plan(m, n, k);
  W4PairParams p{};
  p.m = m; p.n = n; p.group_shift = group_size == 2 * w4p::kBK ? 1 : 0; p.groups = k / group_size;
  p.mchunks = ceil_div(m, 256 * plan.mb); p.ntiles = ceil_div(n, plan.tile_n); p.splits = plan.splits; p.kblocks = k / w4p::kBK;
  p.tile_n = plan.tile_n; p.bufs = 2 * plan.mb * plan.tile_n <= 512 ? 2 : 1;
  p.param_dtype = param_dtype; p.nibble_signed = nibble_signed; p.out_f32 = out_f32;
  p.scales = scales; p.zeros = zeros; p.bias = bias; p.residual = residual; p.out = out; p.partials = partials; p.status = status;
#define XQT_PAIR(T) (plan.mb == 2 ? launch_pair<2, T, false>(x, qw, p, k, stream) : launch_pair<1, T, false>(x, qw, p, k, stream))
  return act_dtype == XQT_B200_BF16 ? XQT_PAIR(__nv_bfloat16) : XQT_PAIR(__half);
#undef XQT_PAIR
}

// h[M, inter] (fp16) = silu(x gate^T) * (x up^T), qw = [gate; up] with 2 * inter rows; x: fp16 [M, K].  act_dtype is the type the
// sums and h are rounded to.
int w4a16_gemm_pair_glu_launch(const void* x, const void* qw, const void* scales, const void* zeros, void* h, int m, int inter, int k,
                               int group_size, int nibble_signed, int act_dtype, int param_dtype, unsigned int* status, cudaStream_t stream) {
  const PairPlan plan = pair_plan(m, 2 * inter, k, 1);
  W4PairParams p{};
  p.m = m; p.n = 2 * inter; p.inter = inter; p.group_shift = group_size == 2 * w4p::kBK ? 1 : 0; p.groups = k / group_size;
  p.mchunks = ceil_div(m, 256 * plan.mb); p.ntiles = ceil_div(2 * inter, plan.tile_n); p.splits = 1; p.kblocks = k / w4p::kBK;
  p.tile_n = plan.tile_n; p.bufs = 2 * plan.mb * plan.tile_n <= 512 ? 2 : 1;
  p.param_dtype = param_dtype; p.nibble_signed = nibble_signed;
  p.scales = scales; p.zeros = zeros; p.out = h; p.status = status;
#define XQT_PAIR(T) (plan.mb == 2 ? launch_pair<2, T, true>(x, qw, p, k, stream) : launch_pair<1, T, true>(x, qw, p, k, stream))
  return act_dtype == XQT_B200_BF16 ? XQT_PAIR(__nv_bfloat16) : XQT_PAIR(__half);
#undef XQT_PAIR
}

}  // namespace xqt_b200
