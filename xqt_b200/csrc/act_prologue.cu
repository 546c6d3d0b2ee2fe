// Activation prologue of the W8A8 / W4A4 / SVDQuant linears in one kernel: block-Hadamard rotation, dynamic
// quantisation and the rank-R down projection of a low-rank branch, so that a token is read once and only its codes,
// scales and R sums are written.  The definitions (butterfly order, scales, rounding, code forms) are those of
// rotate_quant.cu, bit for bit; that file serves the options this one does not.
//
// A warp's unit of work is 4 tokens x 256 features.  Two of the rotation's stages (strides below 16) run on 16
// consecutive features a lane has loaded; the wider ones need features 16 apart, so the unit is transposed once through
// the warp's own shared memory (fp32, conflict-free both ways) and every lane then holds two adjacent features of all
// sixteen 16-feature runs: the wide stages are packed fp32 pairs, and so are the scaling and the rounding to the
// activation type.  The rounded unit stays in shared memory (16-byte chunks exchanged by row, see `chunk_at`), from
// where it is quantised in feature order and multiplied by the down factors (mma.m16n8k16, 16 x 32 sums per warp).
//
// What bounds it: instruction issue (about 18 instructions a feature, half of them the quantisation; counters at 2048 x 4096 int8:
// issue 52 % and the shared-memory pipe 50 % busy with 20 warps an SM, DRAM 11 %, caches cold).  The form before
// it exchanged the wide stages by shuffles (34 a feature) and left the down projection to a kernel of its own, which
// read the rotated token again and was bound by load latency.
//   int8 modes:  the scale needs the whole token, so the CTAs of a token hold it whole (tokens x K x 2 bytes).
//   int4 group-64 mode: everything is local to a 256-feature chunk; a warp runs its chunks on its own.
// A CTA takes 4, 8 or 16 tokens (`pick_split`): 4 unless a low-rank branch makes every CTA read its share of the down
// matrix (64 bytes a feature, from L2).  The features of a token may be split over the CTAs of a cluster: their maxima and
// partial sums meet in distributed shared memory.  That split is what keeps enough warps on an SM: one CTA per 16 tokens
// of a 3072-feature layer (256 CTAs of 6 warps, 10 warps an SM) ran 40 us at 4096 tokens.
#include "common.cuh"
#include "sm100.cuh"

namespace xqt_b200 {

using namespace sm100;

namespace apro {
constexpr int kMaxWarps = 8, kMaxSplit = 8;
constexpr int kUnitRows = 4, kChunk = 256;                 // a unit is kUnitRows x kChunk
constexpr int kXposeStride = kChunk + 16;                  // floats; rows 64 bytes apart modulo 128
constexpr int kXposeBytes = kUnitRows * kXposeStride * 4;  // 4352
constexpr int kRedStride = 33;
constexpr int kSmemMost = 200 * 1024, kSmemOptIn = 220 * 1024;      // the sums of a low-rank branch come on top
constexpr float kMagic = 12582912.f;                       // 1.5 * 2^23: adding it leaves rint(x) in the low mantissa bits
constexpr float kSeventh = 1.0f / 7.0f;
}  // namespace apro

struct ProloguePar {
  const void* x;
  const float* column_scale;   // [rot_block] or null
  int factors_ready;           // the caller vouches that no earlier kernel is writing them: read before griddepcontrol.wait
  int8_t* codes;               // [M, K]
  float* scales;               // int8: [M]; int4: tile-major [ceil(M/128)][K/64][128]
  const void* down;            // [32, K] or null
  void* la;                    // what la_form says
  float lora_scale;
  int la_form;                 // 1: fp32 [M, 32]; 2: bf16 hi|lo operand images (see lowrank_down.cu); 3: T [M, 64], columns 0-31
  int m, k, rot_block, rows, chunks, split;      // split: CTAs of a cluster that share a token's chunks
  int gather_off;                                // shared-memory offset of the sums from the cluster's CTAs: memory of its own
};

// 16-byte chunk c of row r of a rounded tile: rows r, r+1 in different 64-byte halves (a fragment load of two rows), rows
// 0..3 of a unit in different 32-byte quarters (the unit's stores)
__device__ __forceinline__ int chunk_at(int r, int c) { return c ^ (((r & 1) << 2) | (r & 2)); }

// Maxima of packed absolute values propagate NaN, so a maximum also says whether a value was not finite, at no cost to the
// values that are; a NaN does not count towards a scale (see where it is found).
__device__ __forceinline__ uint32_t apro_top(uint32_t v) { return max(v & 0xffffu, v >> 16); }

template <typename T> struct Pack16;
template <> struct Pack16<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 v = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static constexpr uint32_t kInf = 0x7f80;
  static __device__ __forceinline__ uint32_t round2(float a, float b) { const __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&v); }
  static __device__ __forceinline__ float2 wide2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
};
template <> struct Pack16<__half> {
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __half2 v = __hmax2_nan(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static constexpr uint32_t kInf = 0x7c00;
  static __device__ __forceinline__ uint32_t round2(float a, float b) { const __half2 v = __floats2half2_rn(a, b); return *reinterpret_cast<const uint32_t*>(&v); }
  static __device__ __forceinline__ float2 wide2(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
};

__device__ __forceinline__ unsigned long long apro_sub2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

template <typename T>
__device__ __forceinline__ void apro_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (sizeof(T) == 2 && __is_same(T, __half))
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A radix-4 butterfly of the regular family on (a, b, c, d); `Op` adds and subtracts floats or packed pairs.
template <typename V, typename Add, typename Sub>
__device__ __forceinline__ void regular4(V& a, V& b, V& c, V& d, Add add, Sub sub) {
  const V p = add(a, b), q = sub(a, b), r = add(c, d), t = sub(c, d);
  a = add(p, t); b = sub(p, t); c = add(q, r); d = sub(r, q);
}

// Rotates and rounds rows [row0, row0 + 4) x features [256 chunk, +256) of x into the tile at `tile` (row stride
// `stride` bytes, the unit's first row being tile row `tr0`, its first chunk `c0`); rows past M and features past K are
// zeros.  Returns, per lane, the packed absolute maximum of the values it has rounded (row tr0 + lane / 8).
template <typename T, int ROT>
__device__ __forceinline__ uint32_t apro_unit(const ProloguePar& p, int row0, int chunk, unsigned char* tile, int stride, int tr0, int c0,
                                              float* xpose, const float* cs) {
  using namespace apro;
  using P = Pack16<T>;
  const int lane = threadIdx.x & 31;
  const int hh = lane >> 4, l = lane & 15;
  const int f0 = chunk * kChunk + l * 16;
  uint4 raw[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = row0 + 2 * i + hh;
    const bool inside = row < p.m && f0 < p.k;
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + (size_t)row * p.k + f0);
    raw[i][0] = inside ? __ldg(src) : make_uint4(0u, 0u, 0u, 0u);
    raw[i][1] = inside ? __ldg(src + 1) : make_uint4(0u, 0u, 0u, 0u);
  }
  uint32_t top = 0u;
  if constexpr (ROT == 0) {
    // no rotation: the values are rounded already; row tr0 + 2 i + hh, reduced to the lane / 8 form by the caller's rule
    uint32_t mx[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = tr0 + 2 * i + hh;
#pragma unroll
      for (int j = 0; j < 2; ++j)
        *reinterpret_cast<uint4*>(tile + r * stride + chunk_at(r, c0 + 2 * l + j) * 16) = raw[i][j];
      const uint32_t w[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
      mx[i] = 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) mx[i] = Pack16<T>::max2(mx[i], w[j] & 0x7fff7fffu);
      mx[i] = Pack16<T>::max2(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 8));      // lanes l and l ^ 8
    }
    // lane 16 h + l now holds rows h and 2 + h; lane / 8 wants rows 0..3: half 0 keeps rows 0 (l < 8) and 1, half 1 rows 2 and 3
    const uint32_t give = hh ? mx[0] : mx[1];
    const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 16);
    const uint32_t own = hh ? mx[1] : mx[0];                 // half 0: row 0, half 1: row 3
    // half 0 received row 1 (from half 1's mx[0]), half 1 received row 2 (half 0's mx[1])
    top = hh ? ((lane & 8) ? own : got) : ((lane & 8) ? got : own);
    return top;
  } else {
    float* dst[4];                                           // slots of this lane's runs, see below
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = xpose + hh * kXposeStride + 16 * l + 4 * (j ^ ((l >> 1) & 3));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float v[16];
      const uint32_t w[8] = {raw[i][0].x, raw[i][0].y, raw[i][0].z, raw[i][0].w, raw[i][1].x, raw[i][1].y, raw[i][1].z, raw[i][1].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 f = P::wide2(w[j]);
        v[2 * j] = f.x;
        v[2 * j + 1] = f.y;
      }
      auto add = [](float a, float b) { return __fadd_rn(a, b); };
      auto sub = [](float a, float b) { return __fsub_rn(a, b); };
      if constexpr (ROT == 1) {
#pragma unroll
        for (int b = 0; b < 4; ++b) regular4(v[4 * b], v[4 * b + 1], v[4 * b + 2], v[4 * b + 3], add, sub);
#pragma unroll
        for (int b = 0; b < 4; ++b) regular4(v[b], v[4 + b], v[8 + b], v[12 + b], add, sub);
      } else {
#pragma unroll
        for (int st = 1; st <= 8; st *= 2)
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int at = (b / st) * 2 * st + (b % st);
            const float a = v[at], c = v[at + st];
            v[at] = add(a, c);
            v[at + st] = sub(a, c);
          }
      }
      // features 16 l + 4 j .. + 3 at 16-byte slot 4 l + (j ^ (l / 2 mod 4)): eight lanes' stores cover all banks
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4*>(dst[j] + 2 * i * kXposeStride) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    __syncwarp();
    const int r = lane >> 3, tp = lane & 7;                  // row of the unit; features 16 i + 2 tp, + 1
    unsigned long long w[16];
    const float* src[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) src[j] = xpose + r * kXposeStride + 2 * (tp & 1) + 4 * ((tp >> 1) ^ j);
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = *reinterpret_cast<const unsigned long long*>(src[(i >> 1) & 3] + 16 * i);
    auto add = [](unsigned long long a, unsigned long long b) { return f32x2_add(a, b); };
    auto sub = [](unsigned long long a, unsigned long long b) { return apro_sub2(a, b); };
    if constexpr (ROT == 1) {
      if (p.rot_block > 16) {
#pragma unroll
        for (int b = 0; b < 4; ++b) regular4(w[4 * b], w[4 * b + 1], w[4 * b + 2], w[4 * b + 3], add, sub);
      }
      if (p.rot_block > 64) {
#pragma unroll
        for (int b = 0; b < 4; ++b) regular4(w[b], w[4 + b], w[8 + b], w[12 + b], add, sub);
      }
    } else {
#pragma unroll
      for (int st = 1; st <= 8; st *= 2) {
        if (16 * st < p.rot_block) {
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int at = (b / st) * 2 * st + (b % st);
            const unsigned long long a = w[at], c = w[at + st];
            w[at] = add(a, c);
            w[at + st] = sub(a, c);
          }
        }
      }
    }
    // chunk_at(tr, c0 + 2 i + tp / 4): c0 is a multiple of 32 and the row's mask even, so only i's low two bits meet it
    const int tr = tr0 + r, mask = chunk_at(tr, 0) >> 1;
    unsigned char* trow = tile + tr * stride + c0 * 16 + (tp >> 2) * 16 + (tp & 3) * 4;
    unsigned char* out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j] = trow + (j ^ mask) * 32;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const unsigned long long s = f32x2_mul(w[i], *reinterpret_cast<const unsigned long long*>(cs + 16 * i + 2 * tp));
      float a, b;
      f32x2_unpack(s, a, b);
      const uint32_t o = P::round2(a, b);
      top = Pack16<T>::max2(top, o & 0x7fff7fffu);
      *reinterpret_cast<uint32_t*>(out[i & 3] + (i >> 2) * 128) = o;
    }
    return top;
  }
}

// larger half of a packed pair, as fp32
template <typename T>
__device__ __forceinline__ float apro_wide_max(uint32_t v) {
  const float2 f = Pack16<T>::wide2(v);
  return fmaxf(f.x, f.y);
}

// a / b correctly rounded, two quotients at once: Markstein's division step ("Computation of elementary functions on the
// IBM RISC System/6000 processor", 1990): with the correctly rounded reciprocal y, q0 = a y and the exact remainder
// r = a - b q0, q0 + r y is the IEEE quotient (no over- or underflow in between).  No test for values that lie near a
// rounding boundary is needed: 16-bit values hit such boundaries so often that half of the warps took the slow way.
__device__ __forceinline__ unsigned long long apro_div2(unsigned long long a, unsigned long long y, unsigned long long neg_b) {
  const unsigned long long q0 = f32x2_mul(a, y);
  return f32x2_fma(f32x2_fma(neg_b, q0, a), y, q0);
}

// largest absolute value in N words of packed pairs that is not NaN, and no less than mx
template <typename T, int N>
__device__ __forceinline__ float apro_number_max(const uint32_t (&w)[N], float mx) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const float2 f = Pack16<T>::wide2(w[j]);
    mx = fmaxf(mx, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  return mx;
}

// The same over tile row r, whose 16-byte chunks 0 .. chunks - 1 a warp shares
template <typename T>
__device__ __noinline__ float apro_row_number_max(const unsigned char* row, int r, int chunks) {
  float mx = 0.f;
  for (int c = threadIdx.x & 31; c < chunks; c += 32) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + chunk_at(r, c) * 16);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    mx = apro_number_max<T>(w, mx);
  }
#pragma unroll
  for (int off = 1; off <= 16; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  return mx;
}

// Codes of 16 consecutive values (8 packed words): rint of the IEEE quotient value / sc.  `divide`: the quotient may leave
// the code range, the scale is subnormal or a value is not finite (a token's or group's own rule, rare; a NaN quotient takes
// the lowest code).  FORM 0: int8; 1: int4 as sign << 7 | magnitude.
template <typename T, int FORM>
__device__ __forceinline__ uint4 quantise16(const uint32_t (&w)[8], float sc, float rcp, bool divide) {
  using namespace apro;
  const unsigned long long rcp2 = f32x2_pack(rcp, rcp), neg2 = f32x2_pack(-sc, -sc), magic2 = f32x2_pack(kMagic, kMagic);
  uint32_t code[16];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t word = w[j];
    if (FORM == 1) word &= 0x7fff7fffu;
    const float2 f = Pack16<T>::wide2(word);
    float rx, ry;
    f32x2_unpack(f32x2_add(apro_div2(f32x2_pack(f.x, f.y), rcp2, neg2), magic2), rx, ry);
    code[2 * j] = __float_as_uint(rx);
    code[2 * j + 1] = __float_as_uint(ry);
  }
  if (divide) {
    constexpr float low = FORM == 0 ? -128.f : -8.f, high = FORM == 0 ? 127.f : 7.f;
    auto exact = [&](float v) {
      const int c = (int)fminf(fmaxf(rintf(__fdiv_rn(v, sc)), low), high);
      return (uint32_t)(FORM == 0 || c >= 0 ? c : 0x80 - c);
    };
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 f = Pack16<T>::wide2(w[j]);
      code[2 * j] = exact(f.x);
      code[2 * j + 1] = exact(f.y);
    }
  }
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    o[j] = __byte_perm(__byte_perm(code[4 * j], code[4 * j + 1], 0x0040), __byte_perm(code[4 * j + 2], code[4 * j + 3], 0x0040), 0x5410);
    if (FORM == 1 && !divide) {
      // magnitudes are 0..7: the sign bit only where the magnitude is not zero
      const uint32_t sign = __byte_perm(w[2 * j], w[2 * j + 1], 0x7531) & 0x80808080u;
      o[j] |= sign & (o[j] + 0x7f7f7f7fu);
    }
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Partial down projection of a warp: the fragment steps s = first, first + every, .. below `steps`, each 16 tokens x 32
// features of the rounded tile (whose first feature is the layer's `k0`) times the down factors.  Lane t of a quad takes 8
// consecutive features for two MMA steps, both operands alike.  Tokens the CTA does not have repeat its last one: their
// sums are not stored.
template <typename T>
__device__ __forceinline__ void apro_down(const ProloguePar& p, const unsigned char* tile, int stride, int k0, int first, int every, int steps,
                                          float (&acc)[4][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = min(g, p.rows - 1), r1 = min(g + 8, p.rows - 1), m0 = chunk_at(r0, 0), m1 = chunk_at(r1, 0);
  // chunk_at(r, 4 s + t) = 4 (s ^ mask / 4) + (t ^ mask mod 4)
  const unsigned char* a0 = tile + r0 * stride + (t ^ (m0 & 3)) * 16;
  const unsigned char* a1 = tile + r1 * stride + (t ^ (m1 & 3)) * 16;
  const int x0 = m0 >> 2, x1 = m1 >> 2;
  const uint4* b0 = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.down) + (size_t)g * p.k + k0) + t;
  const uint4* b1 = b0 + p.k;                           // eight rows of k elements are k 16-byte pieces
  const uint4* b2 = b1 + p.k;
  const uint4* b3 = b2 + p.k;
#pragma unroll 2
  for (int s = first; s < steps; s += every) {
    const uint4 b[4] = {__ldg(b0 + 4 * s), __ldg(b1 + 4 * s), __ldg(b2 + 4 * s), __ldg(b3 + 4 * s)};
    const uint4 lo = *reinterpret_cast<const uint4*>(a0 + (s ^ x0) * 64), hi = *reinterpret_cast<const uint4*>(a1 + (s ^ x1) * 64);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      apro_mma<T>(acc[j], lo.x, hi.x, lo.y, hi.y, b[j].x, b[j].y);
      apro_mma<T>(acc[j], lo.z, hi.z, lo.w, hi.w, b[j].z, b[j].w);
    }
  }
}

// The chunks of this CTA: [first, last) of p.chunks
__device__ __forceinline__ void apro_share(const ProloguePar& p, int& rank, int& first, int& last) {
  rank = p.split > 1 ? (int)cluster_ctarank() : 0;
  first = rank * p.chunks / p.split;
  last = (rank + 1) * p.chunks / p.split;
}

// Adds the warps' 16 x 32 partial sums in warp order (`part`: one [16][kRedStride] strip per warp), then those of the
// cluster's CTAs in rank order (`gather`: [split][16][32] in the first CTA), and stores them.  The cluster's CTAs are known
// to run when this is called.
template <typename T>
__device__ __forceinline__ void apro_store_down(const ProloguePar& p, float* part, float* gather, const float (&acc)[4][4], int row0, int rank) {
  using namespace apro;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* own = part + warp * 16 * kRedStride;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int col = 8 * j + 2 * t;
    own[g * kRedStride + col] = acc[j][0];
    own[g * kRedStride + col + 1] = acc[j][1];
    own[(g + 8) * kRedStride + col] = acc[j][2];
    own[(g + 8) * kRedStride + col + 1] = acc[j][3];
  }
  __syncthreads();
  const int warps = blockDim.x >> 5;
  const uint32_t remote = p.split > 1 ? cluster_map(smem_addr(gather + rank * 512), 0) : 0u;
  for (int i = threadIdx.x; i < p.rows * 32; i += blockDim.x) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += part[(w * 16 + (i >> 5)) * kRedStride + (i & 31)];
    if (p.split > 1) st_cluster_f32(remote + i * 4, s);
    else gather[i] = s;
  }
  if (p.split > 1) {
    cluster_arrive_release();
    cluster_wait_acquire();
    if (rank != 0) return;
  } else {
    __syncthreads();
  }
  for (int i = threadIdx.x; i < p.rows * 32; i += blockDim.x) {
    const int c = i & 31, row = row0 + (i >> 5);
    if (row >= p.m) break;
    float s = 0.f;
    for (int q = 0; q < p.split; ++q) s += gather[q * 512 + i];
    s *= p.lora_scale;
    if (p.la_form == 1) {
      reinterpret_cast<float*>(p.la)[(size_t)row * 32 + c] = s;
    } else if (p.la_form == 2) {
      unsigned char* dst = reinterpret_cast<unsigned char*>(p.la) + (size_t)row * 128;
      const __nv_bfloat16 hi = __float2bfloat16_rn(s), lo = __float2bfloat16_rn(s - __bfloat162float(hi));
      *reinterpret_cast<__nv_bfloat16*>(dst + (((c >> 3) ^ (row & 7)) << 4) + (c & 7) * 2) = hi;
      *reinterpret_cast<__nv_bfloat16*>(dst + ((((c >> 3) + 4) ^ (row & 7)) << 4) + (c & 7) * 2) = lo;
    } else {
      reinterpret_cast<T*>(p.la)[(size_t)row * 64 + c] = from_float<T>(s);
    }
  }
}

// Read after the wait they cost every CTA a memory latency on its critical path (0.4 of 9.4 us at 77 tokens x 2048, 0.7 of 43.7
// at 2048 x 4096; a prefetch into L2 or loads of x ahead of them do not hide it), read before it nothing.
template <int ROT>
__device__ __forceinline__ void apro_column_scale(const ProloguePar& p, float* cs) {
  if constexpr (ROT != 0)
    for (int i = threadIdx.x; i < apro::kChunk; i += blockDim.x) cs[i] = __ldg(p.column_scale + (i & (p.rot_block - 1)));
}

// int8, one scale per token.  SCALE16: the scale rounded to T (mode 9).
template <typename T, int ROT, bool SCALE16>
__global__ void __launch_bounds__(apro::kMaxWarps * 32, 4)
act_prologue_i8_kernel(const ProloguePar p) {
  using namespace apro;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float cs[kChunk];
  __shared__ int s_top[16], s_peer[kMaxSplit][16], s_nan[17];         // s_nan: per token, then of any
  __shared__ float4 s_scale[16];                       // per token: scale, reciprocal, "divide" (see quantise16)
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int rank, first, last;
  apro_share(p, rank, first, last);
  const int own = last - first, k0 = first * kChunk, k1 = min(p.k, last * kChunk);
  const int stride = own * kChunk * 2;
  unsigned char* tile = smem;
  float* xpose = reinterpret_cast<float*>(smem + p.rows * stride + warp * kXposeBytes);
  const int row0 = (int)(blockIdx.x / p.split) * p.rows;
  if (p.split > 1) cluster_arrive_relaxed();           // "this CTA runs"; waited for before the first remote store
  if (threadIdx.x < 17) s_top[threadIdx.x & 15] = s_nan[threadIdx.x] = 0;
  if (p.factors_ready) apro_column_scale<ROT>(p, cs);
  __syncthreads();
  grid_dependency_wait();
  grid_launch_dependents();
  if (ROT != 0 && !p.factors_ready) {
    apro_column_scale<ROT>(p, cs);
    __syncthreads();
  }
  int chunk = warp;
  for (int ur = 0; ur < p.rows; ur += kUnitRows, chunk -= own) {
    // consecutive units of the CTA go to consecutive warps, also where a token has fewer chunks than there are warps
    for (; chunk < own; chunk += warps) {
      __syncwarp();
      uint32_t top = apro_unit<T, ROT>(p, row0 + ur, first + chunk, tile, stride, ur, chunk * (kChunk / 8), xpose, cs);
#pragma unroll
      for (int off = 1; off <= 4; off <<= 1) top = Pack16<T>::max2(top, __shfl_xor_sync(0xffffffffu, top, off));
      if ((lane & 7) == 0) {
        atomicMax(&s_top[ur + (lane >> 3)], __float_as_int(apro_wide_max<T>(top)));   // values are not negative
        if (apro_top(top) > Pack16<T>::kInf) s_nan[ur + (lane >> 3)] = s_nan[16] = 1;
      }
    }
  }
  __syncthreads();
  if (s_nan[16] != 0) {                                // a NaN in a token: its maximum is that of its other values
    for (int r = warp; r < p.rows; r += warps) {
      if (s_nan[r] == 0) continue;
      const float mx = apro_row_number_max<T>(tile + r * stride, r, own * (kChunk / 8));
      if (lane == 0) s_top[r] = __float_as_int(mx);
    }
    __syncthreads();
  }
  if (p.split > 1) {
    cluster_wait_acquire();
    for (int i = threadIdx.x; i < 16 * p.split; i += blockDim.x)
      st_cluster_f32(cluster_map(smem_addr(&s_peer[rank][i & 15]), i >> 4), __int_as_float(s_top[i & 15]));
    cluster_arrive_release();
    cluster_wait_acquire();
  }
  if (threadIdx.x < p.rows) {
    float mx = __int_as_float(s_top[threadIdx.x]);
    if (p.split > 1)
      for (int q = 0; q < p.split; ++q) mx = fmaxf(mx, __int_as_float(s_peer[q][threadIdx.x]));
    const float s0 = SCALE16 ? to_float<T>(from_float<T>(__fdiv_rn(mx, 127.0f))) : __fdiv_rn(fmaxf(mx, 1e-8f), 127.0f);
    const float sc = SCALE16 ? (s0 > 0.f ? s0 : 1.f) : fmaxf(s0, 1e-8f);
    const float rcp = __frcp_rn(sc);
    s_scale[threadIdx.x] = make_float4(sc, rcp, sc < 1e-30f || !(mx * rcp < 127.4f) || s_nan[threadIdx.x] != 0 ? 1.f : 0.f, 0.f);
    if (rank == 0 && row0 + (int)threadIdx.x < p.m) p.scales[row0 + threadIdx.x] = s0;
  }
  __syncthreads();
  // quantise: a warp takes 32 runs of 16 features of one token at a time
  const int runs = (k1 - k0) / 16, strips = (runs + 31) / 32;
  int r = 0, strip = warp;
  while (strip >= strips) { strip -= strips; ++r; }
  while (r < p.rows && row0 + r < p.m) {
    const int run = strip * 32 + lane;
    if (run < runs) {
      const float4 sc = s_scale[r];
      const uint4 a = *reinterpret_cast<const uint4*>(tile + r * stride + chunk_at(r, 2 * run) * 16);
      const uint4 b = *reinterpret_cast<const uint4*>(tile + r * stride + chunk_at(r, 2 * run + 1) * 16);
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      *reinterpret_cast<uint4*>(p.codes + (size_t)(row0 + r) * p.k + k0 + run * 16) = quantise16<T, 0>(w, sc.x, sc.y, sc.z != 0.f);
    }
    strip += warps;
    while (strip >= strips) { strip -= strips; ++r; }
  }
  if (p.down != nullptr) {
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    apro_down<T>(p, tile, stride, k0, warp, warps, (k1 - k0) / 32, acc);
    __syncthreads();                                  // the tile is read: its space holds the partial sums
    apro_store_down<T>(p, reinterpret_cast<float*>(smem), reinterpret_cast<float*>(smem + p.gather_off), acc, row0, rank);
  }
}

// int4, one scale per token and 64 features, sign-magnitude bytes, scales tile-major (mode 6 of rotate_quant.cu)
template <typename T, int ROT>
__global__ void __launch_bounds__(apro::kMaxWarps * 32, 3)
act_prologue_i4_kernel(const ProloguePar p) {
  using namespace apro;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float cs[kChunk];
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int stride = kChunk * 2;
  int rank, first, last;
  apro_share(p, rank, first, last);
  unsigned char* tile = smem + warp * (p.rows * stride + kXposeBytes);
  float* xpose = reinterpret_cast<float*>(tile + p.rows * stride);
  const int row0 = (int)(blockIdx.x / p.split) * p.rows, groups = p.k / 64;
  if (p.split > 1) cluster_arrive_relaxed();
  if (p.factors_ready) apro_column_scale<ROT>(p, cs);
  __syncthreads();
  grid_dependency_wait();
  grid_launch_dependents();
  if (ROT != 0 && !p.factors_ready) {
    apro_column_scale<ROT>(p, cs);
    __syncthreads();
  }
  float acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  for (int chunk = first + warp; chunk < last; chunk += warps) {
    for (int ur = 0; ur < p.rows && row0 + ur < p.m; ur += kUnitRows) {
      __syncwarp();
      apro_unit<T, ROT>(p, row0 + ur, chunk, tile, stride, ur, 0, xpose, cs);
    }
    __syncwarp();
    // two tokens at a time: lane = 16 hh + l holds features 16 l .. + 15 of token 2 i + hh
    const int hh = lane >> 4, l = lane & 15, f0 = chunk * kChunk + 16 * l;
    const bool inside = f0 < p.k;
    for (int i = 0; i < p.rows / 2 && row0 + 2 * i < p.m; ++i) {
      const int r = 2 * i + hh, row = row0 + r;
      const uint4 a = *reinterpret_cast<const uint4*>(tile + r * stride + chunk_at(r, 2 * l) * 16);
      const uint4 b = *reinterpret_cast<const uint4*>(tile + r * stride + chunk_at(r, 2 * l + 1) * 16);
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      uint32_t top = 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) top = Pack16<T>::max2(top, w[j] & 0x7fff7fffu);
      top = Pack16<T>::max2(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = Pack16<T>::max2(top, __shfl_xor_sync(0xffffffffu, top, 2));
      const float mx = apro_wide_max<T>(top), by7 = mx * kSeventh;
      float sc = fmaxf(fmaf(fmaf(-7.0f, by7, mx), kSeventh, by7), 1e-6f);            // mx / 7, see apro_div2
      const bool odd = apro_top(top) >= Pack16<T>::kInf;                             // infinity or NaN in the group
      if (__any_sync(0xffffffffu, odd)) {
        float number = apro_number_max<T>(w, 0.f);
        number = fmaxf(number, __shfl_xor_sync(0xffffffffu, number, 1));
        number = fmaxf(number, __shfl_xor_sync(0xffffffffu, number, 2));
        if (odd) sc = fmaxf(__fdiv_rn(number, 7.0f), 1e-6f);
      }
      if (inside && row < p.m) {
        if ((l & 3) == 0) p.scales[((size_t)(row >> 7) * groups + f0 / 64) * 128 + (row & 127)] = sc;
        *reinterpret_cast<uint4*>(p.codes + (size_t)row * p.k + f0) = quantise16<T, 1>(w, sc, __frcp_rn(sc), odd);
      }
    }
    if (p.down != nullptr) apro_down<T>(p, tile, stride, chunk * kChunk, 0, 1, min(kChunk, p.k - chunk * kChunk) / 32, acc);
  }
  if (p.split > 1) cluster_wait_acquire();
  if (p.down != nullptr) {
    __syncthreads();
    apro_store_down<T>(p, reinterpret_cast<float*>(smem), reinterpret_cast<float*>(smem + p.gather_off), acc, row0, rank);
  }
}

// ----------------------------------------------------------------------------------------- host

// Modes 8, 9 (int8 per token) and 6 (int4 per 64 features) of rotate_quant.cu; rot_kind / rot_block as there.
bool act_prologue_supported(int k, int rot_kind, int rot_block, int mode) {
  using namespace apro;
  if (k <= 0 || k % 16 != 0 || (mode != 6 && mode != 8 && mode != 9) || (mode == 6 && k % 64 != 0)) return false;
  if (rot_kind != 0 && (rot_kind < 0 || rot_kind > 2 || rot_block < 16 || rot_block > kChunk || kChunk % rot_block != 0 || k % rot_block != 0)) return false;
  if (rot_kind == 1 && rot_block != 16 && rot_block != 64 && rot_block != 256) return false;
  // int8: four tokens over the largest cluster, beside the warps' transposition buffers
  return mode == 6 || (size_t)kUnitRows * ceil_div(ceil_div(k, kChunk), kMaxSplit) * kChunk * 2 + kMaxWarps * kXposeBytes <= (size_t)kSmemMost;
}

template <void (*Kern)(const ProloguePar)>
static int apro_launch(const ProloguePar& p, int warps, size_t smem, cudaStream_t stream) {
  XQT_SMEM_OPT_IN(Kern, apro::kSmemOptIn);
  return launch_pdl_cluster(Kern, dim3((unsigned)(ceil_div(p.m, p.rows) * p.split)), dim3((unsigned)warps * 32), p.split, smem, stream, p);
}

// Tokens per CTA and CTAs per token.  Without a low-rank branch 4 tokens, whole unless a warp would get more than four
// units.  With one: the fewest tokens that still give no more than one CTA row per SM (the down matrix is read once per CTA
// row), at most 16, and then features split until there are two CTAs per SM or a warp has one chunk.
static void pick_split(ProloguePar& p) {
  using namespace apro;
  const int sms = sm_count();
  p.rows = p.down == nullptr || p.m <= 4 * sms ? 4 : (p.m <= 8 * sms ? 8 : 16);
  p.split = 1;
  auto more = [&] { return p.split < kMaxSplit && 2 * p.split <= p.chunks; };
  if (p.down == nullptr) {
    while (more() && ceil_div(p.chunks, p.split) > 4 * kMaxWarps) p.split *= 2;
  } else {
    while (more() && (ceil_div(p.chunks, p.split) > kMaxWarps || (ceil_div(p.m, p.rows) * p.split < 2 * sms && ceil_div(p.chunks, p.split) > 1)))
      p.split *= 2;
  }
}

template <typename T>
static int apro_dispatch(ProloguePar p, int rot_kind, int mode, cudaStream_t stream) {
  using namespace apro;
  p.chunks = ceil_div(p.k, kChunk);
  pick_split(p);
  // the warps' partial sums take the place of the tiles; other CTAs of the cluster may write to `gather` while this one
  // still reads its tiles
  auto with_down = [&](size_t tiles, int warps) {
    const size_t part = (size_t)warps * 16 * kRedStride * 4;
    p.gather_off = (int)((tiles > part || p.down == nullptr ? tiles : part) + 15) & ~15;
    return p.down == nullptr ? tiles : (size_t)p.gather_off + (size_t)p.split * 2048;
  };
  if (mode == 6) {
    const int own = ceil_div(p.chunks, p.split), warps = ceil_div(own, ceil_div(own, kMaxWarps));
    const size_t smem = with_down((size_t)warps * (p.rows * kChunk * 2 + kXposeBytes), warps);
    if (rot_kind == 0) return apro_launch<act_prologue_i4_kernel<T, 0>>(p, warps, smem, stream);
    if (rot_kind == 1) return apro_launch<act_prologue_i4_kernel<T, 1>>(p, warps, smem, stream);
    return apro_launch<act_prologue_i4_kernel<T, 2>>(p, warps, smem, stream);
  }
  auto bytes = [&] { return (size_t)p.rows * ceil_div(p.chunks, p.split) * kChunk * 2 + (rot_kind == 0 ? 0 : (size_t)kMaxWarps * kXposeBytes); };
  while (bytes() > (size_t)kSmemMost && p.split < kMaxSplit && 2 * p.split <= p.chunks) p.split *= 2;
  while (bytes() > (size_t)kSmemMost && p.rows > 4) p.rows /= 2;
  const int units = (p.rows / kUnitRows) * ceil_div(p.chunks, p.split), warps = units < kMaxWarps ? units : kMaxWarps;
  const size_t smem = with_down(bytes(), warps);
#define XQT_APRO_I8(ROT) (mode == 9 ? apro_launch<act_prologue_i8_kernel<T, ROT, true>>(p, warps, smem, stream) \
                                    : apro_launch<act_prologue_i8_kernel<T, ROT, false>>(p, warps, smem, stream))
  if (rot_kind == 0) return XQT_APRO_I8(0);
  return rot_kind == 1 ? XQT_APRO_I8(1) : XQT_APRO_I8(2);
#undef XQT_APRO_I8
}

int act_prologue_launch(const void* x, const float* column_scale, void* codes, float* scales, const void* down, void* la, float lora_scale,
                        int m, int k, int rot_kind, int rot_block, int mode, int la_form, int act_dtype, cudaStream_t stream) {
  const int factors_ready = (rot_kind & XQT_B200_ROT_FACTORS_READY) != 0;
  rot_kind &= ~XQT_B200_ROT_FACTORS_READY;
  XQT_REQUIRE(m > 0 && act_prologue_supported(k, rot_kind, rot_block, mode) && la_form >= 0 && la_form <= 3);
  XQT_REQUIRE(down == nullptr || k % 32 == 0);
  XQT_REQUIRE((down != nullptr) == (la_form != 0) && (down == nullptr || la != nullptr) && (rot_kind == 0 || column_scale != nullptr));
  XQT_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)codes & 15) == 0 && ((uintptr_t)down & 15) == 0 && ((uintptr_t)la & 15) == 0);
  ProloguePar p{};
  p.factors_ready = factors_ready;
  p.x = x; p.column_scale = column_scale; p.codes = (int8_t*)codes; p.scales = scales; p.down = down; p.la = la;
  p.lora_scale = lora_scale; p.la_form = la_form; p.m = m; p.k = k; p.rot_block = rot_block;
  if (act_dtype == XQT_B200_BF16) return apro_dispatch<__nv_bfloat16>(p, rot_kind, mode, stream);
  XQT_REQUIRE(act_dtype == XQT_B200_FP16);
  return apro_dispatch<__half>(p, rot_kind, mode, stream);
}

}  // namespace xqt_b200
