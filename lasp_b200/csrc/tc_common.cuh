// Device helpers shared by the tensor-core kernels: bounded waits that report
// through the fault word, accumulator <-> shared-memory moves with the decay
// mask, and the enumeration of the tiles a persistent CTA walks over.
#pragma once
#include "common.cuh"
#include "sm100.cuh"
#include "span_cut.h"

namespace lasp {
namespace tc {

using namespace sm100;

constexpr int C = kTensorTile;  // 128 tokens per tile
constexpr float kLog2e = 1.4426950408889634f;

// Whether a wait of the CTA has run out (in shared memory).  With a link (LINK) some of its warps may also be waiting for
// another rank, for as long as the hand-over's own limit says; the time of the other warps' waits stands still meanwhile.
template <bool LINK>
struct Health {
  enum { kWell = 0, kGaveUp = 1, kAwaitsPeer = 2 };
  int word;
  __device__ __forceinline__ bool gave_up() const { return *const_cast<const volatile int*>(&word) == kGaveUp; }
  __device__ __forceinline__ void give_up() { *const_cast<volatile int*>(&word) = kGaveUp; }
  __device__ __forceinline__ void peer_wait_begins() { atomicCAS(&word, kWell, kAwaitsPeer); }
  __device__ __forceinline__ void peer_wait_ends() { atomicCAS(&word, kAwaitsPeer, kWell); }
};

// Bounded wait that records a fault once and lets later waits of the CTA give up at once.  There are some thirty of
// these in a walk kernel: the code that a wait normally runs is one probe, and 32-bit clocks keep the rest short.
template <bool LINK>
__device__ __forceinline__ void wait_or_fault(uint64_t* bar, uint32_t parity, Health<LINK>* cta, int32_t* fault, int32_t code) {
  if (mbar_try_wait(bar, parity)) return;
  uint32_t t0 = clock();
  while (!mbar_try_wait(bar, parity)) {
    const int state = *const_cast<const volatile int*>(&cta->word);
    if (state == Health<LINK>::kGaveUp) return;
    if (LINK && state == Health<LINK>::kAwaitsPeer) t0 = clock();
    if ((uint32_t)clock() - t0 > kWaitClocks) {
      cta->give_up();
      atomicOr(fault, code);
      return;
    }
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

__device__ __forceinline__ float decay_pow(float sl2, int k) { return exp2f(-sl2 * (float)k); }

// Tiles that a decay rate s reaches over: a token s * tokens >= 27.6 away has a weight below 1e-12 (exchange_layout.h
// draws the same line between ranks).  At least one; no limit without decay.  The line does not look at magnitudes: what
// it leaves out of a state is at most 1e-12 of what the same token contributes at its own place, far below the rounding
// of an fp32 sum that holds both, but not of one that holds only tokens 1e9 times smaller.  (Summing on to the smallest
// normal number, s * tokens = 87.4: forward / dK,dV 16 x 131072 500 -> 560 / 734 -> 780 us, 36 x 3001 36.8 -> 37.7 /
// 46.9 -> 48.0, 24 x 2048 23.5 -> 24.7 / 29.1 -> 29.9.)
__device__ __forceinline__ int reach_tiles(float s) {
  const float r = 27.6f / (s * (float)C);
  return s > 0.f && r < 1e6f ? (int)r + 1 : 1 << 20;
}

// Arithmetic on pairs: one instruction for two fp32 values (packed operations of this architecture), and a product of
// bf16 pairs with an fp32 factor f in two instead of the five of unpacking, multiplying and packing again:
// f = hi + lo in bf16, x f = fma(x, hi, x lo), rounded once but for the 2^-18 that x lo loses.
struct F2 {
  float x, y;
};
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\t"
      "mov.b64 {%0, %1}, d;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ F2 pair(uint32_t a, uint32_t b) { return {__uint_as_float(a), __uint_as_float(b)}; }
struct SplitFactor {
  __nv_bfloat162 hi, lo;
};
__device__ __forceinline__ SplitFactor split_factor(float f) {
  const __nv_bfloat16 h = __float2bfloat16_rn(f);
  return {__bfloat162bfloat162(h), __float2bfloat162_rn(f - __bfloat162float(h))};
}
__device__ __forceinline__ uint32_t scale_bf16x2(uint32_t u, const SplitFactor& f) {
  const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&u);
  const __nv_bfloat162 r = __hfma2(x, f.hi, __hmul2(x, f.lo));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// acc (32 columns) *= f, in tensor memory
__device__ __forceinline__ void scale_tmem32(uint32_t taddr, float f) {
  uint32_t r[32];
  tmem_ld32(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const F2 v = mul2(pair(r[j], r[j + 1]), {f, f});
    r[j] = __float_as_uint(v.x), r[j + 1] = __float_as_uint(v.y);
  }
  tmem_st32(taddr, r);
}

// tile[row][col0 .. col0+31] = bf16(acc) into a swizzled staging tile of C rows; a TMA store then moves the tile out
__device__ __forceinline__ void stage_row32(uint32_t taddr, uint8_t* tile, int row, int col0) {
  uint32_t a[32];
  tmem_ld32(taddr, a);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    uint4 v = make_uint4(pack_bf16(__uint_as_float(a[j]), __uint_as_float(a[j + 1])),
                         pack_bf16(__uint_as_float(a[j + 2]), __uint_as_float(a[j + 3])),
                         pack_bf16(__uint_as_float(a[j + 4]), __uint_as_float(a[j + 5])),
                         pack_bf16(__uint_as_float(a[j + 6]), __uint_as_float(a[j + 7])));
    *reinterpret_cast<uint4*>(tile + tile_offset(row, col0 + j, C)) = v;
  }
}

// Four 16-byte pieces of a row in each of four neighbouring lanes change hands so that piece i of every lane belongs to the
// i-th of the four rows: stored piece by piece, four lanes then write 64 bytes of one row.  (As they are, the 32 lanes of a
// store write 16 bytes of 32 rows, a cache line each: 64 KB of results took the load-store unit 5600 clocks, in which the
// filling warps' loads stood still too.)
__device__ __forceinline__ void rows_to_lanes(uint4 (&v)[4], int lane) {
#pragma unroll
  for (int s = 1; s <= 2; s *= 2) {
    const bool high = lane & s;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = s == 1 ? 2 * u : u, j = i + s;   // the pair of pieces of which this lane keeps one and sends the other
      uint32_t* a = reinterpret_cast<uint32_t*>(&v[i]);
      uint32_t* b = reinterpret_cast<uint32_t*>(&v[j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, high ? a[q] : b[q], s);
        (high ? a[q] : b[q]) = got;
      }
    }
  }
}

// Decay mask.  32 fp32 accumulator columns at `src` (columns col0 .. col0+31 of a score tile, this thread's lane = row)
// become 16 columns of masked bf16 pairs, which the caller leaves in tensor memory as the A operand of the next MMA.
// Per group of eight columns the factor is built from the group's live column nearest the diagonal away from it by
// repeated multiplication with lambda (short independent chains), so it can only underflow towards the far columns.
// `pre` multiplies every element (the folded q,k scale).
// TRANSPOSED = false: lane = query row r, column = key c:  [r >= c] lambda^(r-c)
// TRANSPOSED = true : lane = key c, column = query row r:  [r >= c] lambda^(r-c)   (the tile is S^T)
template <bool TRANSPOSED>
__device__ __forceinline__ void masked_pack32(uint32_t src, int row, int col0, float sl2, float lam,
                                              uint32_t (&out)[16], float pre = 1.f) {
  const int row0 = row & ~31;
  const bool none = TRANSPOSED ? (col0 + 31 < row0) : (col0 > row0 + 31);   // same for every lane of the warp
  if (none) {
#pragma unroll
    for (int j = 0; j < 16; ++j) out[j] = 0u;
    return;
  }
  uint32_t r[32];
  tmem_ld32(src, r);
  float f[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    // the chain of a group of eight columns starts at its live column nearest the diagonal
    const int start = TRANSPOSED ? max(row, col0 + 8 * g) : min(row, col0 + 8 * g + 7);
    f[g] = pre * decay_pow(sl2, TRANSPOSED ? start - row : row - start);
  }
  tmem_ld_wait();
  if (TRANSPOSED ? (col0 >= row0 + 31) : (col0 + 31 <= row0)) {   // the whole block is below the diagonal
    const F2 step = {lam * lam, lam * lam};   // a pair of columns further from it
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      F2 fac = TRANSPOSED ? F2{f[g], f[g] * lam} : F2{f[g] * lam, f[g]};   // of the group's nearest pair
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int j = TRANSPOSED ? jj : 3 - jj;
        const F2 m = mul2(pair(r[8 * g + 2 * j], r[8 * g + 2 * j + 1]), fac);
        out[4 * g + j] = pack_bf16(m.x, m.y);
        if (jj < 3) fac = mul2(fac, step);
      }
    }
    return;
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float m[8];
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      const int j = TRANSPOSED ? jj : 7 - jj;           // away from the diagonal
      const int col = col0 + 8 * g + j;
      const bool live = TRANSPOSED ? col >= row : col <= row;
      m[j] = live ? __uint_as_float(r[8 * g + j]) * f[g] : 0.f;
      f[g] = live ? f[g] * lam : f[g];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) out[4 * g + j] = pack_bf16(m[2 * j], m[2 * j + 1]);
  }
}

// exp of a pair of bf16 values: the argument is scaled in fp32, the exponential itself is ONE special-function
// operation for the pair (the map passes are bound by that unit)
__device__ __forceinline__ __nv_bfloat162 exp_bf16x2(uint32_t u) {
  const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
  const uint32_t t = pack_bf16(f.x * kLog2e, f.y * kLog2e);
  uint32_t r;
  asm("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(r) : "r"(t));
  return *reinterpret_cast<__nv_bfloat162*>(&r);
}
// elu(x) + 1 on a pair of bf16 values (the feature map of the no-decay linear-transformer configuration):
// x + 1 for x > 0, exp(x) otherwise = max(x, 0) + min(exp(x), 1), without a branch
__device__ __forceinline__ uint32_t elu1_bf16x2(uint32_t u) {
  const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&u);
  const __nv_bfloat162 r = __hadd2(__hmax2(x, __float2bfloat162_rn(0.f)), __hmin2(exp_bf16x2(u), __float2bfloat162_rn(1.f)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// its derivative: 1 for x > 0, exp(x) otherwise = min(exp(x), 1) = min(elu(x) + 1, 1): from x, or from what the map gave
// (MAPPED)
template <bool MAPPED>
__device__ __forceinline__ float2 elu1_slope_bf16x2(uint32_t u) {
  const __nv_bfloat162 y = MAPPED ? *reinterpret_cast<const __nv_bfloat162*>(&u) : exp_bf16x2(u);
  return __bfloat1622float2(__hmin2(y, __float2bfloat162_rn(1.f)));
}

// Multiplies CHUNKS 16-byte pieces of row `row` of a swizzled tile of C rows by w, in place, starting
// at piece `first` (pieces are counted slab by slab; a row keeps its pieces under the swizzle, so the
// physical position inside the row does not matter).  `lane` rotates the order to spread the banks.
// MAP: each element goes through elu(x) + 1 first.
template <int CHUNKS, bool MAP = false>
__device__ __forceinline__ void scale_row_pieces(uint8_t* tile, int row, int first, float w, int lane) {
  static_assert((CHUNKS & (CHUNKS - 1)) == 0, "a power of two");
  const SplitFactor f = split_factor(w);
  uint4 v[CHUNKS];
  uint4* p[CHUNKS];
#pragma unroll
  for (int q = 0; q < CHUNKS; ++q) {   // all loads first: their latencies overlap
    const int piece = first + ((q + lane) & (CHUNKS - 1));
    p[q] = reinterpret_cast<uint4*>(tile + (piece >> 3) * C * 128 + row * 128 + (piece & 7) * 16);
    v[q] = *p[q];
  }
#pragma unroll
  for (int q = 0; q < CHUNKS; ++q) {
    uint32_t* u = reinterpret_cast<uint32_t*>(&v[q]);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (MAP) u[t] = elu1_bf16x2(u[t]);
      if (!MAP || w != 1.f) u[t] = scale_bf16x2(u[t], f);
    }
    *p[q] = v[q];
  }
}

// dst row = w * src row, the same pieces of two tiles of C rows
template <int CHUNKS>
__device__ __forceinline__ void copy_row_pieces(uint8_t* dst, const uint8_t* src, int row, int first, float w, int lane) {
  const SplitFactor f = split_factor(w);
  uint4 v[CHUNKS];
#pragma unroll
  for (int q = 0; q < CHUNKS; ++q) {
    const int piece = first + ((q + lane) & (CHUNKS - 1));
    v[q] = *reinterpret_cast<const uint4*>(src + (piece >> 3) * C * 128 + row * 128 + (piece & 7) * 16);
  }
#pragma unroll
  for (int q = 0; q < CHUNKS; ++q) {
    const int piece = first + ((q + lane) & (CHUNKS - 1));
    uint32_t* u = reinterpret_cast<uint32_t*>(&v[q]);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      u[t] = scale_bf16x2(u[t], f);
    }
    *reinterpret_cast<uint4*>(dst + (piece >> 3) * C * 128 + row * 128 + (piece & 7) * 16) = v[q];
  }
}

// stage_row32 with the chain rule of the folded q,k preprocessing x' = c * map(x): the 32 accumulator values
// (a gradient with respect to x') are multiplied by c * map'(x) on their way to the staging tile.  x, or with MAPPED
// map(x), comes from the q or k that the launch was given (`raw` points at column 0 of this thread's row): raw_row32, which the caller issues ahead of its wait for the
// accumulator, because these loads go through L2 (with the loads behind the wait a dQ walk over 64-wide heads took 86 us - now 79 -
// for 4 x 16 x 4096 tokens, against 35 us without a map).
__device__ __forceinline__ void raw_row32(uint4 (&x)[4], const __nv_bfloat16* raw, int col0) {
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = __ldg(reinterpret_cast<const uint4*>(raw + col0) + j);
}
template <bool MAPPED>
__device__ __forceinline__ void stage_row32_chain(uint32_t taddr, uint8_t* tile, int row, int col0,
                                                  const uint4 (&x)[4], float c, bool elu) {
  uint32_t a[32];
  tmem_ld32(taddr, a);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float m[8];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float sx = c, sy = c;
      if (elu) {
        const float2 sl = elu1_slope_bf16x2<MAPPED>(reinterpret_cast<const uint32_t*>(&x[j])[t]);
        sx *= sl.x, sy *= sl.y;
      }
      m[2 * t] = __uint_as_float(a[8 * j + 2 * t]) * sx;
      m[2 * t + 1] = __uint_as_float(a[8 * j + 2 * t + 1]) * sy;
    }
    *reinterpret_cast<uint4*>(tile + tile_offset(row, col0 + 8 * j, C)) =
        make_uint4(pack_bf16(m[0], m[1]), pack_bf16(m[2], m[3]), pack_bf16(m[4], m[5]), pack_bf16(m[6], m[7]));
  }
}

// The work of a persistent CTA (span_cut.h): items blockIdx.x, + gridDim.x, ..., walked first to last tile or last to
// first.
template <bool BACKWARDS>
struct TileWalk {
  const SpanCut& c;
  bool even;
  int it, bh, sp, t, t0, t1;  // current item, its sequence and span, current tile, the item's tile range [t0, t1)

  __device__ __forceinline__ int span_t0(int s) const { return span_first_tile<BACKWARDS>(c, even, s); }
  __device__ __forceinline__ bool load() {
    if (it >= c.items) return false;
    bh = sequence_of_item(c, it);
    sp = span_of_place<BACKWARDS>(c, even, it - bh * c.nspans);
    t0 = span_t0(sp);
    t1 = span_t0(sp + 1);
    t = BACKWARDS ? t1 - 1 : t0;
    return true;
  }
  __device__ __forceinline__ bool start() {
    it = blockIdx.x;
    return load();
  }
  __device__ __forceinline__ bool next() {
    if (BACKWARDS ? (--t >= t0) : (++t < t1)) return true;
    it += gridDim.x;
    return load();
  }
  __device__ __forceinline__ bool first_of_item() const { return BACKWARDS ? t == t1 - 1 : t == t0; }
  __device__ __forceinline__ bool last_of_item() const { return BACKWARDS ? t == t0 : t == t1 - 1; }
};

}  // namespace tc
}  // namespace lasp
