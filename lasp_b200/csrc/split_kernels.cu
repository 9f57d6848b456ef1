// Full-precision path: fp32 and fp16 tensors, and bf16 shapes the walk kernels do not take (head widths other than
// 64 and 128, sequences shorter than a tile), on the tensor cores without giving up fp32 arithmetic.
//
// An fp32 number is the exact sum of three bf16 numbers (24 bits = 8 + 8 + 8), an fp16 number of two, so a product
// of fp32 matrices is a sum of products of bf16 matrices accumulated in fp32.  (From 2^-110 on: of smaller numbers the
// last term falls below bf16's smallest, 2^-133, which is then the absolute error.  Not from bf16's largest, 3.39e38, on:
// see "outside the terms' range" below.)  Of the nine products of two three-term operands the six with i + j <= 2 are
// kept: what is left out is below 2^-24 of a factor, the rounding of an fp32 product (the method of Henry, Tang and
// Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019).  Small products go first, so that the few additions at full magnitude
// come last.  Inputs in 16-bit types need fewer terms: they are exact in two (fp16) or one (bf16), and the scores, whose
// operands are both inputs, come from fp16 tiles as they are, one exact product.  What is computed on the way - masked
// scores, states, decayed rows - has three terms, 24 bits, for all types.  (With two there, 17 bits, and the scores from
// two terms of fp16 operands, a tenth faster, the rank states of fp16 and bf16 tensors were 3.7e-6 and 2.4e-6 off instead
// of 1.5e-7, and the rounded fp16 results' error against fp64 was larger by 3e-4 of itself.)
//
// Sequences are cut into 128-token chunks (the last one ragged), everything in parallel over chunks:
//   k_split_states  T = sum_c w_c a_c b_c^T of every chunk                       (a,b = k,v or q,do)
//   k_scan          the states at the chunk borders
//   k_split_out     OUT = (X Y^T . M) Z + diag(w) X op(P)
// k_split_out is all of the output kernels: (X,Y,Z,op(P)) = (Q,K,V,P) gives O, (dO,V,K,P^T) dQ, (V,dO,Q,Dn^T) dK and
// (K,Q,dO,Dn) dV, the last two with the mask transposed; the backward pass runs the three as one launch.  Computing
// the scores once per result costs one product in nine and makes every chunk three independent tasks.
//
// One B200, b=2, h=12, n=2048, forward / backward, before (a CTA of 256 FFMA threads per 64-token chunk) and now:
// fp32 d=e=128 730 / 1421 -> 82 / 154 us, fp16 d=128, e=64 365 / 869 -> 48 / 86 us, bf16 d=e=96 363 / 920 -> 44 / 79 us;
// the error against fp64, relative to theirs: fp16 and bf16 results 1.00, rank states of all types 0.5 to 0.97, fp32 results
// 0.65 to 0.97 of 1.3e-7 to 3.2e-7, but for o and dv without decay beyond a chunk, 1.0 to 1.18 of 1.3e-7 to 1.8e-7 (sums
// of numbers of one sign, which the tensor cores' accumulation rounds towards zero; the same calls' dq and dk: 0.8).
#include <type_traits>

#include "tc_common.cuh"

namespace lasp {
namespace {

using namespace tc;

constexpr int NT = 512;           // sixteen worker warps, one of whose threads issues the MMAs
constexpr int kPieces = 4;        // 8-element pieces of a 128 x 128 tile per thread

// terms of the inputs and of intermediate quantities, and the largest i + j of a product that is kept
template <typename T> struct Terms;
template <> struct Terms<float> { static constexpr int in = 3, mid = 3, cut = 2; };
template <> struct Terms<__half> { static constexpr int in = 2, mid = 3, cut = 2; };
template <> struct Terms<__nv_bfloat16> { static constexpr int in = 1, mid = 3, cut = 2; };

// eight elements of a row as they come from global memory
template <typename T> struct Raw { uint4 v; };
template <> struct Raw<float> { uint4 v, w; };

template <typename T> __device__ __forceinline__ void zero_raw(Raw<T>& r) { r.v = make_uint4(0u, 0u, 0u, 0u); }
template <> __device__ __forceinline__ void zero_raw<float>(Raw<float>& r) { r.v = r.w = make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ uint4 ld_nc(const void* p) { return __ldg(static_cast<const uint4*>(p)); }
template <typename T> __device__ __forceinline__ void load_piece(Raw<T>& r, const T* p) { r.v = ld_nc(p); }
template <> __device__ __forceinline__ void load_piece<float>(Raw<float>& r, const float* p) {
  r.v = ld_nc(p), r.w = ld_nc(p + 4);
}
template <typename T> __device__ __forceinline__ void to_floats(const Raw<T>& r, float (&x)[8]);
template <> __device__ __forceinline__ void to_floats<float>(const Raw<float>& r, float (&x)[8]) {
  const uint32_t u[8] = {r.v.x, r.v.y, r.v.z, r.v.w, r.w.x, r.w.y, r.w.z, r.w.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(u[j]);
}
template <> __device__ __forceinline__ void to_floats<__half>(const Raw<__half>& r, float (&x)[8]) {
  const uint32_t u[4] = {r.v.x, r.v.y, r.v.z, r.v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[j]));
    x[2 * j] = f.x, x[2 * j + 1] = f.y;
  }
}
template <> __device__ __forceinline__ void to_floats<__nv_bfloat16>(const Raw<__nv_bfloat16>& r, float (&x)[8]) {
  const uint32_t u[4] = {r.v.x, r.v.y, r.v.z, r.v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) x[2 * j] = __uint_as_float(u[j] << 16), x[2 * j + 1] = __uint_as_float(u[j] & 0xFFFF0000u);
}

// x0, x1 -> N bf16 pairs whose sum is the pair (N = 3: exactly; the last term of N = 2 is rounded): round, take the
// remainder, which is exact, and so on - nine instructions for three terms of a pair
template <int N>
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t (&t)[N]) {
  F2 x = {x0, x1};
#pragma unroll
  for (int i = 0; i < N; ++i) {
    t[i] = pack_bf16(x.x, x.y);
    if (i + 1 < N) x = fma2({__uint_as_float(t[i] << 16), __uint_as_float(t[i] & 0xFFFF0000u)}, {-1.f, -1.f}, x);
  }
}

// the terms of eight elements of row `row` from column `col` on, into the operand tiles (one per term,
// `stride` bytes apart, `rows` rows each)
template <int N>
__device__ __forceinline__ void store_terms(uint8_t* tiles, uint32_t stride, int row, int col, int rows, const float (&x)[8]) {
  uint32_t t[4][N];
#pragma unroll
  for (int j = 0; j < 4; ++j) split_pair<N>(x[2 * j], x[2 * j + 1], t[j]);
  const uint32_t off = tile_offset(row, col, rows);
#pragma unroll
  for (int i = 0; i < N; ++i)
    *reinterpret_cast<uint4*>(tiles + i * stride + off) = make_uint4(t[0][i], t[1][i], t[2][i], t[3][i]);
}

__device__ __forceinline__ int padded(int w) { return w <= 64 ? 64 : 128; }

// A 128 x wp tile (wp = 64 or 128; rows >= len and columns >= w read as zero): piece p of the tile is row p / (wp/8),
// columns 8 (p mod wp/8) on, so that a warp reads whole rows and its shared-memory stores hit every bank once.
template <typename T>
__device__ __forceinline__ void load_tile(Raw<T> (&r)[kPieces], const T* base, int pitch, int len, int w, int wp, int tid) {
  const int sh = wp == 128 ? 4 : 3;
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int p = tid + NT * i, row = p >> sh, col = (p & ((1 << sh) - 1)) * 8;
    zero_raw<T>(r[i]);
    if (row < len && col < w) load_piece<T>(r[i], base + (size_t)row * pitch + col);
  }
}
// ... its terms in shared memory, row `row` multiplied by wt(row) first
template <typename T, int N, bool WEIGHTED, typename W>
__device__ __forceinline__ void store_tile(uint8_t* tiles, const Raw<T> (&r)[kPieces], int wp, int tid, W wt) {
  const int sh = wp == 128 ? 4 : 3;
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int p = tid + NT * i, row = p >> sh, col = (p & ((1 << sh) - 1)) * 8;
    if (row >= C) break;
    if constexpr (N == 1 && !WEIGHTED) {
      *reinterpret_cast<uint4*>(tiles + tile_offset(row, col, C)) = r[i].v;   // bf16 is its own only term
    } else {
      float x[8];
      to_floats<T>(r[i], x);
      if constexpr (WEIGHTED) {
        const float f = wt(row);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] *= f;
      }
      store_terms<N>(tiles, C * wp * 2, row, col, C, x);
    }
  }
}
struct NoWeight {};
// ... as it is, a 16-bit type
template <typename T>
__device__ __forceinline__ void store_raw(uint8_t* tile, const Raw<T> (&r)[kPieces], int wp, int tid) {
  const int sh = wp == 128 ? 4 : 3;
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int p = tid + NT * i, row = p >> sh, col = (p & ((1 << sh) - 1)) * 8;
    if (row >= C) break;
    *reinterpret_cast<uint4*>(tile + tile_offset(row, col, C)) = r[i].v;
  }
}

// a d x e state in lane order (common.cuh), padded to dp x ep: piece p is row p mod dp, columns 8 (p / dp) on
__device__ __forceinline__ void load_state(Raw<float> (&r)[kPieces], const float* state, int d, int e, int dp, int ep, int tid) {
  const int sh = dp == 128 ? 7 : 6;
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int p = tid + NT * i, row = p & (dp - 1), g = p >> sh;   // columns 8 g .. 8 g + 7
    zero_raw<float>(r[i]);
    if (row < d && 8 * g < e) {
      const float4* src = reinterpret_cast<const float4*>(state) + (size_t)(2 * g) * d + row;
      r[i].v = ld_nc(src), r[i].w = ld_nc(src + d);
    }
  }
}
template <int N>
__device__ __forceinline__ void store_state_terms(uint8_t* tiles, const Raw<float> (&r)[kPieces], int dp, int ep, int tid) {
  const int sh = dp == 128 ? 7 : 6;
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int p = tid + NT * i, row = p & (dp - 1), g = p >> sh;
    if (8 * g >= ep) break;
    float x[8];
    to_floats<float>(r[i], x);
    store_terms<N>(tiles, dp * ep * 2, row, 8 * g, dp, x);
  }
}

// One operand of a product in shared memory: its terms lie `stride` bytes apart.
struct TermOperand {
  uint32_t addr, stride, rows;
  bool mn_major;
  __device__ __forceinline__ SmemDesc desc(int term) const { return operand_desc(addr + term * stride, rows, mn_major); }
};
// D[128 x n] = A B: every kept product of terms, the smallest first; issued by one thread
template <int NA, int NB, int CUT, bool FP16 = false>
__device__ __forceinline__ void issue_terms(uint32_t d_tmem, const TermOperand& a, const TermOperand& b, uint32_t n, int ksteps) {
  const uint32_t idesc = umma_idesc(128, n, a.mn_major, b.mn_major, FP16);
  uint32_t acc = 0;
#pragma unroll
  for (int sum = CUT; sum >= 0; --sum) {
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int j = sum - i;
      if (j < 0 || j >= NB) continue;
      const SmemDesc da = a.desc(i), db = b.desc(j);
#pragma unroll 1
      for (int kq = 0; kq < ksteps / 4; ++kq) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          umma(d_tmem, operand_step(da, a.rows, a.mn_major, 4 * kq + u), operand_step(db, b.rows, b.mn_major, 4 * kq + u), idesc, acc);
          acc = 1;
        }
      }
    }
  }
}
// the same with A's terms in tensor memory as mask_terms leaves them: K step ks of terms 0 and 1 in the 32-column block
// ks / 2 of t_s, of term 2 in t_lo
template <int NA, int NB, int CUT>
__device__ __forceinline__ void issue_terms_ts(uint32_t d_tmem, uint32_t t_s, uint32_t t_lo, const TermOperand& b, uint32_t n) {
  const uint32_t idesc = umma_idesc(128, n, false, b.mn_major);
  uint32_t acc = 0;
#pragma unroll
  for (int sum = CUT; sum >= 0; --sum) {
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int j = sum - i;
      if (j < 0 || j >= NB) continue;
      const SmemDesc db = b.desc(j);
#pragma unroll 1
      for (int kq = 0; kq < C / 64; ++kq) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int ks = 4 * kq + u;
          const uint32_t ta = i == 2 ? t_lo + 8 * ks : t_s + 32 * (ks >> 1) + 8 * (ks & 1) + 16 * i;
          umma_ts(d_tmem, ta, operand_step(db, b.rows, b.mn_major, ks), idesc, acc);
          acc = 1;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Outside the terms' range.  Infinities, and finite values above bf16's largest, have an infinite first term and a
// remainder that is NaN or infinite too, so that wherever one of them - an input, a state, a score - takes part, the
// products of terms give no finite number.  Results that are not finite are computed again in plain fp32 arithmetic from
// the tensors: infinities, large numbers and NaN come out as they do there, and reach the tokens that they do there.
// The kernels look at every 16 results at once and come back to those that need it where few registers are live: after
// all of a CTA's tasks, or, where results are added to what a tensor holds, at the end of the task.  (Calls inside the
// epilogue's loop cost fp32 outputs 5 to 12 % by the registers that they take; this way 1.8 %, fp16 nothing, bf16 1 %.)
// ---------------------------------------------------------------------------
// (by their sum: eight packed additions; one that overflows costs a look at results that are finite)
__device__ __forceinline__ bool all_finite(const uint32_t (&r)[16]) {
  F2 z = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 16; j += 2) z = fma2(pair(r[j], r[j + 1]), {1.f, 1.f}, z);
  return isfinite(z.x + z.y);
}
__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }

// ---------------------------------------------------------------------------
// chunk states: T[i][j] = sum_c w_c A[c][i] B[c][j], in lane order
//   forward : A = K, B = V,  w_c = lambda^(len-c);   backward: A = Q, B = dO, w_c = lambda^c
// A task per chunk, persistent CTAs; the next chunk's rows are on their way while the products of this one run.
// Bound by the loads' latency and the splitting arithmetic (one CTA per SM: 192 KB of operand terms for fp32).
// ---------------------------------------------------------------------------
struct StateArgs {
  const void *a, *b;
  const float* s;
  float* states;
  int h, n, nc, tasks, d, e, pitch_a, pitch_b, backward;
  int skip;   // chunk whose state nobody reads (-1: none)
  int32_t* fault;
};

// The elements of a task's state that are not finite, again
template <typename T>
__device__ __forceinline__ void plain_state(const StateArgs& g, int task) {
  const int bh = task / g.nc, chunk = task - bh * g.nc, len = min(C, g.n - chunk * C);
  const size_t tok = (size_t)bh * g.n + (size_t)chunk * C;
  const T *a = static_cast<const T*>(g.a) + tok * g.pitch_a, *b = static_cast<const T*>(g.b) + tok * g.pitch_b;
  const float sh = g.s[bh % g.h];
  float4* state = reinterpret_cast<float4*>(g.states + (size_t)task * g.d * g.e);
  for (int p = threadIdx.x; p < g.d * g.e / 4; p += NT) {   // four columns of a row, in lane order
    const int row = p % g.d, col = p / g.d * 4;
    const float4 old = state[p];
    if (isfinite(old.x + old.y + old.z + old.w)) continue;
    float y[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < len && !(isnan(y[0]) && isnan(y[1]) && isnan(y[2]) && isnan(y[3])); ++c) {
      const float x = to_float(a[(size_t)c * g.pitch_a + row]) * expf(-sh * (float)(g.backward ? c : len - c));
      for (int j = 0; j < 4; ++j) y[j] = fmaf(x, to_float(b[(size_t)c * g.pitch_b + col + j]), y[j]);
    }
    state[p] = make_float4(isfinite(old.x) ? old.x : y[0], isfinite(old.y) ? old.y : y[1], isfinite(old.z) ? old.z : y[2],
                           isfinite(old.w) ? old.w : y[3]);
  }
}

template <typename T>
__global__ void __launch_bounds__(NT, 1) k_split_states(const StateArgs g) {
  using TT = Terms<T>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t done;
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  __shared__ int look_again;   // a state with an element that is not finite has been written
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dp = padded(g.d), ep = padded(g.e);
  uint8_t* sa = align1024(smem_raw);
  uint8_t* sb = sa + TT::mid * C * dp * 2;   // (with dp = 64 the M = 128 MMA reads on from A into B: valid memory)
  if (tid == 0) {
    cta.word = look_again = 0;
    mbar_init(&done, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 128);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const int row_l = (warp & 3) * 32 + lane;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

  Raw<T> ra[kPieces], rb[kPieces];
  const auto fetch = [&](int task) {
    const int bh = task / g.nc, chunk = task - bh * g.nc, len = min(C, g.n - chunk * C);
    const size_t tok = (size_t)bh * g.n + (size_t)chunk * C;
    load_tile<T>(ra, static_cast<const T*>(g.a) + tok * g.pitch_a, g.pitch_a, len, g.d, dp, tid);
    load_tile<T>(rb, static_cast<const T*>(g.b) + tok * g.pitch_b, g.pitch_b, len, g.e, ep, tid);
  };
  const auto skipped = [&](int task) { return task % g.nc == g.skip; };
  int task = blockIdx.x;
  while (task < g.tasks && skipped(task)) task += gridDim.x;
  if (task < g.tasks) fetch(task);
  for (int it = 0; task < g.tasks; ++it) {
    const int bh = task / g.nc, chunk = task - bh * g.nc, len = min(C, g.n - chunk * C);
    const float sh = g.s[bh % g.h];
    const bool backward = g.backward != 0;
    store_tile<T, TT::mid, true>(sa, ra, dp, tid, [&](int row) {
      return expf(-sh * (float)(backward ? row : max(len - row, 0)));
    });
    store_tile<T, TT::in, false>(sb, rb, ep, tid, NoWeight());
    fence_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after_sync();
      issue_terms<TT::mid, TT::in, TT::cut>(tmem, TermOperand{smem_u32(sa), (uint32_t)(C * dp * 2), C, true},
                                            TermOperand{smem_u32(sb), (uint32_t)(C * ep * 2), C, true}, ep, C / 16);
      umma_commit(&done);
    }
    int next = task + gridDim.x;
    while (next < g.tasks && skipped(next)) next += gridDim.x;
    if (next < g.tasks) fetch(next);
    wait_or_fault(&done, it & 1, &cta, g.fault, kFaultMmaWait);
    tc_fence_after_sync();
    float4* out = reinterpret_cast<float4*>(g.states + (size_t)task * g.d * g.e);
    const int per = ep / 4;   // columns of this warp's group
#pragma unroll 1
    for (int c0 = (warp >> 2) * per; c0 < ((warp >> 2) + 1) * per; c0 += 16) {
      uint32_t r[16];
      tmem_ld16(tmem + lane_base + c0, r);
      tmem_ld_wait();
      if (row_l < g.d && c0 < g.e) {
        if (!all_finite(r)) look_again = 1;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          out[(size_t)(c0 / 4 + q) * g.d + row_l] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                               __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
      }
    }
    task = next;
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
  if (look_again) {   // (after the loop, whose registers hold the next chunk's rows)
    for (int u = blockIdx.x; u < g.tasks; u += gridDim.x)
      if (u % g.nc != g.skip) plain_state<T>(g, u);
  }
}

// ---------------------------------------------------------------------------
// outputs: OUT = (X Y^T . M) Z + diag(w) X op(P)
//   rev = 0: M_ij = lambda^(i-j) [i >= j], w_i = lambda^i;   rev = 1: M_ij = lambda^(j-i) [j >= i], w_i = lambda^(len-i)
// Tensor memory: S (terms 0 and 1 of the masked scores over S itself), its term 2, the two products.  Shared memory:
// two sets of term tiles, X then Z in the first, Y (fp16: Y and X as they are) then P in the second.  A task's steps, each product running
// under the next step's work (the loads of a step are issued one step earlier):
//   S = X Y^T | P's terms | O2 = X P | mask, split S; Z's terms | O1 = S_m Z | next task's Y, X terms | next S | epilogue
// ---------------------------------------------------------------------------
struct OutRole {
  const void *x, *y, *z;
  void* out;
  const float* state;      // border states of the chunks in lane order; NULL: all zero
  int wx, wz, pitch_x, pitch_z;
  int transposed;          // op(P) = P^T
  int rev;
  int zero_chunk;          // chunk whose border state is zero (-1: none)
  int add;                 // add to OUT instead of overwriting it
};
struct OutArgs {
  OutRole role[3];
  const float* s;
  int roles, h, n, nc, tasks, d, e;
  uint32_t set_bytes;      // bytes of the first set of term tiles
  int32_t* fault;
};

__device__ __forceinline__ void put16(float* p, const float (&x)[16], bool add) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float4 v = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    float4* dst = reinterpret_cast<float4*>(p) + q;
    if (add) {
      const float4 o = *dst;
      v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
    }
    *dst = v;
  }
}
__device__ __forceinline__ uint32_t pack2(float a, float b, __half) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack2(float a, float b, __nv_bfloat16) { return pack_bf16(a, b); }
__device__ __forceinline__ float2 unpack2(uint32_t u, __half) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
__device__ __forceinline__ float2 unpack2(uint32_t u, __nv_bfloat16) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
template <typename T>
__device__ __forceinline__ void put16(T* p, const float (&x)[16], bool add) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint4* dst = reinterpret_cast<uint4*>(p) + q;
    uint32_t u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = pack2(x[8 * q + 2 * j], x[8 * q + 2 * j + 1], T());
    if (add) {   // the sum of two rounded slices, rounded again
      const uint4 o = *dst;
      const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = unpack2(u[j], T()), b = unpack2(w[j], T());
        u[j] = pack2(a.x + b.x, a.y + b.y, T());
      }
    }
    *dst = make_uint4(u[0], u[1], u[2], u[3]);
  }
}

// Blocks of 16 columns of row `row` of a task's output from column `col` on, those whose bit is set
template <typename T>
__device__ __noinline__ void plain_out(const OutArgs* g, int t, int row, int col, uint32_t blocks) {
  const OutRole& r = g->role[t % g->roles];
  const int u = t / g->roles, bh = u / g->nc, chunk = u - bh * g->nc, len = min(C, g->n - chunk * C);
  const size_t tok = (size_t)bh * g->n + (size_t)chunk * C;
  const T *x = static_cast<const T*>(r.x) + (tok + row) * r.pitch_x, *y = static_cast<const T*>(r.y) + tok * r.pitch_x;
  const float sh = g->s[bh % g->h];
  for (; blocks != 0; blocks >>= 1, col += 16) {
    if ((blocks & 1) == 0) continue;
    const T* z = static_cast<const T*>(r.z) + tok * r.pitch_z + col;
    float sum[16], inter[16];
    for (int j = 0; j < 16; ++j) sum[j] = inter[j] = 0.f;
    bool settled = false;   // all NaN: so they stay
    for (int c = r.rev ? row : 0; !settled && (r.rev ? c < len : c <= row); ++c) {   // the tokens that the mask lets through
      float dot = 0.f;
      for (int i = 0; i < r.wx; i += 8) {
        Raw<T> rx, ry;
        load_piece<T>(rx, x + i), load_piece<T>(ry, y + (size_t)c * r.pitch_x + i);
        float fx[8], fy[8];
        to_floats<T>(rx, fx), to_floats<T>(ry, fy);
        for (int j = 0; j < 8; ++j) dot = fmaf(fx[j], fy[j], dot);
      }
      dot *= expf(-sh * (float)(r.rev ? c - row : row - c));
      settled = true;
      for (int h = 0; h < 16; h += 8) {
        Raw<T> rz;
        load_piece<T>(rz, z + (size_t)c * r.pitch_z + h);
        float fz[8];
        to_floats<T>(rz, fz);
        for (int j = 0; j < 8; ++j) {
          sum[h + j] = fmaf(dot, fz[j], sum[h + j]);
          settled = settled && isnan(sum[h + j]);
        }
      }
    }
    if (!settled && r.state != nullptr && chunk != r.zero_chunk) {
      const float* p = r.state + ((size_t)bh * g->nc + chunk) * g->d * g->e;   // lane order (common.cuh)
      for (int i = 0; i < r.wx; ++i) {
        for (int j = 0; j < 16; ++j) {
          const int pr = r.transposed ? col + j : i, pc = r.transposed ? i : col + j;
          inter[j] = fmaf(to_float(x[i]), p[((size_t)(pc / 4) * g->d + pr) * 4 + pc % 4], inter[j]);
        }
      }
      const float w_row = expf(-sh * (float)(r.rev ? len - row : row));
      for (int j = 0; j < 16; ++j) sum[j] = fmaf(w_row, inter[j], sum[j]);
    }
    put16(static_cast<T*>(r.out) + (tok + row) * r.pitch_z + col, sum, r.add != 0);
  }
}

// ... of a whole task, the blocks of its output that hold such a result
template <typename T>
__device__ __noinline__ void plain_out_where_needed(const OutArgs* g, int t) {
  const OutRole& r = g->role[t % g->roles];
  const int u = t / g->roles, bh = u / g->nc, chunk = u - bh * g->nc, len = min(C, g->n - chunk * C);
  const size_t tok = (size_t)bh * g->n + (size_t)chunk * C;
  for (int p = threadIdx.x; p < C * (r.wz / 16); p += NT) {
    const int row = p % C, col = p / C * 16;
    if (row >= len) continue;
    const T* out = static_cast<const T*>(r.out) + (tok + row) * r.pitch_z + col;
    bool finite = true;
    for (int j = 0; j < 16; ++j) finite = finite && isfinite(to_float(out[j]));
    if (!finite) plain_out<T>(g, t, row, col, 1u);
  }
}

template <typename T, bool ADD>
__global__ void __launch_bounds__(NT, 1) k_split_out(const __grid_constant__ OutArgs g) {
  using TT = Terms<T>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t s_done, o2_done, o1_done;
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  __shared__ int look_again;   // a result that is not finite has been written
  __shared__ float decay[C + 1];   // lambda^0 .. lambda^128 of the task's head
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dp = padded(g.d), ep = padded(g.e);
  uint8_t* set_a = align1024(smem_raw);
  uint8_t* set_b = set_a + g.set_bytes;
  if (tid == 0) {
    cta.word = look_again = 0;
    mbar_init(&s_done, 1);
    mbar_init(&o2_done, 1);
    mbar_init(&o1_done, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t t_s = tmem, t_lo = tmem + 128, t_o1 = tmem + 192, t_o2 = tmem + 320;
  const int quarter = warp & 3, group = warp >> 2;     // tensor-memory lanes and columns of this warp
  const int row_l = quarter * 32 + lane;
  const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
  const uint32_t addr_a = smem_u32(set_a), addr_b = smem_u32(set_b);

  struct Task {
    const OutRole* r;
    int bh, chunk, len;
    size_t tok;
    float sh;
    bool has_state;
  };
  const auto task_of = [&](int t) {
    Task k;
    k.r = &g.role[t % g.roles];
    const int u = t / g.roles;
    k.bh = u / g.nc, k.chunk = u - k.bh * g.nc;
    k.len = min(C, g.n - k.chunk * C);
    k.tok = (size_t)k.bh * g.n + (size_t)k.chunk * C;
    k.sh = g.s[k.bh % g.h];
    k.has_state = k.r->state != nullptr && k.chunk != k.r->zero_chunk;
    return k;
  };
  const auto load_xy = [&](Raw<T> (&dst)[kPieces], const void* p, const Task& k) {
    load_tile<T>(dst, static_cast<const T*>(p) + k.tok * k.r->pitch_x, k.r->pitch_x, k.len, k.r->wx, padded(k.r->wx), tid);
  };
  // the scores' operands: Y and, for fp16, X as they are in the second set, X's terms in the first
  constexpr bool kRawScores = std::is_same<T, __half>::value;
  const auto store_y = [&](const Raw<T> (&ry)[kPieces], const Raw<T> (&rx)[kPieces], int wx) {
    if constexpr (kRawScores) {
      store_raw<T>(set_b, ry, wx, tid);
      store_raw<T>(set_b + C * wx * 2, rx, wx, tid);
    } else {
      store_tile<T, TT::in, false>(set_b, ry, wx, tid, NoWeight());
    }
  };
  const auto issue_s = [&](const Task& k) {
    const int wx = padded(k.r->wx);
    tc_fence_after_sync();
    if constexpr (kRawScores)
      issue_terms<1, 1, 0, true>(t_s, TermOperand{addr_b + (uint32_t)(C * wx * 2), 0, C, false}, TermOperand{addr_b, 0, C, false}, C,
                                 wx / 16);
    else
      issue_terms<TT::in, TT::in, TT::cut>(t_s, TermOperand{addr_a, (uint32_t)(C * wx * 2), C, false},
                                           TermOperand{addr_b, (uint32_t)(C * wx * 2), C, false}, C, wx / 16);
    umma_commit(&s_done);
  };

  int t = blockIdx.x;
  if (t < g.tasks) {
    Task k = task_of(t);
    {
      Raw<T> rx[kPieces], ry[kPieces];
      load_xy(rx, k.r->x, k);
      load_xy(ry, k.r->y, k);
      if (tid <= C) decay[tid] = expf(-k.sh * (float)tid);
      store_y(ry, rx, padded(k.r->wx));
      store_tile<T, TT::in, false>(set_a, rx, padded(k.r->wx), tid, NoWeight());
    }
    fence_async_smem();
    __syncthreads();
    if (tid == 0) issue_s(k);
    int o2_uses = 0;
    for (int it = 0;; ++it) {
      const int wx = padded(k.r->wx), wz = padded(k.r->wz);
      const float w_row = decay[k.r->rev ? max(k.len - row_l, 0) : row_l];
      // ---- P's terms over Y (the scores have read it), O2 = X op(P)
      if (k.has_state) {
        Raw<float> rp[kPieces];
        load_state(rp, k.r->state + ((size_t)k.bh * g.nc + k.chunk) * g.d * g.e, g.d, g.e, dp, ep, tid);
        wait_or_fault(&s_done, it & 1, &cta, g.fault, kFaultMmaWait);
        store_state_terms<TT::mid>(set_b, rp, dp, ep, tid);
        fence_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        if (tid == 0) {
          tc_fence_after_sync();
          issue_terms<TT::in, TT::mid, TT::cut>(t_o2, TermOperand{addr_a, (uint32_t)(C * wx * 2), C, false},
                                                TermOperand{addr_b, (uint32_t)(dp * ep * 2), (uint32_t)dp, k.r->transposed == 0},
                                                wz, wx / 16);
          umma_commit(&o2_done);
        }
      } else {
        wait_or_fault(&s_done, it & 1, &cta, g.fault, kFaultMmaWait);
      }
      // ---- the masked scores' terms, Z's terms over X, O1 = S_m Z
      {
        Raw<T> rz[kPieces];
        load_tile<T>(rz, static_cast<const T*>(k.r->z) + k.tok * k.r->pitch_z, k.r->pitch_z, k.len, k.r->wz, wz, tid);
        tc_fence_after_sync();
        {
          uint32_t hi[16], mid[16], lo[16];
          const bool none = k.r->rev ? group < quarter : group > quarter;   // the block is all masked (as every lane sees it)
          if (none) {
#pragma unroll
            for (int j = 0; j < 16; ++j) hi[j] = mid[j] = lo[j] = 0u;
          } else {
            uint32_t r[32];
            tmem_ld32(t_s + lane_base + 32 * group, r);
            tmem_ld_wait();
            const int rel = k.r->rev ? 32 * group - row_l : row_l - 32 * group;   // distance from the diagonal of column 0
            const int dir = k.r->rev ? 1 : -1;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              float x[2];
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int dist = rel + dir * (j + u);
                x[u] = dist >= 0 ? __uint_as_float(r[j + u]) * decay[max(dist, 0)] : 0.f;
              }
              uint32_t tt[TT::mid];
              split_pair<TT::mid>(x[0], x[1], tt);
              hi[j / 2] = tt[0], mid[j / 2] = tt[1];
              if constexpr (TT::mid == 3) lo[j / 2] = tt[2];
            }
          }
          tmem_st16(t_s + lane_base + 32 * group, hi);
          tmem_st16(t_s + lane_base + 32 * group + 16, mid);
          if constexpr (TT::mid == 3) tmem_st16(t_lo + lane_base + 16 * group, lo);
          tmem_st_wait();
        }
        if (k.has_state) wait_or_fault(&o2_done, o2_uses & 1, &cta, g.fault, kFaultMmaWait);   // O2 has read X
        store_tile<T, TT::in, false>(set_a, rz, wz, tid, NoWeight());
      }
      fence_async_smem();
      tc_fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after_sync();
        issue_terms_ts<TT::mid, TT::in, TT::cut>(t_o1, t_s, t_lo, TermOperand{addr_a, (uint32_t)(C * wz * 2), C, true}, wz);
        umma_commit(&o1_done);
      }
      // ---- the next task's Y and X, its scores
      const int t_next = t + gridDim.x;
      const bool more = t_next < g.tasks;
      Task kn = k;
      if (more) {
        kn = task_of(t_next);
        Raw<T> ry[kPieces], rx[kPieces];
        load_xy(ry, kn.r->y, kn);
        load_xy(rx, kn.r->x, kn);
        if (tid <= C) decay[tid] = expf(-kn.sh * (float)tid);   // this task's masks are done (barrier above)
        store_y(ry, rx, padded(kn.r->wx));   // O2 has read P
        wait_or_fault(&o1_done, it & 1, &cta, g.fault, kFaultMmaWait);
        store_tile<T, TT::in, false>(set_a, rx, padded(kn.r->wx), tid, NoWeight());
        fence_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        if (tid == 0) issue_s(kn);
      } else {
        wait_or_fault(&o1_done, it & 1, &cta, g.fault, kFaultMmaWait);
      }
      // ---- epilogue, under the next scores
      tc_fence_after_sync();
      {
        const int per = wz / 4;
        T* out = static_cast<T*>(k.r->out) + (k.tok + row_l) * k.r->pitch_z;
        uint32_t again = 0;   // blocks of 16 columns with a result that is not finite
#pragma unroll 1
        for (int c0 = group * per; c0 < (group + 1) * per; c0 += 16) {
          uint32_t a1[16], a2[16];
          tmem_ld16(t_o1 + lane_base + c0, a1);
          if (k.has_state) tmem_ld16(t_o2 + lane_base + c0, a2);
          tmem_ld_wait();
          if (row_l < k.len && c0 < k.r->wz) {
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              x[j] = k.has_state ? fmaf(w_row, __uint_as_float(a2[j]), __uint_as_float(a1[j])) : __uint_as_float(a1[j]);
              a1[j] = __float_as_uint(x[j]);
            }
            if constexpr (ADD) {
              if (all_finite(a1))
                put16(out + c0, x, k.r->add != 0);
              else
                again |= 1u << ((c0 - group * per) / 16);
            } else {
              if (!all_finite(a1)) look_again = 1;
              put16(out + c0, x, false);
            }
          }
        }
        if constexpr (ADD) {
          if (again) plain_out<T>(&g, t, row_l, group * per, again);   // (here few registers are live)
        }
      }
      o2_uses += k.has_state ? 1 : 0;
      if (!more) break;
      t = t_next;
      k = kn;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if constexpr (!ADD) {
    if (look_again)   // (after the loop, whose registers are all taken)
      for (int u = blockIdx.x; u < g.tasks; u += gridDim.x) plain_out_where_needed<T>(&g, u);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
int host_padded(int w) { return w <= 64 ? 64 : 128; }

constexpr size_t kMaxSmem = 6 * 32768 + 1024;

template <typename T>
cudaError_t launch_states(const Dims& m, const StateArgs& g, cudaStream_t st) {
  const size_t smem = (size_t)C * 2 * (Terms<T>::mid * host_padded(m.d) + Terms<T>::in * host_padded(m.e)) + 1024;
  cudaError_t err = opt_in_smem<k_split_states<T>>(kMaxSmem);
  if (err != cudaSuccess) return err;
  // (a 64-wide A of the last term reads 16 KB past its tile: the B terms behind it are at least that long)
  const int grid = g.tasks < sm_count() ? g.tasks : sm_count();
  k_split_states<T><<<grid, NT, smem, st>>>(g);
  err = cudaGetLastError();
  if (err != cudaSuccess) g_failed_step = "launch of the chunk-state kernel";
  return err;
}

template <typename T, bool ADD>
cudaError_t launch_out(const Dims& m, OutArgs& g, cudaStream_t st) {
  const int dp = host_padded(m.d), ep = host_padded(m.e), widest = dp > ep ? dp : ep;
  g.set_bytes = (uint32_t)(Terms<T>::in * C * widest * 2);
  const size_t state = (size_t)Terms<T>::mid * dp * ep * 2;
  const size_t smem = g.set_bytes + (state > g.set_bytes ? state : g.set_bytes) + 1024;
  cudaError_t err = opt_in_smem<k_split_out<T, ADD>>(kMaxSmem);
  if (err != cudaSuccess) return err;
  const int grid = g.tasks < sm_count() ? g.tasks : sm_count();
  k_split_out<T, ADD><<<grid, NT, smem, st>>>(g);
  err = cudaGetLastError();
  if (err != cudaSuccess) g_failed_step = "launch of the output kernel";
  return err;
}

template <typename F>
cudaError_t by_dtype(int dtype, F&& f) {
  switch (dtype) {
    case LASP_F32: return f(float());
    case LASP_F16: return f(__half());
    case LASP_BF16: return f(__nv_bfloat16());
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t split_chunk_states(const Dims& m, const void* a, const void* bten, const float* s, float* states,
                               bool backward, bool alone, cudaStream_t st) {
  StateArgs g = {};
  g.a = a, g.b = bten, g.s = s, g.states = states;
  g.h = m.h, g.n = m.n, g.nc = m.nc, g.tasks = m.b * m.h * m.nc;
  g.d = m.d, g.e = m.e, g.pitch_a = m.pitch_d, g.pitch_b = m.pitch_e, g.backward = backward ? 1 : 0;
  g.skip = alone ? (backward ? 0 : m.nc - 1) : -1;   // nobody follows the sequence's end
  const cudaError_t err = fault_word_address(&g.fault);
  if (err != cudaSuccess) return err;
  return by_dtype(m.dtype, [&](auto t) { return launch_states<decltype(t)>(m, g, st); });
}

cudaError_t split_fwd_output(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                             const float* prefix, void* o, bool alone, bool add_o, cudaStream_t st) {
  OutArgs g = {};
  g.role[0] = {q, k, v, o, m.nc == 1 && alone ? nullptr : prefix, m.d, m.e, m.pitch_d, m.pitch_e, 0, 0, alone ? 0 : -1, add_o};
  g.roles = 1;
  g.s = s, g.h = m.h, g.n = m.n, g.nc = m.nc, g.d = m.d, g.e = m.e, g.tasks = m.b * m.h * m.nc;
  const cudaError_t err = fault_word_address(&g.fault);
  if (err != cudaSuccess) return err;
  return by_dtype(m.dtype, [&](auto t) { return g.role[0].add || g.role[1].add || g.role[2].add ? launch_out<decltype(t), true>(m, g, st) : launch_out<decltype(t), false>(m, g, st); });
}

cudaError_t split_bwd_grads(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, const float* s,
                            const float* prefix, const float* suffix, void* dq, void* dk, void* dv, bool alone,
                            bool add_qk, bool add_v, cudaStream_t st) {
  OutArgs g = {};
  const int first = alone ? 0 : -1, last = alone ? m.nc - 1 : -1;
  if (m.nc == 1 && alone) prefix = suffix = nullptr;
  g.role[0] = {d_o, v, k, dq, prefix, m.e, m.d, m.pitch_e, m.pitch_d, 1, 0, first, add_qk};
  g.role[1] = {v, d_o, q, dk, suffix, m.e, m.d, m.pitch_e, m.pitch_d, 1, 1, last, add_qk};
  g.role[2] = {k, q, d_o, dv, suffix, m.d, m.e, m.pitch_d, m.pitch_e, 0, 1, last, add_v};
  g.roles = 3;
  g.s = s, g.h = m.h, g.n = m.n, g.nc = m.nc, g.d = m.d, g.e = m.e, g.tasks = 3 * m.b * m.h * m.nc;
  const cudaError_t err = fault_word_address(&g.fault);
  if (err != cudaSuccess) return err;
  return by_dtype(m.dtype, [&](auto t) { return g.role[0].add || g.role[1].add || g.role[2].add ? launch_out<decltype(t), true>(m, g, st) : launch_out<decltype(t), false>(m, g, st); });
}

}  // namespace lasp
