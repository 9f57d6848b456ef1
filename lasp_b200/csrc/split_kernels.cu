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
//   k_scan          the states at the chunk borders, in terms
//   k_split_out     OUT = (X Y^T . M) Z + diag(w) X op(P)
// k_split_out is all of the output kernels: (X,Y,Z,op(P)) = (Q,K,V,P) gives O, (dO,V,K,P^T) dQ, (V,dO,Q,Dn^T) dK and
// (K,Q,dO,Dn) dV, the last two with the mask transposed; the backward pass runs the three as one launch.  Computing
// the scores once per result costs one product in nine and makes every chunk three independent tasks.
//
// What bounds them: fp32, the shared memory between the fillers' stores and the products (an SS product of 128 x 128 reads
// 128 bytes a clock, all there is: 48 of a task's 144 MMAs take 87 clocks with A in tensor memory, the others 105 to 125 of
// 64); 16-bit types, the chain scores - mask - O1 of a task.  In step instead of in roles (sixteen warps loading,
// splitting, storing and meeting at barriers, results written 16 bytes of 32 rows at a time, the states split once per
// product) a dQ, dK or dV task of fp32 took 32000 clocks, now 22000; of bf16 16000, now 8400.
//
// One B200, b=2, h=12, n=2048, forward / backward in us, in step and now: fp32 d=e=128 82.7 / 160 -> 69.5 / 119, fp16 d=128, e=64
// 47.8 / 90 -> 44 / 72, fp16 d=e=128 57.7 / 111 -> 53.4 / 82, bf16 d=e=96 44.3 / 83 -> 36.8 / 55.  The error against
// fp64, relative to what it was then: fp32 results 0.79 to 0.87, rank states of all types 0.61 to 0.87, fp16 and bf16 results 1.00
// (a chunk of 64 elements of K is summed in an accumulator of its own, and the tensor cores' additions round towards zero).
#include <type_traits>
#include <utility>

#include "state_terms.cuh"
#include "tc_common.cuh"

namespace lasp {
namespace {

using namespace tc;

// Warps in four roles, by warpgroups: control (one warp issues the MMAs, one the TMA loads), readers of the accumulators
// (mask, split, epilogue), and fillers, which load, split and store operand chunks (two groups of them in the chunk-state
// kernel, one per chunk).
constexpr int kFillers = 256;     // threads of one group
constexpr int kUnit = 16384;      // one term of a chunk: 128 x 64 or 64 x 128 bf16
constexpr int kBox = 8192;        // what one TMA load brings: 64 x 64
constexpr int kPieces = 4;        // 8-element pieces of a chunk per filling thread

// terms of the inputs and of intermediate quantities, and the largest i + j of a product that is kept
template <typename T> struct Terms;
template <> struct Terms<float> { static constexpr int in = 3, mid = 3, cut = 2; };
template <> struct Terms<__half> { static constexpr int in = 2, mid = 3, cut = 2; };
template <> struct Terms<__nv_bfloat16> { static constexpr int in = 1, mid = 3, cut = 2; };

// eight elements of a row as they come from global memory
template <typename T> struct Raw { uint4 v; };
template <> struct Raw<float> { uint4 v, w; };

// (not by the read-only path: the kernel before may write them while this one's CTAs are there already)
__device__ __forceinline__ uint4 ld16(const void* p) { return *static_cast<const uint4*>(p); }
template <typename T> __device__ __forceinline__ void load_piece(Raw<T>& r, const T* p) { r.v = ld16(p); }
template <> __device__ __forceinline__ void load_piece<float>(Raw<float>& r, const float* p) {
  r.v = ld16(p), r.w = ld16(p + 4);
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

// A chunk is 64 elements of a product's K dimension of one operand, all its terms, in units of 16 KB: 128 rows of a
// K-major operand (X, Y, P^T) or 64 rows of an MN-major one (A, B, Z, P).  States' terms, and 16-bit tiles where they enter
// a product as they are, come by TMA; everything else through the fillers.  Piece p of a filled chunk is eight elements of
// a row; pieces run along the rows, so that a warp reads whole rows and its shared-memory stores hit every bank once.
struct Chunk {
  const char* src;     // this thread's first piece
  uint32_t stride;     // bytes from one of its pieces to the next
  int row0, drow;      // rows of its pieces
  int col;             // their columns, in eights
  int rows, live, cols;   // rows of the chunk, those from `live` on being zero; columns in eights
};
template <typename T>
__device__ __forceinline__ Chunk tensor_chunk(const T* p, int pitch, int rows, int live, int cols, bool wide, int tid) {
  const int sh = wide ? 4 : 3, row0 = tid >> sh, col = tid & ((1 << sh) - 1), drow = kFillers >> sh;
  return {reinterpret_cast<const char*>(p + (size_t)row0 * pitch + 8 * col), (uint32_t)(drow * pitch * (int)sizeof(T)), row0, drow, col, rows, live,
          cols / 8};
}

template <typename T>
struct RawChunk {   // a thread's pieces on their way
  Raw<T> piece[kPieces];
};
template <typename T>
__device__ __forceinline__ void load_chunk_piece(RawChunk<T>& r, const Chunk& c, int i) {
  Raw<T>& e = r.piece[i];
  e.v = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (std::is_same<T, float>::value) e.w = e.v;
  if (c.row0 + i * c.drow < c.live && c.col < c.cols) load_piece<T>(e, reinterpret_cast<const T*>(c.src + (size_t)i * c.stride));
}
struct NoWeight {};
// ... N terms of them in shared memory, units of 16 KB from `units` on, row `row` multiplied by wt(row).  The registers of a
// piece that is stored take the next chunk's: next(i).
template <typename T, int N, typename F, typename W = NoWeight>
__device__ __forceinline__ void store_chunk(uint8_t* units, const RawChunk<T>& r, const Chunk& c, F next, W wt = W()) {
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int row = c.row0 + i * c.drow;
    if (row < c.rows && c.col < c.cols) {
      uint8_t* dst = units + tile_offset(row, 8 * c.col, c.rows);
      float x[8];
      to_floats<T>(r.piece[i], x);
      if constexpr (!std::is_same<W, NoWeight>::value) {
        const float f = wt(row);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] *= f;
      }
      uint32_t t[4][N];
#pragma unroll
      for (int j = 0; j < 4; ++j) split_pair<N>(x[2 * j], x[2 * j + 1], t[j]);
#pragma unroll
      for (int k = 0; k < N; ++k) *reinterpret_cast<uint4*>(dst + k * kUnit) = make_uint4(t[0][k], t[1][k], t[2][k], t[3][k]);
    }
    next(i);
  }
}

// One operand of a product over a chunk: descriptors of its terms (16 KB apart) and of the steps of 16 K elements
struct TermOperand {
  SmemDesc first;
  uint32_t step;   // in units of 16 bytes
  __device__ __forceinline__ TermOperand(uint32_t addr, uint32_t rows, bool mn_major)
      : first(operand_desc(addr, rows, mn_major)), step(mn_major ? 128 : 2) {}
  __device__ __forceinline__ SmemDesc desc(int term, int ks) const { return {first.lo + term * (kUnit / 16) + ks * step, first.hi}; }
};
// The masked scores' terms in tensor memory, as the readers leave them: K step ks of terms 0 and 1 in the columns of t_s
// that held the step's sixteen scores, of term 2 in those of t_lo
struct ScoreOperand {
  uint32_t t_s, t_lo;
  __device__ __forceinline__ uint32_t addr(int term, int ks) const { return (term == 2 ? t_lo : t_s + 8 * term) + 16 * ks; }
};
// The products of terms whose indexes sum to FROM, FROM - 1, ..., TO, over one chunk.  A whole warp computes what the
// instructions take (uniform values, so that they live in uniform registers), its lane `leader` issues them.  (One thread
// in loops took 155 clocks for an MMA of 64, the warp unrolled 100 to 125 with lane 0 as the leader, less with an elected
// one; the warp in loops 10 % longer for the whole kernel.)
template <int NA, int NB, int FROM, int TO, typename A>
__device__ __forceinline__ void issue_terms(uint32_t d_tmem, const A& a, const TermOperand& b, uint32_t idesc, int ksteps, uint32_t& acc,
                                            bool leader) {
#pragma unroll
  for (int sum = FROM; sum >= TO; --sum) {
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int j = sum - i;
      if (j < 0 || j >= NB) continue;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks < ksteps) {
          if constexpr (std::is_same<A, ScoreOperand>::value)
            umma_ts(d_tmem, a.addr(i, ks), b.desc(j, ks), idesc, acc, leader);
          else
            umma(d_tmem, a.desc(i, ks), b.desc(j, ks), idesc, acc, leader);
          acc = 1;
        }
      }
    }
  }
}
__device__ __forceinline__ int ksteps_of(int width, int chunk) { return max(min(width - 64 * chunk, 64), 0) / 16; }

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
// chunk states: T[i][j] = sum_c w_c A[c][i] B[c][j], row-major
//   forward : A = K, B = V,  w_c = lambda^(len-c);   backward: A = Q, B = dO, w_c = lambda^c
// A task per chunk of the sequence, persistent CTAs.  The 64 tokens of a chunk of the operands are summed in an accumulator
// of their own, so that the next task's can follow at once; the readers add the two.
// ---------------------------------------------------------------------------
struct StateArgs {
  const void *a, *b;
  const float* s;
  float* states;
  int h, n, nc, tasks, d, e, pitch_a, pitch_b, backward;
  int skip;   // chunk whose state nobody reads (-1: none)
  int32_t* fault;
};

constexpr int kStateReaders = 256, kStateThreads = 128 + kStateReaders + 2 * kFillers;

// The elements of a task's state that are not finite, again
template <typename T>
__device__ __forceinline__ void plain_state(const StateArgs& g, int task) {
  const int bh = task / g.nc, chunk = task - bh * g.nc, len = min(C, g.n - chunk * C);
  const size_t tok = (size_t)bh * g.n + (size_t)chunk * C;
  const T *a = static_cast<const T*>(g.a) + tok * g.pitch_a, *b = static_cast<const T*>(g.b) + tok * g.pitch_b;
  const float sh = g.s[bh % g.h];
  float4* state = reinterpret_cast<float4*>(g.states + (size_t)task * g.d * g.e);
  for (int p = threadIdx.x - 128; p < g.d * g.e / 4; p += kStateThreads - 128) {   // four columns of a row
    const int row = p / (g.e / 4), col = p % (g.e / 4) * 4;
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
struct StatePlan {   // units of 16 KB: A's chunk, then B's, of the first 64 tokens and of the others
  static constexpr int kChunk = Terms<T>::mid + Terms<T>::in;
  static constexpr size_t kSmem = (size_t)2 * kChunk * kUnit + 1024;
  static constexpr bool kTmaB = Terms<T>::in == 1;   // bf16 is its own only term
};

template <typename T>
__global__ void __launch_bounds__(kStateThreads, 1) k_split_states(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ StateArgs g) {
  using TT = Terms<T>;
  using Plan = StatePlan<T>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_a[2], full_b[2], done[2], result[2], acc_free[2];   // by chunk; result, acc_free: by the task's parity
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  __shared__ int look_again;   // a state with an element that is not finite has been written
  const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
  uint8_t* smem = align1024(smem_raw);
  if (tid == 0) {
    cta.word = look_again = 0;
    for (int j = 0; j < 2; ++j) {
      mbar_init(&full_a[j], kFillers / 32);
      mbar_init(&full_b[j], Plan::kTmaB ? 1 : kFillers / 32);
      mbar_init(&done[j], 1), mbar_init(&result[j], 1), mbar_init(&acc_free[j], kStateReaders / 32);
    }
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;   // [parity of the task][chunk], 128 columns each
  after_previous();
  let_next_start();
  const auto next_task = [&](int t) {
    while (t < g.tasks && t % g.nc == g.skip) t += gridDim.x;
    return t;
  };

  if (warp < 4) {
    set_regs_dec<40>();
    if (warp == 0) {
      const uint32_t idesc = umma_idesc(128, g.e, true, true), base = uniform(smem_u32(smem)), t_acc = uniform(tmem);
      const bool leader = elect_one();
      int it = 0;
      for (int t = next_task(blockIdx.x); t < g.tasks; t = next_task(t + gridDim.x), ++it) {
        const int len = min(C, g.n - (t % g.nc) * C);
        if (it >= 2) wait_or_fault(&acc_free[it & 1], ((it >> 1) - 1) & 1, &cta, g.fault, kFaultMmaWait);
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          wait_or_fault(&full_a[c], it & 1, &cta, g.fault, kFaultTmaWait);
          wait_or_fault(&full_b[c], it & 1, &cta, g.fault, kFaultTmaWait);
          tc_fence_after_wait();
          const uint32_t at = base + c * Plan::kChunk * kUnit;
          uint32_t acc = 0;
          issue_terms<TT::mid, TT::in, TT::cut, 0>(t_acc + 256 * (it & 1) + 128 * c, TermOperand(at, 64, true),
                                                   TermOperand(at + TT::mid * kUnit, 64, true), idesc, ksteps_of(len + 15, c), acc, leader);
          if (leader) umma_commit(&done[c]);
        }
        if (leader) umma_commit(&result[it & 1]);
        __syncwarp();
      }
    } else if (Plan::kTmaB && warp == 1 && lane == 0) {
      int it = 0;
      for (int t = next_task(blockIdx.x); t < g.tasks; t = next_task(t + gridDim.x), ++it) {
        const int bh = t / g.nc, chunk = t - bh * g.nc, slabs = g.e > 64 ? 2 : 1;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          if (it > 0) wait_or_fault(&done[c], (it - 1) & 1, &cta, g.fault, kFaultMmaWait);
          mbar_expect_tx(&full_b[c], slabs * kBox);
          for (int u = 0; u < slabs; ++u)
            tma_load_3d(smem_u32(smem) + (c * Plan::kChunk + TT::mid) * kUnit + u * kBox, &map_b, &full_b[c], 64 * u, chunk * C + 64 * c, bh);
        }
      }
    }
  } else if (warp < 4 + kStateReaders / 32) {
    set_regs_inc<88>();
    const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;   // tensor-memory lanes and columns of this warp
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int it = 0;
    for (int t = next_task(blockIdx.x); t < g.tasks; t = next_task(t + gridDim.x), ++it) {
      const uint32_t acc = tmem + 256 * (it & 1) + lane_base;
      wait_or_fault(&result[it & 1], (it >> 1) & 1, &cta, g.fault, kFaultMmaWait);
      tc_fence_after_wait();
      const bool two = g.n - (t % g.nc) * C > 64;   // tokens in the second chunk
      float* out = g.states + ((size_t)t * g.d + (row & ~3)) * g.e + 4 * (lane & 3);
#pragma unroll 1
      for (int c0 = 16 * half; c0 < g.e; c0 += 32) {
        uint32_t r[16], r2[16];
        __syncwarp();   // (rows that do not exist are not stored)
        tmem_ld16(acc + c0, r);
        if (two) tmem_ld16(acc + 128 + c0, r2);
        tmem_ld_wait();
        if (two) {
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
        }
        if (row < g.d && !all_finite(r)) look_again = 1;
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
        rows_to_lanes(v, lane);
        if (row < g.d) {   // (widths are multiples of 16: four neighbouring rows exist together)
#pragma unroll
          for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(out + (size_t)i * g.e + c0) = v[i];
        }
      }
      tc_fence_before_sync();
      warp_arrive(&acc_free[it & 1]);
    }
  } else {
    const int c = warp >= 4 + (kStateReaders + kFillers) / 32 ? 1 : 0, ft = tid & (kFillers - 1);   // this group's chunk
    struct Task {
      int len;
      size_t tok;
      float sh;
    };
    const auto task_of = [&](int t) {
      const int bh = t / g.nc, chunk = t - bh * g.nc;
      return Task{min(C, g.n - chunk * C), (size_t)bh * g.n + (size_t)chunk * C, g.s[bh % g.h]};
    };
    const auto chunk_of = [&](const Task& k, bool is_b) {
      const int w = is_b ? g.e : g.d, pitch = is_b ? g.pitch_b : g.pitch_a;
      return tensor_chunk<T>(static_cast<const T*>(is_b ? g.b : g.a) + (k.tok + 64 * c) * pitch, pitch, 64, k.len - 64 * c, w, w > 64, ft);
    };
    int t = next_task(blockIdx.x), it = 0;
    bool is_b = false;
    if (t < g.tasks) {
      Task k = task_of(t);
      Chunk cur = chunk_of(k, false);
      RawChunk<T> r;
#pragma unroll
      for (int i = 0; i < kPieces; ++i) load_chunk_piece<T>(r, cur, i);
      while (true) {
        const int prev = it - 1, len = k.len;
        const float sh = k.sh;
        const bool b_now = is_b;
        if (Plan::kTmaB || is_b) {
          is_b = false, ++it;
          t = next_task(t + gridDim.x);
          if (t < g.tasks) k = task_of(t);
        } else {
          is_b = true;
        }
        Chunk next = chunk_of(k, is_b);
        if (t >= g.tasks) next.cols = 0;
        if (prev >= 0 && !b_now) wait_or_fault(&done[c], prev & 1, &cta, g.fault, kFaultMmaWait);
        const auto load_next = [&](int i) { load_chunk_piece<T>(r, next, i); };
        uint8_t* units = smem + c * Plan::kChunk * kUnit;
        if (b_now) {
          store_chunk<T, TT::in>(units + TT::mid * kUnit, r, cur, load_next);
        } else {
          const bool backward = g.backward != 0;
          store_chunk<T, TT::mid>(units, r, cur, load_next, [&](int row) {
            return expf(-sh * (float)(backward ? 64 * c + row : max(len - 64 * c - row, 0)));
          });
        }
        fence_async_smem();
        warp_arrive(b_now ? &full_b[c] : &full_a[c]);
        if (t >= g.tasks) break;
        cur = next;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
  // (after the loops, whose registers hold the next chunk's rows; the control warps have given theirs away)
  if (look_again && warp >= 4) {
    for (int u = blockIdx.x; u < g.tasks; u += gridDim.x)
      if (u % g.nc != g.skip) plain_state<T>(g, u);
  }
}

// ---------------------------------------------------------------------------
// outputs: OUT = (X Y^T . M) Z + diag(w) X op(P)
//   rev = 0: M_ij = lambda^(i-j) [i >= j], w_i = lambda^i;   rev = 1: M_ij = lambda^(j-i) [j >= i], w_i = lambda^(len-i)
// A task - one result of one chunk of the sequence - is up to eight chunks of operands (two of X, Y, P and Z each) and
// three products:
//   S = X Y^T (an accumulator per chunk) | O2 = X op(P), while the readers mask and split S | O1 = S_m Z
// and under the next task's S the readers write OUT.  All of it meets at mbarriers, one phase per task each; every chunk
// is announced for every task, also one that the task has no use for, so that no barrier gets two phases ahead of a waiter.
// ---------------------------------------------------------------------------
enum Kind { kX0, kX1, kY0, kY1, kP0, kP1, kZ0, kZ1 };
enum Done { kS0, kS, kO2, kO1 };   // products of a task that have read their operands: S of chunk 0, S, O2, O1
constexpr int kPrev = 4, kAny = 8;  // (of the task before; whatever the same warps have waited for before)

// Where a chunk lies (in units of 16 KB) and what has to have read the chunk that was there before; fill_*: of what the
// fillers store, where a tile also comes as it is.
template <typename T> struct OutPlan;
// fp32: 192 KB hold X and Y and nothing else, so P follows Y, Z follows X and P, and the places of the next task's X and Y are
// those that are free first: it has them the other way round.
template <> struct OutPlan<float> {
  static constexpr int kUnits = 12, kTurn = 6, kReaders = 256, kReaderRegs = 112, kControlRegs = 64;
  static constexpr bool kFillXZ = true, kFillY = true, kRawXY = false;
  static constexpr uint32_t kFills = 6, kFillOrder = kX0 | kY0 << 4 | kX1 << 8 | kY1 << 12 | kZ0 << 16 | kZ1 << 20;
  static constexpr int place(int kind) {
    return kind == kX0 || kind == kZ0 ? 0 : kind == kX1 ? 6 : kind == kY1 || kind == kP1 ? 9 : 3;
  }
  static constexpr int after(int kind) {
    return kind == kX0 ? kO2 + kPrev : kind == kX1 ? kO1 + kPrev : kind == kP0 ? kS0 : kind == kP1 ? kS : kind == kZ0 || kind == kZ1 ? kO2 : kAny;
  }
  static constexpr int fill_place(int kind) { return place(kind); }
  static constexpr int fill_after(int kind) { return after(kind); }
};
// fp16: X as it is, X in two terms, Y as it is, P; Z follows X and Y as they are, which only the scores need
template <> struct OutPlan<__half> {
  static constexpr int kUnits = 14, kTurn = 0, kReaders = 256, kReaderRegs = 112, kControlRegs = 64;
  static constexpr bool kFillXZ = true, kFillY = false, kRawXY = true;
  static constexpr uint32_t kFills = 4, kFillOrder = kX0 | kX1 << 4 | kZ0 << 8 | kZ1 << 12;
  static constexpr int place(int kind) {
    return kind == kX0 || kind == kZ0 ? 0 : kind == kX1 ? 1 : kind == kY0 || kind == kZ1 ? 2 : kind == kY1 ? 3 : kind == kP0 ? 8 : 11;
  }
  static constexpr int fill_place(int kind) { return kind == kX0 ? 4 : kind == kX1 ? 6 : place(kind); }
  static constexpr int after(int kind) { return kind == kX0 ? kO1 + kPrev : kind == kP0 ? kO2 + kPrev : kind == kZ0 || kind == kZ1 ? kS : kAny; }
  static constexpr int fill_after(int kind) { return kind == kX0 || kind == kX1 ? kO2 + kPrev : kS; }
};
// bf16: room for everything
template <> struct OutPlan<__nv_bfloat16> {
  static constexpr int kUnits = 12, kTurn = 0, kReaders = 512, kReaderRegs = 104, kControlRegs = 64;
  static constexpr bool kFillXZ = false, kFillY = false, kRawXY = true;
  static constexpr int place(int kind) { return kind <= kP0 ? kind : kind == kP1 ? 7 : kind == kZ0 ? 10 : 11; }
  static constexpr int after(int kind) { return kind == kX0 ? kO2 + kPrev : kind == kZ0 ? kO1 + kPrev : kAny; }
  static constexpr int fill_place(int kind) { return place(kind); }
};
template <typename T>
constexpr int kOutThreads = 128 + OutPlan<T>::kReaders + (OutPlan<T>::kFillXZ ? kFillers : 0);
// (looked up at run time: the eight values of a function, four bits each, in a constant)
template <int (*F)(int)>
constexpr uint32_t packed_plan() {
  uint32_t v = 0;
  for (int k = 0; k < 8; ++k) v |= (uint32_t)F(k) << (4 * k);
  return v;
}
template <int (*F)(int)>
struct PackedPlan {
  static constexpr uint32_t value = packed_plan<F>();
};
template <int (*F)(int)>
__device__ __forceinline__ int plan_at(int k) {
  return (int)(PackedPlan<F>::value >> (4 * k)) & 15;
}

struct OutRole {
  const void *x, *y, *z;
  void* out;
  const __nv_bfloat16* state;   // border states of the chunks in terms; NULL: all zero
  int mx, my, mz, mp;      // their tensor maps
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
  int32_t* fault;
};
enum Map { kMapQ, kMapK, kMapV, kMapDo, kMapPrefix, kMapSuffix, kMaps };
struct OutMaps {
  CUtensorMap m[kMaps];
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
      const size_t elems = (size_t)g->d * g->e;
      const __nv_bfloat16* p = r.state + ((size_t)bh * g->nc + chunk) * 3 * elems;
      for (int i = 0; i < r.wx; ++i) {
        for (int j = 0; j < 16; ++j) {
          const int pr = r.transposed ? col + j : i, pc = r.transposed ? i : col + j;
          inter[j] = fmaf(to_float(x[i]), state_of_terms(p, (size_t)pr * g->e + pc, elems), inter[j]);
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
  for (int p = threadIdx.x - 128; p < C * (r.wz / 16); p += blockDim.x - 128) {
    const int row = p % C, col = p / C * 16;
    if (row >= len) continue;
    const T* out = static_cast<const T*>(r.out) + (tok + row) * r.pitch_z + col;
    bool finite = true;
    for (int j = 0; j < 16; ++j) finite = finite && isfinite(to_float(out[j]));
    if (!finite) plain_out<T>(g, t, row, col, 1u);
  }
}

template <typename T, bool ADD>
__global__ void __launch_bounds__(kOutThreads<T>, 1) k_split_out(const __grid_constant__ OutMaps maps, const __grid_constant__ OutArgs g) {
  using TT = Terms<T>;
  using Plan = OutPlan<T>;
  constexpr bool kRawScores = std::is_same<T, __half>::value;   // S of fp16 tiles is one product of the tiles as they are
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[8], done[4], sm_ready, acc_free;
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  __shared__ int look_again;   // a result that is not finite has been written
  // What the scores of a block of 32 columns on the diagonal take: line[k] = lambda^(31 - k) up to k = 31 and 0 beyond (the
  // transposed mask: lambda^(k - 31) from k = 31 on and 0 before), of which row r of the block starts at 31 - r.  Four
  // copies shifted by 0 to 3 elements, so that every row reads 16 bytes at a time, and as far apart as keeps eight
  // neighbouring rows on different banks.  (With a look-up and a comparison for every element a block on the diagonal took
  // 2300 clocks, one beside it 600.)
  __shared__ __align__(16) float line[4][72];
  __shared__ OutArgs args;   // (for the functions that are called: a parameter whose address is taken is not read as one)
  const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
  uint8_t* smem = align1024(smem_raw);
  if (tid == 0) {
    cta.word = look_again = 0;
    for (int j = 0; j < 8; ++j) {
      const bool filled = j < kY0 || j >= kZ0 ? Plan::kFillXZ : j < kP0 ? Plan::kFillY : false;
      const bool loaded = j >= kP0 && j < kZ0 ? true : j >= kZ0 ? !Plan::kFillXZ : Plan::kRawXY;
      mbar_init(&full[j], (filled ? kFillers / 32 : 0) + (loaded ? 1 : 0));
    }
    for (int j = 0; j < 4; ++j) mbar_init(&done[j], 1);
    mbar_init(&sm_ready, Plan::kReaders / 32);
    mbar_init(&acc_free, Plan::kReaders / 32);
    fence_mbar_init();
  }
  if (tid == 32) args = g;
  if (warp == 2) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  after_previous();
  let_next_start();

  struct Task {
    OutRole r;
    int bh, chunk, len;
    size_t tok;
    bool has_state;
  };
  const auto task_of = [&](int t) {
    Task k;
    k.r = g.role[t % g.roles];
    const int u = t / g.roles;
    k.bh = u / g.nc, k.chunk = u - k.bh * g.nc;
    k.len = min(C, g.n - k.chunk * C);
    k.tok = (size_t)k.bh * g.n + (size_t)k.chunk * C;
    k.has_state = k.r.state != nullptr && k.chunk != k.r.zero_chunk;
    return k;
  };
  const auto turned = [&](int unit, int it) {
    return Plan::kTurn && (it & 1) ? (unit >= Plan::kTurn ? unit - Plan::kTurn : unit + Plan::kTurn) : unit;
  };
  // (dep: what was in the place of a chunk of the CTA's task `it` has been read)
  const auto await_place = [&](int dep, int it) {
    const int of = dep == kAny ? -1 : it - (dep >> 2);
    if (of >= 0) wait_or_fault(&done[dep & 3], of & 1, &cta, g.fault, kFaultMmaWait);
  };

  if (warp < 4) {
    set_regs_dec<Plan::kControlRegs>();
    if (warp == 0) {
      const bool leader = elect_one();
      const uint32_t base = uniform(smem_u32(smem)), tm = uniform(tmem);
      const uint32_t t_s = tm, t_s1 = tm + 128, t_o1 = tm + 256, t_o2 = tm + 384;
      int it = 0;
      for (int t = blockIdx.x; t < g.tasks; t += gridDim.x, ++it) {
        const Task k = task_of(t);
        const OutRole& r = k.r;
        const auto await = [&](int kind) {
          wait_or_fault(&full[kind], it & 1, &cta, g.fault, kFaultTmaWait);
          tc_fence_after_wait();
        };
        const auto addr = [&](int kind) { return base + turned(plan_at<Plan::place>(kind), it) * kUnit; };
        const auto addr_terms = [&](int kind) { return base + turned(plan_at<Plan::fill_place>(kind), it) * kUnit; };
        const int chunks = r.wx > 64 ? 2 : 1;
        // S; its accumulators hold the masked scores of the task before until O1 has read them
        if (it > 0) wait_or_fault(&done[kO1], (it - 1) & 1, &cta, g.fault, kFaultMmaWait);
        const uint32_t idesc_s = umma_idesc(128, C, false, false, kRawScores);
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          await(kX0 + c);
          await(kY0 + c);
          if (c < chunks) {
            uint32_t acc = 0;
            constexpr int kIn = kRawScores ? 1 : TT::in, kCut = kIn == 1 ? 0 : TT::cut;
            issue_terms<kIn, kIn, kCut, 0>(c ? t_s1 : t_s, TermOperand(addr(kX0 + c), C, false), TermOperand(addr(kY0 + c), C, false),
                                           idesc_s, ksteps_of(r.wx, c), acc, leader);
          }
          if (leader) umma_commit(&done[c ? kS : kS0]);
        }
        // O2: the smaller products of both chunks, then the largest
        if (it > 0) wait_or_fault(&acc_free, (it - 1) & 1, &cta, g.fault, kFaultMmaWait);
        {
          const bool p_mn = r.transposed == 0;
          const uint32_t idesc = umma_idesc(128, r.wz, false, p_mn);
          const int p_rows = p_mn ? 64 : g.d, o2_chunks = k.has_state ? chunks : 0;
          uint32_t acc = 0;
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            await(kP0 + c);
            if (c < o2_chunks) issue_terms<TT::in, TT::mid, TT::cut, 1>(t_o2, TermOperand(addr_terms(kX0 + c), C, false),
                                                     TermOperand(addr(kP0 + c), p_rows, p_mn), idesc, ksteps_of(r.wx, c), acc, leader);
          }
#pragma unroll 1
          for (int c = 0; c < o2_chunks; ++c)
            issue_terms<1, 1, 0, 0>(t_o2, TermOperand(addr_terms(kX0 + c), C, false), TermOperand(addr(kP0 + c), p_rows, p_mn), idesc,
                                    ksteps_of(r.wx, c), acc, leader);
        }
        if (leader) umma_commit(&done[kO2]);
        // O1
        wait_or_fault(&sm_ready, it & 1, &cta, g.fault, kFaultMmaWait);
        {
          const uint32_t idesc = umma_idesc(128, r.wz, false, true);
          uint32_t acc = 0;
          const int zs = k.len > 64 ? 2 : 1;
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            await(kZ0 + c);
            if (c < zs) issue_terms<TT::mid, TT::in, TT::cut, 1>(t_o1, ScoreOperand{t_s + 64 * c, t_s1 + 64 * c}, TermOperand(addr_terms(kZ0 + c), 64, true),
                                                     idesc, 4, acc, leader);
          }
#pragma unroll 1
          for (int c = 0; c < zs; ++c)
            issue_terms<1, 1, 0, 0>(t_o1, ScoreOperand{t_s + 64 * c, t_s1 + 64 * c}, TermOperand(addr_terms(kZ0 + c), 64, true), idesc, 4, acc, leader);
        }
        if (leader) umma_commit(&done[kO1]);
        __syncwarp();
      }
    } else if (warp == 1 && lane == 0) {
      // ---- TMA: states' terms, tiles that enter a product as they are
      int it = 0;
      for (int t = blockIdx.x; t < g.tasks; t += gridDim.x, ++it) {
        const Task k = task_of(t);
        const OutRole& r = k.r;
        const auto load = [&](int kind, int map, int c0, int rows, int matrix, int row_step, int boxes, int terms) {
          // `boxes` boxes that lie one behind the other, 64 rows or 64 columns further each, of every term
          await_place(plan_at<Plan::after>(kind), it);
          if (boxes == 0) {
            mbar_arrive(&full[kind]);
            return;
          }
          mbar_expect_tx(&full[kind], boxes * terms * kBox);
          const uint32_t at = smem_u32(smem) + turned(plan_at<Plan::place>(kind), it) * kUnit;
          for (int i = 0; i < terms; ++i)
            for (int u = 0; u < boxes; ++u)
              tma_load_3d(at + i * kUnit + u * kBox, &maps.m[map], &full[kind], c0 + (64 - row_step) * u, rows + row_step * u, matrix + i);
        };
        const int row0 = k.chunk * C, state = 3 * (k.bh * g.nc + k.chunk);
        const auto load_xy = [&] {
#pragma unroll 1
          for (int u = 0; u < 4; ++u) {
            const int c = u & 1;
            load((u < 2 ? kX0 : kY0) + c, u < 2 ? r.mx : r.my, 64 * c, row0, k.bh, 64, r.wx > 64 * c ? 2 : 0, 1);
          }
        };
        if (Plan::kRawXY && !Plan::kFillXZ) load_xy();
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          const bool live = k.has_state && r.wx > 64 * c;
          if (r.transposed)
            load(kP0 + c, r.mp, 64 * c, 0, state, 64, live ? (g.d > 64 ? 2 : 1) : 0, 3);
          else
            load(kP0 + c, r.mp, 0, 64 * c, state, 0, live ? (g.e > 64 ? 2 : 1) : 0, 3);
        }
        if (Plan::kRawXY && Plan::kFillXZ) {   // (fp16: they wait for more than P does)
          // Y, which nobody else has asked for, comes into L2 while its place is taken: 24 x 2048 tokens, 128/128, forward
          // 52.8 -> 51.1 us, backward 81.4 -> 80.7.  (The next task's X, Y and Z, a task ahead: forward 3 us slower.)
#pragma unroll 1
          for (int u = 0; u < 4; ++u)
            if (64 * (u & 1) < r.wx) tma_prefetch_3d(&maps.m[r.my], 64 * (u & 1), row0 + 64 * (u >> 1), k.bh);
          load_xy();
        }
        if (!Plan::kFillXZ) {
#pragma unroll 1
          for (int c = 0; c < 2; ++c) load(kZ0 + c, r.mz, 0, row0 + 64 * c, k.bh, 0, k.len > 64 * c ? (r.wz > 64 ? 2 : 1) : 0, 1);
        }
      }
    }
  } else if (warp < 4 + Plan::kReaders / 32) {
    set_regs_inc<Plan::kReaderRegs>();
    const uint32_t t_s = tmem, t_s1 = tmem + 128, t_o1 = tmem + 256, t_o2 = tmem + 384;
    const int rid = tid - 128, quarter = warp & 3, part = (rid >> 7);   // tensor-memory lanes and columns of this warp
    constexpr int kParts = Plan::kReaders / 128;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const auto decay_of = [&](int t) { return g.s[t / g.roles / g.nc % g.h]; };
    const auto write_line = [&](int t) {
      if (rid < 256) {
        const int k = (rid & 63) + (rid >> 6), dist = g.role[t % g.roles].rev ? k - 31 : 31 - k;
        line[rid >> 6][rid & 63] = dist >= 0 ? expf(-decay_of(t) * (float)dist) : 0.f;
      }
    };
    write_line(blockIdx.x);
    int it = 0;
    for (int t = blockIdx.x; t < g.tasks; t += gridDim.x, ++it) {
      const Task k = task_of(t);
      const OutRole& r = k.r;
      const float sh = decay_of(t);
      const float w_row = expf(-sh * (float)(r.rev ? max(k.len - row, 0) : row));
      named_sync(1, Plan::kReaders);
      // ---- the masked scores' terms over the scores
      wait_or_fault(&done[kS], it & 1, &cta, g.fault, kFaultMmaWait);
      tc_fence_after_wait();
      const bool two = r.wx > 64;
      // Sixteen columns at a time, in a loop: the code runs once a task, so most of what is straight-line is fetched anew
      // every time.
#pragma unroll 1
      for (int u = 2 * part; u < 8; u = (u & 1) ? u + 2 * kParts - 1 : u + 1) {
        const int blk = u >> 1;
        uint32_t hi[8], mid[8], lo[8];
        const uint32_t at = lane_base + 16 * u;
        if (r.rev ? blk < quarter : blk > quarter) {   // all masked
#pragma unroll
          for (int j = 0; j < 8; ++j) hi[j] = mid[j] = lo[j] = 0u;
        } else {
          uint32_t x[16], y[16];
          tmem_ld16(t_s + at, x);
          if (two) tmem_ld16(t_s1 + at, y);
          // lambda^distance: beside the diagonal the row's distance to the block's nearer edge times the column's to it
          const bool diagonal = blk == quarter;
          const float edge = diagonal ? 1.f : expf(-sh * (float)(r.rev ? 32 * blk - row : row - 32 * blk - 31));
          const int first = (diagonal ? 31 - lane : r.rev ? 31 : 0) + 16 * (u & 1);
          const float4* factors = reinterpret_cast<const float4*>(&line[first & 3][first & ~3]);
          tmem_ld_wait();
          if (two) {
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
              const F2 sum = fma2(pair(y[j], y[j + 1]), {1.f, 1.f}, pair(x[j], x[j + 1]));
              x[j] = __float_as_uint(sum.x), x[j + 1] = __float_as_uint(sum.y);
            }
          }
          if (diagonal) {   // (a masked score that is not finite must not leave a trace)
            const uint32_t live = (r.rev ? 0xffffffffu << lane : 0xffffffffu >> (31 - lane)) >> (16 * (u & 1));
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = live & (1u << j) ? x[j] : 0u;
          }
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const float4 f = factors[j / 4];
#pragma unroll
            for (int v = 0; v < 4; v += 2) {
              const F2 m = mul2(pair(x[j + v], x[j + v + 1]), mul2(v ? F2{f.z, f.w} : F2{f.x, f.y}, {edge, edge}));
              uint32_t tt[3];
              split_pair<3>(m.x, m.y, tt);
              hi[(j + v) / 2] = tt[0], mid[(j + v) / 2] = tt[1], lo[(j + v) / 2] = tt[2];
            }
          }
        }
        tmem_st8(t_s + at, hi);
        tmem_st8(t_s + at + 8, mid);
        tmem_st8(t_s1 + at, lo);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      warp_arrive(&sm_ready);
      named_sync(1, Plan::kReaders);
      if (t + (int)gridDim.x < g.tasks) write_line(t + gridDim.x);
      // ---- epilogue
      wait_or_fault(&done[kO1], it & 1, &cta, g.fault, kFaultMmaWait);
      tc_fence_after_wait();
      const auto result16 = [&](int c0, uint32_t (&a1)[16]) {   // sixteen results of this thread's row from column c0 on
        uint32_t a2[16];
        __syncwarp();   // (rows past the end are not stored)
        tmem_ld16(t_o1 + lane_base + c0, a1);
        if (k.has_state) tmem_ld16(t_o2 + lane_base + c0, a2);
        tmem_ld_wait();
        if (k.has_state) {
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const F2 x = fma2({w_row, w_row}, pair(a2[j], a2[j + 1]), pair(a1[j], a1[j + 1]));
            a1[j] = __float_as_uint(x.x), a1[j + 1] = __float_as_uint(x.y);
          }
        }
      };
      if constexpr (ADD) {
        T* out = static_cast<T*>(r.out) + (k.tok + row) * r.pitch_z;
        uint32_t again = 0;   // blocks of 16 columns with a result that is not finite
#pragma unroll 1
        for (int c0 = 16 * part; c0 < r.wz; c0 += 16 * kParts) {
          uint32_t a1[16];
          result16(c0, a1);
          if (row < k.len) {
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(a1[j]);
            if (all_finite(a1))
              put16(out + c0, x, r.add != 0);
            else
              again |= 1u << (c0 / 16);
          }
        }
        tc_fence_before_sync();
        warp_arrive(&acc_free);
        if (again) plain_out<T>(&args, t, row, 0, again);   // (here few registers are live)
      } else {
        // 64 bytes of a row at a time: sixteen fp32 results, or two times sixteen
        constexpr int kCols = 64 / (int)sizeof(T), kPer = 16 / (int)sizeof(T);
        const int my_col = (lane & 3) * kPer;
        T* out = static_cast<T*>(r.out) + (k.tok + (row & ~3)) * r.pitch_z + my_col;
        const int rows_left = k.len - (row & ~3);
#pragma unroll 1
        for (int c0 = kCols * part; c0 < r.wz; c0 += kParts * kCols) {
          uint4 v[4];
#pragma unroll
          for (int u = 0; u < kCols / 16; ++u) {
            uint32_t a1[16];
            if (u > 0 && c0 + 16 * u >= r.wz) {
#pragma unroll
              for (int j = 0; j < 16; ++j) a1[j] = 0u;
            } else {
              result16(c0 + 16 * u, a1);
            }
            if (row < k.len && !all_finite(a1)) look_again = 1;
            if constexpr (std::is_same<T, float>::value) {
#pragma unroll
              for (int q = 0; q < 4; ++q) v[q] = make_uint4(a1[4 * q], a1[4 * q + 1], a1[4 * q + 2], a1[4 * q + 3]);
            } else {
              uint32_t h[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) h[j] = pack2(__uint_as_float(a1[2 * j]), __uint_as_float(a1[2 * j + 1]), T());
              v[2 * u] = make_uint4(h[0], h[1], h[2], h[3]), v[2 * u + 1] = make_uint4(h[4], h[5], h[6], h[7]);
            }
          }
          rows_to_lanes(v, lane);
          if (c0 + my_col < r.wz) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i < rows_left) *reinterpret_cast<uint4*>(out + (size_t)i * r.pitch_z + c0) = v[i];
          }
        }
        tc_fence_before_sync();
        warp_arrive(&acc_free);
      }
    }
  } else if constexpr (Plan::kFillXZ) {
    // ---- fillers
    const int ft = (tid - 128 - Plan::kReaders) & (kFillers - 1);
    // what a task's chunks are made of: its first token's rows
    struct Source {
      const T *x, *y, *z;
      int pitch_x, pitch_z, wx, wz, len;
    };
    const auto source_of = [&](int t) {
      const Task k = task_of(t);
      return Source{static_cast<const T*>(k.r.x) + k.tok * k.r.pitch_x, static_cast<const T*>(k.r.y) + k.tok * k.r.pitch_x,
                    static_cast<const T*>(k.r.z) + k.tok * k.r.pitch_z, k.r.pitch_x, k.r.pitch_z, k.r.wx, k.r.wz, k.len};
    };
    const auto chunk_of = [&](const Source& k, int kind) {
      const int c = kind & 1;
      if (kind >= kZ0)
        return tensor_chunk<T>(k.z + (size_t)64 * c * k.pitch_z, k.pitch_z, 64, k.len - 64 * c, k.len > 64 * c ? k.wz : 0, k.wz > 64, ft);
      return tensor_chunk<T>((kind >= kY0 ? k.y : k.x) + 64 * c, k.pitch_x, C, k.len, min(k.wx - 64 * c, 64), false, ft);
    };
    int t = blockIdx.x, it = 0;
    uint32_t u = 0;
    if (t < g.tasks) {
      Source task = source_of(t);
      Chunk cur = chunk_of(task, Plan::kFillOrder & 15), next;
      RawChunk<T> r;
      const auto load_next = [&](int i) { load_chunk_piece<T>(r, next, i); };
#pragma unroll
      for (int i = 0; i < kPieces; ++i) load_chunk_piece<T>(r, cur, i);
      while (true) {
        const int now = (Plan::kFillOrder >> (4 * u)) & 15, it_now = it;
        if (++u == Plan::kFills) {
          u = 0, ++it;
          t += gridDim.x;
          if (t < g.tasks) task = source_of(t);
        }
        next = chunk_of(task, (Plan::kFillOrder >> (4 * u)) & 15);
        if (t >= g.tasks) next.cols = 0;
        await_place(plan_at<Plan::fill_after>(now), it_now);
        store_chunk<T, TT::in>(smem + turned(plan_at<Plan::fill_place>(now), it_now) * kUnit, r, cur, load_next);
        fence_async_smem();
        warp_arrive(&full[now]);
        if (t >= g.tasks) break;
        cur = next;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
  if constexpr (!ADD) {
    // (after the loops, whose registers are all taken; the control warps have given theirs away)
    if (look_again && warp >= 4)
      for (int u = blockIdx.x; u < g.tasks; u += gridDim.x) plain_out_where_needed<T>(&args, u);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
cudaError_t matrix_map(CUtensorMap* map, const void* base, size_t count, int rows, int width, int pitch) {
  const cudaError_t err = make_matrix_map(map, base, count, (uint64_t)rows, (uint32_t)width, (uint32_t)pitch);
  if (err != cudaSuccess) g_failed_step = "tensor map of the full-precision path";
  return err;
}

template <typename T>
cudaError_t launch_states(const Dims& m, const StateArgs& g, cudaStream_t st) {
  CUtensorMap map_b = {};
  cudaError_t err;
  if (StatePlan<T>::kTmaB && (err = matrix_map(&map_b, g.b, (size_t)m.b * m.h, m.n, m.e, m.pitch_e)) != cudaSuccess) return err;
  if ((err = opt_in_smem<k_split_states<T>>(StatePlan<T>::kSmem)) != cudaSuccess) return err;
  const int grid = g.tasks < sm_count() ? g.tasks : sm_count();
  err = launch_following(k_split_states<T>, dim3(grid), kStateThreads, StatePlan<T>::kSmem, st, map_b, g);
  if (err != cudaSuccess) g_failed_step = "launch of the chunk-state kernel";
  return err;
}

template <typename T, bool ADD>
cudaError_t launch_out(const OutMaps& maps, const OutArgs& g, cudaStream_t st) {
  constexpr size_t smem = (size_t)OutPlan<T>::kUnits * kUnit + 1024;
  cudaError_t err = opt_in_smem<k_split_out<T, ADD>>(smem);
  if (err != cudaSuccess) return err;
  const int grid = g.tasks < sm_count() ? g.tasks : sm_count();
  err = launch_following(k_split_out<T, ADD>, dim3(grid), kOutThreads<T>, smem, st, maps, g);
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

namespace {
// the launch of one (o) or three (dq, dk, dv) results; maps only of what the kernels of this type load by TMA
cudaError_t split_outputs(const Dims& m, OutArgs& g, const void* q, const void* k, const void* v, const void* d_o, const void* prefix,
                          const void* suffix, cudaStream_t st) {
  g.h = m.h, g.n = m.n, g.nc = m.nc, g.d = m.d, g.e = m.e, g.tasks = g.roles * m.b * m.h * m.nc;
  cudaError_t err = fault_word_address(&g.fault);
  if (err != cudaSuccess) return err;
  OutMaps maps = {};
  const size_t seqs = (size_t)m.b * m.h;
  for (const auto& [i, p] : {std::pair<int, const void*>{kMapPrefix, prefix}, {kMapSuffix, suffix}})
    if (p && (err = matrix_map(&maps.m[i], p, seqs * m.nc * 3, m.d, m.e, m.e)) != cudaSuccess) return err;
  if (m.dtype != LASP_F32) {
    for (const auto& [i, p] : {std::pair<int, const void*>{kMapQ, q}, {kMapK, k}})
      if ((err = matrix_map(&maps.m[i], p, seqs, m.n, m.d, m.pitch_d)) != cudaSuccess) return err;
    for (const auto& [i, p] : {std::pair<int, const void*>{kMapV, v}, {kMapDo, d_o}})
      if (p && (err = matrix_map(&maps.m[i], p, seqs, m.n, m.e, m.pitch_e)) != cudaSuccess) return err;
  }
  const bool add = g.role[0].add || g.role[1].add || g.role[2].add;
  return by_dtype(m.dtype, [&](auto t) { return add ? launch_out<decltype(t), true>(maps, g, st) : launch_out<decltype(t), false>(maps, g, st); });
}
}  // namespace

cudaError_t split_fwd_output(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                             const void* prefix, void* o, bool alone, bool add_o, cudaStream_t st) {
  if (m.nc == 1 && alone) prefix = nullptr;
  OutArgs g = {};
  g.s = s, g.roles = 1;
  g.role[0] = {q, k, v, o, static_cast<const __nv_bfloat16*>(prefix), kMapQ, kMapK, kMapV, kMapPrefix, m.d, m.e, m.pitch_d, m.pitch_e,
               0, 0, alone ? 0 : -1, add_o};
  return split_outputs(m, g, q, k, v, nullptr, prefix, nullptr, st);
}

cudaError_t split_bwd_grads(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, const float* s,
                            const void* prefix, const void* suffix, void* dq, void* dk, void* dv, bool alone,
                            bool add_qk, bool add_v, cudaStream_t st) {
  if (m.nc == 1 && alone) prefix = suffix = nullptr;
  const int first = alone ? 0 : -1, last = alone ? m.nc - 1 : -1;
  const auto *p = static_cast<const __nv_bfloat16*>(prefix), *dn = static_cast<const __nv_bfloat16*>(suffix);
  OutArgs g = {};
  g.s = s, g.roles = 3;
  g.role[0] = {d_o, v, k, dq, p, kMapDo, kMapV, kMapK, kMapPrefix, m.e, m.d, m.pitch_e, m.pitch_d, 1, 0, first, add_qk};
  g.role[1] = {v, d_o, q, dk, dn, kMapV, kMapDo, kMapQ, kMapSuffix, m.e, m.d, m.pitch_e, m.pitch_d, 1, 1, last, add_qk};
  g.role[2] = {k, q, d_o, dv, dn, kMapK, kMapQ, kMapDo, kMapSuffix, m.d, m.e, m.pitch_d, m.pitch_e, 0, 1, last, add_v};
  return split_outputs(m, g, q, k, v, d_o, prefix, suffix, st);
}

}  // namespace lasp
