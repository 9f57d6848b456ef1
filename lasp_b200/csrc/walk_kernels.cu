// Tensor-core path (tcgen05 MMAs, accumulators in tensor memory, operands staged by TMA) with the
// running KV / dKV state kept ON CHIP.  bf16 inputs, fp32 accumulation, one rounding on store.
//
// A sequence of one (batch, head) is cut into 128-token tiles and the tiles into spans of `span`
// consecutive tiles; a span is the unit of work of a persistent CTA.  Per direction:
//
//   k_span_totals   T_span = sum over the span's tokens of decay * a_j b_j^T  (a,b = k,v or q,do)
//   (scan over the few span totals of a sequence: k_scan of state_kernels.cu, seeded with the rank's
//    incoming state; gives every span its fp32 state at the span border)
//   k_walk_out      walks a span first to last tile with the d x e state in registers (fp32) and in
//                   shared memory (bf16 MMA operand):  OUT = (X Y^T . M) Z + diag(lambda^r) X op(P),
//                   then P <- lambda^C P + K^T diag(w) V.  Forward: (X,Y,Z,OUT) = (Q,K,V,O), op(P)=P;
//                   the same kernel gives dQ with (X,Y,Z,OUT) = (dO,V,K,dQ), op(P)=P^T.
//   k_walk_dkv      walks a span last to first tile with the suffix state Dn on chip: dK, dV.
//
// So K and V (Q and dO) are read twice per direction and nothing else is: no per-tile state is written
// to or read from global memory.  Every tile in shared memory is in the swizzled slab format of
// sm100.cuh; all buffers are 32 KB so that a tile's buffer can be reused for the decay-masked score
// tile and for the staging tile of the TMA store.  All waits are bounded (see tc_common.cuh).
#include <stdio.h>
#include <stdlib.h>

#include "exchange_layout.h"
#include "tc_common.cuh"

namespace lasp {

namespace {

using namespace tc;

constexpr int kBuf = 32768;       // one shared-memory buffer: a 128 x 128 bf16 tile

// Two buffers of a double-buffered tile / two accumulators, addressed by arithmetic: an array of two pointers
// indexed by the tile's parity would live in local memory, and the tile loops look these up all the time.
struct BufPair {
  uint8_t* base;
  __device__ __forceinline__ uint8_t* operator[](int p) const { return base + p * kBuf; }
};
struct TmemPair {
  uint32_t base;
  __device__ __forceinline__ uint32_t operator[](int p) const { return base + p * 128; }
};
template <int G>
struct Group {   // a worker group as a compile-time constant: 0 = A, 1 = B
  static constexpr int value = G;
};
struct IntPair {
  int a, b;
  __device__ __forceinline__ int get(int p) const { return p ? b : a; }
  __device__ __forceinline__ void set(int p, int v) {
    if (p) b = v; else a = v;
  }
};
constexpr int kWorkers = 256;     // threads of one group of eight worker warps
// The walk kernels run five warpgroups: producer and issuer in the first (its other two warps idle), two for each
// worker group.  They are launched with 96 registers a thread (640 x 96 = 61440) and share them out anew: 64 + 2 x 72
// + 2 x 136 per warpgroup of 128 threads, the state being held by group B.
constexpr int kFirstWorker = 128;
constexpr int kThreads = kFirstWorker + 2 * kWorkers;
constexpr int kRegsFront = 64, kRegsA = 72, kRegsB = 136;
static_assert(128 * kRegsFront + kWorkers * kRegsA + kWorkers * kRegsB <= kThreads * 96, "registers of the launch");

// Global-memory image of a d x e span state in lane order (see common.cuh): this thread's part is row
// `row`, columns [col0, col0 + N).
template <int N, int ROWS, bool COHERENT>
__device__ __forceinline__ void load_state(const float* state, int row, int col0, float (&P)[N]) {
  const float4* src = reinterpret_cast<const float4*>(state) + (size_t)(col0 / 4) * ROWS + row;
#pragma unroll
  for (int q = 0; q < N / 4; ++q) {
    const float4 v = COHERENT ? __ldcg(src + (size_t)q * ROWS) : src[(size_t)q * ROWS];
    P[4 * q] = v.x, P[4 * q + 1] = v.y, P[4 * q + 2] = v.z, P[4 * q + 3] = v.w;
  }
}
template <int N, int ROWS>
__device__ __forceinline__ void fma_state(const float* state, int row, int col0, float dec, float (&P)[N]) {
  const float4* src = reinterpret_cast<const float4*>(state) + (size_t)(col0 / 4) * ROWS + row;
  constexpr int kBatch = N / 4 < 8 ? N / 4 : 8;   // loads in flight per thread (registers)
#pragma unroll
  for (int q0 = 0; q0 < N / 4; q0 += kBatch) {
    float4 v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) v[u] = __ldcg(src + (size_t)(q0 + u) * ROWS);   // written by another CTA of this launch
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int q = q0 + u;
      P[4 * q] = fmaf(dec, v[u].x, P[4 * q]), P[4 * q + 1] = fmaf(dec, v[u].y, P[4 * q + 1]);
      P[4 * q + 2] = fmaf(dec, v[u].z, P[4 * q + 2]), P[4 * q + 3] = fmaf(dec, v[u].w, P[4 * q + 3]);
    }
  }
}
template <int N, int ROWS>
__device__ __forceinline__ void store_state(float* state, int row, int col0, const float (&P)[N]) {
  float4* dst = reinterpret_cast<float4*>(state) + (size_t)(col0 / 4) * ROWS + row;
#pragma unroll
  for (int q = 0; q < N / 4; ++q) dst[(size_t)q * ROWS] = make_float4(P[4 * q], P[4 * q + 1], P[4 * q + 2], P[4 * q + 3]);
}
// 32 accumulator columns of this thread's row -> lane-order state
template <int ROWS>
__device__ __forceinline__ void store_state32(float* state, int row, int col0, const uint32_t (&r)[32]) {
  float4* dst = reinterpret_cast<float4*>(state) + (size_t)(col0 / 4) * ROWS + row;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    dst[(size_t)q * ROWS] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                        __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
}


// ---------------------------------------------------------------------------
// span totals: totals[item][i][j] = sum_c w_c A[c][i] B[c][j] over the span's tokens
//   forward  (A,B) = (K,V):  w = lambda^(span end - position)      (decayed to the end of the span)
//   backward (A,B) = (Q,dO): w = lambda^(position - span start)    (decayed to the start of the span)
// Ten warps: warp 0 producer (three-stage ring of A,B tiles), warp 1 tensor-core issuer (accumulator
// double buffered over items), warps 2-5 scale the rows of A in place, warps 6-9 write the totals.
// ---------------------------------------------------------------------------
template <int D, int E>
__global__ void __launch_bounds__(320, 1) k_span_totals(const __grid_constant__ CUtensorMap map_a,
                                                        const __grid_constant__ CUtensorMap map_b,
                                                        const float* __restrict__ s, float* __restrict__ totals,
                                                        int h, int n, const __grid_constant__ SpanCut cut,
                                                              int reverse, int32_t* fault) {
  constexpr int kStages = 3;
  constexpr int kA = C * D * 2, kB = C * E * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  // per stage: A then B (with D = 64 the M = 128 MMA reads on from A into B, which is valid memory)
  __shared__ uint64_t full[kStages], scaled[kStages], empty[kStages], acc_full[2], acc_free[2];
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    cta.word = 0;
    for (int j = 0; j < kStages; ++j) {
      mbar_init(&full[j], 1);
      mbar_init(&scaled[j], 128);
      mbar_init(&empty[j], 1);
    }
    for (int j = 0; j < 2; ++j) {
      mbar_init(&acc_full[j], 1);
      mbar_init(&acc_free[j], 128);
    }
    fence_mbar_init();
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
  }
  if (warp == 2) tmem_alloc(&tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  TileWalk<false> w{cut, false};

  if (warp == 0) {
    if (lane == 0) {
      int g = 0;
      for (bool ok = w.start(); ok; ok = w.next(), ++g) {
        const int j = g % kStages, use = g / kStages;
        if (use >= 1) wait_or_fault(&empty[j], (use - 1) & 1, &cta, fault, kFaultMmaWait);
        uint8_t* sa = smem + j * (kA + kB);
        mbar_expect_tx(&full[j], kA + kB);
        tma_load_4d(sa, &map_a, &full[j], 0, w.t * C, 0, w.bh);
        tma_load_4d(sa + kA, &map_b, &full[j], 0, w.t * C, 0, w.bh);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int g = 0, li = -1;
      for (bool ok = w.start(); ok; ok = w.next(), ++g) {
        const int j = g % kStages, use = g / kStages;
        if (w.first_of_item()) {
          ++li;
          if (li >= 2) wait_or_fault(&acc_free[li & 1], ((li >> 1) - 1) & 1, &cta, fault, kFaultMmaWait);
        }
        wait_or_fault(&scaled[j], use & 1, &cta, fault, kFaultTmaWait);
        tc_fence_after_sync();
        uint8_t* sa = smem + j * (kA + kB);
        umma_gemm<true, true, E, C>(tmem + 128 * (li & 1), smem_u32(sa), C, smem_u32(sa + kA), C, !w.first_of_item());
        umma_commit(&empty[j]);
        if (w.last_of_item()) umma_commit(&acc_full[li & 1]);
      }
    }
  } else if (warp < 6) {
    const int row = tid - 64;  // the token of the tile this thread scales
    int g = 0;
    for (bool ok = w.start(); ok; ok = w.next(), ++g) {
      const int j = g % kStages, use = g / kStages;
      const float sl2 = s[w.bh % h] * kLog2e;
      const int pos = w.t * C + row;
      const int dist = reverse ? pos - w.t0 * C : min(w.t1 * C, n) - pos;
      const float wt = decay_pow(sl2, max(dist, 0));  // rows past the end of the sequence are zero anyway
      wait_or_fault(&full[j], use & 1, &cta, fault, kFaultTmaWait);
      scale_row_pieces<D / 8>(smem + j * (kA + kB), row, 0, wt, lane);
      fence_async_smem();
      mbar_arrive(&scaled[j]);
    }
  } else {
    const int row = (warp & 3) * 32 + lane;  // tensor-memory lane = row of the state; warps 6..9 -> quarters 2,3,0,1
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int li = -1;
    for (bool ok = w.start(); ok; ok = w.next()) {
      if (!w.last_of_item()) continue;
      ++li;
      wait_or_fault(&acc_full[li & 1], (li >> 1) & 1, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      if (row < D) {
#pragma unroll
        for (int c0 = 0; c0 < E; c0 += 32) {
          uint32_t a[32];
          tmem_ld32(tmem + 128 * (li & 1) + lane_base + c0, a);
          tmem_ld_wait();
          store_state32<D>(totals + (size_t)w.it * D * E, row, c0, a);
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&acc_free[li & 1]);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------
// flags between the CTAs of one launch (fused kernels)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_volatile_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// A flag between CTAs of a launch: what its writer's CTA wrote ahead of a barrier before the release is there for everyone
// behind a barrier after the acquire.
__device__ __forceinline__ void st_release_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_inc(uint32_t* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
// spins until *flag == want or `limit` clocks pass
__device__ __forceinline__ bool wait_flag_eq(const uint32_t* flag, uint32_t want, long long limit) {
  if (ld_acquire_u32(flag) == want) return true;
  const long long t0 = clock64();
  while (ld_acquire_u32(flag) != want) {
    if (clock64() - t0 > limit) return false;
  }
  return true;
}

// The peer-mapped buffers of a sequence-parallel group for one direction (word format, slots and
// acknowledgements as in relay_kernels.cu).  With a link the fused kernels hand the rank state over
// themselves: the CTA that owns the last span of a sequence (in walk order) stores the sequence's total
// into the slots of the ranks after this one as soon as the span totals exist, and every CTA adds what
// the ranks before stored here to its border state - one launch per direction computes AND exchanges.
struct Link {
  const uint2* my_slots;                 // local: slots[parity][source][element] of {value, step} words
  uint2* dst_slots[xl::kMaxRanks];       // peer: each destination's slots
  uint32_t* src_acks[xl::kMaxRanks];     // peer: acknowledgement words in each source's memory
  const uint32_t* my_acks;               // local acknowledgement words [destination]
  uint32_t* counters;                    // local: [0] = last completed step
  int ranks;                             // group size; 0 = no link
  int me;                                // this rank's place in the chain order
  long long wait_clocks;
};

__device__ __forceinline__ uint4 ld_volatile_v4(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_volatile_v4(void* p, uint4 v) {
  asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

// Where the two 16-byte halves of the four {value, step} words of float4 chunk g, row `row`, of a
// sequence sit among its slots (in words): per chunk two planes of ROWS x 16 bytes, so that the 32 rows
// of a warp write - and read - 512 contiguous bytes with each instruction.
template <int ROWS>
__device__ __forceinline__ size_t link_word(int g, int row, int plane) {
  return (size_t)g * ROWS * 4 + (size_t)plane * ROWS * 2 + (size_t)row * 2;
}

// This thread's part (row `row`, columns [col0, col0 + N)) of a sequence's outgoing total, dec * P + own,
// written over `own` (the total of the sequence's last span in walk order, which no other CTA reads).
template <int N, int ROWS>
__device__ __forceinline__ void link_make_total(float* own, int row, int col0, float dec, const float (&P)[N]) {
  float4* t = reinterpret_cast<float4*>(own) + (size_t)(col0 / 4) * ROWS + row;
#pragma unroll 4
  for (int q = 0; q < N / 4; ++q) {
    const float4 o = __ldcg(t + (size_t)q * ROWS);
    t[(size_t)q * ROWS] = make_float4(fmaf(dec, P[4 * q], o.x), fmaf(dec, P[4 * q + 1], o.y),
                                      fmaf(dec, P[4 * q + 2], o.z), fmaf(dec, P[4 * q + 3], o.w));
  }
}

// One CTA's share of the sending: of this thread's float4 chunks of the sequence's total, those whose index
// is `part` modulo `parts`, stored as {value, step} words into the slots of every rank after this one
// that the state still reaches.  All CTAs of a sequence send, each its share: one SM alone pushes slowly.
template <int N, int ROWS>
__device__ __forceinline__ void link_send_part(const Link& l, uint32_t step, long long elems, size_t seq_off, int row,
                                               int col0, const float* total, float sn, int part, int parts) {
  const float4* src = reinterpret_cast<const float4*>(total) + (size_t)(col0 / 4) * ROWS + row;
  const int n_dst = l.ranks - 1 - l.me;
#pragma unroll 4
  for (int q = 0; q < N / 4; ++q) {
    if ((col0 / 4 + q) % parts != part) continue;
    const float4 t = __ldcg(src + (size_t)q * ROWS);
    for (int di = 0; di < n_dst; ++di) {
      if (!xl::reaches(sn, di)) break;   // farther ranks are out of reach too
      uint2* out = l.dst_slots[l.me + 1 + di] + xl::slot_offset(step & 1, l.ranks, l.me, elems) + seq_off;
      st_volatile_v4(out + link_word<ROWS>(col0 / 4 + q, row, 0),
                     make_uint4(__float_as_uint(t.x), step, __float_as_uint(t.y), step));
      st_volatile_v4(out + link_word<ROWS>(col0 / 4 + q, row, 1),
                     make_uint4(__float_as_uint(t.z), step, __float_as_uint(t.w), step));
    }
  }
}

// The whole of this thread's part of the total, dec * P + own, straight from registers to the NEXT rank
// only (for sequences whose state reaches no farther: nothing to share out, no detour through memory).
template <int N, int ROWS>
__device__ __forceinline__ void link_send_next(const Link& l, uint32_t step, long long elems, size_t seq_off, int row,
                                               int col0, float dec, const float (&P)[N], const float* own) {
  const float4* src = reinterpret_cast<const float4*>(own) + (size_t)(col0 / 4) * ROWS + row;
  uint2* out = l.dst_slots[l.me + 1] + xl::slot_offset(step & 1, l.ranks, l.me, elems) + seq_off;
#pragma unroll 4
  for (int q = 0; q < N / 4; ++q) {
    const float4 o = __ldcg(src + (size_t)q * ROWS);
    const float4 t = make_float4(fmaf(dec, P[4 * q], o.x), fmaf(dec, P[4 * q + 1], o.y), fmaf(dec, P[4 * q + 2], o.z),
                                 fmaf(dec, P[4 * q + 3], o.w));
    st_volatile_v4(out + link_word<ROWS>(col0 / 4 + q, row, 0),
                   make_uint4(__float_as_uint(t.x), step, __float_as_uint(t.y), step));
    st_volatile_v4(out + link_word<ROWS>(col0 / 4 + q, row, 1),
                   make_uint4(__float_as_uint(t.z), step, __float_as_uint(t.w), step));
  }
}

// P += dec * sum over the ranks before this one of exp(-sn)^(hops) * their total of this sequence, each word
// awaited until it carries `step`.  Returns false when a wait ran out (P is then NaN).
template <int N, int ROWS>
__device__ __forceinline__ bool link_receive(const Link& l, uint32_t step, long long elems, size_t seq_off, int row,
                                             int col0, float dec, float (&P)[N], float sn) {
  bool late = false;
  for (int src = l.me - 1; src >= 0; --src) {
    const int hops = l.me - 1 - src;
    if (!xl::reaches(sn, hops)) break;   // farther ranks are out of reach too
    const float wgt = dec * expf(-sn * (float)hops);
    const uint2* in = l.my_slots + xl::slot_offset(step & 1, l.ranks, src, elems) + seq_off;
    // wait with pauses on this thread's last word before touching the rest: thousands of threads
    // re-reading all their words would only get in the way of the stores that are arriving
    {
      const uint2* p = in + link_word<ROWS>(col0 / 4 + N / 4 - 1, row, 1);
      const long long t0 = clock64();
      while (!late && ld_volatile_v4(p).w != step) {
        __nanosleep(100);
        if (clock64() - t0 > l.wait_clocks) late = true;
      }
    }
    constexpr int kBatch = 4;   // float4 chunks in flight
#pragma unroll
    for (int q0 = 0; q0 < N / 4; q0 += kBatch) {
      uint4 w0[kBatch], w1[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        w0[u] = ld_volatile_v4(in + link_word<ROWS>(col0 / 4 + q0 + u, row, 0));
        w1[u] = ld_volatile_v4(in + link_word<ROWS>(col0 / 4 + q0 + u, row, 1));
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        if (!late && (w0[u].y != step || w0[u].w != step || w1[u].y != step || w1[u].w != step)) {
          const long long t0 = clock64();   // after one wait has run out this thread waits no more
          do {
            w0[u] = ld_volatile_v4(in + link_word<ROWS>(col0 / 4 + q0 + u, row, 0));
            w1[u] = ld_volatile_v4(in + link_word<ROWS>(col0 / 4 + q0 + u, row, 1));
            if (clock64() - t0 > l.wait_clocks) {
              late = true;
              break;
            }
          } while (w0[u].y != step || w0[u].w != step || w1[u].y != step || w1[u].w != step);
        }
        const int j = 4 * (q0 + u);
        P[j] = fmaf(wgt, __uint_as_float(w0[u].x), P[j]);
        P[j + 1] = fmaf(wgt, __uint_as_float(w0[u].z), P[j + 1]);
        P[j + 2] = fmaf(wgt, __uint_as_float(w1[u].x), P[j + 2]);
        P[j + 3] = fmaf(wgt, __uint_as_float(w1[u].z), P[j + 3]);
      }
    }
  }
  if (late) {   // a state that did not arrive must not look like one that did
#pragma unroll
    for (int j = 0; j < N; ++j) P[j] = __int_as_float(0x7fc00000);
  }
  return !late;
}

// spins until *flag >= want (as a step number) or `limit` clocks pass
__device__ __forceinline__ bool wait_flag_ge(const uint32_t* flag, uint32_t want, long long limit) {
  if ((int32_t)(ld_volatile_u32(flag) - want) >= 0) return true;
  const long long t0 = clock64();
  while ((int32_t)(ld_volatile_u32(flag) - want) < 0) {
    if (clock64() - t0 > limit) return false;
  }
  return true;
}

// The span-total phase streams its tiles through a ring over tile buffers that the walk is not using yet: three stages of
// 64 KB (128-wide heads) or four of 48 KB over all six, or four of 32 KB (64-wide heads) over four, whose first is
// BASE, so that the walk's first loads into the other two can come in meanwhile.  With two stages a tile took a load's
// latency and a half: 131072 tokens, 16 heads, forward 414 -> 404 us; 4 x 16 x 4096 tokens, 64-wide, folded
// preprocessing, 86 -> 75 us.
// Where the number of stages is even the worker groups take the tiles in turn; where it is odd each takes half of every
// tile, because a group has to see every phase of a barrier that it waits for.
template <int D, int E, int BASE>
struct Ring {
  static constexpr int kStage = C * (D + E) * 2;
  static constexpr bool kNarrow = D + E == 128;   // over four buffers
  static constexpr int kStages = (kNarrow ? 4 : 6) * kBuf / kStage;
  static constexpr bool kInTurn = kStages % 2 == 0;
  uint8_t* smem;
  __device__ __forceinline__ uint8_t* a(int j) const { return smem + (kNarrow ? BASE : 0) * kBuf + j * kStage; }
  __device__ __forceinline__ uint8_t* b(int j) const { return a(j) + C * D * 2; }
  // a group's share of the row scaling of stage j
  template <int GRP, bool MAP>
  __device__ __forceinline__ void scale(int j, int row, int half, float w, int lane) const {
    if constexpr (kInTurn)
      scale_row_pieces<D / 16, MAP>(a(j), row, half * (D / 16), w, lane);
    else
      scale_row_pieces<D / 32, MAP>(a(j), row, (2 * half + GRP) * (D / 32), w, lane);
  }
};
constexpr int kMaxRing = 4;

struct WalkArgs {
  const float* s;
  const float* p0;     // not fused: fp32 state of every span at its border, [items][D][E] (from the scan)
  float* p0_save;      // fused: where the border states are kept for the backward pass (may be NULL)
  float* totals;       // fused: span totals [items][D][E], exchanged between the CTAs of the launch
  uint32_t* sync;      // fused: [0] launch counter, [1] CTAs done, [kSyncFlags + item] "total written" flags,
                       // [kSyncFlags + kSyncSecondBank + sequence] "sequence total written" flags (4 KB in all)
  const float* x_in;   // fused: incoming rank state (b,h,d,e) or NULL
  float* x_out;        // fused: outgoing rank state (b,h,d,e) or NULL
  int h, n;
  SpanCut cut;
  float qk_scale;      // q and k enter as qk_scale * map(q), qk_scale * map(k)
  int elu;             // map = elu(x) + 1 (otherwise the identity)
  const void* raw;     // backward with a map: q (dQ walk) or k (dK/dV walk) for the chain rule, raw or (PRE = 2) mapped
  int raw_pitch;       // ... and its row pitch in elements
  int even;            // the tiles of a sequence are shared out evenly among its spans (see TileWalk); a fused
                       // forward records it in sync[kSyncEven], the dQ walk reads it from the forward's workspace
  const uint32_t* even_word;   // dQ: where the forward pass recorded how it cut the sequences (NULL: a.even)
  int all_totals;      // fused: the last span of a sequence computes its total too
  int coop;            // fused: every CTA has exactly one span and the CTAs synchronise (several spans per
                       // sequence, or a link)
  int add_out, add_out2;       // the stores of OUT (dK, dV) add to what the tensors hold
  long long wait_clocks;
  int32_t* fault;
  Link link;           // fused: hand the rank state over inside the launch (link.ranks > 0)
};
constexpr int kSyncEven = 2;
constexpr int kSyncFlags = 32;
// A span's flag counts the parts of its total that are there, the launch's number above the count: no launch takes another's
// for its own until the number has gone round, which is 2^27 launches.
constexpr uint32_t kTotalParts = 2 * kWorkers / 32;
__device__ __forceinline__ uint32_t nothing_published(uint32_t step) { return step * 32; }
__device__ __forceinline__ uint32_t published(uint32_t step) { return step * 32 + kTotalParts; }
static_assert(kTotalParts < 32, "the count's bits");
constexpr int kSyncSecondBank = 480;   // [kSyncFlags + kSyncSecondBank + sequence]: "the sequence's total is written"

// bf16 image of this thread's part of the state (row `row`, columns [col0, col0 + N)) in the operand tile
template <int N>
__device__ __forceinline__ void write_state_operand(uint8_t* tile, int rows, int row, int col0, const float (&P)[N]) {
#pragma unroll
  for (int j = 0; j < N; j += 8)
    *reinterpret_cast<uint4*>(tile + tile_offset(row, col0 + j, rows)) =
        make_uint4(pack_bf16(P[j], P[j + 1]), pack_bf16(P[j + 2], P[j + 3]), pack_bf16(P[j + 4], P[j + 5]),
                   pack_bf16(P[j + 6], P[j + 7]));
}

// ---------------------------------------------------------------------------
// walk, first to last tile:  OUT = (X Y^T . M) Z + diag(lambda^r) X op(P);  P <- lambda^C P + K^T diag(w) V
//
//   DQ = false: X,Y = Q,K (width D), Z,OUT = V,O (width E), op(P) = P
//   DQ = true : X,Y = dO,V (width E), Z,OUT = K,dQ (width D), op(P) = P^T
// P is the d x e state in both: fp32 in the registers of the eight group-B warps (thread = one row and
// half of the columns) and bf16 in shared memory as the operand of X op(P).
//
// Shared memory: X, Y, Z double buffered and the state operand, seven 32 KB buffers.  A buffer's life
// inside a tile:  X: tile -> free after S and O2
//                 Y: tile -> (after S) rows scaled in place -> free after L
//                 Z: tile -> free after L and O1 -> staging tile of OUT
// (OUT is staged over Z, which is the last one read: X and Y of the tile after next are on their way early)
// Tensor memory: S (two buffers; the masked scores are packed to bf16 over S itself and feed O1 as its A
// operand from tensor memory), O (X op(P), rows scaled by lambda^r in place, += S_m Z), L = the state update.
//   warp 0 (one lane)  producer: loads, and the TMA stores of the finished staging tiles
//   warps 1-3          tensor-core issuers
//   warps 4-11  (A)    mask of the scores, epilogue
//   warps 12-19 (B)    the state chain: scaling of Y's rows, of O2's rows, state update
// Two groups because one group of eight warps doing all of it was the serial chain of a tile: 5300 clocks against
// the 5600 that its bytes take at the measured HBM rate, with nothing left to make up for the ramps of a launch.
//
// FUSED = false: the state of every span at its border comes from the scan (a.p0).
// FUSED = true : one launch does everything.  With more than one span per sequence every CTA has
//   exactly one span (one CTA per SM at most; each waits for the totals of lower block indexes only).  It first sums its own span,
//   T = sum_c lambda^(span end - c) k_c v_c^T, streaming K and V once through a ring of stages, writes
//   T to global memory and raises a flag; then it adds up the totals of the spans before it (and the
//   incoming rank state) with their decays - that is its border state - and walks.  The last span of a sequence
//   needs no total unless a.all_totals; the outgoing rank state is the state after the last tile of the last span.
//   Tokens and totals that the head's decay has brought below 1e-12 are left out of the sums (reach_tiles: the same
//   line as for the ranks of a group), so on a long sequence only the tiles next to the border are read twice.
// ---------------------------------------------------------------------------
// PRE: what becomes of q and k - 0 nothing, 1 all of it (the map on tiles in shared memory, the scale, the chain rule),
// 2 the scale and the chain rule of q and k that are mapped already
template <int D, int E, bool DQ, bool FUSED, int PRE, bool LINK>
__global__ void __launch_bounds__(kThreads, 1) k_walk_out(const __grid_constant__ CUtensorMap map_x,
                                                     const __grid_constant__ CUtensorMap map_y,
                                                     const __grid_constant__ CUtensorMap map_z,
                                                     const __grid_constant__ CUtensorMap map_out,
                                                     const __grid_constant__ WalkArgs a) {
  static_assert(!(DQ && FUSED), "dQ walks over states the forward pass kept");
  constexpr int WX = DQ ? E : D;  // width of X and Y
  constexpr int WZ = DQ ? D : E;  // width of Z and OUT
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const BufPair sx{smem};
  const BufPair sy{smem + 2 * kBuf};
  const BufPair sz{smem + 4 * kBuf};
  uint8_t* sp = smem + 6 * kBuf;
  using R = Ring<WX, WZ, 2>;
  const R ring{smem};
  __shared__ uint64_t x_full[2], y_full[2], z_full[2], s_full[2], sm_ready[2], o_full[2], o2_full[2], l_full[2], staged[2];
  __shared__ uint64_t p_ready, l_free, o_free, ys_ready, o2s_ready;
  __shared__ uint64_t mapped[2];   // with a feature map: the workers have mapped the tile's X, Y (dQ: Z) in place
  __shared__ uint64_t ring_full[kMaxRing], ring_scaled[kMaxRing], ring_empty[kMaxRing], sum_done;   // the span-total phase
  __shared__ uint32_t tmem_slot, step_s, step_x, even_s;
  __shared__ Health<LINK> cta;
  const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
  int32_t* fault = a.fault;
  // Thread 0 is also the producer: it asks for its first tiles before the CTA-wide barrier below, so that their
  // flight overlaps the rest of the set-up (what it issued is remembered in early_*; only its copy matters).
  bool early_ring = false;
  int early_x = 0;
  if (tid == 0) {
    cta.word = 0;
    // the words this launch reads from global memory, all in flight while the barriers are set up
    const uint32_t ev = a.even_word != nullptr ? ld_volatile_u32(a.even_word) : (uint32_t)a.even;
    uint32_t ss = 0, sx_ = 0;
    if constexpr (FUSED) {
      if (a.coop) ss = ld_volatile_u32(a.sync);
      if (LINK && a.link.ranks > 0) sx_ = ld_volatile_u32(a.link.counters);
    }
    for (int p = 0; p < 2; ++p) {
      mbar_init(&x_full[p], 1);
      mbar_init(&y_full[p], 1);
      mbar_init(&z_full[p], 1);
      mbar_init(&s_full[p], 1);
      mbar_init(&sm_ready[p], kWorkers);
      mbar_init(&o_full[p], 1);
      mbar_init(&o2_full[p], 1);
      mbar_init(&l_full[p], 1);
      mbar_init(&staged[p], kWorkers);
      mbar_init(&mapped[p], 2 * kWorkers);
    }
    if constexpr (FUSED) {
      for (int j = 0; j < R::kStages; ++j) {
        mbar_init(&ring_full[j], 1);
        mbar_init(&ring_scaled[j], (R::kInTurn ? 1 : 2) * kWorkers / 32);
        mbar_init(&ring_empty[j], 1);
      }
    }
    mbar_init(&p_ready, kWorkers);
    mbar_init(&l_free, kWorkers);
    mbar_init(&o_free, kWorkers);
    mbar_init(&ys_ready, kWorkers);
    mbar_init(&o2s_ready, kWorkers);
    mbar_init(&sum_done, 1);
    fence_mbar_init();
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_y);
    prefetch_tensormap(&map_z);
    prefetch_tensormap(&map_out);
    even_s = ev;
    if constexpr (FUSED) {
      step_s = a.coop ? ss + 1 : 0;                              // this launch among those on the workspace
      step_x = LINK && a.link.ranks > 0 ? sx_ + 1 : 0;           // this hand-over in the group
    }
    TileWalk<false> w0{a.cut, ev != 0};
    if (w0.start()) {
      const int sp0 = w0.sp;
      if (FUSED && a.coop && (sp0 < a.cut.nspans - 1 || a.all_totals)) {   // first stage of the span-total ring
        mbar_expect_tx(&ring_full[0], C * (WX + WZ) * 2);
        tma_load_4d(ring.a(0), &map_y, &ring_full[0], 0, (w0.t1 - 1) * C, 0, w0.bh);
        tma_load_4d(ring.b(0), &map_z, &ring_full[0], 0, (w0.t1 - 1) * C, 0, w0.bh);
        early_ring = true;
      } else {                                                          // X of the first tile of the walk
        mbar_expect_tx(&x_full[0], C * WX * 2);
        tma_load_4d(smem, &map_x, &x_full[0], 0, w0.t * C, 0, w0.bh);
        early_x = 1;
      }
    }
  }
  if (warp == 2) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const TmemPair t_s{tmem};
  const uint32_t t_o = tmem + 256, t_l = tmem + 384;
  TileWalk<false> w{a.cut, even_s != 0};
  // the span-total phase: only with several spans per sequence, and then this CTA has one span.  The tiles are
  // summed from the span's end backwards, as far as the head's decay reaches.
  int sums = 0, sum_t1 = 0, my_bh = 0;
  if constexpr (FUSED) {
    if (a.coop && w.start()) {
      my_bh = w.bh;
      sum_t1 = w.t1;
      if (w.sp < a.cut.nspans - 1 || a.all_totals) sums = min(w.t1 - w.t0, reach_tiles(a.s[my_bh % a.h]));
    }
  }

  const int wid = (tid - kFirstWorker) & (kWorkers - 1);   // 0..255 inside the group
  const int row = (warp & 3) * 32 + lane;      // tensor-memory lane quarter of this warp
  const int half = wid >> 7;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  constexpr int kHalfE = E / 2;
  // q and k enter as c * map(q), c * map(k): the map is applied to the tiles in shared memory, c is folded
  // into factors that exist anyway (dQ: the state already carries k's c)
  // (PRE = 0: instantiations without any of this, for callers who bring q and k as they are)
  const float c = PRE ? a.qk_scale : 1.f;
  const bool elu = PRE == 1 && a.elu != 0;           // tiles are mapped here
  const bool slope = PRE != 0 && a.elu != 0;         // results take the map's derivative
  // brings tile j (buffers of parity j & 1) through the feature map once its loads have landed, each group its share
  auto map_tile = [&](int j, auto group) {
    constexpr int grp = decltype(group)::value;
    const int q = j & 1, uq = (j >> 1) & 1;
    if constexpr (!DQ) {
      wait_or_fault(grp ? &y_full[q] : &x_full[q], uq, &cta, fault, kFaultTmaWait);
      scale_row_pieces<WX / 16, true>(grp ? sy[q] : sx[q], row, half * (WX / 16), 1.f, lane);
    } else {
      wait_or_fault(&z_full[q], uq, &cta, fault, kFaultTmaWait);
      scale_row_pieces<WZ / 32, true>(sz[q], row, (2 * half + grp) * (WZ / 32), 1.f, lane);
    }
    fence_async_smem();
    mbar_arrive(&mapped[q]);
  };
  auto span_total = [&](auto group) {
    constexpr int grp = decltype(group)::value;
    if (sums == 0) return;
    // ---- this span's total, written where the CTAs of the later spans find it; the groups take the stages in turn
    const float sl2 = a.s[my_bh % a.h] * kLog2e;
    const int span_end = min(sum_t1 * C, a.n);
#pragma unroll 1
    for (int g = R::kInTurn ? grp : 0; g < sums; g += R::kInTurn ? 2 : 1) {
      const int j = g % R::kStages;
      wait_or_fault(&ring_full[j], (g / R::kStages) & 1, &cta, fault, kFaultTmaWait);
      const float wt = c * decay_pow(sl2, max(span_end - ((sum_t1 - 1 - g) * C + row), 0));
      if (elu)
        ring.template scale<grp, true>(j, row, half, wt, lane);
      else
        ring.template scale<grp, false>(j, row, half, wt, lane);
      fence_async_smem();
      warp_arrive(&ring_scaled[j]);
    }
    wait_or_fault(&sum_done, 0, &cta, fault, kFaultMmaWait);
    tc_fence_after_wait();
    const int c0 = half * kHalfE + grp * 32;
    if (row < D && grp * 32 < kHalfE) {
      uint32_t r[32];
      tmem_ld32(t_l + lane_base + c0, r);
      tmem_ld_wait();
      store_state32<D>(a.totals + (size_t)blockIdx.x * D * E, row, c0, r);
    }
    tc_fence_before_sync();
    named_sync(2, 2 * kWorkers);   // every worker's part of the total is written ...
    if (tid == kFirstWorker) st_release_u32(a.sync + kSyncFlags + blockIdx.x, published(step_s));   // ... and visible before the flag is
  };
  // The three kinds of warps part for good here: each branch sets its registers and is compiled for them.
  if (warp < kFirstWorker / 32) {
    set_regs_dec<kRegsFront>();
    if (warp == 0) {
      if (lane == 0) {
        int x_issued = early_x;
        if (sums > 0) {
#pragma unroll 1
          for (int g = 0; g < sums; ++g) {
            const int j = g % R::kStages, t = sum_t1 - 1 - g;
            if (g >= R::kStages) wait_or_fault(&ring_empty[j], (g / R::kStages - 1) & 1, &cta, fault, kFaultMmaWait);
            if (!(g == 0 && early_ring)) {
              mbar_expect_tx(&ring_full[j], R::kStage);
              tma_load_4d(ring.a(j), &map_y, &ring_full[j], 0, t * C, 0, my_bh);
              tma_load_4d(ring.b(j), &map_z, &ring_full[j], 0, t * C, 0, my_bh);
            }
            if (R::kNarrow && (g == 1 || g == sums - 1)) {
              // X of the first two tiles of the walk can come in during the sums - behind the first ring
              // stages, which every CTA of the launch asks for at the same moment and the sums wait for
#pragma unroll 1
              for (bool ok = x_issued == 0 && w.start(); ok && x_issued < 2; ok = w.next(), ++x_issued) {
                mbar_expect_tx(&x_full[x_issued], C * WX * 2);
                tma_load_4d(sx[x_issued], &map_x, &x_full[x_issued], 0, w.t * C, 0, w.bh);
              }
            }
          }
          wait_or_fault(&sum_done, 0, &cta, fault, kFaultMmaWait);   // the MMAs have read every ring stage
        }
        int i = 0;
        IntPair out_row{0, 0}, out_bh{0, 0};
#pragma unroll 1
        for (bool ok = w.start(); ok; ok = w.next(), ++i) {
          const int p = i & 1, u = i >> 1;
          if (i >= x_issued) {
            if (i >= 2) {   // S, O2 of tile i-2 read X
              wait_or_fault(&s_full[p], (u - 1) & 1, &cta, fault, kFaultMmaWait);
              wait_or_fault(&o2_full[p], (u - 1) & 1, &cta, fault, kFaultMmaWait);
            }
            mbar_expect_tx(&x_full[p], C * WX * 2);
            tma_load_4d(sx[p], &map_x, &x_full[p], 0, w.t * C, 0, w.bh);
          }
          if (i >= 2) wait_or_fault(&l_full[p], (u - 1) & 1, &cta, fault, kFaultMmaWait);   // S, L of tile i-2 read Y
          mbar_expect_tx(&y_full[p], C * WX * 2);
          tma_load_4d(sy[p], &map_y, &y_full[p], 0, w.t * C, 0, w.bh);
          if (i >= 2) {
            // the output of tile i-2 is staged in Z's buffer: store it, then reuse the buffer
            wait_or_fault(&staged[p], (u - 1) & 1, &cta, fault, kFaultMmaWait);
            tma_store_or_add_4d(&map_out, sz[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out);
            bulk_commit();
            bulk_wait_read<0>();
          }
          mbar_expect_tx(&z_full[p], C * WZ * 2);
          tma_load_4d(sz[p], &map_z, &z_full[p], 0, w.t * C, 0, w.bh);
          out_row.set(p, w.t * C);
          out_bh.set(p, w.bh);
        }
#pragma unroll 1
        for (int j = (i >= 2 ? i - 2 : 0); j < i; ++j) {   // the last two tiles
          const int p = j & 1, u = j >> 1;
          wait_or_fault(&staged[p], u & 1, &cta, fault, kFaultMmaWait);
          tma_store_or_add_4d(&map_out, sz[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out);
          bulk_commit();
        }
        bulk_wait_all<0>();
      }
    } else {
      // Three issuing warps, so that no product waits behind another one's issue and none of them has to poll for what is
      // ready.  A whole warp each, an elected lane of which issues (see umma): a thread of its own took 130 to 160 clocks for
      // an instruction of 64.  8 x 32 x 2048 111 / 108 / 170 -> 99 / 94 / 153 us, 3 x 12 x 3001 36.9 / 26.4 / 47.0 -> 35.1 /
      // 26.1 / 43.8, 16 x 16384 71.5 / 53.9 / 98 -> 67.4 / 49.7 / 90:
      //   warp 1  the span total; O2 = X op(P), then O1 = S_m Z on top of the row-scaled O2
      //   warp 2  L = K^T diag(w) V (d x e), the scaled rows being Y's
      //   warp 3  S = X Y^T of the next tile
      const bool leader = elect_one();
      const bool map_xy = PRE == 1 && a.elu && !DQ, map_z = PRE == 1 && a.elu && DQ;
      if (warp == 1 && sums > 0) {
#pragma unroll 1
        for (int g = 0; g < sums; ++g) {
          const int j = g % R::kStages;
          wait_or_fault(&ring_scaled[j], (g / R::kStages) & 1, &cta, fault, kFaultTmaWait);
          tc_fence_after_wait();
          umma_gemm<true, true, E, C>(t_l, smem_u32(ring.a(j)), C, smem_u32(ring.b(j)), C, g > 0, leader);
          if (leader) umma_commit(&ring_empty[j]);
        }
        if (leader) umma_commit(&sum_done);
      }
      int total = 0;
#pragma unroll 1
      for (bool ok = w.start(); ok; ok = w.next()) ++total;
      if (warp == 1) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, ph = (i >> 1) & 1, one = i & 1;
          // the state operand of this tile is written, the epilogue has drained O
          wait_or_fault(&p_ready, one, &cta, fault, kFaultMmaWait);
          if (i >= 1) wait_or_fault(&o_free, one ^ 1, &cta, fault, kFaultMmaWait);
          wait_or_fault(&x_full[p], ph, &cta, fault, kFaultTmaWait);
          if (map_xy) wait_or_fault(&mapped[p], ph, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          if constexpr (!DQ)  // X P: the state tile as [K = d rows] x [N = e columns]
            umma_gemm<false, true, E, D>(t_o, smem_u32(sx[p]), C, smem_u32(sp), D, false, leader);
          else                // X P^T: the state tile as [N = d rows] x [K = e columns]
            umma_gemm<false, false, D, E>(t_o, smem_u32(sx[p]), C, smem_u32(sp), D, false, leader);
          if (leader) umma_commit(&o2_full[p]);
          // the masked scores are read from tensor memory
          wait_or_fault(&sm_ready[p], ph, &cta, fault, kFaultMmaWait);
          wait_or_fault(&z_full[p], ph, &cta, fault, kFaultTmaWait);
          if (map_z) wait_or_fault(&mapped[p], ph, &cta, fault, kFaultMmaWait);
          wait_or_fault(&o2s_ready, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm_ts<true, WZ, 64>(t_o, t_s[p], smem_u32(sz[p]), C, true, leader);
          if (leader) umma_commit(&o_full[p]);
        }
      } else if (warp == 2) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, ph = (i >> 1) & 1, one = i & 1;
          wait_or_fault(&z_full[p], ph, &cta, fault, kFaultTmaWait);
          if (map_z) wait_or_fault(&mapped[p], ph, &cta, fault, kFaultMmaWait);
          if (i >= 1) wait_or_fault(&l_free, one ^ 1, &cta, fault, kFaultMmaWait);   // the state update has read the previous L
          wait_or_fault(&ys_ready, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          if constexpr (!DQ)
            umma_gemm<true, true, E, C>(t_l, smem_u32(sy[p]), C, smem_u32(sz[p]), C, false, leader);
          else
            umma_gemm<true, true, E, C>(t_l, smem_u32(sz[p]), C, smem_u32(sy[p]), C, false, leader);
          if (leader) umma_commit(&l_full[p]);
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, ph = (i >> 1) & 1;
          if (i >= 2) wait_or_fault(&o_full[p], ph ^ 1, &cta, fault, kFaultMmaWait);   // O1 of tile i-2 has read S_m
          wait_or_fault(&x_full[p], ph, &cta, fault, kFaultTmaWait);
          wait_or_fault(&y_full[p], ph, &cta, fault, kFaultTmaWait);
          if (map_xy) wait_or_fault(&mapped[p], ph, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<false, false, C, WX>(t_s[p], smem_u32(sx[p]), C, smem_u32(sy[p]), C, false, leader);
          if (leader) umma_commit(&s_full[p]);
        }
      }
    }
  } else if (warp < (kFirstWorker + kWorkers) / 32) {
    set_regs_dec<kRegsA>();
    const Group<0> grp;
    span_total(grp);
    int total = 0;
    if (elu) {
#pragma unroll 1
      for (bool ok = w.start(); ok; ok = w.next()) ++total;
      if (total > 0) map_tile(0, grp);
    }
    // ---- group A
    const float c_mask = DQ ? c : c * c;
    float sl2 = 0.f, lam = 1.f;
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int p = i & 1, ph = (i >> 1) & 1;
      if (w.first_of_item()) {
        sl2 = a.s[w.bh % a.h] * kLog2e;
        lam = exp2f(-sl2);
      }
      wait_or_fault(&s_full[p], ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      // masked scores, packed to bf16 in place: they are the A operand of O1 straight from tensor memory
#pragma unroll 1
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t packed[16];
        masked_pack32<false>(t_s[p] + lane_base + half * 64 + cc * 32, row, half * 64 + cc * 32, sl2, lam, packed, c_mask);
        tmem_st16(t_s[p] + lane_base + half * 64 + cc * 16, packed);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(&sm_ready[p]);
      if (elu && i + 1 < total) map_tile(i + 1, grp);   // the next tile's S can then go out under this tile's work
      // dq = dq' * c * map'(q), q (PRE = 2: mapped) read from its tensor (rows past the end of the sequence are not stored)
      const bool chain = PRE && DQ && (slope || c != 1.f);
      const bool live = row < a.n - w.t * C;
      const __nv_bfloat16* raw = nullptr;
      uint4 raw_x[4];
      if (PRE && DQ && slope) {
        raw = static_cast<const __nv_bfloat16*>(a.raw) + ((size_t)w.bh * a.n + (size_t)w.t * C + (live ? row : 0)) * a.raw_pitch;
        raw_row32(raw_x, raw, half * (WZ / 2));
      }
      // epilogue: OUT staged in Z's buffer, once L and O1 have read it
      wait_or_fault(&l_full[p], ph, &cta, fault, kFaultMmaWait);
      wait_or_fault(&o_full[p], ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      if (chain) {
#pragma unroll 1
        for (int cc = 0; cc < WZ / 64; ++cc) {
          const int col0 = half * (WZ / 2) + cc * 32;
          stage_row32_chain<PRE == 2>(t_o + lane_base + col0, sz[p], row, col0, raw_x, c, slope && live);
          if (WZ > 64 && cc == 0 && slope) raw_row32(raw_x, raw, col0 + 32);
        }
      } else {
#pragma unroll 1
        for (int cc = 0; cc < WZ / 64; ++cc) {
          const int col0 = half * (WZ / 2) + cc * 32;
          stage_row32(t_o + lane_base + col0, sz[p], row, col0);
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&o_free);
      fence_async_smem();
      mbar_arrive(&staged[p]);
    }
  } else {
    set_regs_inc<kRegsB>();
    const Group<1> grp;
    span_total(grp);
    int total = 0;
    if (elu) {
#pragma unroll 1
      for (bool ok = w.start(); ok; ok = w.next()) ++total;
      if (total > 0) map_tile(0, grp);
    }
    // ---- group B
    const float c_o2 = DQ ? 1.f : c;
    float P[kHalfE];  // this thread's part of the state: row `row`, columns [half * E/2, (half+1) * E/2)
    float sl2 = 0.f;
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int p = i & 1, ph = (i >> 1) & 1;
      const int len = min(C, a.n - w.t * C);     // tokens really in the tile
      if (w.first_of_item()) sl2 = a.s[w.bh % a.h] * kLog2e;
      wait_or_fault(&s_full[p], ph, &cta, fault, kFaultMmaWait);   // S has read Y
      wait_or_fault(&y_full[p], ph, &cta, fault, kFaultTmaWait);   // completed long ago: makes Y's bytes visible here
      scale_row_pieces<WX / 16>(sy[p], row, half * (WX / 16), c * decay_pow(sl2, max(len - row, 0)), lane);
      fence_async_smem();
      mbar_arrive(&ys_ready);
      if (elu && i + 1 < total) map_tile(i + 1, grp);
      if (__builtin_expect(w.first_of_item(), 0)) {   // once per span: kept out of the tiles' straight-line code
        // the state at the span border; the O2 MMA that read the operand tile of the previous item has completed
        if constexpr (!FUSED) {
          if (row < D) load_state<kHalfE, D, false>(a.p0 + (size_t)w.it * D * E, row, half * kHalfE, P);
        } else {
          const int sp_idx = w.sp;
          const size_t mine = (size_t)row * E + half * kHalfE;
          // incoming rank state, decayed from the first token of the sequence to the first of the span
          if (a.x_in != nullptr && row < D) {
            const float dec = decay_pow(sl2, w.t0 * C);
            const float4* src = reinterpret_cast<const float4*>(a.x_in + (size_t)w.bh * D * E + mine);
#pragma unroll
            for (int j = 0; j < kHalfE / 4; ++j) {
              const float4 v = src[j];
              P[4 * j] = dec * v.x, P[4 * j + 1] = dec * v.y, P[4 * j + 2] = dec * v.z, P[4 * j + 3] = dec * v.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < kHalfE; ++j) P[j] = 0.f;
          }
          // totals of the spans before this one (each decayed to its own end) that still reach this one; one
          // thread per flag
          const int reach = reach_tiles(a.s[w.bh % a.h]);
          int first = sp_idx;
          while (first > 0 && w.t0 - w.span_t0(first) < reach) --first;
          if (wid < sp_idx && wid >= first && !cta.gave_up()) {
            if (!wait_flag_eq(a.sync + kSyncFlags + w.bh * a.cut.nspans + wid, published(step_s), a.wait_clocks)) {
              cta.give_up();
              atomicOr(fault, kFaultFlagWait);
            }
          }
          named_sync(1, kWorkers);
#pragma unroll 1
          for (int j = first; j < sp_idx; ++j) {   // each total is decayed to the end of its span
            if (row < D)
              fma_state<kHalfE, D>(a.totals + (size_t)(w.bh * a.cut.nspans + j) * D * E, row, half * kHalfE,
                                   decay_pow(sl2, (w.t0 - w.span_t0(j + 1)) * C), P);
          }
          if (LINK && a.link.ranks > 0) {
            // hand-over of the rank state inside the launch.  P holds the local part of the border state.
            // The waits for peers below may take longer than any other (a.link.wait_clocks).
            if (wid == 0) cta.peer_wait_begins();
            const float sn = a.s[w.bh % a.h] * (float)a.n;
            const long long elems = (long long)(a.cut.items / a.cut.nspans) * D * E;
            const size_t seq_off = (size_t)w.bh * D * E;
            const int n_dst = a.link.ranks - 1 - a.link.me;
            if (n_dst > 0) {
              const int owner = w.bh * a.cut.nspans + a.cut.nspans - 1;   // the CTA that owns the end of the sequence
              const bool far = n_dst > 1 && xl::reaches(sn, 1);   // the state reaches beyond the next rank
              uint32_t* ready = a.sync + kSyncFlags + kSyncSecondBank + w.bh;
              if (w.it == owner && far) {
                // the sequence's total, lambda^(n - start) P + T, where the other CTAs of the sequence find it
                if (row < D)
                  link_make_total<kHalfE, D>(a.totals + (size_t)owner * D * E, row, half * kHalfE,
                                             decay_pow(sl2, a.n - w.t0 * C), P);
                named_sync(1, kWorkers);
                if (wid == 0) st_release_u32(ready, step_s);
              }
              if (far || w.it == owner) {
                // the readers of the ranks after this one have acknowledged the slots' previous use
                if (!cta.gave_up()) {
                  bool ok2 = true;
                  if (xl::needs_ack_wait(step_x) && wid < n_dst)
                    ok2 = wait_flag_ge(a.link.my_acks + xl::ack_index(a.link.me + 1 + wid, 0), step_x - 2,
                                       a.link.wait_clocks);
                  if (far && wid == xl::kMaxRanks && w.it != owner) ok2 = wait_flag_eq(ready, step_s, a.link.wait_clocks);
                  if (!ok2) {
                    cta.give_up();
                    atomicOr(fault, kFaultRelayWait);
                  }
                }
                named_sync(1, kWorkers);
                if (row < D) {
                  if (far)   // several destinations: every CTA of the sequence sends its share
                    link_send_part<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                              a.totals + (size_t)owner * D * E, sn, sp_idx, a.cut.nspans);
                  else       // the next rank only: straight from the owner's registers
                    link_send_next<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                              decay_pow(sl2, a.n - w.t0 * C), P, a.totals + (size_t)owner * D * E);
                }
              }
            }
            if (a.link.me > 0 && row < D) {
              // what the ranks before this one sent, decayed from the first token of the sequence to the span
              if (!link_receive<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                           decay_pow(sl2, w.t0 * C), P, sn))
                atomicOr(fault, kFaultRelayWait);
            }
            named_sync(1, kWorkers);
            if (wid == 0) cta.peer_wait_ends();
          }
        }
        if (row < D) write_state_operand<kHalfE>(sp, D, row, half * kHalfE, P);
        fence_async_smem();
        mbar_arrive(&p_ready);
        if constexpr (FUSED) {   // kept for the backward pass
          if (a.p0_save != nullptr && row < D) store_state<kHalfE, D>(a.p0_save + (size_t)w.it * D * E, row, half * kHalfE, P);
        }
      }
      // O2's rows take their decay lambda^row in tensor memory; O1 then accumulates on top
      wait_or_fault(&o2_full[p], ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      {
        const float qd = c_o2 * decay_pow(sl2, row);
#pragma unroll 1
        for (int cc = 0; cc < WZ / 64; ++cc) scale_tmem32(t_o + lane_base + half * (WZ / 2) + cc * 32, qd);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(&o2s_ready);
      // state: P <- lambda^len P + L
      wait_or_fault(&l_full[p], ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      if (row < D) {
        const float lam_c = decay_pow(sl2, len);
#pragma unroll
        for (int c0 = 0; c0 < kHalfE; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(t_l + lane_base + half * kHalfE + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const F2 v = fma2({lam_c, lam_c}, {P[c0 + j], P[c0 + j + 1]}, pair(r[j], r[j + 1]));
            P[c0 + j] = v.x, P[c0 + j + 1] = v.y;
          }
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&l_free);
      if (!w.last_of_item()) {
        if (row < D) write_state_operand<kHalfE>(sp, D, row, half * kHalfE, P);
        fence_async_smem();
        mbar_arrive(&p_ready);
      } else if constexpr (FUSED) {
        // the state after the last tile of the sequence is the outgoing rank state
        if (a.x_out != nullptr && w.t == a.cut.tiles - 1 && row < D) {
          float4* dst = reinterpret_cast<float4*>(a.x_out + (size_t)w.bh * D * E + (size_t)row * E + half * kHalfE);
#pragma unroll
          for (int q = 0; q < kHalfE / 4; ++q) dst[q] = make_float4(P[4 * q], P[4 * q + 1], P[4 * q + 2], P[4 * q + 3]);
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
  if constexpr (!DQ) {   // how this pass cut the sequences, for the dQ walk over the border states it leaves
    if (tid == 0 && blockIdx.x == 0 && a.sync != nullptr) st_volatile_u32(a.sync + kSyncEven, even_s);
  }
  if constexpr (FUSED) {
    // the last CTA to finish advances the launch counter: the flags of this launch are stale from then on;
    // with a link it also tells the ranks before this one that their words have been read (they may
    // overwrite them two hand-overs later) and completes the hand-over
    if (tid == 0 && a.coop) {
      __threadfence();
      if (atomicAdd(a.sync + 1, 1u) == gridDim.x - 1) {
        st_volatile_u32(a.sync + 1, 0u);
        __threadfence();
        st_volatile_u32(a.sync, step_s);
        if (LINK && a.link.ranks > 0) {
          for (int q = 0; q < a.link.me; ++q) st_volatile_u32(a.link.src_acks[q] + xl::ack_index(a.link.me, 0), step_x);
          st_volatile_u32(a.link.counters, step_x);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// walk, last to first tile, with the suffix state Dn (d x e) on chip:
//   dK = dS_m^T Q + diag(lambda^(len-c)) V Dn^T
//   dV = S_m^T dO + diag(lambda^(len-c)) K Dn
//   Dn <- lambda^len Dn + Q^T diag(lambda^r) dO          (len = tokens in the tile, 128 but for a ragged tail)
//
// Shared memory: Q, dO double buffered, K, V, the state operand: seven 32 KB buffers.
//   Q, dO: tile -> (after the last product that reads them) staging tiles of dK, dV
//   K, V : free after the four products of the next lines that read them, so the next tile's are on their way early
//   Dn   : state operand -> (after the state products) row-scaled copy of Q for the state update -> new state operand
// Tensor memory, four 128-column regions:
//   T_S : S^T = K Q^T   -> masked and packed to bf16 in place, queries 0..63 in columns [0,32), 64..127 in [96,128),
//                          the A operand of S_m^T dO; the columns between hold the left half of L = Q_s^T dO
//   T_dS: dS^T = V dO^T -> the same for dS_m^T Q and the right half of L
//   T_dK: V Dn^T, rows scaled  -> += dS_m^T Q                  = dK
//   T_dV: K Dn, rows scaled    -> += S_m^T dO                  = dV
// Roles as in k_walk_out:
//   warp 0 producer;  warp 1 state products, then the two products on top of them;  warp 2 L;  warp 3 S^T, dS^T
//   warps 4-11 (A)  masks, epilogue;  warps 12-19 (B)  scaling, copy of Q, state update
// With one group of eight warps, masked scores in shared memory and Q, dO single buffered, a tile was a chain of
// 9300 clocks in which products and workers took turns; its bytes take 8400 at the measured HBM rate.
//
// FUSED: as in k_walk_out - the CTA first sums its span, T = sum_r lambda^(r - span start) q_r do_r^T,
// through the Q and dO buffers, publishes it, adds up the totals of the LATER spans of its sequence (and
// the incoming rank state) and walks; the outgoing rank state is the state after the first tile of the
// sequence.
// ---------------------------------------------------------------------------
template <int D, int E, bool FUSED, int PRE, bool LINK>
__global__ void __launch_bounds__(kThreads, 1) k_walk_dkv(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
    const __grid_constant__ CUtensorMap map_dk, const __grid_constant__ CUtensorMap map_dv,
    const __grid_constant__ WalkArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  const BufPair sq{smem};
  const BufPair sdo{smem + 2 * kBuf};
  uint8_t* sk = smem + 4 * kBuf;
  uint8_t* sv = smem + 5 * kBuf;
  uint8_t* sdn = smem + 6 * kBuf;
  using R = Ring<D, E, 0>;
  const R ring_buf{smem};
  __shared__ uint64_t qdo_full[2], staged[2];
  __shared__ uint64_t kv_full, dn_ready, st_done, s_done, ds_done, sm_ready, dsm_ready, qs_ready, scaled, l_done, l_free, b_done, e_free;
  __shared__ uint64_t mapped;   // with a feature map: the workers have mapped the tile's Q and K in place
  __shared__ uint64_t ring_full[kMaxRing], ring_scaled[kMaxRing], ring_empty[kMaxRing], sum_done, total_read;   // the span-total phase
  __shared__ uint32_t tmem_slot, step_s, step_x;
  __shared__ Health<LINK> cta;
  const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
  int32_t* fault = a.fault;
  // this CTA's span among all spans (the places of a sequence count down, see span_of_place)
  const auto item_of = [&](int bh) { return (2 * bh + 1) * a.cut.nspans - 1 - (int)blockIdx.x; };
  // thread 0 is also the producer: its first loads go out before the CTA-wide barrier (see k_walk_out)
  bool early_ring = false, early_q = false;
  if (tid == 0) {
    cta.word = 0;
    uint32_t ss = 0, sx_ = 0;   // in flight while the barriers are set up
    if constexpr (FUSED) {
      if (a.coop) ss = ld_volatile_u32(a.sync);
      if (LINK && a.link.ranks > 0) sx_ = ld_volatile_u32(a.link.counters);
    }
    for (int p = 0; p < 2; ++p) {
      mbar_init(&qdo_full[p], 1);
      mbar_init(&staged[p], kWorkers);
    }
    if constexpr (FUSED) {
      for (int j = 0; j < R::kStages; ++j) {
        mbar_init(&ring_full[j], 1);
        mbar_init(&ring_scaled[j], (R::kInTurn ? 1 : 2) * kWorkers / 32);
        mbar_init(&ring_empty[j], 1);
      }
    }
    mbar_init(&mapped, 2 * kWorkers);
    mbar_init(&kv_full, 1);
    mbar_init(&st_done, 1);
    mbar_init(&s_done, 1);
    mbar_init(&ds_done, 1);
    mbar_init(&l_done, 1);
    mbar_init(&b_done, 1);
    mbar_init(&sum_done, 1);
    mbar_init(&total_read, 2 * kWorkers / 32);
    mbar_init(&dn_ready, kWorkers);
    mbar_init(&sm_ready, kWorkers);
    mbar_init(&dsm_ready, kWorkers);
    mbar_init(&qs_ready, kWorkers);
    mbar_init(&scaled, kWorkers);
    mbar_init(&l_free, kWorkers);
    mbar_init(&e_free, kWorkers);
    fence_mbar_init();
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    prefetch_tensormap(&map_do);
    prefetch_tensormap(&map_dk);
    prefetch_tensormap(&map_dv);
    if constexpr (FUSED) {
      step_s = a.coop ? ss + 1 : 0;                              // this launch among those on the workspace
      step_x = LINK && a.link.ranks > 0 ? sx_ + 1 : 0;           // this hand-over in the group
    }
    TileWalk<true> w0{a.cut, a.even != 0};
    if (w0.start()) {
      const bool ring = FUSED && a.coop && (w0.sp > 0 || a.all_totals);
      const int t = ring ? w0.t0 : w0.t;   // first stage of the span-total ring, or Q, dO of the walk's first tile
      if (ring) st_volatile_u32(a.sync + kSyncFlags + item_of(w0.bh), nothing_published(step_s));
      uint64_t* bar = ring ? &ring_full[0] : &qdo_full[0];
      mbar_expect_tx(bar, C * (D + E) * 2);
      tma_load_4d(sq[0], &map_q, bar, 0, t * C, 0, w0.bh);   // (where the first ring stage begins too)
      tma_load_4d(ring ? ring_buf.b(0) : sdo[0], &map_do, bar, 0, t * C, 0, w0.bh);
      early_ring = ring;
      early_q = !ring;
    }
  }
  if (warp == 2) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t t_s = tmem, t_ds = tmem + 128, t_dk = tmem + 256, t_dv = tmem + 384;
  TileWalk<true> w{a.cut, a.even != 0};
  // the span-total phase (see k_walk_out): from the span's start onwards, as far as the head's decay reaches
  int sums = 0, sum_t0 = 0, my_bh = 0;
  if constexpr (FUSED) {
    if (a.coop && w.start()) {
      my_bh = w.bh;
      sum_t0 = w.t0;
      if (w.sp > 0 || a.all_totals) sums = min(w.t1 - w.t0, reach_tiles(a.s[my_bh % a.h]));
    }
  }
  const auto my_item = [&] { return item_of(my_bh); };   // (not kept in a register)
  const int row = (warp & 3) * 32 + lane;      // workers: tensor-memory lane quarter of this warp
  const int wid = (tid - kFirstWorker) & (kWorkers - 1);   // 0..255 inside the group
  const int half = wid >> 7;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  constexpr int kHalfE = E / 2;
  // q and k enter as c * map(q), c * map(k): the map is applied to the tiles in shared memory, c is folded
  // into factors that exist anyway
  // (PRE = 0: instantiations without any of this, for callers who bring q and k as they are)
  const float c = PRE ? a.qk_scale : 1.f;
  const bool elu = PRE == 1 && a.elu != 0;
  const bool slope = PRE != 0 && a.elu != 0;
  auto span_total = [&](auto group) {
    constexpr int grp = decltype(group)::value;
    if (sums == 0) return;
    const float sl2 = a.s[my_bh % a.h] * kLog2e;
#pragma unroll 1
    for (int g = R::kInTurn ? grp : 0; g < sums; g += R::kInTurn ? 2 : 1) {
      const int j = g % R::kStages;
      wait_or_fault(&ring_full[j], (g / R::kStages) & 1, &cta, fault, kFaultTmaWait);
      const float wt = c * decay_pow(sl2, g * C + row);
      if (elu)
        ring_buf.template scale<grp, true>(j, row, half, wt, lane);
      else
        ring_buf.template scale<grp, false>(j, row, half, wt, lane);
      fence_async_smem();
      warp_arrive(&ring_scaled[j]);
    }
    wait_or_fault(&sum_done, 0, &cta, fault, kFaultMmaWait);
    tc_fence_after_wait();
    const int c0 = half * kHalfE + grp * 32;
    if (row < D && grp * 32 < kHalfE) {
      uint32_t r[32];
      tmem_ld32(t_s + lane_base + c0, r);
      tmem_ld_wait();
      store_state32<D>(a.totals + (size_t)my_item() * D * E, row, c0, r);
    }
    tc_fence_before_sync();
    warp_arrive(&total_read);      // (S^T takes the total's place in tensor memory)
    // Every warp releases its own part, so that they wait for their stores side by side: the flag is complete with the last
    // one.  24 x 2048 tokens, 128/128 and 128/64, 25.2 / 21.4 us; released by one thread behind a fence of each and a barrier 26.0 /
    // 23.0; behind the barrier alone 26.6 / 22.8; a fence of each, a barrier and a plain store, which is no release, 25.4 / 22.0.
    // (The forward pass, whose totals are further from its first tile's work: even.)  The barrier orders nothing: without it the
    // compiler spills more in the 64-wide kernels with a chain rule (64 x 4096 tokens 71.4 -> 78.9 us).
    __syncwarp();
    if (lane == 0) red_release_inc(a.sync + kSyncFlags + my_item());
    named_sync(2, 2 * kWorkers);
  };

  if (warp < kFirstWorker / 32) {
    set_regs_dec<kRegsFront>();
    if (warp == 0) {
      if (lane == 0) {
        bool kv_issued = false;
        if (sums > 0) {
#pragma unroll 1
          for (int g = 0; g < sums; ++g) {
            const int j = g % R::kStages, t = sum_t0 + g;
            if (g >= R::kStages) wait_or_fault(&ring_empty[j], (g / R::kStages - 1) & 1, &cta, fault, kFaultMmaWait);
            if (!(g == 0 && early_ring)) {
              mbar_expect_tx(&ring_full[j], R::kStage);
              tma_load_4d(ring_buf.a(j), &map_q, &ring_full[j], 0, t * C, 0, my_bh);
              tma_load_4d(ring_buf.b(j), &map_do, &ring_full[j], 0, t * C, 0, my_bh);
            }
            // K, V of the first tile of the walk can come in during the sums, behind the first ring stages
            if (R::kNarrow && (g == 1 || g == sums - 1) && !kv_issued && w.start()) {
              mbar_expect_tx(&kv_full, C * (D + E) * 2);
              tma_load_4d(sk, &map_k, &kv_full, 0, w.t * C, 0, w.bh);
              tma_load_4d(sv, &map_v, &kv_full, 0, w.t * C, 0, w.bh);
              kv_issued = true;
            }
          }
          wait_or_fault(&sum_done, 0, &cta, fault, kFaultMmaWait);   // the MMAs have read every ring stage
        }
        int i = 0;
        IntPair out_row{0, 0}, out_bh{0, 0};
#pragma unroll 1
        for (bool ok = w.start(); ok; ok = w.next(), ++i) {
          const int p = i & 1, u = i >> 1;
          if (i >= 2) {
            // dK and dV of tile i-2 are staged in this parity's Q and dO buffers
            wait_or_fault(&staged[p], (u - 1) & 1, &cta, fault, kFaultMmaWait);
            tma_store_or_add_4d(&map_dk, sq[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out);
            tma_store_or_add_4d(&map_dv, sdo[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out2);
            bulk_commit();
            bulk_wait_read<0>();
          }
          if (!(i == 0 && early_q)) {
            mbar_expect_tx(&qdo_full[p], C * (D + E) * 2);
            tma_load_4d(sq[p], &map_q, &qdo_full[p], 0, w.t * C, 0, w.bh);
            tma_load_4d(sdo[p], &map_do, &qdo_full[p], 0, w.t * C, 0, w.bh);
          }
          if (i >= 1) {   // K, V of tile i-1 are read
            wait_or_fault(&s_done, (i - 1) & 1, &cta, fault, kFaultMmaWait);
            wait_or_fault(&ds_done, (i - 1) & 1, &cta, fault, kFaultMmaWait);
            wait_or_fault(&st_done, (i - 1) & 1, &cta, fault, kFaultMmaWait);
          }
          if (i >= 1 || !kv_issued) {
            mbar_expect_tx(&kv_full, C * (D + E) * 2);
            tma_load_4d(sk, &map_k, &kv_full, 0, w.t * C, 0, w.bh);
            tma_load_4d(sv, &map_v, &kv_full, 0, w.t * C, 0, w.bh);
          }
          out_row.set(p, w.t * C);
          out_bh.set(p, w.bh);
        }
#pragma unroll 1
        for (int j = (i >= 2 ? i - 2 : 0); j < i; ++j) {   // the last two tiles
          const int p = j & 1, u = j >> 1;
          wait_or_fault(&staged[p], u & 1, &cta, fault, kFaultMmaWait);
          tma_store_or_add_4d(&map_dk, sq[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out);
          tma_store_or_add_4d(&map_dv, sdo[p], 0, out_row.get(p), 0, out_bh.get(p), a.add_out2);
          bulk_commit();
        }
        bulk_wait_all<0>();
      }
    } else {
      const bool leader = elect_one();   // (see k_walk_out)
      if (warp == 1 && sums > 0) {
#pragma unroll 1
        for (int g = 0; g < sums; ++g) {
          const int j = g % R::kStages;
          wait_or_fault(&ring_scaled[j], (g / R::kStages) & 1, &cta, fault, kFaultTmaWait);
          tc_fence_after_wait();
          umma_gemm<true, true, E, C>(t_s, smem_u32(ring_buf.a(j)), C, smem_u32(ring_buf.b(j)), C, g > 0, leader);
          if (leader) umma_commit(&ring_empty[j]);
        }
        if (leader) umma_commit(&sum_done);
      }
      int total = 0;
#pragma unroll 1
      for (bool ok = w.start(); ok; ok = w.next()) ++total;
      if (warp == 1) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, one = i & 1;
          // the state tile as [N = d rows] x [K = e columns] (V Dn^T) and as [K = d rows] x [N = e columns] (K Dn);
          // the epilogue has drained T_dK, T_dV
          wait_or_fault(&kv_full, one, &cta, fault, kFaultTmaWait);
          if (elu) wait_or_fault(&mapped, one, &cta, fault, kFaultMmaWait);
          wait_or_fault(&dn_ready, one, &cta, fault, kFaultMmaWait);
          if (i >= 1) wait_or_fault(&e_free, one ^ 1, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<false, false, D, E>(t_dk, smem_u32(sv), C, smem_u32(sdn), D, false, leader);
          umma_gemm<false, true, E, D>(t_dv, smem_u32(sk), C, smem_u32(sdn), D, false, leader);
          if (leader) umma_commit(&st_done);
          // the masked scores' products on top, A operands from tensor memory
          wait_or_fault(&sm_ready, one, &cta, fault, kFaultMmaWait);
          wait_or_fault(&scaled, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm_ts<true, E, 96>(t_dv, t_s, smem_u32(sdo[p]), C, true, leader);    // += S_m^T dO
          wait_or_fault(&dsm_ready, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm_ts<true, D, 96>(t_dk, t_ds, smem_u32(sq[p]), C, true, leader);    // += dS_m^T Q
          if (leader) umma_commit(&b_done);
        }
      } else if (warp == 2) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, one = i & 1;
          // L = Q_s^T dO in the columns that the packed scores leave free; the scaled copy of Q is in the state
          // operand's buffer
          wait_or_fault(&sm_ready, one, &cta, fault, kFaultMmaWait);
          if (E > 64) wait_or_fault(&dsm_ready, one, &cta, fault, kFaultMmaWait);
          wait_or_fault(&qs_ready, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<true, true, 64, C>(t_s + 32, smem_u32(sdn), C, smem_u32(sdo[p]), C, false, leader);
          if constexpr (E > 64)   // columns 64..127 of dO: its second slab
            umma_gemm<true, true, 64, C>(t_ds + 32, smem_u32(sdn), C, smem_u32(sdo[p]) + C * kSlabRowBytes, C, false, leader);
          if (leader) umma_commit(&l_done);
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int p = i & 1, one = i & 1;
          if (i >= 1) {   // the masked scores and L of tile i-1 have been read
            wait_or_fault(&b_done, one ^ 1, &cta, fault, kFaultMmaWait);
            wait_or_fault(&l_free, one ^ 1, &cta, fault, kFaultMmaWait);
          } else if (sums > 0) {
            wait_or_fault(&total_read, 0, &cta, fault, kFaultMmaWait);
          }
          wait_or_fault(&qdo_full[p], (i >> 1) & 1, &cta, fault, kFaultTmaWait);
          wait_or_fault(&kv_full, one, &cta, fault, kFaultTmaWait);
          if (elu) wait_or_fault(&mapped, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<false, false, C, D>(t_s, smem_u32(sk), C, smem_u32(sq[p]), C, false, leader);
          if (leader) umma_commit(&s_done);
          umma_gemm<false, false, C, E>(t_ds, smem_u32(sv), C, smem_u32(sdo[p]), C, false, leader);
          if (leader) umma_commit(&ds_done);
        }
      }
    }
  } else if (warp < (kFirstWorker + kWorkers) / 32) {
    // ---- group A
    set_regs_dec<kRegsA>();
    span_total(Group<0>());
    float sl2 = 0.f, lam = 1.f;
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int p = i & 1, one = i & 1;
      if (w.first_of_item()) {
        sl2 = a.s[w.bh % a.h] * kLog2e;
        lam = exp2f(-sl2);
      }
      if (elu) {   // K of this tile through the feature map before any product reads it
        wait_or_fault(&kv_full, one, &cta, fault, kFaultTmaWait);
        scale_row_pieces<D / 16, true>(sk, row, half * (D / 16), 1.f, lane);
        fence_async_smem();
        mbar_arrive(&mapped);
      }
      // S_m^T, then dS_m^T (times Q's c): one piece of code for the four blocks of 32 queries.  The second half of the
      // queries goes from right to left, packed against the right end, so that every block is read before it is
      // written over.
#pragma unroll 1
      for (int u = 0; u < 4; ++u) {
        if ((u & 1) == 0) {
          wait_or_fault(u == 0 ? &s_done : &ds_done, one, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
        }
        const int blk = half == 0 ? (u & 1) : 3 - (u & 1);
        const uint32_t t = (u < 2 ? t_s : t_ds) + lane_base;
        uint32_t packed[16];
        masked_pack32<true>(t + 32 * blk, row, 32 * blk, sl2, lam, packed, u < 2 ? c * c : c);
        tmem_st16(t + (half == 0 ? 16 * blk : 96 + 16 * (blk - 2)), packed);
        if ((u & 1) == 1) {
          tmem_st_wait();
          tc_fence_before_sync();
          mbar_arrive(u == 1 ? &sm_ready : &dsm_ready);
        }
      }
      // dk = dk' * c * map'(k), k (PRE = 2: mapped) read from its tensor (rows past the end of the sequence are not stored)
      const bool live = row < a.n - w.t * C;
      const __nv_bfloat16* raw = nullptr;
      uint4 raw_x[4];
      if (PRE && slope) {
        raw = static_cast<const __nv_bfloat16*>(a.raw) + ((size_t)w.bh * a.n + (size_t)w.t * C + (live ? row : 0)) * a.raw_pitch;
        raw_row32(raw_x, raw, half * (D / 2));
      }
      // epilogue: dK and dV staged over Q and dO, which every product has read
      wait_or_fault(&l_done, one, &cta, fault, kFaultMmaWait);
      wait_or_fault(&b_done, one, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      if (PRE && (slope || c != 1.f)) {
#pragma unroll 1
        for (int cc = 0; cc < D / 64; ++cc) {
          const int col0 = half * (D / 2) + cc * 32;
          stage_row32_chain<PRE == 2>(t_dk + lane_base + col0, sq[p], row, col0, raw_x, c, slope && live);
          if (D > 64 && cc == 0 && slope) raw_row32(raw_x, raw, col0 + 32);
        }
      }
      // dV's blocks, and dK's too unless the chain rule above has staged them: one loop
#pragma unroll 1
      for (int u = (slope || c != 1.f) ? D / 64 : 0; u < D / 64 + E / 64; ++u) {
        const bool dv_part = u >= D / 64;
        const int cc = dv_part ? u - D / 64 : u;
        const int col0 = half * ((dv_part ? E : D) / 2) + cc * 32;
        stage_row32((dv_part ? t_dv : t_dk) + lane_base + col0, (dv_part ? sdo : sq)[p], row, col0);
      }
      tc_fence_before_sync();
      mbar_arrive(&e_free);
      fence_async_smem();
      mbar_arrive(&staged[p]);
    }
  } else {
    // ---- group B
    set_regs_inc<kRegsB>();
    span_total(Group<1>());
    float Dn[kHalfE];  // this thread's part of the suffix state: row `row`, columns [half * E/2, (half+1) * E/2)
    float sl2 = 0.f;
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int p = i & 1, one = i & 1;
      const int len = min(C, a.n - w.t * C);
      if (__builtin_expect(w.first_of_item(), 0)) {   // once per span: kept out of the tiles' straight-line code
        sl2 = a.s[w.bh % a.h] * kLog2e;
        if constexpr (!FUSED) {
          if (row < D) load_state<kHalfE, D, false>(a.p0 + (size_t)w.it * D * E, row, half * kHalfE, Dn);
        } else {
          const int sp_idx = w.sp;
          const int span_end = min(w.t1 * C, a.n);
          const size_t mine = (size_t)row * E + half * kHalfE;
          // incoming rank state, decayed from the end of the sequence to the end of the span
          if (a.x_in != nullptr && row < D) {
            const float dec = decay_pow(sl2, a.n - span_end);
            const float4* src = reinterpret_cast<const float4*>(a.x_in + (size_t)w.bh * D * E + mine);
#pragma unroll
            for (int j = 0; j < kHalfE / 4; ++j) {
              const float4 v = src[j];
              Dn[4 * j] = dec * v.x, Dn[4 * j + 1] = dec * v.y, Dn[4 * j + 2] = dec * v.z, Dn[4 * j + 3] = dec * v.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < kHalfE; ++j) Dn[j] = 0.f;
          }
          // totals of the spans after this one (each decayed to its own start) that still reach this one; one thread
          // per flag
          const int reach = reach_tiles(a.s[w.bh % a.h]);
          int past = sp_idx + 1;
          while (past < a.cut.nspans && w.span_t0(past) - w.t1 < reach) ++past;
          if (wid < past - 1 - sp_idx && !cta.gave_up()) {
            if (!wait_flag_eq(a.sync + kSyncFlags + w.bh * a.cut.nspans + sp_idx + 1 + wid, published(step_s), a.wait_clocks)) {
              cta.give_up();
              atomicOr(fault, kFaultFlagWait);
            }
          }
          named_sync(1, kWorkers);
#pragma unroll 1
          for (int j = sp_idx + 1; j < past; ++j) {   // each total is decayed to the start of its span
            if (row < D)
              fma_state<kHalfE, D>(a.totals + (size_t)(w.bh * a.cut.nspans + j) * D * E, row, half * kHalfE,
                                   decay_pow(sl2, (w.span_t0(j) - w.t1) * C), Dn);
          }
          if (LINK && a.link.ranks > 0) {
            // hand-over of the rank state inside the launch.  Dn holds the local part of the border state.
            // The waits for peers below may take longer than any other (a.link.wait_clocks).
            if (wid == 0) cta.peer_wait_begins();
            const float sn = a.s[w.bh % a.h] * (float)a.n;
            const long long elems = (long long)(a.cut.items / a.cut.nspans) * D * E;
            const size_t seq_off = (size_t)w.bh * D * E;
            const int n_dst = a.link.ranks - 1 - a.link.me;
            if (n_dst > 0) {
              const int owner = w.bh * a.cut.nspans;   // the CTA that owns the start of the sequence
              const bool far = n_dst > 1 && xl::reaches(sn, 1);   // the state reaches beyond the next rank
              uint32_t* ready = a.sync + kSyncFlags + kSyncSecondBank + w.bh;
              if (sp_idx == 0 && far) {
                // the sequence's total, lambda^(span end) Dn + T, where the other CTAs of the sequence find it
                if (row < D)
                  link_make_total<kHalfE, D>(a.totals + (size_t)owner * D * E, row, half * kHalfE,
                                             decay_pow(sl2, span_end), Dn);
                named_sync(1, kWorkers);
                if (wid == 0) st_release_u32(ready, step_s);
              }
              if (far || sp_idx == 0) {
                // the readers of the ranks after this one in the chain order (the ranks BEFORE it in the
                // sequence) have acknowledged the slots' previous use
                if (!cta.gave_up()) {
                  bool ok2 = true;
                  if (xl::needs_ack_wait(step_x) && wid < n_dst)
                    ok2 = wait_flag_ge(a.link.my_acks + xl::ack_index(a.link.me + 1 + wid, 0), step_x - 2,
                                       a.link.wait_clocks);
                  if (far && wid == xl::kMaxRanks && sp_idx != 0) ok2 = wait_flag_eq(ready, step_s, a.link.wait_clocks);
                  if (!ok2) {
                    cta.give_up();
                    atomicOr(fault, kFaultRelayWait);
                  }
                }
                named_sync(1, kWorkers);
                if (row < D) {
                  if (far)
                    link_send_part<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                              a.totals + (size_t)owner * D * E, sn, sp_idx, a.cut.nspans);
                  else
                    link_send_next<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                              decay_pow(sl2, span_end), Dn, a.totals + (size_t)owner * D * E);
                }
              }
            }
            if (a.link.me > 0 && row < D) {
              // what came from the ranks after this one in the sequence, decayed from its end to the span's
              if (!link_receive<kHalfE, D>(a.link, step_x, elems, seq_off, row, half * kHalfE,
                                           decay_pow(sl2, a.n - span_end), Dn, sn))
                atomicOr(fault, kFaultRelayWait);
            }
            named_sync(1, kWorkers);
            if (wid == 0) cta.peer_wait_ends();
          }
        }
        // the MMAs that read the operand tile of the previous item have completed (l_done was waited for)
        if (row < D) write_state_operand<kHalfE>(sdn, D, row, half * kHalfE, Dn);
        fence_async_smem();
        mbar_arrive(&dn_ready);
      }
      wait_or_fault(&qdo_full[p], (i >> 1) & 1, &cta, fault, kFaultTmaWait);
      if (elu) {   // Q of this tile through the feature map before any product reads it
        scale_row_pieces<D / 16, true>(sq[p], row, half * (D / 16), 1.f, lane);
        fence_async_smem();
        mbar_arrive(&mapped);
      }
      wait_or_fault(&st_done, one, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      // row-scaled copy of Q over the state operand (the state products have read it)
      copy_row_pieces<D / 16>(sdn, sq[p], row, half * (D / 16), c * decay_pow(sl2, row), lane);
      fence_async_smem();
      mbar_arrive(&qs_ready);
      // the two state products take their row decay in place (32 columns at a time, dV's blocks then dK's)
      const float kd = decay_pow(sl2, max(len - row, 0));
#pragma unroll 1
      for (int u = 0; u < D / 64 + E / 64; ++u) {
        const bool dk_part = u >= E / 64;
        const int cc = dk_part ? u - E / 64 : u;
        scale_tmem32((dk_part ? t_dk + half * (D / 2) : t_dv + half * (E / 2)) + lane_base + cc * 32, dk_part ? kd : kd * c);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(&scaled);
      // state: Dn <- lambda^len Dn + L, this thread's half of the columns being the one in T_S or in T_dS
      wait_or_fault(&l_done, one, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      if (row < D) {
        const float lam_len = decay_pow(sl2, len);
        const uint32_t t_l = lane_base + 32 + (E > 64 ? (half ? t_ds : t_s) : t_s + half * 32);
#pragma unroll
        for (int c0 = 0; c0 < kHalfE; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(t_l + c0, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const F2 v = fma2({lam_len, lam_len}, {Dn[c0 + j], Dn[c0 + j + 1]}, pair(r[j], r[j + 1]));
            Dn[c0 + j] = v.x, Dn[c0 + j + 1] = v.y;
          }
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&l_free);
      if (!w.last_of_item()) {
        if (row < D) write_state_operand<kHalfE>(sdn, D, row, half * kHalfE, Dn);
        fence_async_smem();
        mbar_arrive(&dn_ready);
      } else if constexpr (FUSED) {
        // the state after the first tile of the sequence is the outgoing rank state
        if (a.x_out != nullptr && w.t == 0 && row < D) {
          float4* dst = reinterpret_cast<float4*>(a.x_out + (size_t)w.bh * D * E + (size_t)row * E + half * kHalfE);
#pragma unroll
          for (int q = 0; q < kHalfE / 4; ++q) dst[q] = make_float4(Dn[4 * q], Dn[4 * q + 1], Dn[4 * q + 2], Dn[4 * q + 3]);
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
  if constexpr (FUSED) {
    if (tid == 0 && a.coop) {
      __threadfence();
      if (atomicAdd(a.sync + 1, 1u) == gridDim.x - 1) {
        st_volatile_u32(a.sync + 1, 0u);
        __threadfence();
        st_volatile_u32(a.sync, step_s);
        if (LINK && a.link.ranks > 0) {
          for (int q = 0; q < a.link.me; ++q) st_volatile_u32(a.link.src_acks[q] + xl::ack_index(a.link.me, 0), step_x);
          st_volatile_u32(a.link.counters, step_x);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
cudaError_t seq_map(CUtensorMap* map, const void* base, const Dims& m, int width, int pitch, const char* what) {
  cudaError_t err = make_seq_tile_map(map, base, (uint64_t)m.b * m.h, (uint64_t)m.n, (uint32_t)width, C, (uint32_t)pitch);
  if (err != cudaSuccess) {
    static thread_local char text[160];
    snprintf(text, sizeof(text), "tensor map (%s): CUresult %d, base %p, b*h %d, n %d, width %d", what,
             last_encode_result(), base, m.b * m.h, m.n, width);
    g_failed_step = text;
  }
  return err;
}

cudaError_t launched(const char* what) {
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) g_failed_step = what;
  return err;
}

int grid_for(int items) {
  const int sms = sm_count();
  return items < sms ? items : sms;
}

template <int D, int E>
cudaError_t launch_span_totals(const Dims& m, const void* a, const void* bten, const float* s, float* totals,
                               bool reverse, cudaStream_t st) {
  CUtensorMap ma, mb;
  cudaError_t err;
  if ((err = seq_map(&ma, a, m, D, m.pitch_d, "span totals, first operand")) != cudaSuccess) return err;
  if ((err = seq_map(&mb, bten, m, E, m.pitch_e, "span totals, second operand")) != cudaSuccess) return err;
  int32_t* fault = nullptr;
  if ((err = fault_word_address(&fault)) != cudaSuccess) return err;
  const size_t smem = (size_t)3 * C * (D + E) * 2 + 1024;
  if ((err = opt_in_smem<k_span_totals<D, E>>(smem)) != cudaSuccess) return err;
  const int items = m.b * m.h * m.nc;
  k_span_totals<D, E><<<grid_for(items), 320, smem, st>>>(ma, mb, s, totals, m.h, m.n,
                                                          make_span_cut(items, m.nc, m.span, m.tiles), reverse ? 1 : 0, fault);
  return launched("launch of the span-total kernel");
}

// The CTAs of a fused launch wait for one another's totals.  They are at most one per SM (the host side
// checks), so all of them become resident as soon as whatever ran before has drained; their waits are
// bounded all the same and report through the fault word.
template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(void (*kernel)(KArgs...), int grid, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

constexpr long long kFlagWaitClocks = 1000000000LL;   // about half a second

template <int D, int E, bool DQ, bool FUSED, int PRE, bool LINK>
cudaError_t launch_walk_out_pre(const Dims& m, const void* x, const void* y, const void* z, void* out, WalkArgs a,
                            cudaStream_t st) {
  constexpr int WX = DQ ? E : D, WZ = DQ ? D : E;
  CUtensorMap mx, my, mz, mo;
  cudaError_t err;
  if ((err = seq_map(&mx, x, m, WX, DQ ? m.pitch_e : m.pitch_d, DQ ? "do" : "q")) != cudaSuccess) return err;
  if ((err = seq_map(&my, y, m, WX, DQ ? m.pitch_e : m.pitch_d, DQ ? "v" : "k")) != cudaSuccess) return err;
  if ((err = seq_map(&mz, z, m, WZ, DQ ? m.pitch_d : m.pitch_e, DQ ? "k" : "v")) != cudaSuccess) return err;
  if ((err = seq_map(&mo, out, m, WZ, DQ ? m.pitch_d : m.pitch_e, DQ ? "dq" : "o")) != cudaSuccess) return err;
  if ((err = fault_word_address(&a.fault)) != cudaSuccess) return err;
  const size_t smem = (size_t)7 * kBuf + 1024;
  if ((err = opt_in_smem<k_walk_out<D, E, DQ, FUSED, PRE, LINK>>(smem)) != cudaSuccess) return err;
  a.h = m.h, a.n = m.n, a.cut = make_span_cut(m.b * m.h * m.nc, m.nc, m.span, m.tiles);
  a.wait_clocks = kFlagWaitClocks;
  a.qk_scale = m.qk_scale, a.elu = m.qk_map, a.raw_pitch = m.pitch_d;
  const bool waits = FUSED && (m.nc > 1 || a.link.ranks > 0);   // CTAs wait for one another: one span each, all resident
  a.coop = waits ? 1 : 0;
  if (waits) a.even = 1;
  if (a.link.ranks > 0 && a.link.me < a.link.ranks - 1) a.all_totals = 1;   // the sequence totals are sent on
  if (waits && a.cut.items > sm_count()) {
    g_failed_step = "fused walk kernel: more spans than SMs";
    return cudaErrorInvalidConfiguration;
  }
  if ((err = launch_kernel(k_walk_out<D, E, DQ, FUSED, PRE, LINK>, grid_for(a.cut.items), kThreads, smem, st, mx, my, mz, mo, a)) !=
      cudaSuccess) {
    g_failed_step = "launch of a walk kernel";
    return err;
  }
  return launched(DQ ? "launch of the dq walk kernel" : "launch of the forward walk kernel");
}

template <int D, int E, bool FUSED, int PRE, bool LINK>
cudaError_t launch_walk_dkv_pre(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, void* dk,
                            void* dv, WalkArgs a, cudaStream_t st) {
  CUtensorMap mq, mk, mv, mdo, mdk, mdv;
  cudaError_t err;
  if ((err = seq_map(&mq, q, m, D, m.pitch_d, "q")) != cudaSuccess) return err;
  if ((err = seq_map(&mk, k, m, D, m.pitch_d, "k")) != cudaSuccess) return err;
  if ((err = seq_map(&mv, v, m, E, m.pitch_e, "v")) != cudaSuccess) return err;
  if ((err = seq_map(&mdo, d_o, m, E, m.pitch_e, "do")) != cudaSuccess) return err;
  if ((err = seq_map(&mdk, dk, m, D, m.pitch_d, "dk")) != cudaSuccess) return err;
  if ((err = seq_map(&mdv, dv, m, E, m.pitch_e, "dv")) != cudaSuccess) return err;
  if ((err = fault_word_address(&a.fault)) != cudaSuccess) return err;
  a.raw = k;   // for the chain rule of a folded k preprocessing
  const size_t smem = (size_t)7 * kBuf + 1024;
  if ((err = opt_in_smem<k_walk_dkv<D, E, FUSED, PRE, LINK>>(smem)) != cudaSuccess) return err;
  a.h = m.h, a.n = m.n, a.cut = make_span_cut(m.b * m.h * m.nc, m.nc, m.span, m.tiles);
  a.wait_clocks = kFlagWaitClocks;
  a.qk_scale = m.qk_scale, a.elu = m.qk_map, a.raw_pitch = m.pitch_d;
  const bool waits = FUSED && (m.nc > 1 || a.link.ranks > 0);
  a.coop = waits ? 1 : 0;
  if (waits) a.even = 1;
  if (a.link.ranks > 0 && a.link.me < a.link.ranks - 1) a.all_totals = 1;
  if (waits && a.cut.items > sm_count()) {
    g_failed_step = "fused walk kernel: more spans than SMs";
    return cudaErrorInvalidConfiguration;
  }
  if ((err = launch_kernel(k_walk_dkv<D, E, FUSED, PRE, LINK>, grid_for(a.cut.items), kThreads, smem, st, mq, mk, mv, mdo, mdk, mdv, a)) !=
      cudaSuccess) {
    g_failed_step = "launch of the dk/dv walk kernel";
    return err;
  }
  return launched("launch of the dk/dv walk kernel");
}

// the instantiations with the q,k preprocessing only where it is asked for: the others keep the short code
template <int D, int E, bool DQ, bool FUSED>
cudaError_t launch_walk_out(const Dims& m, const void* x, const void* y, const void* z, void* out, WalkArgs a,
                            cudaStream_t st) {
  // ... and the hand-over code only in the launches of a sequence-parallel rank
  const bool linked = a.link.ranks > 0;
  if (has_qk_preprocessing(m)) {
    const bool map_tiles = m.qk_map == LASP_QK_ELU1;
    if constexpr (FUSED) {
      if (linked) return launch_walk_out_pre<D, E, DQ, true, 1, true>(m, x, y, z, out, a, st);
      if (map_tiles) return launch_walk_out_pre<D, E, DQ, true, 1, false>(m, x, y, z, out, a, st);
      return m.qk_scale == 1.f ? launch_walk_out_pre<D, E, DQ, true, 0, false>(m, x, y, z, out, a, st)   // mapped: nothing is left to do
                               : launch_walk_out_pre<D, E, DQ, true, 2, false>(m, x, y, z, out, a, st);
    } else if constexpr (DQ) {
      return map_tiles ? launch_walk_out_pre<D, E, true, false, 1, false>(m, x, y, z, out, a, st)
                       : launch_walk_out_pre<D, E, true, false, 2, false>(m, x, y, z, out, a, st);
    }
    g_failed_step = "q,k preprocessing is not part of the phase-by-phase schedule";
    return cudaErrorInvalidValue;
  }
  if constexpr (FUSED) {
    if (linked) return launch_walk_out_pre<D, E, DQ, true, 0, true>(m, x, y, z, out, a, st);
  }
  return launch_walk_out_pre<D, E, DQ, FUSED, 0, false>(m, x, y, z, out, a, st);
}
template <int D, int E, bool FUSED>
cudaError_t launch_walk_dkv(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, void* dk,
                            void* dv, WalkArgs a, cudaStream_t st) {
  const bool linked = a.link.ranks > 0;
  if (has_qk_preprocessing(m)) {
    if constexpr (FUSED) {
      if (linked) return launch_walk_dkv_pre<D, E, true, 1, true>(m, q, k, v, d_o, dk, dv, a, st);
      return m.qk_map == LASP_QK_ELU1 ? launch_walk_dkv_pre<D, E, true, 1, false>(m, q, k, v, d_o, dk, dv, a, st)
                                      : launch_walk_dkv_pre<D, E, true, 2, false>(m, q, k, v, d_o, dk, dv, a, st);
    }
    g_failed_step = "q,k preprocessing is not part of the phase-by-phase schedule";
    return cudaErrorInvalidValue;
  }
  if constexpr (FUSED) {
    if (linked) return launch_walk_dkv_pre<D, E, true, 0, true>(m, q, k, v, d_o, dk, dv, a, st);
  }
  return launch_walk_dkv_pre<D, E, FUSED, 0, false>(m, q, k, v, d_o, dk, dv, a, st);
}

}  // namespace

#define LASP_DISPATCH_DE(m, CALL)                                        \
  do {                                                                    \
    if ((m).d == 128 && (m).e == 128) return CALL(128, 128);              \
    if ((m).d == 128 && (m).e == 64) return CALL(128, 64);                \
    if ((m).d == 64 && (m).e == 128) return CALL(64, 128);                \
    if ((m).d == 64 && (m).e == 64) return CALL(64, 64);                  \
    return cudaErrorInvalidValue;                                         \
  } while (0)

cudaError_t walk_span_totals(const Dims& m, const void* a, const void* bten, const float* s, float* totals,
                             bool reverse, cudaStream_t st) {
#define LASP_CALL(DD, EE) launch_span_totals<DD, EE>(m, a, bten, s, totals, reverse, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

cudaError_t walk_fwd_output(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                            const float* prefix, uint32_t* sync, void* o, bool add_o, cudaStream_t st) {
  WalkArgs a = {};
  a.add_out = add_o;
  a.s = s, a.p0 = prefix, a.sync = sync;   // sync: only the word that says how the sequences were cut
#define LASP_CALL(DD, EE) launch_walk_out<DD, EE, false, false>(m, q, k, v, o, a, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

// the walk kernels' view of the caller's peer-mapped buffers (NULL: no link)
static Link make_link(const lasp_exchange_args* x) {
  Link l = {};
  if (x == nullptr) return l;
  l.my_slots = static_cast<const uint2*>(x->my_slots);
  l.my_acks = x->my_acks;
  l.counters = x->counters;
  for (int i = 0; i < xl::kMaxRanks; ++i) {
    l.src_acks[i] = x->peer_acks[i];
    l.dst_slots[i] = static_cast<uint2*>(x->peer_slots[i]);
  }
  l.ranks = x->ranks;
  l.me = x->position;
  l.wait_clocks = x->wait_clocks > 0 ? x->wait_clocks : 20000000000LL;   // about ten seconds
  return l;
}

cudaError_t walk_fwd_fused(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                           const float* x_in, float* x_out, uint32_t* sync, float* totals, float* prefix, void* o,
                           const lasp_exchange_args* link, bool add_o, cudaStream_t st) {
  WalkArgs a = {};
  a.add_out = add_o;
  a.link = make_link(link);
  a.s = s, a.x_in = x_in, a.x_out = x_out, a.sync = sync, a.totals = totals, a.p0_save = prefix;
#define LASP_CALL(DD, EE) launch_walk_out<DD, EE, false, true>(m, q, k, v, o, a, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

cudaError_t walk_bwd_dq(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, const float* s,
                        const float* prefix, const uint32_t* fwd_sync, bool even, void* dq, bool add_dq, cudaStream_t st) {
  WalkArgs a = {};
  a.add_out = add_dq;
  a.s = s, a.p0 = prefix, a.even = even;   // the sequences are cut as the forward pass did
  if (fwd_sync != nullptr) a.even_word = fwd_sync + kSyncEven;
  a.raw = q;                                                    // for the chain rule of a folded q preprocessing
#define LASP_CALL(DD, EE) launch_walk_out<DD, EE, true, false>(m, d_o, v, k, dq, a, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

cudaError_t walk_bwd_dkv(const Dims& m, const void* q, const void* k, const void* v, const void* d_o,
                         const float* s, const float* suffix, void* dk, void* dv, bool add_dk, bool add_dv,
                         cudaStream_t st) {
  WalkArgs a = {};
  a.add_out = add_dk, a.add_out2 = add_dv;
  a.s = s, a.p0 = suffix;
#define LASP_CALL(DD, EE) launch_walk_dkv<DD, EE, false>(m, q, k, v, d_o, dk, dv, a, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

cudaError_t walk_bwd_dkv_fused(const Dims& m, const void* q, const void* k, const void* v, const void* d_o,
                               const float* s, const float* x_in, float* x_out, uint32_t* sync, float* totals,
                               void* dk, void* dv, const lasp_exchange_args* link, bool add_dk, bool add_dv,
                               cudaStream_t st) {
  WalkArgs a = {};
  a.add_out = add_dk, a.add_out2 = add_dv;
  a.link = make_link(link);
  a.s = s, a.x_in = x_in, a.x_out = x_out, a.sync = sync, a.totals = totals;
#define LASP_CALL(DD, EE) launch_walk_dkv<DD, EE, true>(m, q, k, v, d_o, dk, dv, a, st)
  LASP_DISPATCH_DE(m, LASP_CALL);
#undef LASP_CALL
}

}  // namespace lasp
