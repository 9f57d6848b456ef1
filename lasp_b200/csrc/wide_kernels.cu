// Heads of 256 (q, k and v alike) on the tensor-core path in one pass per result: bf16 operands, fp32 accumulation and state,
// as in walk_kernels.cu.
//
// Cut in 128-wide slices (the general way) such a call is four operators, each of which reads its slices of all inputs and
// adds its contribution to results in memory: every input and every result moves four times, and the scores of the two
// q,k slices are rounded, masked and applied one by one.  Here a CTA walks a sequence tile by tile for 128 columns of one
// result, the state that those need, 256 x 128, being on chip:
//
//   OUT = (X Y^T . M) Z + diag(w_out) X G;   G <- lambda^len G + Y^T diag(w_in) Z
//
//   o   : X, Y, Z = Q, K, V slice       first to last tile      w_out = lambda^r,        w_in = lambda^(len - r)
//   dq  : X, Y, Z = dO, V, K slice      first to last
//   dk  : X, Y, Z = V, dO, Q slice      last to first, M transposed, w_out = lambda^(len - r), w_in = lambda^r
//   dv  : X, Y, Z = K, Q, dO slice      last to first
//
// One launch forward, one backward: an item is a sequence, a result and a half of its columns, so that the CTAs that read the
// same tiles are neighbours and HBM sees each tile once or twice.  Nothing is kept for the backward pass: its walks start
// at the ends of the sequences.
//
// What bounds it: the chain of a tile (S, mask, O1, state update and operand, all tiles of a step in single buffers: X, Y,
// the state operand 64 KB each, Z 32 KB), then HBM.  A tile takes 5400 clocks, 3584 of them tensor work, for 192 KB.  b=4, h=16,
// n=4096, no decay, slices and now: forward 326 -> 138 us, training 984 -> 476 (1044 -> 544 under the power cap); with decay 306 -> 162
// and 934 -> 556.  Error against fp64 2.3e-3 to 3.1e-3 -> 1.7e-3 to 2.4e-3.  The next tile's X, Y, Z asked into L2 ahead: 8 % slower.
#include "tc_common.cuh"

namespace lasp {
namespace {

using namespace tc;

constexpr int W = 256, N = 128;               // width of X and Y; columns of Z, OUT
constexpr int kWide = C * W * 2, kNarrow = C * N * 2;
// Four warpgroups: producer and issuers (warps 0-3); A, masks and results (warps 4-7); B, the state (warps 8-15), 128 fp32
// numbers in the registers of each of its threads.  Launched with 128 registers a thread.
constexpr int kThreadsA = 128, kThreadsB = 256, kThreads = 128 + kThreadsA + kThreadsB;
constexpr int kRegsFront = 40, kRegsA = 104, kRegsB = 184;
static_assert(128 * kRegsFront + kThreadsA * kRegsA + kThreadsB * kRegsB <= kThreads * 128, "registers of the launch");

enum Tensor { kQ, kK, kV, kDo, kInputs, kDq = kInputs, kDk, kDv, kTensors };   // o takes dq's place in a forward launch
struct WideRole {
  int x, y, z, out, backwards;
};
struct WideMaps {
  CUtensorMap m[kInputs];
};
struct WideArgs {
  WideRole role[3];
  int roles, items, h, n, tiles;
  const float* s;
  __nv_bfloat16* out[kTensors];   // results by their place among the tensors
  int32_t* fault;
};

// the tiles of a persistent CTA's items: item = (sequence, role, half of the columns)
struct Walk {
  const WideArgs& a;
  int it, bh, half, t;
  WideRole r;
  __device__ __forceinline__ bool load() {
    if (it >= a.items) return false;
    half = it & 1;
    const int u = it >> 1;
    bh = u / a.roles;
    r = a.role[u - bh * a.roles];
    t = r.backwards ? a.tiles - 1 : 0;
    return true;
  }
  __device__ __forceinline__ bool start() {
    it = blockIdx.x;
    return load();
  }
  __device__ __forceinline__ bool next() {
    if (r.backwards ? --t >= 0 : ++t < a.tiles) return true;
    it += gridDim.x;
    return load();
  }
  __device__ __forceinline__ bool first() const { return t == (r.backwards ? a.tiles - 1 : 0); }
  __device__ __forceinline__ bool last() const { return t == (r.backwards ? 0 : a.tiles - 1); }
};

__global__ void __launch_bounds__(kThreads, 1) k_walk_wide(const __grid_constant__ WideMaps maps, const __grid_constant__ WideArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sx = align1024(smem_raw);
  uint8_t* sy = sx + kWide;
  uint8_t* sz = sy + kWide;
  uint8_t* sh = sz + kNarrow;   // the state as an operand: G^T, 128 rows (columns of Z) of 256
  __shared__ uint64_t x_full, y_full, z_full, s_done, sm_ready, o2_done, o2_scaled, o_done, o_free, ys_ready, l_done, l_free, g_ready;
  __shared__ uint32_t tmem_slot;
  __shared__ Health<false> cta;
  const int tid = threadIdx.x, warp = (int)uniform(tid >> 5), lane = tid & 31;
  int32_t* fault = a.fault;
  if (tid == 0) {
    cta.word = 0;
    mbar_init(&x_full, 1), mbar_init(&y_full, 1), mbar_init(&z_full, 1);
    mbar_init(&s_done, 1), mbar_init(&o2_done, 1), mbar_init(&o_done, 1), mbar_init(&l_done, 1);
    mbar_init(&sm_ready, kThreadsA), mbar_init(&o_free, kThreadsA);
    mbar_init(&o2_scaled, kThreadsB), mbar_init(&ys_ready, kThreadsB), mbar_init(&l_free, kThreadsB), mbar_init(&g_ready, kThreadsB);
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(&tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t t_s = tmem, t_o = tmem + 128, t_l = tmem + 256;   // scores, OUT, L^T = Z^T diag(w_in) Y (256 columns)
  Walk w{a};

  if (warp < 4) {
    set_regs_dec<kRegsFront>();
    if (warp == 0) {
      if (lane == 0) {
        int i = 0;
#pragma unroll 1
        for (bool ok = w.start(); ok; ok = w.next(), ++i) {
          const int prev = (i - 1) & 1;
          if (i > 0) {   // S and O2 of the tile before have read X
            wait_or_fault(&s_done, prev, &cta, fault, kFaultMmaWait);
            wait_or_fault(&o2_done, prev, &cta, fault, kFaultMmaWait);
          }
          mbar_expect_tx(&x_full, kWide);
          tma_load_4d(sx, &maps.m[w.r.x], &x_full, 0, w.t * C, 0, w.bh);
          tma_load_4d(sx + kNarrow, &maps.m[w.r.x], &x_full, 0, w.t * C, 2, w.bh);
          if (i > 0) wait_or_fault(&l_done, prev, &cta, fault, kFaultMmaWait);   // S and L have read Y
          mbar_expect_tx(&y_full, kWide);
          tma_load_4d(sy, &maps.m[w.r.y], &y_full, 0, w.t * C, 0, w.bh);
          tma_load_4d(sy + kNarrow, &maps.m[w.r.y], &y_full, 0, w.t * C, 2, w.bh);
          if (i > 0) wait_or_fault(&o_done, prev, &cta, fault, kFaultMmaWait);   // L and O1 have read Z
          mbar_expect_tx(&z_full, kNarrow);
          tma_load_4d(sz, &maps.m[w.r.z], &z_full, 0, w.t * C, 2 * w.half, w.bh);
        }
      }
    } else {
      // a whole warp each, an elected lane of which issues
      const bool leader = elect_one();
      const uint32_t x = uniform(smem_u32(sx)), y = uniform(smem_u32(sy)), z = uniform(smem_u32(sz)), g = uniform(smem_u32(sh)), tm = uniform(tmem);
      const uint32_t t_s = tm, t_o = tm + 128, t_l = tm + 256;
      int total = 0;
#pragma unroll 1
      for (int it = blockIdx.x; it < a.items; it += gridDim.x) total += a.tiles;
      if (warp == 1) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int ph = i & 1;
          wait_or_fault(&x_full, ph, &cta, fault, kFaultTmaWait);
          wait_or_fault(&y_full, ph, &cta, fault, kFaultTmaWait);
          if (i > 0) wait_or_fault(&o_done, ph ^ 1, &cta, fault, kFaultMmaWait);   // O1 has read the masked scores
          tc_fence_after_wait();
          umma_gemm<false, false, C, W>(t_s, x, C, y, C, false, leader);
          if (leader) umma_commit(&s_done);
          __syncwarp();
        }
      } else if (warp == 2) {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int ph = i & 1;
          wait_or_fault(&x_full, ph, &cta, fault, kFaultTmaWait);
          wait_or_fault(&g_ready, ph, &cta, fault, kFaultMmaWait);
          if (i > 0) wait_or_fault(&o_free, ph ^ 1, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<false, false, N, W>(t_o, x, C, g, N, false, leader);
          if (leader) umma_commit(&o2_done);
          __syncwarp();
          wait_or_fault(&z_full, ph, &cta, fault, kFaultTmaWait);
          wait_or_fault(&o2_scaled, ph, &cta, fault, kFaultMmaWait);
          wait_or_fault(&sm_ready, ph, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm_ts<true, N, 32>(t_o, t_s, z, C, true, leader);
          if (leader) umma_commit(&o_done);
          __syncwarp();
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < total; ++i) {
          const int ph = i & 1;
          wait_or_fault(&z_full, ph, &cta, fault, kFaultTmaWait);
          wait_or_fault(&ys_ready, ph, &cta, fault, kFaultMmaWait);
          if (i > 0) wait_or_fault(&l_free, ph ^ 1, &cta, fault, kFaultMmaWait);
          tc_fence_after_wait();
          umma_gemm<true, true, W, C>(t_l, z, C, y, C, false, leader);
          if (leader) umma_commit(&l_done);
          __syncwarp();
        }
      }
    }
  } else if (warp < 8) {
    // ---- A: masks, results
    set_regs_dec<kRegsA>();
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    float sl2 = 0.f, lam = 1.f;
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int ph = i & 1;
      if (w.first()) {
        sl2 = a.s[w.bh % a.h] * kLog2e;
        lam = exp2f(-sl2);
      }
      wait_or_fault(&s_done, ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      // packed from left to right: sixteen columns for the thirty-two that have been read
#pragma unroll 1
      for (int b = 0; b < 4; ++b) {
        uint32_t packed[16];
        if (w.r.backwards)
          masked_pack32<true>(t_s + lane_base + 32 * b, row, 32 * b, sl2, lam, packed);
        else
          masked_pack32<false>(t_s + lane_base + 32 * b, row, 32 * b, sl2, lam, packed);
        tmem_st16(t_s + lane_base + 16 * b, packed);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(&sm_ready);
      wait_or_fault(&o_done, ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      // Straight to memory, four lanes 64 bytes of a row, so that Z's buffer is free for the next tile at once.  (Through a
      // staging tile over Z and a TMA store, no decay: 4 x 16 x 4096 training 505 instead of 476 us, 2 x 24 x 2048 215 instead
      // of 197; with decay, where the scaling of rows is longer than Z's way, even.)
      const int row4 = w.t * C + (row & ~3);
      __nv_bfloat16* out = a.out[w.r.out] + ((size_t)w.bh * a.n + row4) * W + N * w.half + 8 * (lane & 3);
#pragma unroll 1
      for (int c0 = 0; c0 < N; c0 += 32) {
        uint32_t r[32];
        __syncwarp();   // (rows past the end are not stored)
        tmem_ld32(t_o + lane_base + c0, r);
        tmem_ld_wait();
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          v[u] = make_uint4(pack_bf16(__uint_as_float(r[8 * u]), __uint_as_float(r[8 * u + 1])),
                            pack_bf16(__uint_as_float(r[8 * u + 2]), __uint_as_float(r[8 * u + 3])),
                            pack_bf16(__uint_as_float(r[8 * u + 4]), __uint_as_float(r[8 * u + 5])),
                            pack_bf16(__uint_as_float(r[8 * u + 6]), __uint_as_float(r[8 * u + 7])));
        rows_to_lanes(v, lane);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (row4 + u < a.n) *reinterpret_cast<uint4*>(out + (size_t)u * W + c0) = v[u];
      }
      tc_fence_before_sync();
      mbar_arrive(&o_free);
    }
  } else {
    // ---- B: the state.  This thread's part of G^T: row `row` (a column of Z), columns [128 half, 128 half + 128)
    set_regs_inc<kRegsB>();
    const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    float G[128];
    float sl2 = 0.f;
    const auto write_operand = [&] {
#pragma unroll
      for (int j = 0; j < 128; j += 8)
        *reinterpret_cast<uint4*>(sh + tile_offset(row, half * 128 + j, N)) =
            make_uint4(pack_bf16(G[j], G[j + 1]), pack_bf16(G[j + 2], G[j + 3]), pack_bf16(G[j + 4], G[j + 5]), pack_bf16(G[j + 6], G[j + 7]));
      fence_async_smem();
      mbar_arrive(&g_ready);
    };
    int i = 0;
#pragma unroll 1
    for (bool ok = w.start(); ok; ok = w.next(), ++i) {
      const int ph = i & 1;
      const int len = min(C, a.n - w.t * C);
      if (__builtin_expect(w.first(), 0)) {   // (O2 of the item before has read its operand)
        sl2 = a.s[w.bh % a.h] * kLog2e;
#pragma unroll
        for (int j = 0; j < 128; ++j) G[j] = 0.f;
        write_operand();
      }
      const bool decays = sl2 != 0.f;   // (otherwise every weight is 1)
      const int from_end = max(len - row, 0);
      wait_or_fault(&s_done, ph, &cta, fault, kFaultMmaWait);   // S has read Y
      if (decays) {
        wait_or_fault(&y_full, ph, &cta, fault, kFaultTmaWait);   // completed long ago: makes Y's bytes visible here
        const float wt = decay_pow(sl2, w.r.backwards ? row : from_end);
        scale_row_pieces<8>(sy, row, 16 * half, wt, lane);
        scale_row_pieces<8>(sy, row, 16 * half + 8, wt, lane);
        fence_async_smem();
      }
      mbar_arrive(&ys_ready);
      wait_or_fault(&o2_done, ph, &cta, fault, kFaultMmaWait);
      if (decays) {
        tc_fence_after_wait();
        const float wt = decay_pow(sl2, w.r.backwards ? from_end : row);
#pragma unroll 1
        for (int c0 = 64 * half; c0 < 64 * half + 64; c0 += 32) scale_tmem32(t_o + lane_base + c0, wt);
        tmem_st_wait();
        tc_fence_before_sync();
      }
      mbar_arrive(&o2_scaled);
      wait_or_fault(&l_done, ph, &cta, fault, kFaultMmaWait);
      tc_fence_after_wait();
      const float lam_len = decay_pow(sl2, len);
#pragma unroll
      for (int c0 = 0; c0 < 128; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(t_l + lane_base + 128 * half + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const F2 v = fma2({lam_len, lam_len}, {G[c0 + j], G[c0 + j + 1]}, pair(r[j], r[j + 1]));
          G[c0 + j] = v.x, G[c0 + j + 1] = v.y;
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&l_free);
      if (!w.last()) write_operand();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
}

cudaError_t launch_wide(int b, int h, int n, WideArgs& g, const WideMaps& maps, cudaStream_t st) {
  cudaError_t err = fault_word_address(&g.fault);
  if (err != cudaSuccess) return err;
  g.h = h, g.n = n, g.tiles = (n + C - 1) / C, g.items = 2 * g.roles * b * h;
  constexpr size_t smem = 3 * (size_t)kWide + kNarrow + 1024;
  if ((err = opt_in_smem<k_walk_wide>(smem)) != cudaSuccess) return err;
  const int sms = sm_count();
  k_walk_wide<<<g.items < sms ? g.items : sms, kThreads, smem, st>>>(maps, g);
  err = cudaGetLastError();
  if (err != cudaSuccess) g_failed_step = "launch of the walk over 256-wide heads";
  return err;
}

cudaError_t wide_map(CUtensorMap* map, const void* base, int b, int h, int n) {   // boxes of 128 tokens x 128 columns
  const cudaError_t err = make_seq_tile_map(map, base, (uint64_t)b * h, (uint64_t)n, W, C, W, N / 64);
  if (err != cudaSuccess) g_failed_step = "tensor map of a 256-wide tensor";
  return err;
}

}  // namespace

cudaError_t wide_forward(int b, int h, int n, const void* q, const void* k, const void* v, const float* s, void* o, cudaStream_t st) {
  WideMaps maps = {};
  const void* tensor[] = {q, k, v};
  for (int i = 0; i < 3; ++i) {
    const cudaError_t err = wide_map(&maps.m[i], tensor[i], b, h, n);
    if (err != cudaSuccess) return err;
  }
  WideArgs g = {};
  g.out[kDq] = static_cast<__nv_bfloat16*>(o);
  g.s = s, g.roles = 1;
  g.role[0] = {kQ, kK, kV, kDq, 0};
  return launch_wide(b, h, n, g, maps, st);
}

cudaError_t wide_backward(int b, int h, int n, const void* q, const void* k, const void* v, const void* d_o, const float* s, void* dq,
                          void* dk, void* dv, cudaStream_t st) {
  WideMaps maps = {};
  const void* tensor[] = {q, k, v, d_o};
  for (int i = 0; i < kInputs; ++i) {
    const cudaError_t err = wide_map(&maps.m[i], tensor[i], b, h, n);
    if (err != cudaSuccess) return err;
  }
  WideArgs g = {};
  g.out[kDq] = static_cast<__nv_bfloat16*>(dq), g.out[kDk] = static_cast<__nv_bfloat16*>(dk), g.out[kDv] = static_cast<__nv_bfloat16*>(dv);
  g.s = s, g.roles = 3;
  g.role[0] = {kDo, kV, kK, kDq, 0};
  g.role[1] = {kV, kDo, kQ, kDk, 1};
  g.role[2] = {kK, kQ, kDo, kDv, 1};
  return launch_wide(b, h, n, g, maps, st);
}

}  // namespace lasp
