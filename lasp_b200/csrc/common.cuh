// Shared declarations of the lasp_b200 CUDA library (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "lasp_b200.h"

namespace lasp {

// Workspace layout (forward and backward use the same one), with S = b*h*nc*d*e
// and nc the number of states kept per sequence.  The chunk-state phase writes
// the LOCAL states, the scan reads them and writes the PREFIX states (exclusive,
// seeded with the incoming rank state) that the output / gradient kernels read:
//   FULL PRECISION : one state per 128-token chunk, row-major:
//                      [0, S*6) prefix states, each as the three bf16 matrices that its terms make up
//                               (state_terms.cuh), as the output kernels' tensor-core operands need them
//                      [S*6, S*10) local states, fp32
//   TENSOR path      : one state per SPAN of `span` 128-token tiles (a few per
//                      sequence; inside a span the state lives on chip):
//                      [0, 4096)            words the CTAs of the fused kernels
//                                           synchronise through (zeroed once by
//                                           the caller, kept by the library)
//                      [4096, 4096 + S*4)   local states: fp32 span totals
//                      [4096 + S*4, + S*4)  prefix states: fp32 states at the span borders
// The running prefix inside the scan is always fp32.
constexpr int kTensorTile = 128;  // one tcgen05 M=128 tile
constexpr int kAbiChunk = 64;     // the reference's block size: the unit in which the C ABI states the chunks of the
                                  // full-precision path and sizes its workspace (8 bytes per element of a state; the
                                  // kernels use 10 per chunk of their own, which are two of these)

struct Dims {
  int b, h, n, d, e;
  int chunk;  // tokens per state kept in the workspace
  int nc;     // states per sequence
  int dtype;
  int path;
  int walk;   // 1 on the tensor path: the state is carried on chip along a span of tiles
  int tiles;  // tensor path: 128-token tiles per sequence
  int span;   // tensor path: tiles per span (chunk = span * 128)
  int pitch_d, pitch_e;  // elements between the rows of consecutive tokens in q,k,dq,dk and in v,o,do,dv
  int qk_map;      // q and k enter as qk_scale * map(x): a lasp_qk_map
  float qk_scale;  // (1 when the caller left it 0)
};

inline bool has_qk_preprocessing(const Dims& m) { return m.qk_map != 0 || m.qk_scale != 1.f; }

// SM count of the current device (cached per device ordinal)
int sm_count();

inline size_t state_elems(const Dims& m) { return (size_t)m.b * m.h * m.nc * m.d * m.e; }

// The states of the tensor path in a workspace are kept in "lane order": the float4 holding
// columns 4g..4g+3 of row r of a d x e state sits at float4 index g*d + r, so that the 32 rows a warp
// owns are contiguous for each of its accesses.  Rank states handed in and out by the caller stay
// row-major.
__host__ __device__ inline int lane_order_to_row_major(int f4, int rows, int cols) {
  const int g = f4 / rows, r = f4 - g * rows;
  return r * (cols / 4) + g;
}
constexpr size_t kWalkSyncBytes = 4096;
inline uint32_t* ws_walk_sync(void* ws) { return reinterpret_cast<uint32_t*>(ws); }
inline const uint32_t* ws_walk_sync(const void* ws) { return reinterpret_cast<const uint32_t*>(ws); }
inline float* ws_walk_totals(void* ws) { return reinterpret_cast<float*>(static_cast<char*>(ws) + kWalkSyncBytes); }
inline float* ws_walk_border(void* ws, const Dims& m) {
  return reinterpret_cast<float*>(static_cast<char*>(ws) + kWalkSyncBytes + state_elems(m) * 4);
}
inline const float* ws_walk_border(const void* ws, const Dims& m) {
  return reinterpret_cast<const float*>(static_cast<const char*>(ws) + kWalkSyncBytes + state_elems(m) * 4);
}
// where the chunk-state phase writes / where the scan writes and the output kernels read (fp32 on the tensor path, terms
// on the full-precision path)
inline float* ws_local(void* ws, const Dims& m) {
  return m.walk ? ws_walk_totals(ws) : reinterpret_cast<float*>(static_cast<char*>(ws) + state_elems(m) * 6);
}
inline void* ws_prefix(void* ws, const Dims& m) { return m.walk ? ws_walk_border(ws, m) : ws; }
// bits of the sticky per-device fault word (fault_word.cu owns the word)
enum : int32_t {
  kFaultNone = 0,
  kFaultTmaWait = 1,   // a bounded wait on a TMA mbarrier ran out
  kFaultMmaWait = 2,   // a bounded wait on a tcgen05.commit mbarrier ran out
  kFaultRelayWait = 4, // a bounded wait on a peer's flag ran out (state relay)
  kFaultFlagWait = 8,  // a bounded wait on another CTA's flag ran out (fused kernels)
};
cudaError_t read_fault_word(int32_t* host, bool clear, cudaStream_t st);
// device address of the current device's fault word (for kernels in other translation units)
cudaError_t fault_word_address(int32_t** out);

// name of the host-side step that produced the last cudaError_t (for error text)
extern thread_local const char* g_failed_step;

// Lets a kernel ask for up to `bytes` (the most that it ever takes) of dynamic shared memory; once per kernel and device,
// the attribute call costs the host about as much as a launch.
template <auto fn>
cudaError_t opt_in_smem(size_t bytes) {
  static bool done[64] = {};
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess && dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
  if (err == cudaSuccess)
    err = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (err != cudaSuccess)
    g_failed_step = "cudaFuncSetAttribute(max dynamic shared memory)";
  else if (dev >= 0 && dev < 64)
    done[dev] = true;
  return err;
}

// The kernels of the full-precision path follow one another closely (states, scan, outputs): each lets the next one's CTAs
// take an SM as soon as its own have left it, and waits itself, before it touches global memory, for what came before it to
// be complete.  Training passes of 2 x 12 x 2048: fp32 219 -> 212 us, fp16 122 -> 116.5 (with the
// next one let in ahead of the wait; behind it 213.7 -> 211.2 and 116.6 -> 114.8); the walk kernels' passes got 1 to 2 %
// longer with it.
//   after_previous   every thread, before its first access to global memory, and after the CTA has its tensor memory: a CTA
//                    that waited for columns while it kept the CTA that holds them from starting would wait for good.
//                    Tiles that a kernel wrote with ordinary stores are read by TMA, another proxy: hence the fence.
//   let_next_start   behind after_previous: whatever starts early finds everything but this kernel complete - a kernel of a
//                    caller's that reads what it takes for long written ahead of its own wait, and the L1 of its SM.  A
//                    kernel whose stores the next one's TMA reads calls it behind them and their fence.
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  fence_async_global();
}
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... KArgs, typename... Args>
cudaError_t launch_following(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, const Args&... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ---- launchers implemented in the .cu files (return cudaError_t) -----------
// Full-precision path (split_kernels.cu).  `alone`: no rank state comes in or goes out, so the states at the
// sequence's ends are zero or unread.
cudaError_t split_chunk_states(const Dims& m, const void* a, const void* bten, const float* s, float* states,
                               bool backward, bool alone, cudaStream_t st);
cudaError_t split_fwd_output(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                             const void* prefix, void* o, bool alone, bool add_o, cudaStream_t st);
cudaError_t split_bwd_grads(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, const float* s,
                            const void* prefix, const void* suffix, void* dq, void* dk, void* dv, bool alone,
                            bool add_qk, bool add_v, cudaStream_t st);
cudaError_t scan_states(const Dims& m, const float* s, const float* local, void* prefix, const float* x_in,
                        float* x_out, bool reverse, cudaStream_t st);
cudaError_t state_combine(int b, int h, int d, int e, int n, const float* s, const float* x_in,
                          const float* x_local, float* x_out, cudaStream_t st);

cudaError_t map_qk(const void* q, const void* k, void* q_out, void* k_out, int64_t elements, cudaStream_t st);

// state relay (relay_kernels.cu)
cudaError_t exchange_scan(const Dims& m, const lasp_exchange_args& a, const float* local, void* prefix,
                          cudaStream_t st);

// tcgen05 path
bool tensor_path_supported(const Dims& m);

// 256-wide heads in one pass per result (wide_kernels.cu)
cudaError_t wide_forward(int b, int h, int n, const void* q, const void* k, const void* v, const float* s, void* o, cudaStream_t st);
cudaError_t wide_backward(int b, int h, int n, const void* q, const void* k, const void* v, const void* d_o, const float* s, void* dq,
                          void* dk, void* dv, cudaStream_t st);

// tcgen05 path with the state carried on chip (walk_kernels.cu)
cudaError_t walk_span_totals(const Dims& m, const void* a, const void* bten, const float* s, float* totals,
                             bool reverse, cudaStream_t st);
cudaError_t walk_fwd_output(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                            const float* prefix, uint32_t* sync, void* o, bool add_o, cudaStream_t st);
cudaError_t walk_fwd_fused(const Dims& m, const void* q, const void* k, const void* v, const float* s,
                           const float* x_in, float* x_out, uint32_t* sync, float* totals, float* prefix, void* o,
                           const lasp_exchange_args* link, bool add_o, cudaStream_t st);
// fwd_sync: the forward's synchronisation words, which say how it cut the sequences; NULL: `even` says it
cudaError_t walk_bwd_dq(const Dims& m, const void* q, const void* k, const void* v, const void* d_o, const float* s,
                        const float* prefix, const uint32_t* fwd_sync, bool even, void* dq, bool add_dq, cudaStream_t st);
cudaError_t walk_bwd_dkv(const Dims& m, const void* q, const void* k, const void* v, const void* d_o,
                         const float* s, const float* suffix, void* dk, void* dv, bool add_dk, bool add_dv,
                         cudaStream_t st);
cudaError_t walk_bwd_dkv_fused(const Dims& m, const void* q, const void* k, const void* v, const void* d_o,
                               const float* s, const float* x_in, float* x_out, uint32_t* sync, float* totals,
                               void* dk, void* dv, const lasp_exchange_args* link, bool add_dk, bool add_dv,
                               cudaStream_t st);

}  // namespace lasp
