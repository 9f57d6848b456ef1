// Forward pass for callers that cannot allocate device memory.
//
// Some hosts of this library hand every byte of the GPU to a pool of their own
// at start-up (an inference server that pre-reserves the device), or call the
// operator from a section where cudaMalloc / cudaFree - which may synchronise
// the whole device - are not allowed (a latency-critical serving loop).  Such
// a caller has nowhere to get the chunk-state workspace from.  This file gives
// the forward pass a workspace that lives inside the library image: a
// file-scope __device__ array that every GPU loading the library holds until
// the process exits.
#include <mutex>

#include "common.cuh"

namespace {

// the workspace itself: LASP_B200_STATIC_SCRATCH_BYTES on every device
static __device__ __align__(256) unsigned char g_static_scratch[LASP_B200_STATIC_SCRATCH_BYTES];
// The words that the CTAs of a tensor-path launch synchronise through.  The launches keep them consistent from one to the
// next, so they are not part of the workspace, which calls on the full-precision path fill with states from its start.
static __device__ __align__(256) uint32_t g_static_sync[lasp::kWalkSyncBytes / 4];

constexpr int kMaxDevices = 64;
std::mutex g_setup_lock;
struct Addresses {
  void *scratch, *sync;
};
Addresses g_addr[kMaxDevices] = {};      // device addresses of the two arrays, per device ordinal

// In host code the arrays' names are only handles for the runtime, not
// addresses a kernel can use: the device addresses are asked for once per
// device, with that device current, and cached.
cudaError_t scratch_addresses(Addresses* out) {
  int dev = -1;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> guard(g_setup_lock);
  if (!g_addr[dev].scratch) {
    Addresses at = {};
    if ((err = cudaGetSymbolAddress(&at.scratch, g_static_scratch)) != cudaSuccess) return err;
    if ((err = cudaGetSymbolAddress(&at.sync, g_static_sync)) != cudaSuccess) return err;
    if (!at.scratch || !at.sync) return cudaErrorInvalidSymbol;
    g_addr[dev] = at;
  }
  *out = g_addr[dev];
  return cudaSuccess;
}

}  // namespace

extern "C" int lasp_b200_forward_static(const lasp_problem* p, const lasp_fwd_args* a, void* stream) {
  if (!p || !a) return LASP_ERR_NULL;
  const int path = lasp_b200_resolve_path(p);  // full shape / dtype validation
  if (path < 0) return path;
  const size_t need = lasp_b200_fwd_workspace_bytes(p);
  if (need == 0 || need > (size_t)LASP_B200_STATIC_SCRATCH_BYTES) return LASP_ERR_TOO_LARGE;
  Addresses at;
  if (scratch_addresses(&at) != cudaSuccess) return LASP_ERR_CUDA;
  lasp_fwd_args with_ws = *a;
  with_ws.ws = at.scratch;
  with_ws.ws_bytes = (size_t)LASP_B200_STATIC_SCRATCH_BYTES;
  // every chunk state the scan and the output kernel read is written by the
  // chunk-state kernel of this same call, so nothing has to be cleared first
  const lasp_call_options opt = {static_cast<uint32_t*>(at.sync), 1, 0, 0};
  return lasp_b200_forward_opt(p, &with_ws, &opt, stream);
}
