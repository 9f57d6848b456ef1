// Elementwise kernels: on the fp32 d x e states the scan over the chunks (or spans) of a sequence and the update of
// a rank state; the feature map on q and k.
#include "state_terms.cuh"
#include "tc_common.cuh"

namespace lasp {
namespace {

// ---------------------------------------------------------------------------
// scan over chunks, elementwise in (d,e).  forward: exclusive prefix seeded
// with x_in; reverse: exclusive suffix.  k_scan reads the fp32 local states
// and writes the prefix states to a second array: fp32 in lane order (tensor path), or row-major in terms
// (TERMS, full-precision path).  Loads of a batch of chunks are issued before the
// dependent recurrence so that their latencies overlap.
// ---------------------------------------------------------------------------
constexpr int kScanBatch = 8;

template <bool TERMS>
__global__ void __launch_bounds__(256) k_scan(const float* __restrict__ s, const float* __restrict__ local,
                                              void* __restrict__ prefix, const float* __restrict__ x_in,
                                              float* __restrict__ x_out, int h,
                                              int n, int de, int nc, int chunk, int reverse, int rows,
                                              int cols) {
  if (TERMS) after_previous();
  const int bh = blockIdx.y;
  const int el = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (el >= de) return;
  // where this float4 of a state in lane order lives in the caller's row-major rank states
  const int ext = TERMS ? el : lane_order_to_row_major(el / 4, rows, cols) * 4;
  const float sh = s[bh % h];
  const float full = expf(-sh * (float)chunk);
  const int last_len = n - (nc - 1) * chunk;
  const float tail = expf(-sh * (float)last_len);
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
  // (around the read-only path: the kernel before writes these while this one's CTAs may be there already)
  if (x_in) p = __ldcg(reinterpret_cast<const float4*>(x_in + (size_t)bh * de + ext));
  const float* base = local + (size_t)bh * nc * de + el;
  for (int i0 = 0; i0 < nc; i0 += kScanBatch) {
    float4 loc[kScanBatch];
#pragma unroll
    for (int u = 0; u < kScanBatch; ++u) {
      const int i = i0 + u;
      if (i < nc) loc[u] = __ldcg(reinterpret_cast<const float4*>(base + (size_t)(reverse ? nc - 1 - i : i) * de));
    }
#pragma unroll
    for (int u = 0; u < kScanBatch; ++u) {
      const int i = i0 + u;
      if (i < nc) {
        const int c = reverse ? nc - 1 - i : i;
        const float dec = (c == nc - 1) ? tail : full;
        const size_t state = (size_t)bh * nc + c;
        if (TERMS)
          store_state_terms(static_cast<__nv_bfloat16*>(prefix) + state * 3 * de, el, de, p);
        else
          *reinterpret_cast<float4*>(static_cast<float*>(prefix) + state * de + el) = p;
        p.x = fmaf(dec, p.x, loc[u].x);
        p.y = fmaf(dec, p.y, loc[u].y);
        p.z = fmaf(dec, p.z, loc[u].z);
        p.w = fmaf(dec, p.w, loc[u].w);
      }
    }
  }
  if (x_out) *reinterpret_cast<float4*>(x_out + (size_t)bh * de + ext) = p;
  if (TERMS) {   // (the output kernels read the terms by TMA)
    fence_async_global();
    let_next_start();
  }
}

__global__ void __launch_bounds__(256) k_state_combine(const float* __restrict__ s, const float* __restrict__ x_in,
                                                       const float* __restrict__ x_local, float* __restrict__ x_out,
                                                       int h, int de, int n) {
  const int bh = blockIdx.y;
  const int el = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (el >= de) return;
  const float dec = expf(-s[bh % h] * (float)n);
  float4 loc = *reinterpret_cast<const float4*>(x_local + (size_t)bh * de + el);
  if (x_in) {
    float4 p = *reinterpret_cast<const float4*>(x_in + (size_t)bh * de + el);
    loc.x = fmaf(dec, p.x, loc.x);
    loc.y = fmaf(dec, p.y, loc.y);
    loc.z = fmaf(dec, p.z, loc.z);
    loc.w = fmaf(dec, p.w, loc.w);
  }
  *reinterpret_cast<float4*>(x_out + (size_t)bh * de + el) = loc;
}

// elu(x) + 1 of q (blockIdx.y = 0) and k (1).  Bound by HBM: 8 bytes an element.
constexpr int kMapPieces = 4;   // 16-byte loads in flight per thread
__global__ void __launch_bounds__(256) k_map_qk(const uint4* __restrict__ q, const uint4* __restrict__ k, uint4* __restrict__ q_out,
                                                uint4* __restrict__ k_out, int64_t pieces) {
  const uint4* in = blockIdx.y ? k : q;
  uint4* out = blockIdx.y ? k_out : q_out;
  const int64_t first = (int64_t)blockIdx.x * (256 * kMapPieces) + threadIdx.x;
  uint4 v[kMapPieces];
#pragma unroll
  for (int i = 0; i < kMapPieces; ++i)
    if (first + 256 * i < pieces) v[i] = __ldg(in + first + 256 * i);
#pragma unroll
  for (int i = 0; i < kMapPieces; ++i)
    if (first + 256 * i < pieces)
      out[first + 256 * i] = make_uint4(tc::elu1_bf16x2(v[i].x), tc::elu1_bf16x2(v[i].y), tc::elu1_bf16x2(v[i].z), tc::elu1_bf16x2(v[i].w));
}

}  // namespace

cudaError_t map_qk(const void* q, const void* k, void* q_out, void* k_out, int64_t elements, cudaStream_t st) {
  const int64_t pieces = elements / 8, blocks = (pieces + 256 * kMapPieces - 1) / (256 * kMapPieces);
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  k_map_qk<<<dim3((unsigned)blocks, 2), 256, 0, st>>>(static_cast<const uint4*>(q), static_cast<const uint4*>(k), static_cast<uint4*>(q_out),
                                                      static_cast<uint4*>(k_out), pieces);
  return cudaGetLastError();
}

cudaError_t scan_states(const Dims& m, const float* s, const float* local, void* prefix, const float* x_in,
                        float* x_out, bool reverse, cudaStream_t st) {
  const int de = m.d * m.e;
  dim3 grid((de / 4 + 255) / 256, m.b * m.h);
  if (!m.walk)
    return launch_following(k_scan<true>, grid, 256, 0, st, s, local, prefix, x_in, x_out, m.h, m.n, de, m.nc, m.chunk, reverse ? 1 : 0, m.d,
                            m.e);
  k_scan<false><<<grid, 256, 0, st>>>(s, local, prefix, x_in, x_out, m.h, m.n, de, m.nc, m.chunk, reverse ? 1 : 0, m.d, m.e);
  return cudaGetLastError();
}


cudaError_t state_combine(int b, int h, int d, int e, int n, const float* s, const float* x_in,
                          const float* x_local, float* x_out, cudaStream_t st) {
  const int de = d * e;
  dim3 grid((de / 4 + 255) / 256, b * h);
  k_state_combine<<<grid, 256, 0, st>>>(s, x_in, x_local, x_out, h, de, n);
  return cudaGetLastError();
}

}  // namespace lasp
