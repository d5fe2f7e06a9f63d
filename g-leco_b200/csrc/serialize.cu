// serialize.cu -- a column's version-5 blob written to device memory by one kernel, and an uploaded
// blob's metadata dealt out to a column's arrays.
//
// The blob is a 120-byte header, seven metadata arrays and the bitstream, each from an 8-byte
// boundary with zeros between them (api/G-LeCo.cuh:1878-2047 copies them one by one).  As eight
// copies, the padding's memsets and the header's host-to-device copy, a blob of 330 KB took 13
// operations of about 1.5 us with 2 to 5 us between them; here the header travels in the launch's
// parameters and every word of the blob is written once, by the same launch.
//
// Small blobs are bound by that one launch (2^20 int32 values in partitions of 1024, compress and
// serialize together: 94 -> 66 us), large ones by memory: the bitstream is copied in 16-byte
// stores, four in flight per thread (339 MB: 114 us, 5.9 TB/s read and written, as a device copy).
#include <algorithm>
#include "glc_internal.h"

namespace glc {

constexpr int kSerThreads = 256;
constexpr int kSerUnroll = 4;

// 16 bytes from a 4-byte aligned address; ALIGN is the alignment it is known to have.
template <int ALIGN> __device__ __forceinline__ uint4 load16(const uint32_t* p) {
  if (ALIGN == 16) return __ldg(reinterpret_cast<const uint4*>(p));
  if (ALIGN == 8) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(p)), b = __ldg(reinterpret_cast<const uint2*>(p) + 1);
    return make_uint4(a.x, a.y, b.x, b.y);
  }
  return make_uint4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

template <int ALIGN>
__device__ __forceinline__ void copy16(uint4* __restrict__ dst, const uint32_t* __restrict__ src, int64_t n16) {
  const int64_t step = (int64_t)kSerThreads * kSerUnroll;
  for (int64_t b = (int64_t)blockIdx.x * step; b < n16; b += (int64_t)gridDim.x * step) {
    uint4 v[kSerUnroll];
#pragma unroll
    for (int u = 0; u < kSerUnroll; u++) {
      const int64_t i = b + u * kSerThreads + threadIdx.x;
      if (i < n16) v[u] = load16<ALIGN>(src + 4 * i);
    }
#pragma unroll
    for (int u = 0; u < kSerUnroll; u++) {
      const int64_t i = b + u * kSerThreads + threadIdx.x;
      if (i < n16) dst[i] = v[u];
    }
  }
}

__global__ void __launch_bounds__(kSerThreads) serialize_kernel(const __grid_constant__ SerializeArgs a) {
  const int64_t tid = (int64_t)blockIdx.x * kSerThreads + threadIdx.x, nthreads = (int64_t)gridDim.x * kSerThreads;
  uint32_t* __restrict__ out = reinterpret_cast<uint32_t*>(a.dst);
  // header and metadata, word by word: the piece that holds word w, or the padding after it
  const int64_t nmeta = (int64_t)(a.off[kSerPieces - 1] >> 2);
  for (int64_t w = tid; w < nmeta; w += nthreads) {
    uint32_t v = 0u;
    if (w < kSerHeaderWords) {
      v = a.header[w];
    } else {
      int j = 0;
#pragma unroll
      for (int k = 1; k < kSerPieces - 1; k++) j += w >= (int64_t)(a.off[k] >> 2);
      const int64_t i = w - (int64_t)(a.off[j] >> 2);
      if (i >= 0 && i < (int64_t)(a.bytes[j] >> 2)) v = __ldg(reinterpret_cast<const uint32_t*>(a.src[j]) + i);
    }
    out[w] = v;
  }
  // the bitstream: words to the first 16-byte boundary of the blob, 16-byte groups of whole source
  // words, then the last words (a partial one with its unused bytes zero) and the zeros up to the end
  const uint32_t* src = reinterpret_cast<const uint32_t*>(a.src[kSerPieces - 1]);
  uint32_t* dst = out + nmeta;
  const int64_t bytes = (int64_t)a.bytes[kSerPieces - 1];
  const int64_t nall = (int64_t)((a.total - a.off[kSerPieces - 1]) >> 2), nfull = bytes >> 2;
  int64_t head = (int64_t)((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15) >> 2;
  head = head < nfull ? head : nfull;
  const int64_t n16 = (nfull - head) >> 2;
  const uintptr_t s0 = reinterpret_cast<uintptr_t>(src + head);
  uint4* dst16 = reinterpret_cast<uint4*>(dst + head);
  if ((s0 & 15) == 0) copy16<16>(dst16, src + head, n16);
  else if ((s0 & 7) == 0) copy16<8>(dst16, src + head, n16);
  else copy16<4>(dst16, src + head, n16);
  const int64_t rest = head + 4 * n16;  // words [0, head) and [rest, nall): at most a dozen
  const int64_t nedge = head + (nall - rest);
  for (int64_t k = tid; k < nedge; k += nthreads) {
    const int64_t w = k < head ? k : rest + (k - head);
    uint32_t v = 0u;
    if (w < nfull) v = __ldg(src + w);
    else if (w == nfull && (bytes & 3)) v = __ldg(src + w) & ((1u << (8 * (bytes & 3))) - 1u);
    dst[w] = v;
  }
}

__global__ void __launch_bounds__(kSerThreads) scatter_kernel(const __grid_constant__ ScatterArgs a) {
  const int64_t tid = (int64_t)blockIdx.x * kSerThreads + threadIdx.x, nthreads = (int64_t)gridDim.x * kSerThreads;
#pragma unroll
  for (int j = 0; j < kSerPieces - 1; j++)
    for (int64_t w = tid; w < (int64_t)a.words[j]; w += nthreads) a.dst[j][w] = __ldg(a.src[j] + w);
}

cudaError_t launch_scatter(const ScatterArgs& a, int num_sms, cudaStream_t s) {
  uint64_t most = 0;
  for (uint64_t w : a.words) most = std::max(most, w);
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(((int64_t)most + kSerThreads - 1) / kSerThreads, (int64_t)num_sms * 8));
  scatter_kernel<<<(unsigned)grid, kSerThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_serialize(const SerializeArgs& a, int num_sms, cudaStream_t s) {
  const int64_t meta = (int64_t)a.off[kSerPieces - 1] / 4, per = (int64_t)kSerThreads * kSerUnroll;
  const int64_t groups = (int64_t)a.bytes[kSerPieces - 1] / 16;
  int64_t grid = std::max((groups + per - 1) / per, (meta + kSerThreads - 1) / kSerThreads);
  grid = std::max<int64_t>(1, std::min<int64_t>(grid, (int64_t)num_sms * 8));  // 8 CTAs of 256 threads fill an SM
  serialize_kernel<<<(unsigned)grid, kSerThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace glc
