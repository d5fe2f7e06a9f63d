// glc_scan.cuh -- device-wide exclusive prefix sum (reduce-then-scan) for any trivially
// copyable value type with operator+ (int64, 128-bit integers, pairs of them).
//
// Up to 16384 items of 8 bytes: one CTA, one launch (the totals of a column's tiles or partitions
// are usually that few, and each launch of a chain costs 3 to 5 us, its gap included: 13,725
// widths took 14 us in three launches, 5 us in one).  More than that, where one SM's loads would
// bound it, or wider items:
// three launches: each 1024-thread CTA scans a tile of 4096 items (1024 of 32 bytes) and writes its total;
// one CTA scans the tile totals (looping with a carry, so any count works); each CTA then adds
// its tile's base.  The bit offsets of the bitstream are this scan over len * bits
// (the reference computes each offset with an O(P) loop per partition,
// compression/CompressionKernels.cuh:222-238).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "glc_device.cuh"

namespace glc {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

template <typename V> __device__ __forceinline__ V shfl_up_any(V v, int d) {
  static_assert(sizeof(V) % 4 == 0, "scan values are multiples of 4 bytes");
  int w[sizeof(V) / 4];
  memcpy(w, &v, sizeof(V));
#pragma unroll
  for (int k = 0; k < (int)(sizeof(V) / 4); k++) w[k] = __shfl_up_sync(FULL_MASK, w[k], d);
  V r;
  memcpy(&r, w, sizeof(V));
  return r;
}

// Exclusive scan of one value per thread across the CTA; returns the CTA total in *total.
template <typename V> __device__ V block_exclusive_scan(V x, V* total, V* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  V inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    V y = shfl_up_any(inc, d);
    if (lane >= d) inc = inc + y;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    V w = (lane < nwarps) ? s_warp[lane] : V();
    V winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      V y = shfl_up_any(winc, d);
      if (lane >= d) winc = winc + y;
    }
    if (lane < nwarps) s_warp[lane] = winc;  // inclusive warp totals
  }
  __syncthreads();
  V base = (warp > 0) ? s_warp[warp - 1] : V();
  *total = s_warp[nwarps - 1];
  V excl = shfl_up_any(inc, 1);
  if (lane == 0) excl = V();
  __syncthreads();
  return base + excl;
}

// One item, in one access where it is 32 bytes (and its array 32-byte aligned, as 32-byte items' are here).
template <typename V> __device__ __forceinline__ V scan_load(const V* p) {
  if constexpr (sizeof(V) == 32) {
    const Bytes32 r = load32(p);
    V v;
    memcpy(&v, &r, 32);
    return v;
  } else {
    return *p;
  }
}
template <typename V> __device__ __forceinline__ void scan_store(V* p, const V& v) {
  if constexpr (sizeof(V) == 32) {
    Bytes32 r;
    memcpy(&r, &v, 32);
    store32(p, r);
  } else {
    *p = v;
  }
}

// Items per thread of a tile: four of 8 bytes, one of 32 (a column of 3M values has 23,439 block sums of
// 32 bytes, which six tiles of 4096 left to six SMs).
template <typename V> __host__ __device__ constexpr int scan_items() { return sizeof(V) == 32 ? 1 : kScanItems; }
template <typename V> __host__ __device__ constexpr int scan_tile() { return kScanThreads * scan_items<V>(); }

template <typename V> __global__ void __launch_bounds__(kScanThreads)
scan_tiles_kernel(const V* __restrict__ in, V* __restrict__ out, int64_t count, V* __restrict__ tile_totals) {
  __shared__ V s_warp[32];
  constexpr int kItems = scan_items<V>();
  const int64_t base = (int64_t)blockIdx.x * scan_tile<V>() + (int64_t)threadIdx.x * kItems;
  V items[kItems];
  V sum = V();
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    items[k] = (base + k < count) ? scan_load(in + base + k) : V();
    sum = sum + items[k];
  }
  V total;
  V ex = block_exclusive_scan(sum, &total, s_warp);
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    if (base + k < count) scan_store(out + base + k, ex);
    ex = ex + items[k];
  }
  if (threadIdx.x == 0) tile_totals[blockIdx.x] = total;
}

template <typename V> __global__ void __launch_bounds__(kScanThreads)
scan_totals_kernel(V* __restrict__ totals, int64_t ntiles, V* __restrict__ grand_total) {
  __shared__ V s_warp[32];
  __shared__ V s_carry;
  if (threadIdx.x == 0) s_carry = V();
  __syncthreads();
  for (int64_t off = 0; off < ntiles; off += kScanTile) {
    const int64_t base = off + (int64_t)threadIdx.x * kScanItems;
    V items[kScanItems];
    V sum = V();
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      items[k] = (base + k < ntiles) ? totals[base + k] : V();
      sum = sum + items[k];
    }
    V total;
    V ex = block_exclusive_scan(sum, &total, s_warp);
    V carry = s_carry;
    ex = ex + carry;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      if (base + k < ntiles) totals[base + k] = ex;
      ex = ex + items[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) s_carry = carry + total;
    __syncthreads();
  }
  if (threadIdx.x == 0 && grand_total) *grand_total = s_carry;
}

template <typename V> __global__ void __launch_bounds__(kScanThreads)
scan_add_kernel(V* __restrict__ out, int64_t count, const V* __restrict__ tile_bases) {
  constexpr int kItems = scan_items<V>();
  const V b = tile_bases[blockIdx.x];
  const int64_t base = (int64_t)blockIdx.x * scan_tile<V>() + (int64_t)threadIdx.x * kItems;
#pragma unroll
  for (int k = 0; k < kItems; k++)
    if (base + k < count) scan_store(out + base + k, scan_load(out + base + k) + b);
}

// The whole scan in one CTA: up to four chunks of 4 items per thread, all of them loaded before the
// barriers and stored after them (in and out may alias).  The chunks' warp scans are independent,
// and warp c scans the warp totals of chunk c, so four chunks cost two barriers like one.  A
// thread's four 8-byte items are one 32-byte access where in and out allow it (one SM writes a
// sector per cycle: 13,725 items in 8-byte stores took 11 us).
constexpr int kScanOneChunks = 4;
constexpr int kScanOneMax = kScanTile * kScanOneChunks;

template <typename V> __global__ void __launch_bounds__(kScanThreads)
scan_one_kernel(const V* in, V* out, int count, V* grand_total) {
  __shared__ V s_warp[kScanOneChunks][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int chunk = (int)blockDim.x * kScanItems;
  static_assert(sizeof(V) * kScanItems == 32, "a thread's items of a chunk are one 32-byte access");
  const bool vec_in = (reinterpret_cast<uintptr_t>(in) & 31) == 0, vec_out = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  V items[kScanOneChunks][kScanItems], sum[kScanOneChunks], inc[kScanOneChunks];
#pragma unroll
  for (int c = 0; c < kScanOneChunks; c++) {
    const int base = c * chunk + (int)threadIdx.x * kScanItems;
    sum[c] = V();
    if (vec_in && base + kScanItems <= count) {
      const Bytes32 r = load32(in + base);
      memcpy(items[c], &r, 32);
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; k++) items[c][k] = (base + k < count) ? in[base + k] : V();
    }
#pragma unroll
    for (int k = 0; k < kScanItems; k++) sum[c] = sum[c] + items[c][k];
    inc[c] = sum[c];
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int c = 0; c < kScanOneChunks; c++) {
      const V y = shfl_up_any(inc[c], d);
      if (lane >= d) inc[c] = inc[c] + y;
    }
  }
  if (lane == 31) {
#pragma unroll
    for (int c = 0; c < kScanOneChunks; c++) s_warp[c][warp] = inc[c];
  }
  __syncthreads();
  for (int c = warp; c < kScanOneChunks; c += nwarps) {
    V w = lane < nwarps ? s_warp[c][lane] : V();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const V y = shfl_up_any(w, d);
      if (lane >= d) w = w + y;
    }
    if (lane < nwarps) s_warp[c][lane] = w;  // inclusive
  }
  __syncthreads();
  V before = V();  // the chunks before chunk c
#pragma unroll
  for (int c = 0; c < kScanOneChunks; c++) {
    const int base = c * chunk + (int)threadIdx.x * kScanItems;
    V ex = before + (warp > 0 ? s_warp[c][warp - 1] : V()) + inc[c] - sum[c];
    V res[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      res[k] = ex;
      ex = ex + items[c][k];
    }
    if (vec_out && base + kScanItems <= count) {
      Bytes32 r;
      memcpy(&r, res, 32);
      store32(out + base, r);
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; k++)
        if (base + k < count) out[base + k] = res[k];
    }
    before = before + s_warp[c][nwarps - 1];
  }
  if (threadIdx.x == 0 && grand_total) *grand_total = before;
}

template <typename V = int64_t> int64_t scan_num_tiles(int64_t count) { return (count + scan_tile<V>() - 1) / scan_tile<V>(); }

// Scratch: one V per tile.  in and out may alias.  *grand_total (device) may be null.
template <typename V>
cudaError_t exclusive_scan(const V* in, V* out, int64_t count, V* grand_total, V* tile_scratch, cudaStream_t s) {
  if (count <= 0) {
    if (grand_total) return cudaMemsetAsync(grand_total, 0, sizeof(V), s);
    return cudaSuccess;
  }
  if constexpr (sizeof(V) == 8) {
    if (count <= kScanOneMax) {
      const int need = (int)((count + kScanItems - 1) / kScanItems + 31) & ~31;
      const int threads = need < kScanThreads ? need : kScanThreads;
      scan_one_kernel<V><<<1, threads, 0, s>>>(in, out, (int)count, grand_total);
      return cudaGetLastError();
    }
  }
  int64_t nt = scan_num_tiles<V>(count);
  scan_tiles_kernel<V><<<(unsigned)nt, kScanThreads, 0, s>>>(in, out, count, tile_scratch);
  scan_totals_kernel<V><<<1, kScanThreads, 0, s>>>(tile_scratch, nt, grand_total);
  scan_add_kernel<V><<<(unsigned)nt, kScanThreads, 0, s>>>(out, count, tile_scratch);
  return cudaGetLastError();
}

}  // namespace glc
