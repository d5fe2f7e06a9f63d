// partition_v6.cu -- the reference's GPU partitioner (compress with use_gpu_partitioning = true,
// GPUVariableLengthPartitionerV6, compression/GpuPartitioner.cuh:34-214), kept as a fast mode
// whose partition boundaries match the reference's.
//
// The reference's algorithm (compression/PartitioningKernels.cuh:647-727):
//  1. cut the column into variance blocks of 8 x base values (base = 2048 in compress,
//     api/G-LeCo.cuh:384-387);
//  2. per block, a "variance" from 128 threads: thread t Kahan-sums v and v^2 over positions
//     start + t + 128k in double, each warp reduces its 32 pairs with a shuffle-down tree, and
//     every warp adds float(S2/n - (S1/n)^2) (n = the block's length) into the block's value;
//  3. thresholds = the values of rank nb/4, nb/2 and 3nb/4 of the sorted block values;
//  4. block i gets partitions of 4 x base values when the i-th SMALLEST block value is below the
//     first threshold, 2 x base below the second, base below the third, otherwise base / 2: the
//     reference sorts the value array in place (GpuPartitioner.cuh:60-61) before the partition
//     kernel reads it by block index, so with distinct values the sizes follow block position
//     and the values only matter through ties; the last partition of a block is cut at the
//     block's (or the column's) end.
// The boundaries are all that the compressor keeps of the partitioner: compress refits every
// partition afterwards (api/G-LeCo.cuh:512-530), exactly as for the other modes.
//
// Here the same arithmetic runs with explicit IEEE operations (Kahan adds, v*v - c as one fma
// and S2/n - m*m as one fma, as the reference's compiler contracts them) so the oracle can
// restate it bit for bit; the four warp values are added in warp order (the reference adds them
// with float atomics in whatever order the warps finish).  The thresholds come from a radix
// select instead of a sort.  "The i-th smallest value is below threshold k" is "i < the number of
// values below threshold k", so only those three counts are needed; the sizes then are four runs of
// blocks, and partition o is computed from o instead of atomics followed by a sort.
#include "glc_internal.h"

namespace glc {
namespace {

constexpr int kV6Threads = 128;  // compression/GpuPartitioner.cuh:52

__device__ __forceinline__ double as_double(int32_t v) { return (double)v; }
__device__ __forceinline__ double as_double(uint32_t v) { return (double)v; }
__device__ __forceinline__ double as_double(int64_t v) { return __ll2double_rn(v); }
__device__ __forceinline__ double as_double(uint64_t v) { return __ull2double_rn(v); }

template <typename T>
__global__ void __launch_bounds__(kV6Threads)
v6_variance_kernel(const T* __restrict__ data, int64_t n, int64_t block_len, float* __restrict__ var) {
  const int64_t start = (int64_t)blockIdx.x * block_len;
  const int64_t end = start + block_len < n ? start + block_len : n;
  double s1 = 0.0, s2 = 0.0, c1 = 0.0, c2 = 0.0;
#pragma unroll 4
  for (int64_t i = start + threadIdx.x; i < end; i += kV6Threads) {
    const double v = as_double(__ldg(data + i));
    const double y1 = __dsub_rn(v, c1);
    const double t1 = __dadd_rn(s1, y1);
    c1 = __dsub_rn(__dsub_rn(t1, s1), y1);
    s1 = t1;
    const double y2 = __fma_rn(v, v, -c2);
    const double t2 = __dadd_rn(s2, y2);
    c2 = __dsub_rn(__dsub_rn(t2, s2), y2);
    s2 = t2;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s1 = __dadd_rn(s1, __shfl_down_sync(FULL_MASK, s1, off));
    s2 = __dadd_rn(s2, __shfl_down_sync(FULL_MASK, s2, off));
  }
  __shared__ float warp_val[kV6Threads / 32];
  if ((threadIdx.x & 31) == 0) {
    const double dn = (double)(end - start);
    const double m = __ddiv_rn(s1, dn);
    warp_val[threadIdx.x >> 5] = __double2float_rn(__fma_rn(-m, m, __ddiv_rn(s2, dn)));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < kV6Threads / 32; w++) acc = __fadd_rn(acc, warp_val[w]);
    var[blockIdx.x] = acc;
  }
}

// Total order of floats as unsigned keys (negative values reversed below the positive ones).
__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Everything between the block values and the partitions, in one CTA (as five launches, with one
// thread walking the bins, it took 70 us of a 30M-value column's 380; 10 us here): the values of rank
// nb/4, nb/2, 3nb/4 (0-based, ascending) by a most-significant-digit radix select, 8 bits per pass, a
// warp per rank; how many block values lie below each (float comparison, as the reference's); and
// the number of partitions.
//
// edge[k], k < 3: blocks [edge[k - 1], edge[k]) (edge[-1] = 0) have partitions of 4, 2 and 1 times the
// base, those from edge[2] on of half the base.
struct V6Plan {
  int64_t edge[3];
  int64_t total;
};

// Partitions of the blocks before block i (all of them full).
__device__ __forceinline__ int64_t v6_before(int64_t i, const int64_t* e) {
  const int64_t a = i < e[0] ? i : e[0], b = i < e[1] ? i : e[1], c = i < e[2] ? i : e[2];
  return 2 * a + 4 * (b - a) + 8 * (c - b) + 16 * (i - c);
}
// Partition size of block i: its rank among the sorted values against the three counts.
__device__ __forceinline__ int64_t v6_size(int64_t i, const int64_t* e, int64_t base) {
  return i < e[0] ? 4 * base : (i < e[1] ? 2 * base : (i < e[2] ? base : base / 2));
}

__global__ void __launch_bounds__(1024)
v6_select_kernel(const float* __restrict__ var, int64_t nb, int64_t n, int64_t base, V6Plan* __restrict__ plan) {
  __shared__ unsigned int hist[3][256];
  __shared__ uint32_t s_prefix[3];
  __shared__ long long s_rank[3];
  __shared__ unsigned int s_below[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 3) {
    s_rank[tid] = tid == 0 ? nb / 4 : (tid == 1 ? nb / 2 : 3 * nb / 4);
    s_prefix[tid] = 0u;
    s_below[tid] = 0u;
  }
  uint32_t mask = 0u;
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (tid < 768) hist[tid >> 8][tid & 255] = 0u;
    __syncthreads();
    const uint32_t p0 = s_prefix[0], p1 = s_prefix[1], p2 = s_prefix[2];
    for (int64_t i = tid; i < nb; i += 1024) {
      const uint32_t k = float_key(var[i]), bin = (k >> shift) & 255u, pre = k & mask;
      if (pre == p0) atomicAdd(&hist[0][bin], 1u);
      if (pre == p1) atomicAdd(&hist[1][bin], 1u);
      if (pre == p2) atomicAdd(&hist[2][bin], 1u);
    }
    __syncthreads();
    if (warp < 3) {  // lane l holds bins [8 l, 8 l + 8): the first bin whose running count passes the rank
      unsigned int c[8], sum = 0u;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        c[j] = hist[warp][8 * lane + j];
        sum += c[j];
      }
      unsigned int inc = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned int y = __shfl_up_sync(FULL_MASK, inc, d);
        if (lane >= d) inc += y;
      }
      const long long rank = s_rank[warp];
      const unsigned hit = __ballot_sync(FULL_MASK, (long long)inc > rank);
      const int l = hit ? __ffs(hit) - 1 : 31;
      __syncwarp();
      if (lane == l) {
        long long r = rank - (long long)(inc - sum);
        int j = 0;
        for (; j < 7; j++) {
          if (r < (long long)c[j]) break;
          r -= c[j];
        }
        s_prefix[warp] |= (uint32_t)(8 * lane + j) << shift;
        s_rank[warp] = r;
      }
    }
    mask |= 0xffu << shift;
    __syncthreads();
  }
  const float t0 = key_float(s_prefix[0]), t1 = key_float(s_prefix[1]), t2 = key_float(s_prefix[2]);
  unsigned int c0 = 0, c1 = 0, c2 = 0;
  for (int64_t i = tid; i < nb; i += 1024) {
    const float x = var[i];
    c0 += x < t0;
    c1 += x < t1;
    c2 += x < t2;
  }
  c0 = __reduce_add_sync(FULL_MASK, c0);
  c1 = __reduce_add_sync(FULL_MASK, c1);
  c2 = __reduce_add_sync(FULL_MASK, c2);
  if (lane == 0) {
    atomicAdd(&s_below[0], c0);
    atomicAdd(&s_below[1], c1);
    atomicAdd(&s_below[2], c2);
  }
  __syncthreads();
  if (tid == 0) {
    int64_t e[3];
    e[0] = s_below[0];
    e[1] = s_below[1] > e[0] ? s_below[1] : e[0];
    e[2] = s_below[2] > e[1] ? s_below[2] : e[1];
    const int64_t last = n - (nb - 1) * 8 * base, size = v6_size(nb - 1, e, base);
    for (int k = 0; k < 3; k++) plan->edge[k] = e[k];
    plan->total = v6_before(nb - 1, e) + (last + size - 1) / size;
  }
}

__global__ void v6_emit_kernel(int64_t nb, const V6Plan* __restrict__ plan, int64_t n, int64_t base, int64_t P,
                               int32_t* __restrict__ starts, int32_t* __restrict__ ends, int32_t* __restrict__ unit_first) {
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= P) return;
  int64_t e[3];
#pragma unroll
  for (int k = 0; k < 3; k++) e[k] = plan->edge[k];
  int64_t i = nb - 1;  // the partition's block
  const int64_t c0 = 2 * e[0], c1 = c0 + 4 * (e[1] - e[0]), c2 = c1 + 8 * (e[2] - e[1]);
  if (o < v6_before(nb - 1, e)) i = o < c0 ? o / 2 : o < c1 ? e[0] + (o - c0) / 4 : o < c2 ? e[1] + (o - c1) / 8 : e[2] + (o - c2) / 16;
  const int64_t size = v6_size(i, e, base), end = 8 * base * (i + 1) < n ? 8 * base * (i + 1) : n;
  const int64_t s = 8 * base * i + (o - v6_before(i, e)) * size;
  starts[o] = (int32_t)s;
  ends[o] = (int32_t)(s + size < end ? s + size : end);
  if (unit_first) {  // (a block is a whole number of units, and every size divides it)
    if (s % kFitShort == 0) unit_first[s / kFitShort] = (int32_t)o;
    if (o == P - 1) unit_first[(n + kFitShort - 1) / kFitShort] = (int32_t)P;
  }
}

template <typename T>
cudaError_t v6_typed(glc_ctx* ctx, const T* values, int64_t n, int64_t base, const PartOut& out, cudaStream_t s) {
  const int64_t block_len = 8 * base;
  const int64_t nb = (n + block_len - 1) / block_len;
  V6Plan* plan = nullptr;  // then the block values
  cudaError_t e = pool_alloc(ctx, &plan, sizeof(V6Plan) + 4 * (size_t)nb, s);
  if (e != cudaSuccess) return e;
  float* var = (float*)(plan + 1);
  int32_t *starts = nullptr, *ends = nullptr;
  v6_variance_kernel<T><<<(unsigned)nb, kV6Threads, 0, s>>>(values, n, block_len, var);
  v6_select_kernel<<<1, 1024, 0, s>>>(var, nb, n, base, plan);
  if ((e = cudaGetLastError()) == cudaSuccess &&
      (e = cudaMemcpyAsync(ctx->h_stats, &plan->total, 8, cudaMemcpyDeviceToHost, s)) == cudaSuccess)
    e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) {
    const int64_t P = ctx->h_stats[0];
    if (out.column) {
      out.column->P = P;
      if ((e = out.alloc(out.column, s)) == cudaSuccess) {
        starts = out.column->d_start;
        ends = out.column->d_end;
        if (out.unit_first) e = pool_alloc(ctx, out.unit_first, 4 * (size_t)((n + kFitShort - 1) / kFitShort + 1), s);
      }
    } else {
      *out.P = P;
      if ((e = pool_alloc(ctx, out.starts, 4 * P, s)) == cudaSuccess && (e = pool_alloc(ctx, out.ends, 4 * P, s)) == cudaSuccess) {
        starts = *out.starts;
        ends = *out.ends;
      }
    }
    if (e == cudaSuccess) {
      v6_emit_kernel<<<(unsigned)((P + 255) / 256), 256, 0, s>>>(nb, plan, n, base, P, starts, ends,
                                                                 out.unit_first ? *out.unit_first : nullptr);
      e = cudaGetLastError();
    }
  }
  cudaFreeAsync(plan, s);
  return e;
}

}  // namespace

cudaError_t launch_partition_v6(glc_ctx* ctx, glc_dtype dt, const void* values, int64_t n, int32_t base,
                                const PartOut& out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  switch (dt) {
    case GLC_I32: return v6_typed<int32_t>(ctx, (const int32_t*)values, n, base, out, s);
    case GLC_I64: return v6_typed<int64_t>(ctx, (const int64_t*)values, n, base, out, s);
    case GLC_U64: return v6_typed<uint64_t>(ctx, (const uint64_t*)values, n, base, out, s);
    case GLC_U32: return v6_typed<uint32_t>(ctx, (const uint32_t*)values, n, base, out, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace glc
