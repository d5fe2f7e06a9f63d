// compress_fixed.cu -- one-pass compression of a column with fixed partitions whose length L
// divides the 4096-value tile and is at least 256 (L = 256, 512, 1024, 2048, 4096; the
// reference's TILE_SIZE is 4096, core/CudaUtils.cuh:18).
//
// Replaces, for those columns, the separate fit, bit-offset scan, table build and pack passes
// (fit.cu, glc_scan.cuh, pack.cu; in the reference wprocessPartitionsKernel,
// setBitOffsetsKernel and packDeltasKernelOptimized, compression/CompressionKernels.cuh:45-372,
// which read the values four times) with ONE kernel that reads every value once.  Every partition
// lies inside a tile (L divides 4096), so a CTA fits, measures and packs its tile alone: its words
// go into its own slot of a scratch array (slots of the worst-case size of a tile, bit offsets
// relative to the tile), with the partitions' descriptors and max errors and the tile's bit count.
// Then an exclusive scan of the tiles' bit counts gives every tile's first bit, and
// fixed_place_kernel (one CTA per tile) copies each tile's words to their place in the column
// and writes the metadata arrays from the descriptors.  No tile waits for another.
//
// The column's word array is allocated at its exact size between the two kernels (the scan gives
// the total); the slots cost one extra write and read of the compressed bits.
//
// The partition-length choice of a batch (choose_lengths_kernel) measures three lengths at once and
// packs the usual choice, 4096, on the way.
#include <type_traits>
#include "glc_group.cuh"
#include "glc_internal.h"
#include "glc_scan.cuh"

namespace glc {

constexpr int kCfMinLen = 256;
constexpr int kCfMaxParts = kDecodeTile / kCfMinLen;  // 16 partitions per tile at L = 256
constexpr int kCfMaxSegs = 16;                        // reduction segments (8 lanes each at L = 256)

// A launch: work item i = one 4096-value tile of column owner[i] (every column of one element
// type, tiles in order), or of `single` when cols is null.
struct FixedCompressArgs {
  const CfColumn* cols;
  const int32_t* owner;
  CfColumn single;
  int64_t nitems;
  uint32_t* slots;            // item i's words at slots + i * slot_words (tile-relative bits)
  int64_t slot_words;
  int64_t* tile_bits;         // per item: bits of the tile (nitems + 1 entries: the scan's input)
  const int64_t* tile_first;  // per item: exclusive scan of tile_bits over the launch (nitems + 1)
  unsigned long long* status; // the place: DEVERR_BOUNDS when a column's words would pass its array
  PartDesc* tdesc;            // the length choice that also packs at 4096: per item, the tile's one
  long long* terr;            // partition's descriptor (tile-relative offset) and max error
};

// ---- pieces of the compute warps -----------------------------------------------------------

// Per value, for the range tests of the partition: uint64 keeps the max of the high words, above
// 2^21 when some value exceeds 2^53 (direct copy; exactly 2^21 is decided by a rescan of the
// partition, cg_overflows) and below 2^19 iff every value is below 2^51; int64 keeps the OR of
// hi ^ (hi >> 31), below 2^19 iff every value is in [-2^51, 2^51); 4-byte values always fit.
template <typename T> __device__ __forceinline__ void value_flag(uint32_t& f, T y) {
  if (sizeof(T) == 8) {
    const uint32_t hi = (uint32_t)((uint64_t)y >> 32);
    if (TypeTraits<T>::is_signed) f |= hi ^ (uint32_t)((int32_t)hi >> 31);
    else f = hi > f ? hi : f;
  }
}
// Direct copy for the range flag of the partition whose `len` values start at value j0 of the tile (the
// reference copies a uint64 partition with a value above 2^53 directly): a largest high word of exactly
// 2^21 is decided by its values.
template <typename T> __device__ __forceinline__ bool cg_overflows(uint32_t flag, const uint8_t* stage, int j0, int len) {
  if (TypeTraits<T>::is_signed || sizeof(T) != 8) return false;
  bool over = flag > 0x200000u;
  if (flag == 0x200000u) {
#pragma unroll 1
    for (int j = j0; j < j0 + len && !over; j++) over = (uint64_t)*reinterpret_cast<const T*>(stage + cg_at<T>(j)) > (1ull << 53);
  }
  return over;
}

// K + y as a double from the bits of y (|y| <= 2^51).
template <typename T> __device__ __forceinline__ double magic_of(T y) {
  if (sizeof(T) == 8) {
    const uint64_t u = (uint64_t)y;
    return __hiloint2double((int)((uint32_t)(u >> 32) + 0x43380000u), (int)(uint32_t)u);
  } else if (TypeTraits<T>::is_signed) {
    return __hiloint2double((int)(0x43380000u + (uint32_t)((int32_t)y >> 31)), (int)y);
  } else {
    return __hiloint2double(0x43380000, (int)(uint32_t)y);
  }
}
__device__ __forceinline__ uint64_t madw_u(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
__device__ __forceinline__ int64_t madw_s(int32_t a, int32_t b, int64_t c) {
  int64_t d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// ---- the compress kernel ---------------------------------------------------------------------
// One CTA of 128 threads per 4096-value tile, six CTAs per SM; thread G owns the 32 consecutive values
// of group G.  A partition is a whole number of groups (L is a multiple of 32), so a group's fields,
// at the partition's width b, are exactly b whole words: the thread keeps its 32 fields in registers
// from the residual pass to the packing, and no field passes through shared memory.
//   load      16-byte asynchronous copies; group G's row starts G * (32 sizeof(T) + 16) bytes into
//             the stage, so the lanes of a warp read their rows in 16-byte pieces without bank
//             conflicts (rows without the 16 bytes would put every lane on the same banks);
//   A         exact sums of y and j y over the group from 32-bit halves, added over the partition;
//   solve     lane p of warp 0 fits partition p (fit.cu's arithmetic) and picks its residual mode;
//   B         residuals in 64-bit integers against an FP64 prediction rounded without conversion
//             instructions; their smallest, largest and a test that all fit 32 bits;
//   C         widths and offsets (every warp for itself, from the partitions' maxima), fields to
//             words with the width a compile-time constant (one funnel shift each), words through
//             shared memory (over the warp's values) to the tile's slot in 16-byte stores.
// A tile with a width above 31, a direct copy, a general-mode partition or an incomplete group takes
// the slow path: 64-bit residuals value by value, each group packed in its own row.  Its last group
// aside, a column of full tiles reaches it where a residual passes 2^30 (a jump inside a partition).
// What bounds it: instruction issue (56 % of the slots, about 50 instructions per value and lane, the
// sums' 64-bit additions and the residuals' integer tests first) and the five barriers of a tile,
// which the other CTAs of the SM cover in part; memory is at 39 %.  200M uint64 values at L = 4096:
// 903 -> 498 us (3.9 TB/s), against persistent CTAs of 256 compute threads, three per SM,
// that passed every field through shared memory and packed with half of their threads.
// Exact sums of a group (values past the column's end are zero): s = sum y_f, x = sum (i0 + f) y_f, by
// halves.  Every partial is below 32 * 2^12 * 2^32 = 2^49 in magnitude.
template <typename T>
__device__ __forceinline__ void cg_sums(const uint8_t* __restrict__ row, int i0, HalfSums<T>& hs, uint32_t& flag) {
  typedef typename HalfSums<T>::Acc Acc;
  Acc s_lo = 0, s_hi = 0, t_lo = 0, t_hi = 0;
#pragma unroll
  for (int k = 0; k < 32 / CgVec<T>::N; k++) {
    const CgVec<T> vec(row + 16 * k);
#pragma unroll
    for (int u = 0; u < CgVec<T>::N; u++) {
      const int f = k * CgVec<T>::N + u;
      const T y = vec.v[u];
      value_flag<T>(flag, y);
      if (sizeof(T) == 8) {
        const uint32_t yl = (uint32_t)(uint64_t)y, yh = (uint32_t)((uint64_t)y >> 32);
        s_lo = (Acc)madw_u(yl, 1u, (uint64_t)s_lo);
        if (f) t_lo = (Acc)madw_u(yl, (uint32_t)f, (uint64_t)t_lo);
        if (TypeTraits<T>::is_signed) {
          s_hi = (Acc)madw_s((int32_t)yh, 1, (int64_t)s_hi);
          if (f) t_hi = (Acc)madw_s((int32_t)yh, f, (int64_t)t_hi);
        } else {
          s_hi = (Acc)madw_u(yh, 1u, (uint64_t)s_hi);
          if (f) t_hi = (Acc)madw_u(yh, (uint32_t)f, (uint64_t)t_hi);
        }
      } else if (TypeTraits<T>::is_signed) {
        s_lo = (Acc)madw_s((int32_t)y, 1, (int64_t)s_lo);
        if (f) t_lo = (Acc)madw_s((int32_t)y, f, (int64_t)t_lo);
      } else {
        s_lo = (Acc)madw_u((uint32_t)y, 1u, (uint64_t)s_lo);
        if (f) t_lo = (Acc)madw_u((uint32_t)y, (uint32_t)f, (uint64_t)t_lo);
      }
    }
  }
  hs.s_lo = s_lo;
  hs.s_hi = s_hi;
  hs.x_lo = (Acc)i0 * s_lo + t_lo;
  hs.x_hi = (Acc)i0 * s_hi + t_hi;
}

// The residuals of a full group in one of the fast modes: y - pred as 64-bit integers, pred from the
// bits of K + pred (or K - pred, K + pred - c).  Keeps their low 32 bits in fl and the largest
// magnitude; false when some residual does not fit 32 bits (then only the slow path knows them: a
// difference taken modulo 2^64 that fits 32 bits is the difference, |y - pred| < 2^64 + 2^51 here and
// within 2^32 of a multiple of 2^64 only near 0).
template <typename T, int MODE>
__device__ __forceinline__ bool cg_resid(const uint8_t* __restrict__ row, int i0, double t0, double t1, double c,
                                         long long ci, uint32_t (&fl)[32], uint32_t& mag) {
  constexpr long long kBits = 0x4338000000000000ll;  // the bits of K
  double xd = (double)i0;
  int mn = 0, mx = 0;
  uint32_t wide = 0u;
#pragma unroll
  for (int k = 0; k < 32 / CgVec<T>::N; k++) {
    const CgVec<T> vec(row + 16 * k);
#pragma unroll
    for (int u = 0; u < CgVec<T>::N; u++) {
      const int f = k * CgVec<T>::N + u;
      const double x = __fma_rn(t1, xd, t0);
      xd = __dadd_rn(xd, 1.0);
      uint64_t d = TypeTraits<T>::is_signed ? (uint64_t)(long long)vec.v[u] : (uint64_t)vec.v[u];
      if (MODE == CF_NONNEG) {
        d -= (uint64_t)(__double_as_longlong(__dadd_rz(__dadd_rn(x, kHalfBias), kMagic)) - kBits);
      } else if (MODE == CF_NONPOS) {
        d += (uint64_t)(__double_as_longlong(__dadd_rz(__dsub_rn(kHalfBias, x), kMagic)) - kBits);
      } else {
        d -= (uint64_t)ci;
        d -= (uint64_t)(__double_as_longlong(__dadd_rz(__dadd_rn(__dsub_rn(x, c), 0.5), kMagic)) - kBits);
      }
      const int lo = (int)(uint32_t)d;
      fl[f] = (uint32_t)d;
      wide |= (uint32_t)(d >> 32) ^ (uint32_t)(lo >> 31);
      mn = min(mn, lo);
      mx = max(mx, lo);
    }
  }
  mag = max((uint32_t)mx, 0u - (uint32_t)mn);
  return wide == 0u;
}

template <typename T> __global__ void __launch_bounds__(kCgThreads, 6)
fixed_compress_kernel(const __grid_constant__ FixedCompressArgs a) {
  extern __shared__ __align__(128) uint8_t stage[];
  __shared__ long long s_acc[kCfMaxSegs][4];  // the segments' exact partial sums and range flags
  __shared__ uint32_t s_flag[kCfMaxSegs];
  __shared__ double s_t0[kCfMaxParts], s_t1[kCfMaxParts], s_c[kCfMaxParts];
  __shared__ long long s_ci[kCfMaxParts];
  __shared__ int s_mode[kCfMaxParts];
  __shared__ unsigned long long s_mx[kCfMaxSegs];
  const int tid = threadIdx.x, lane = tid & 31;

  const int64_t item = blockIdx.x;
  const CfColumn& col = a.cols ? a.cols[a.owner ? a.owner[item] : 0] : a.single;
  const int64_t t = item - col.item_base, e0 = t * kDecodeTile;
  const int64_t left = col.n - e0;
  const int cnt = (int)(left < kDecodeTile ? left : kDecodeTile);
  const int L = col.L, lg = 31 - __clz(L) - 5;  // groups per partition: 2^lg, 8 to 128
  const int np = (cnt + L - 1) / L;
  const int p = tid >> lg, i0 = 32 * (tid & ((1 << lg) - 1));  // this group's partition, its first index there
  const int lgW = lg < 5 ? lg : 5, W = 1 << lgW;               // lanes of a reduction segment
  const int seg = tid >> lgW, segs = 1 << (lg - lgW);          // segments of a partition: 1, 2 or 4
  const int glen = cnt - 32 * tid < 32 ? cnt - 32 * tid : 32;  // values of the group (<= 0: none)
  uint8_t* row = stage + tid * cg_row_bytes<T>();

  cg_load<T>(stage, reinterpret_cast<const T*>(col.values) + e0, cnt, tid);
  cg_load_wait();
  __syncthreads();

  {  // ---- A: exact sums and range flags per segment ----
    HalfSums<T> hs;
    uint32_t flag = 0;
    cg_sums<T>(row, i0, hs, flag);
    const long long c0 = seg_sum50((long long)hs.s_lo, W);
    const long long c1 = sizeof(T) == 8 ? seg_sum50((long long)hs.s_hi, W) : 0;
    const long long c2 = seg_sum50((long long)hs.x_lo, W);
    const long long c3 = sizeof(T) == 8 ? seg_sum50((long long)hs.x_hi, W) : 0;
    flag = TypeTraits<T>::is_signed ? seg_or_u32(flag, W) : seg_max_u32(flag, W);
    if ((tid & (W - 1)) == 0) {
      s_acc[seg][0] = c0;
      s_acc[seg][1] = c1;
      s_acc[seg][2] = c2;
      s_acc[seg][3] = c3;
      s_flag[seg] = flag;
    }
  }
  __syncthreads();
  if (tid < np) {  // ---- the lines ----
    long long a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    uint32_t flag = 0;
    for (int s = tid * segs; s < (tid + 1) * segs; s++) {
      a0 += s_acc[s][0];
      a1 += s_acc[s][1];
      a2 += s_acc[s][2];
      a3 += s_acc[s][3];
      flag = TypeTraits<T>::is_signed ? (flag | s_flag[s]) : (s_flag[s] > flag ? s_flag[s] : flag);
    }
    const int len = (cnt - tid * L) < L ? (cnt - tid * L) : L;
    const bool ovf = cg_overflows<T>(flag, stage, tid * L, len);  // a value above 2^53: direct copy
    const bool vsafe = sizeof(T) == 4 || flag < 0x80000u;
    double t0 = 0.0, t1 = 0.0, c = 0.0;
    long long ci = 0;
    int mode = CF_DIRECT;
    if (!ovf) {
      solve_line(len, (i128)a0 + (i128)a1 * ((i128)1 << 32), (i128)a2 + (i128)a3 * ((i128)1 << 32), t0, t1);
      mode = cf_mode<T>(t0, t1, len, vsafe, c, ci);
    }
    s_t0[tid] = t0;
    s_t1[tid] = t1;
    s_c[tid] = c;
    s_ci[tid] = ci;
    s_mode[tid] = mode;
  }
  __syncthreads();

  // ---- B: the residuals: low 32 bits kept, max |residual| per segment ----
  uint32_t fl[32];
  bool slow = false;
  {
    unsigned long long mx = 0;
    if (glen > 0) {
      const int mode = s_mode[p];
      const double t0 = s_t0[p], t1 = s_t1[p];
      uint32_t mag = 0u;
      bool ok = glen == 32;
      if (ok) {
        if (mode == CF_NONNEG) ok = cg_resid<T, CF_NONNEG>(row, i0, t0, t1, 0.0, 0, fl, mag);
        else if (TypeTraits<T>::is_signed && mode == CF_NONPOS) ok = cg_resid<T, CF_NONPOS>(row, i0, t0, t1, 0.0, 0, fl, mag);
        else if (sizeof(T) == 8 && mode == CF_OFFSET) ok = cg_resid<T, CF_OFFSET>(row, i0, t0, t1, s_c[p], s_ci[p], fl, mag);
        else ok = false;
      }
      mx = mag;
      slow = !ok;
      if (slow && mode != CF_DIRECT) {
        mx = 0;
        const double c = s_c[p];
        const long long ci = s_ci[p];
        double xi = (double)i0;
#pragma unroll 1
        for (int f = 0; f < glen; f++) {
          const T y = *reinterpret_cast<const T*>(row + f * (int)sizeof(T));
          const unsigned long long ad = (unsigned long long)abs_ref(cg_field<T>(y, xi, mode, t0, t1, c, ci));
          xi = __dadd_rn(xi, 1.0);
          mx = ad > mx ? ad : mx;
        }
      }
    }
    mx = seg_max_u64(mx, W);
    if ((tid & (W - 1)) == 0) s_mx[seg] = mx;
  }
  slow = __syncthreads_or(slow);

  // ---- widths and tile-relative offsets: lane q of every warp for partition q ----
  int b = 0, bl = 0, total;
  {
    int nb = 0;
    unsigned long long m = 0;
    if (lane < np) {
      for (int s = lane * segs; s < (lane + 1) * segs; s++) m = s_mx[s] > m ? s_mx[s] : m;
      const bool direct = s_mode[lane] == CF_DIRECT;
      b = direct ? (int)sizeof(T) * 8 : bits_for((long long)m);
      if (direct) m = 0;
      nb = ((cnt - lane * L) < L ? (cnt - lane * L) : L) * b;
    }
    int inc = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(FULL_MASK, inc, o);
      if (lane >= o) inc += v;
    }
    bl = inc - nb;
    total = __shfl_sync(FULL_MASK, inc, 31);
    const int bmax = (int)__reduce_max_sync(FULL_MASK, (unsigned)b);
    slow = slow || bmax > 31;
    if (tid < np) {
      // the descriptor with the tile-relative offset and the max error; fixed_place_kernel
      // completes the offset and writes the other metadata arrays from the descriptor
      const int64_t gp = t * col.parts_per_tile + tid;
      PartDesc d;
      d.theta0 = s_t0[tid];
      d.theta1 = s_t1[tid];
      d.bit_off = bl;
      d.start = (int32_t)(e0 + (int64_t)tid * L);
      d.bits_type = (b & 0xff) | ((s_mode[tid] == CF_DIRECT ? MODEL_DIRECT_COPY : MODEL_LINEAR) << 8);
      col.desc[gp] = d;
      col.err[gp] = (long long)m;
    }
    if (tid == 0) {
      a.tile_bits[item] = total;
      if (bmax > 0) atomicMax(col.stats + 1, (unsigned long long)bmax);
    }
  }

  uint32_t* out = a.slots + item * a.slot_words;
  const int bp = __shfl_sync(FULL_MASK, b, p & 31), blp = __shfl_sync(FULL_MASK, bl, p & 31);
  if (!slow) {
    // ---- C: the group's words, staged over its warp's rows (read by no other warp), then to the
    // slot, a reduction segment at a time: its groups are consecutive words of one partition ----
    uint32_t* stg = reinterpret_cast<uint32_t*>(stage + (tid & ~31) * cg_row_bytes<T>());
    __syncwarp();
    if (glen > 0) cg_pack_dispatch(bp, fl, stg + (lane & ~(W - 1)) * 32 + (lane & (W - 1)) * (bp | 1));
    __syncwarp();
    const int o0 = (blp >> 5) + (i0 >> 5) * bp;  // this group's first word in the tile
    for (int l = 0; l < 32; l += W) {
      const int bs = __shfl_sync(FULL_MASK, bp, l), os = __shfl_sync(FULL_MASK, o0, l);
      const int groups = __popc(__ballot_sync(FULL_MASK, glen > 0) >> l & (uint32_t)((1ull << W) - 1ull));
      // (16-byte aligned: a segment holds at least 8 groups)
      cg_copy_words<true>(stg + l * 32, out + os, groups * bs, bs, lane);
    }
    return;
  }
  // ---- slow path: each group's words in its own row, then to the slot, one thread per word ----
  if (glen > 0 && bp > 0) cg_pack_slow<T>(row, glen, i0, bp, s_mode[p], s_t0[p], s_t1[p], s_c[p], s_ci[p]);
  __syncthreads();
  for (int q = 0; q < np; q++) {
    const int bq = __shfl_sync(FULL_MASK, b, q), blq = __shfl_sync(FULL_MASK, bl, q);
    if (bq <= 0) continue;
    const int len = (cnt - q * L) < L ? (cnt - q * L) : L;
    const int nwp = (int)(((long long)len * bq + 31) >> 5);
    const uint32_t mb = bq > 1 ? 0xffffffffu / (uint32_t)bq + 1u : 0u;  // w / b by a multiply-high (w < 2^13)
    const uint8_t* rows = stage + (q << lg) * cg_row_bytes<T>();
    uint32_t* ow = out + (blq >> 5);
    for (int w = tid; w < nwp; w += kCgThreads) {
      const int g = bq > 1 ? (int)__umulhi((uint32_t)w, mb) : w;
      ow[w] = *reinterpret_cast<const uint32_t*>(rows + g * cg_row_bytes<T>() + 4 * (w - g * bq));
    }
  }
}

// The largest |residual| of a group's `len` values against one line, in mode MODE (0 where it is a
// direct copy): in 32 bits, or again in 64 where one does not fit.
template <typename T, int MODE>
__device__ __forceinline__ unsigned long long cg_max(const uint8_t* __restrict__ row, int len, int i0, double t0, double t1,
                                                     double c, long long ci) {
  int mn = 0, mx = 0;
  uint32_t wide = 0u;
  double xi = (double)i0;
#pragma unroll 4
  for (int f = 0; f < len; f++) {
    const long long d = cg_field<T>(*reinterpret_cast<const T*>(row + f * (int)sizeof(T)), xi, MODE, t0, t1, c, ci);
    xi = __dadd_rn(xi, 1.0);
    const int lo = (int)(uint32_t)(unsigned long long)d;
    wide |= (uint32_t)((unsigned long long)d >> 32) ^ (uint32_t)(lo >> 31);
    mn = min(mn, lo);
    mx = max(mx, lo);
  }
  if (!wide) return max((uint32_t)mx, 0u - (uint32_t)mn);
  unsigned long long m = 0;
  xi = (double)i0;
#pragma unroll 1
  for (int f = 0; f < len; f++) {
    const unsigned long long ad = (unsigned long long)abs_ref(
        cg_field<T>(*reinterpret_cast<const T*>(row + f * (int)sizeof(T)), xi, MODE, t0, t1, c, ci));
    xi = __dadd_rn(xi, 1.0);
    m = ad > m ? ad : m;
  }
  return m;
}
template <typename T>
__device__ __forceinline__ unsigned long long cg_max_mode(const uint8_t* __restrict__ row, int len, int i0, int mode, double t0,
                                                          double t1, double c, long long ci) {
  if (mode == CF_DIRECT) return 0;
  if (mode == CF_NONNEG) return cg_max<T, CF_NONNEG>(row, len, i0, t0, t1, c, ci);
  if (TypeTraits<T>::is_signed && mode == CF_NONPOS) return cg_max<T, CF_NONPOS>(row, len, i0, t0, t1, c, ci);
  if (sizeof(T) == 8 && mode == CF_OFFSET) return cg_max<T, CF_OFFSET>(row, len, i0, t0, t1, c, ci);
  return cg_max<T, CF_GENERAL>(row, len, i0, t0, t1, c, ci);
}

// A full group against the quarter's, the half's and the tile's line, all of them CF_NONNEG (the usual
// case), each value read once.  A width needs only the bit length of the largest |residual|, i.e. its
// FP64 exponent: the largest high word of |d| for the lines that only count bits.  With PACK the
// tile's line keeps its fields and exact maximum, as cg_resid does (false: one does not fit 32 bits).
template <typename T, bool PACK>
__device__ __forceinline__ bool cg_three(const uint8_t* __restrict__ row, const double (&t0)[3], const double (&t1)[3],
                                         const int (&i0)[3], uint32_t (&fl)[32], unsigned long long (&m)[3]) {
  constexpr long long kBits = 0x4338000000000000ll;
  double xd[3];
  uint32_t mh[3] = {0u, 0u, 0u}, wide = 0u;
  int mn = 0, mx = 0;
#pragma unroll
  for (int c = 0; c < 3; c++) xd[c] = (double)i0[c];
#pragma unroll
  for (int k = 0; k < 32 / CgVec<T>::N; k++) {
    const CgVec<T> vec(row + 16 * k);
#pragma unroll
    for (int u = 0; u < CgVec<T>::N; u++) {
      const int f = k * CgVec<T>::N + u;
      const double yc = magic_of<T>(vec.v[u]);  // K + y
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double pm = __dadd_rz(__dadd_rn(__fma_rn(t1[c], xd[c], t0[c]), kHalfBias), kMagic);  // K + pred
        xd[c] = __dadd_rn(xd[c], 1.0);
        if (PACK && c == 2) {
          const uint64_t y = TypeTraits<T>::is_signed ? (uint64_t)(long long)vec.v[u] : (uint64_t)vec.v[u];
          const uint64_t d = y - (uint64_t)(__double_as_longlong(pm) - kBits);
          const int lo = (int)(uint32_t)d;
          fl[f] = (uint32_t)d;
          wide |= (uint32_t)(d >> 32) ^ (uint32_t)(lo >> 31);
          mn = min(mn, lo);
          mx = max(mx, lo);
        } else {
          const uint32_t h = (uint32_t)__double2hiint(__dsub_rn(yc, pm)) & 0x7fffffffu;
          mh[c] = max(mh[c], h);
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++) m[c] = mh[c] ? (1ull << ((mh[c] >> 20) - 1023)) : 0ull;  // the same bit length
  if (PACK) m[2] = max((uint32_t)mx, 0u - (uint32_t)mn);
  return wide == 0u;
}

// The partition-length choice of the batched compress, a CTA of 128 threads per tile as in
// fixed_compress_kernel, a warp per 1024-value quarter: the tile's quarters, its two halves and the
// whole tile are fitted from exact per-quarter sums (the index offsets of a half or the tile added
// exactly); every value's residual is measured against the three lines that cover it, and the bits of
// each candidate length are added into the column's choice_bits[0..2] (1024, 2048, 4096).  The widths
// are the ones the compress at that length computes, so the column's size is exact.  With PACK the
// tile is also compressed at length 4096 -- the usual choice -- exactly as fixed_compress_kernel
// would (the tile's line from the same exact sums, the same residual modes and packing): its words
// into its slot, its descriptor and max error into tdesc / terr, its bits into tile_bits.
// Bound by instruction issue (three lines per value).  169M values of 1024 int32, int64 and uint64
// columns: 1068 -> 620 us in all, against persistent CTAs of 256 compute threads that staged the fields.
template <typename T, bool PACK> __global__ void __launch_bounds__(kCgThreads, 5)
choose_lengths_kernel(const __grid_constant__ FixedCompressArgs a) {
  extern __shared__ __align__(128) uint8_t stage[];
  __shared__ long long s_acc[4][4];  // per quarter: exact partial sums and range flags
  __shared__ uint32_t s_flag[4];
  __shared__ double s_t0[7], s_t1[7], s_c[7];  // line 0 the tile, 1-2 its halves, 3-6 its quarters
  __shared__ long long s_ci[7];
  __shared__ int s_mode[7], s_len[7];
  __shared__ unsigned long long s_m[4][3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t item = blockIdx.x;
  const CfColumn& col = a.cols[a.owner[item]];
  const int64_t e0 = (item - col.item_base) * kDecodeTile, left = col.n - e0;
  const int cnt = (int)(left < kDecodeTile ? left : kDecodeTile);
  const int glen = cnt - 32 * tid < 32 ? cnt - 32 * tid : 32;  // values of the group (<= 0: none)
  uint8_t* row = stage + tid * cg_row_bytes<T>();
  cg_load<T>(stage, reinterpret_cast<const T*>(col.values) + e0, cnt, tid);
  cg_load_wait();
  __syncthreads();
  {  // exact sums per quarter and the range flags
    HalfSums<T> hs;
    uint32_t flag = 0;
    cg_sums<T>(row, 32 * lane, hs, flag);
    const long long c0 = seg_sum50((long long)hs.s_lo, 32);
    const long long c1 = sizeof(T) == 8 ? seg_sum50((long long)hs.s_hi, 32) : 0;
    const long long c2 = seg_sum50((long long)hs.x_lo, 32);
    const long long c3 = sizeof(T) == 8 ? seg_sum50((long long)hs.x_hi, 32) : 0;
    flag = TypeTraits<T>::is_signed ? seg_or_u32(flag, 32) : seg_max_u32(flag, 32);
    if (lane == 0) {
      s_acc[warp][0] = c0;
      s_acc[warp][1] = c1;
      s_acc[warp][2] = c2;
      s_acc[warp][3] = c3;
      s_flag[warp] = flag;
    }
  }
  __syncthreads();
  if (tid < 7) {  // the lines
    const int l = tid;
    const int q0 = l == 0 ? 0 : (l < 3 ? (l - 1) * 2 : l - 3);
    const int q1 = l == 0 ? 4 : (l < 3 ? q0 + 2 : q0 + 1);
    i128 sy = 0, sxy = 0;
    uint32_t flag = 0;
    for (int q = q0; q < q1; q++) {
      flag = TypeTraits<T>::is_signed ? (flag | s_flag[q]) : (s_flag[q] > flag ? s_flag[q] : flag);
      const i128 qy = (i128)s_acc[q][0] + (i128)s_acc[q][1] * ((i128)1 << 32);
      sy += qy;
      sxy += (i128)s_acc[q][2] + (i128)s_acc[q][3] * ((i128)1 << 32) + (i128)(1024 * (q - q0)) * qy;  // quarter index -> line index
    }
    int len = cnt - 1024 * q0;
    len = len < 0 ? 0 : (len < 1024 * (q1 - q0) ? len : 1024 * (q1 - q0));
    const bool ovf = len > 0 && cg_overflows<T>(flag, stage, 1024 * q0, len);
    const bool vsafe = sizeof(T) == 4 || flag < 0x80000u;
    double t0 = 0.0, t1 = 0.0, c = 0.0;
    long long ci = 0;
    int mode = CF_DIRECT;
    if (len > 0 && !ovf) {
      solve_line(len, sy, sxy, t0, t1);
      mode = cf_mode<T>(t0, t1, len, vsafe, c, ci);
    }
    s_t0[l] = t0;
    s_t1[l] = t1;
    s_c[l] = c;
    s_ci[l] = ci;
    s_mode[l] = mode;
    s_len[l] = len;
  }
  __syncthreads();
  uint32_t fl[32];  // PACK: the low 32 bits of each value's residual against the tile's line
  bool slow = false;
  {  // max |residual| of each value against its quarter's, its half's and the tile's line
    const int ls[3] = {3 + warp, 1 + (warp >> 1), 0};
    const int i0[3] = {32 * lane, 32 * (tid & 63), 32 * tid};
    unsigned long long mx[3] = {0, 0, 0};
    if (glen > 0) {
      bool fused = glen == 32, tile_done = false;
#pragma unroll
      for (int c = 0; c < 3; c++) fused = fused && s_mode[ls[c]] == CF_NONNEG;
      if (fused) {
        const double t0[3] = {s_t0[ls[0]], s_t0[ls[1]], s_t0[ls[2]]}, t1[3] = {s_t1[ls[0]], s_t1[ls[1]], s_t1[ls[2]]};
        tile_done = cg_three<T, PACK>(row, t0, t1, i0, fl, mx);
        slow = PACK && !tile_done;
      } else {
#pragma unroll 1
        for (int c = 0; c < 2; c++) {  // (one body for both lines)
          const int l = c ? 1 + (warp >> 1) : 3 + warp, i = c ? 32 * (tid & 63) : 32 * lane;
          const unsigned long long m = cg_max_mode<T>(row, glen, i, s_mode[l], s_t0[l], s_t1[l], s_c[l], s_ci[l]);
          if (c) mx[1] = m;
          else mx[0] = m;
        }
        if (PACK && glen == 32) {
          const int mode = s_mode[0];
          uint32_t mag = 0u;
          if (mode == CF_NONNEG) tile_done = cg_resid<T, CF_NONNEG>(row, i0[2], s_t0[0], s_t1[0], 0.0, 0, fl, mag);
          else if (TypeTraits<T>::is_signed && mode == CF_NONPOS)
            tile_done = cg_resid<T, CF_NONPOS>(row, i0[2], s_t0[0], s_t1[0], 0.0, 0, fl, mag);
          else if (sizeof(T) == 8 && mode == CF_OFFSET)
            tile_done = cg_resid<T, CF_OFFSET>(row, i0[2], s_t0[0], s_t1[0], s_c[0], s_ci[0], fl, mag);
          mx[2] = mag;
        }
        slow = PACK && !tile_done;
      }
      if (!tile_done) mx[2] = cg_max_mode<T>(row, glen, i0[2], s_mode[0], s_t0[0], s_t1[0], s_c[0], s_ci[0]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) mx[c] = seg_max_u64(mx[c], 32);
    if (lane == 0) {
      s_m[warp][0] = mx[0];
      s_m[warp][1] = mx[1];
      s_m[warp][2] = mx[2];
    }
  }
  slow = __syncthreads_or(slow);
  // lane l < 7 (of every warp): line l's width and bits; the three lengths' sums by shuffles
  unsigned long long add[3] = {0, 0, 0}, m_line = 0;
  int b_line = 0;
  if (lane < 7 && s_len[lane] > 0) {
    const int l = lane;
    const int c = l == 0 ? 2 : (l < 3 ? 1 : 0);                  // index into s_m's lines
    const int w0 = l == 0 ? 0 : (l < 3 ? 2 * (l - 1) : l - 3);   // the line's quarters
    const int w1 = l == 0 ? 4 : (l < 3 ? w0 + 2 : w0 + 1);
    for (int w = w0; w < w1; w++) m_line = s_m[w][c] > m_line ? s_m[w][c] : m_line;
    b_line = s_mode[l] == CF_DIRECT ? (int)sizeof(T) * 8 : bits_for((long long)m_line);
    add[c] = (unsigned long long)s_len[l] * (unsigned long long)b_line;
  }
  if (warp == 0) {
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) add[c] += __shfl_xor_sync(FULL_MASK, add[c], o);  // lanes 0-7
  }
  if (tid == 0) {
    for (int c = 0; c < 3; c++)
      if (add[c]) atomicAdd(col.choice_bits + c, add[c]);
    if (PACK) {  // the tile as one partition of 4096 (line 0): width, descriptor, max error, bits
      const bool direct = s_mode[0] == CF_DIRECT;
      PartDesc d;
      d.theta0 = s_t0[0];
      d.theta1 = s_t1[0];
      d.bit_off = 0;
      d.start = (int32_t)e0;
      d.bits_type = (b_line & 0xff) | ((direct ? MODEL_DIRECT_COPY : MODEL_LINEAR) << 8);
      a.tdesc[item] = d;
      a.terr[item] = direct ? 0 : (long long)m_line;
      a.tile_bits[item] = (int64_t)cnt * b_line;
      if (b_line > 0) atomicMax(col.stats + 1, (unsigned long long)b_line);
    }
  }
  if (!PACK) return;
  const int b = __shfl_sync(FULL_MASK, b_line, 0);
  uint32_t* out = a.slots + item * a.slot_words;
  if (!slow && b <= 31) {  // each warp's groups, staged over its rows and copied (fixed_compress_kernel)
    uint32_t* stg = reinterpret_cast<uint32_t*>(stage + (tid & ~31) * cg_row_bytes<T>());
    if (glen > 0) cg_pack_dispatch(b, fl, stg + lane * (b | 1));
    __syncwarp();
    const int groups = __popc(__ballot_sync(FULL_MASK, glen > 0));
    cg_copy_words<true>(stg, out + 32 * warp * b, groups * b, b, lane);
    return;
  }
  if (glen > 0 && b > 0) cg_pack_slow<T>(row, glen, 32 * tid, b, s_mode[0], s_t0[0], s_t1[0], s_c[0], s_ci[0]);
  __syncwarp();
  for (int l = 0; l < 32; l++) {
    const int gl = __shfl_sync(FULL_MASK, glen, l);
    if (gl <= 0) break;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(stage + ((tid & ~31) + l) * cg_row_bytes<T>());
    const int nw = (gl * b + 31) >> 5;
    for (int w = lane; w < nw; w += 32) out[(32 * warp + l) * b + w] = q[w];
  }
}

// Places every tile of the launch in its column, one CTA per tile: the tile's first bit F (the
// scan of the tiles' bits, relative to the column's first tile) is added to its partitions'
// descriptors, whose fields also fill the other metadata arrays (starts, ends, types, params,
// bits, offsets), the tile's decode-table entry is written, and the words whose first bit lies in the
// tile are written -- from the tile's slot with a funnel shift, ORed with the first bits of every
// later tile of the column that starts inside the same word (tiles without bits are skipped).  The
// column's last tile writes the final decode-table entry and the total, and zeroes the padding.
//
// Word w of the column, when its bits all lie in the tile, is funnelshift(slot[i], slot[i + 1], r)
// with i = w - (first word the tile owns) and r = -F mod 32: each thread loads kPlaceUnroll slot
// words before it uses one (the copy is bound by memory latency, so many loads are kept in
// flight), and takes slot[i + 1] from the next lane.
constexpr int kPlaceThreads = 128;
constexpr int kPlaceUnroll = 4;
constexpr int kPlaceVec = 4;

__global__ void __launch_bounds__(kPlaceThreads, 8) fixed_place_kernel(FixedCompressArgs a) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int64_t item = blockIdx.x; item < a.nitems; item += gridDim.x) {
    const CfColumn& col = a.cols ? a.cols[a.owner ? a.owner[item] : 0] : a.single;
    if (!col.words) continue;  // a column this launch does not place
    const int64_t t = item - col.item_base;
    const int64_t col_end = col.item_base + col.ntiles;  // the column's items are [item_base, col_end)
    const int64_t base = a.tile_first[col.item_base];
    const int64_t first = a.tile_first[item] - base;
    const int64_t bits = a.tile_bits[item];
    uint32_t* __restrict__ words = col.words;
    const int64_t e0 = t * kDecodeTile;
    const int cnt = (int)((col.n - e0) < kDecodeTile ? (col.n - e0) : kDecodeTile);
    const int np = (cnt + col.L - 1) / col.L;
    if (tid < np) {  // the tile's partitions: their metadata arrays from the descriptor
      const int64_t gp = t * col.parts_per_tile + tid;
      PartDesc d;
      if (a.tdesc) {  // packed by the length choice: the tile is one partition
        d = a.tdesc[item];
        col.err[gp] = a.terr[item];
      } else {
        d = col.desc[gp];
      }
      const int64_t off = d.bit_off + first;
      const int len = (cnt - tid * col.L) < col.L ? (cnt - tid * col.L) : col.L;
      d.bit_off = off;
      col.desc[gp] = d;
      col.starts[gp] = d.start;
      col.ends[gp] = d.start + len;
      col.types[gp] = d.bits_type >> 8;
      col.params[4 * gp] = d.theta0;
      col.params[4 * gp + 1] = d.theta1;
      col.params[4 * gp + 2] = 0.0;
      col.params[4 * gp + 3] = 0.0;
      col.bits[gp] = d.bits_type & 0xff;
      col.offs[gp] = off;
    }
    const int64_t total = a.tile_first[col_end - 1] - base + a.tile_bits[col_end - 1];
    if (tid == 0) {
      TileInfo ti;
      ti.bit_lo = first;
      ti.p_first = (int32_t)(t * col.parts_per_tile);
      ti.p_last = (int32_t)(t * col.parts_per_tile + np - 1);
      col.tiles[t] = ti;
      if (t == col.ntiles - 1) {
        TileInfo te;
        te.bit_lo = total;
        te.p_first = te.p_last = (int32_t)(col.P - 1);
        col.tiles[col.ntiles] = te;
        col.stats[0] = (unsigned long long)total;
      }
    }
    // words [w_begin, w_end) have their first bit in the tile; [w_begin, w_begin + nfull) lie in it
    const int64_t w_begin = (first + 31) >> 5, w_end = (first + bits + 31) >> 5;
    if (w_end > col.words_cap) {  // the caller sized the array from another count: report, write nothing
      if (tid == 0) atomicExch(a.status, (unsigned long long)DEVERR_BOUNDS);
      continue;
    }
    const uint32_t* __restrict__ slot = a.slots + item * a.slot_words;
    if ((first & 127) == 0 && ((bits & 31) == 0 || item == col_end - 1) &&
        (reinterpret_cast<uintptr_t>(words + w_begin) & 15) == 0) {
      // the usual case: every partition holds L * width bits with L a multiple of 256, so every
      // tile starts on a 16-byte boundary of its column and only a column's last tile ends inside
      // a word -- a vector copy of the slot's first nw words
      const int64_t nw = w_end - w_begin;
      const uint4* __restrict__ src = reinterpret_cast<const uint4*>(slot);
      uint4* __restrict__ dst = reinterpret_cast<uint4*>(words + w_begin);
      const int64_t n4 = nw >> 2;
      for (int64_t i0 = 0; i0 < n4; i0 += (int64_t)kPlaceThreads * kPlaceVec) {
        uint4 v[kPlaceVec];
#pragma unroll
        for (int u = 0; u < kPlaceVec; u++) {
          const int64_t i = i0 + tid + u * kPlaceThreads;
          if (i < n4) v[u] = __ldg(src + i);
        }
#pragma unroll
        for (int u = 0; u < kPlaceVec; u++) {
          const int64_t i = i0 + tid + u * kPlaceThreads;
          if (i < n4) dst[i] = v[u];
        }
      }
      if (tid < (int)(nw & 3)) words[w_begin + 4 * n4 + tid] = slot[4 * n4 + tid];
    } else {
      const int64_t nfull = ((first + bits) >> 5) - w_begin;  // may be negative: the tile owns no full word
      const int r = (int)((32 * w_begin - first) & 31);
      // slot words [0, nfull] are read (the one after the last full word feeds its funnel shift; the
      // slot holds one word more than the widest tile's bits)
      for (int64_t i0 = 0; i0 < nfull; i0 += (int64_t)kPlaceThreads * kPlaceUnroll) {
        uint32_t lo[kPlaceUnroll], hi[kPlaceUnroll];
#pragma unroll
        for (int u = 0; u < kPlaceUnroll; u++) {
          const int64_t i = i0 + tid + u * kPlaceThreads;
          lo[u] = i <= nfull ? __ldg(slot + i) : 0u;
          hi[u] = (lane == 31 && i + 1 <= nfull) ? __ldg(slot + i + 1) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kPlaceUnroll; u++) {
          const uint32_t nx = __shfl_down_sync(FULL_MASK, lo[u], 1);
          const uint32_t h = lane == 31 ? hi[u] : nx;
          const int64_t i = i0 + tid + u * kPlaceThreads;
          if (i < nfull) words[w_begin + i] = __funnelshift_r(lo[u], h, r);
        }
      }
      if (tid == 0 && w_end > w_begin && ((first + bits) & 31) != 0) {
        // the tile ends inside its last word: that word's tile bits, then the next tiles' first bits
        const int64_t w = w_end - 1, i = w - w_begin;
        const int64_t avail = first + bits - 32 * w;  // 1..31 tile bits in the word
        uint32_t v = __funnelshift_r(slot[i], slot[i + 1], r) & ((1u << avail) - 1u);
        int64_t pos = first + bits;  // column bit where the next tile starts
        for (int64_t u = item + 1; u < col_end && pos < 32 * w + 32; u++) {
          const int64_t ub = a.tile_bits[u];
          if (ub == 0) continue;
          const int64_t take = (32 * w + 32 - pos) < ub ? (32 * w + 32 - pos) : ub;
          uint32_t f = a.slots[u * a.slot_words];
          if (take < 32) f &= (1u << take) - 1u;
          v |= f << (pos - 32 * w);
          pos += ub;
        }
        words[w] = v;
      }
    }
    if (t == col.ntiles - 1 && col.nwords_alloc > 0) {  // the decoders' zeroed read-ahead after the bitstream
      const int64_t wt = (total + 31) >> 5;
      int64_t pad_end = ((wt + 3) & ~3ll) + 8;
      pad_end = pad_end < col.nwords_alloc ? pad_end : col.nwords_alloc;
      for (int64_t w = wt + tid; w < pad_end && w < col.words_cap; w += kPlaceThreads) words[w] = 0u;
    }
  }
}

template <typename T> static cudaError_t launch_fixed_compress_t(const FixedCompressArgs& a, cudaStream_t s) {
  // (34 KB per CTA for 8-byte types, 18 KB for 4-byte ones: within the default limit)
  fixed_compress_kernel<T><<<(unsigned)a.nitems, kCgThreads, cg_stage_bytes<T>(), s>>>(a);
  return cudaGetLastError();
}

static cudaError_t launch_fixed_compress_dt(glc_dtype dt, const FixedCompressArgs& a, cudaStream_t s) {
  switch (dt) {
    case GLC_I32: return launch_fixed_compress_t<int32_t>(a, s);
    case GLC_I64: return launch_fixed_compress_t<int64_t>(a, s);
    case GLC_U64: return launch_fixed_compress_t<uint64_t>(a, s);
    case GLC_U32: return launch_fixed_compress_t<uint32_t>(a, s);
  }
  return cudaErrorInvalidValue;
}

template <typename T, bool PACK> static cudaError_t launch_choose_t(const FixedCompressArgs& a, cudaStream_t s) {
  choose_lengths_kernel<T, PACK><<<(unsigned)a.nitems, kCgThreads, cg_stage_bytes<T>(), s>>>(a);
  return cudaGetLastError();
}

static void carve(FixedCompressArgs& a, glc_dtype dt, void* scratch);

cudaError_t launch_choose_lengths(glc_dtype dt, const CfColumn* cols, const int32_t* owner, int64_t nitems,
                                  cudaStream_t s, void* scratch, PartDesc* tdesc, long long* terr) {
  if (nitems <= 0) return cudaSuccess;
  FixedCompressArgs a{};
  a.cols = cols;
  a.owner = owner;
  a.nitems = nitems;
  const bool pack = scratch != nullptr;
  if (pack) {
    carve(a, dt, scratch);
    a.tdesc = tdesc;
    a.terr = terr;
  }
  switch (dt) {
    case GLC_I32: return pack ? launch_choose_t<int32_t, true>(a, s) : launch_choose_t<int32_t, false>(a, s);
    case GLC_I64: return pack ? launch_choose_t<int64_t, true>(a, s) : launch_choose_t<int64_t, false>(a, s);
    case GLC_U64: return pack ? launch_choose_t<uint64_t, true>(a, s) : launch_choose_t<uint64_t, false>(a, s);
    case GLC_U32: return pack ? launch_choose_t<uint32_t, true>(a, s) : launch_choose_t<uint32_t, false>(a, s);
  }
  return cudaErrorInvalidValue;
}

int64_t fixed_compress_worst_words(glc_dtype dt, int64_t n) {
  const int64_t per_value = (dt == GLC_I64 || dt == GLC_U64) ? 64 : 33;  // widest field of the type
  return (n * per_value + 31) / 32 + 12;  // + the decoders' zeroed read-ahead
}

bool fixed_compress_supported(int64_t n, int32_t L) {
  return n > 0 && L >= kCfMinLen && L <= kDecodeTile && (kDecodeTile % L) == 0;
}

// Words of one tile's slot: the widest fields of the type (64 bits for 8-byte types, 33 for 4-byte
// ones) plus the word the placing funnel shift reads after the last, rounded to 16 bytes.
int64_t fixed_compress_slot_words(glc_dtype dt) {
  const int64_t per_value = (dt == GLC_I64 || dt == GLC_U64) ? 64 : 33;
  return ((kDecodeTile * per_value + 31) / 32 + 1 + 3) & ~3ll;
}

// Scratch of a launch over nitems tiles: slots, the tiles' bits, their scan and its tile sums.
size_t fixed_compress_scratch_bytes(glc_dtype dt, int64_t nitems) {
  return (size_t)nitems * fixed_compress_slot_words(dt) * 4 + (size_t)(nitems + 1) * 16 +
         (size_t)(scan_num_tiles(nitems + 1) + 1) * 8 + 256;
}

static void carve(FixedCompressArgs& a, glc_dtype dt, void* scratch) {
  uint8_t* sp = reinterpret_cast<uint8_t*>(scratch);
  a.slot_words = fixed_compress_slot_words(dt);
  a.slots = reinterpret_cast<uint32_t*>(sp);
  sp += (size_t)a.nitems * a.slot_words * 4;
  a.tile_bits = reinterpret_cast<int64_t*>(sp);
  sp += (size_t)(a.nitems + 1) * 8;
  a.tile_first = reinterpret_cast<int64_t*>(sp);
}

// Pass 1 for one launch: fit, residuals and each tile's words into its slot, the tiles' bits, and
// their exclusive scan (all the launch's bits into *total where it is given).
static cudaError_t compress_pass(glc_dtype dt, FixedCompressArgs& a, void* scratch, int64_t* total, cudaStream_t s) {
  carve(a, dt, scratch);
  cudaError_t e;
  if ((e = launch_fixed_compress_dt(dt, a, s)) != cudaSuccess) return e;
  int64_t* first = const_cast<int64_t*>(a.tile_first);
  int64_t* tmp = first + a.nitems + 1;
  return exclusive_scan<int64_t>(a.tile_bits, first, a.nitems, total, tmp, s);
}

static cudaError_t place_pass(const FixedCompressArgs& a, int num_sms, cudaStream_t s) {
  const int64_t cap = (int64_t)num_sms * 8;  // eight CTAs of 128 threads per SM (twice the tiles in flight of four of 256: 33 -> 26 us per 32M values)
  int64_t grid = a.nitems < cap ? a.nitems : cap;
  if (grid < 1) grid = 1;
  fixed_place_kernel<<<(unsigned)grid, kPlaceThreads, 0, s>>>(a);
  return cudaGetLastError();
}

// One column: values (n of dt, fixed partitions of L) into c's metadata arrays and tables
// (allocated by the caller for P = ceil(n / L) partitions); scratch holds
// fixed_compress_scratch_bytes(dt, ntiles) bytes.  Pass 1 leaves stats[0] = the column's total bits,
// stats[1] = its widest field (stats[0..3] zeroed here); the caller reads them, allocates the words
// and calls launch_fixed_place.
cudaError_t launch_fixed_compress(glc_dtype dt, const void* values, glc_column* c, int32_t L, void* scratch,
                                  unsigned long long* stats, cudaStream_t s) {
  FixedCompressArgs a{};
  CfColumn& col = a.single;
  col.values = values;
  col.n = c->n;
  col.L = L;
  col.parts_per_tile = kDecodeTile / L;
  col.P = c->P;
  col.ntiles = c->ntiles;
  col.item_base = 0;
  col.starts = c->d_start;
  col.ends = c->d_end;
  col.types = c->d_types;
  col.params = c->d_params;
  col.bits = c->d_bits;
  col.offs = c->d_offs;
  col.err = c->d_err;
  col.desc = c->d_desc;
  col.tiles = c->d_tiles;
  col.stats = stats;
  a.nitems = c->ntiles;
  cudaError_t e;
  if ((e = cudaMemsetAsync(stats, 0, 4 * sizeof(unsigned long long), s)) != cudaSuccess) return e;
  // the total: the scan's grand total (the column is the whole launch)
  return compress_pass(dt, a, scratch, (int64_t*)stats, s);
}

// Pass 2 for one column: its words into c->d_words (c->nwords_alloc words), its offsets, descriptors
// and decode-table entries completed.  Same arguments as launch_fixed_compress.
cudaError_t launch_fixed_place(glc_dtype dt, glc_column* c, int32_t L, void* scratch, unsigned long long* stats,
                               cudaStream_t s) {
  FixedCompressArgs a{};
  CfColumn& col = a.single;
  col.n = c->n;
  col.L = L;
  col.parts_per_tile = kDecodeTile / L;
  col.P = c->P;
  col.ntiles = c->ntiles;
  col.item_base = 0;
  col.nwords_alloc = c->nwords_alloc;
  col.words_cap = c->nwords_alloc;
  col.starts = c->d_start;
  col.ends = c->d_end;
  col.types = c->d_types;
  col.params = c->d_params;
  col.bits = c->d_bits;
  col.offs = c->d_offs;
  col.desc = c->d_desc;
  col.tiles = c->d_tiles;
  col.words = c->d_words;
  col.stats = stats;
  a.nitems = c->ntiles;
  a.status = stats + 2;
  carve(a, dt, scratch);
  return place_pass(a, c->ctx ? c->ctx->num_sms : 148, s);
}

// The columns packed at 4096 by launch_choose_lengths (same cols layout and owner list, same
// scratch, tdesc and terr): the scan of the tiles' bits and the place of every column whose words
// are set in cols (the others are skipped).
cudaError_t launch_place_prepacked(glc_dtype dt, const CfColumn* cols, const int32_t* owner, int64_t nitems,
                                   void* scratch, PartDesc* tdesc, long long* terr, unsigned long long* status,
                                   int num_sms, cudaStream_t s) {
  if (nitems <= 0) return cudaSuccess;
  FixedCompressArgs a{};
  a.cols = cols;
  a.owner = owner;
  a.nitems = nitems;
  a.status = status;
  a.tdesc = tdesc;
  a.terr = terr;
  carve(a, dt, scratch);
  int64_t* first = const_cast<int64_t*>(a.tile_first);
  cudaError_t e = exclusive_scan<int64_t>(a.tile_bits, first, a.nitems, nullptr, first + a.nitems + 1, s);
  if (e != cudaSuccess) return e;
  return place_pass(a, num_sms, s);
}

// Many columns of one element type: cols (device, each with its own arrays, its exact word array
// and words_cap, stats zeroed) and owner (device, nitems entries: the column of each item, items in
// column order); both passes in stream order.  scratch: fixed_compress_scratch_bytes(dt, nitems).
cudaError_t launch_fixed_compress_batch(glc_dtype dt, const CfColumn* cols, const int32_t* owner, int64_t nitems,
                                        void* scratch, unsigned long long* status, int num_sms, cudaStream_t s) {
  if (nitems <= 0) return cudaSuccess;
  FixedCompressArgs a{};
  a.cols = cols;
  a.owner = owner;
  a.nitems = nitems;
  a.status = status;
  cudaError_t e;
  if ((e = compress_pass(dt, a, scratch, nullptr, s)) != cudaSuccess) return e;
  return place_pass(a, num_sms, s);
}

}  // namespace glc
