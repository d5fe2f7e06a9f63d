// partition.cu -- variable-length partitioning by model cost, on the device.
//
// Replaces VariableLengthPartitioner<T>::partition (compression/CpuPartitioner.cuh:342-422),
// which the reference runs single-threaded on the host (its GPU alternative,
// GPUVariableLengthPartitionerV6, sizes partitions by a variance heuristic and never merges).
//
// Cost of a partition [a, b): 80 + (b - a) * bits / 8 bytes (CpuPartitioner.cuh:128-138), with
// bits from the exact-sum least-squares fit of [a, b) (glc_device.cuh).
//
// Split.  The reference walks from 0: at start s it tries sizes 128..3712 (steps of 128 up to
// 640, then 256 up to 2176, then 512; CpuPartitioner.cuh:150-175), keeps the first size with
// the lowest cost per value and jumps there.  Every start on that walk is a multiple of 128 and
// the best end of a start depends on nothing else.  Short columns evaluate every start (one warp
// each).  Longer ones are cut into ranges: each range is walked from its first block and from the
// block where the previous range's first walk leaves it (one warp per range, each start's best end
// evaluated on the way), and the ranges are chained through the exits of the visited starts; when
// the walk from 0 enters a range at a start no walk visited, every start is evaluated after all and
// the ranges are chained through the exits of all their possible entry points.  The max |delta| each
// evaluation measured for the partition it chose is kept, so the split partitions' costs need no
// second pass over the values.
//
// Merge.  The reference absorbs right neighbours left to right while the merged cost is lower
// (CpuPartitioner.cuh:198-242).  Here merging runs in rounds: the profitable adjacent pairs
// with (index + round) even merge, so the chosen pairs never overlap; rounds stop when no pair is
// profitable (at most 64 rounds).
//
// Fits use exact 128-bit sums from a prefix over 128-value blocks (every boundary here is a
// multiple of 128 or n), so each candidate's line costs O(1) and only its max |delta| needs a
// pass over the values.  The CPU oracle restates this algorithm step for step.
#include <algorithm>
#include "glc_internal.h"
#include "glc_scan.cuh"

namespace glc {

constexpr int kNumSizes = 14;
__constant__ int c_sizes[kNumSizes] = {128, 256, 384, 512, 640, 896, 1152, 1408, 1664, 1920, 2176, 2688, 3200, 3712};
__host__ __device__ constexpr int split_size(int k) {
  return k < 5 ? 128 * (k + 1) : k < 11 ? 640 + 256 * (k - 4) : 2176 + 512 * (k - 10);
}
static_assert(split_size(0) == 128 && split_size(4) == 640 && split_size(5) == 896 && split_size(10) == 2176 &&
              split_size(11) == 2688 && split_size(13) == 3712, "candidate sizes");
constexpr int kMaxJumpBlocks = 29;  // 3712 / 128
constexpr int kMaxRangeBlocks = kMaxJumpBlocks * 128;
constexpr int kWalksPerSM = 7;  // range walks (one warp each) whose reaches fit an SM's shared memory
// Columns up to this many blocks (8.4M values) have every start evaluated, all in parallel; longer
// ones walk.  A walk's starts follow one another (about 10 us each), so short columns are bound by
// its longest chain: 3M timestamps took 3070 us of walks of 2048 blocks and take 141 us this way;
// 200M values would take 26 times the evaluations of the walks.  A whole compress, every start / walks,
// of piecewise values: 4M 522 / 704 us, 8M 694 / 741, 12M 921 / 860, 32M 1744 / 1082; of lines of about
// 600 values: 8M 667 / 979, 16M 1091 / 1125, 32M 1895 / 1261; of timestamps: 8M 658 / 1075, 16M 1059 / 1270,
// 24M 1434 / 1341; of one line: 8M 669 / 1011, 64M 3152 / 3510.  The line lies where no kind loses yet.
constexpr int64_t kAllStartsBlocks = 65536;
constexpr int32_t kUnknown = -1;  // best end of a start not evaluated

struct SumPair {  // trivially constructible: SumPair() value-initialises to zero
  i128 y;
  i128 iy;
  __device__ __forceinline__ SumPair operator+(const SumPair& o) const {
    SumPair r;
    r.y = y + o.y;
    r.iy = iy + o.iy;
    return r;
  }
};

// ---- block sums -----------------------------------------------------------------------
// Eight lanes per block, 16 values each (all loads in flight before the sums), from 64-bit partials of
// the values' halves with the index inside the block.  ovf (uint64 only): the block holds a value
// above 2^53, so its partition is copied.
template <typename T> __global__ void __launch_bounds__(256)
block_sums_kernel(const T* __restrict__ v, int64_t n, int64_t nb, SumPair* __restrict__ out, uint8_t* __restrict__ ovf) {
  const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int l = threadIdx.x & 7;
  const int64_t i0 = j * kMinPart;
  T y[16];
#pragma unroll
  for (int k = 0; k < 16; k++) y[k] = i0 + 8 * k + l < n ? __ldg(v + i0 + 8 * k + l) : (T)0;
  HalfSums<T> h;
  bool over = false;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    h.add(y[k], 8 * k + l);
    over |= overflows_double<T>(y[k]);
  }
#pragma unroll
  for (int m = 4; m > 0; m >>= 1) {  // (a block's sums of halves and of index * half stay inside 64 bits)
    h.s_lo += __shfl_xor_sync(FULL_MASK, h.s_lo, m);
    h.x_lo += __shfl_xor_sync(FULL_MASK, h.x_lo, m);
    if (sizeof(T) == 8) {
      h.s_hi += __shfl_xor_sync(FULL_MASK, h.s_hi, m);
      h.x_hi += __shfl_xor_sync(FULL_MASK, h.x_hi, m);
    }
  }
  const unsigned any = __ballot_sync(FULL_MASK, over);
  if (l == 0 && j < nb) {
    SumPair s;
    s.y = h.sy();
    s.iy = h.sxy() + (i128)i0 * s.y;
    out[j] = s;
    if (!TypeTraits<T>::is_signed && sizeof(T) == 8) ovf[j] = ((any >> (threadIdx.x & 24)) & 0xffu) != 0;
  }
}

struct RangeSums {
  const SumPair* pre;  // nb + 1 entries
  int64_t n, nb;
  __device__ __forceinline__ int64_t blk(int64_t pos) const { return pos >= n ? nb : pos / kMinPart; }
  // exact sums of [a, b): sum y and sum (i - a) * y
  __device__ __forceinline__ void get(int64_t a, int64_t b, i128& sy, i128& sxy) const {
    const SumPair pb = pre[blk(b)], pa = pre[blk(a)];
    sy = pb.y - pa.y;
    sxy = (pb.iy - pa.iy) - (i128)a * sy;
  }
  __device__ __forceinline__ void line(int64_t a, int64_t b, double& t0, double& t1) const {
    i128 sy, sxy;
    get(a, b, sy, sxy);
    solve_line(b - a, sy, sxy, t0, t1);
  }
};

__device__ __forceinline__ double part_cost(int64_t len, int bits) {
  return __dadd_rn(kModelBytes, __ddiv_rn(__dmul_rn(__ll2double_rn(len), (double)bits), 8.0));
}

// ---- split: the best end of a start -----------------------------------------------------------
// Copies vals[0, count) to win[0, count) (16-byte aligned) with asynchronous copies (16 bytes each, or
// an element each where the values' address does not allow it); the caller waits with cp_async_wait_all + __syncwarp.
template <typename T>
__device__ __forceinline__ void stage_reach(const T* __restrict__ vals, T* win, int count, int lane) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(win);
  if ((reinterpret_cast<uintptr_t>(vals) & 15) == 0) {  // (counts are multiples of 128)
    constexpr int kPer = 16 / (int)sizeof(T);
    for (int o = lane * kPer; o < count; o += 32 * kPer)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + o * (int)sizeof(T)), "l"(vals + o) : "memory");
  } else {
    for (int o = lane; o < count; o += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst + o * (int)sizeof(T)), "l"(vals + o),
                   "n"((int)sizeof(T))
                   : "memory");
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A value of the start's reach: from global memory (read-only path) or from the warp's staged copy.
template <bool SMEM, typename T> __device__ __forceinline__ T ld_val(const T* p) {
  if constexpr (SMEM) return *p;
  else return __ldg(p);
}

// The doubles of [2^52, 2^53) are the integers, one per bit pattern: 1.5 * 2^52 + y for |y| < 2^51 is a
// 64-bit addition to the constant's pattern, and back, with no conversion instruction.
constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52
constexpr long long kMagicBits = 0x4338000000000000ll;
__device__ __forceinline__ double magic_plus(long long y) { return __longlong_as_double(kMagicBits + y); }
// The bits in which a value's high word differs from its sign: below 2^k when -2^(32 + k) <= value < 2^(32 + k).
__device__ __forceinline__ uint32_t high_bits(long long y) {
  const int32_t h = (int32_t)(y >> 32);
  return (uint32_t)(h ^ (h >> 31));
}

// How a line's residuals over offsets [0, len) are taken; the forms give the same integers.
//   kNonNeg  predictions in [-0.25, 2^51] and inside T: round half away is trunc(x + 0.5 - 2^-54),
//            the truncation the sum with 1.5 * 2^52 rounded toward zero, and the prediction the
//            integer of that sum's bit pattern.
//   kOffset  8-byte predictions beyond 2^51: every argument x in [2^51, 2^62] (a multiple of 0.5
//            there, and no saturation) and within 2^50 of the integer d.  Round half away is
//            floor(x + 0.5), so pred - d = floor((x - d) + 0.5), where x - d and the + 0.5 are exact
//            and the floor is the sum with 1.5 * 2^52 rounded down.
//   kSigned  predictions and values inside +-2^51 (abs_resid_fp64).
//   kExact   the format's saturating integer arithmetic.
enum : int { kNonNeg = 0, kOffset = 1, kSigned = 2, kExact = 3 };

// (over offsets [o0, o1]: the prediction argument is monotone between them)
template <typename T> __device__ __forceinline__ int line_form(double t0, double t1, int64_t o0, int64_t o1, double& d) {
  const double xa = __fma_rn(t1, (double)o0, t0), xb = __fma_rn(t1, (double)o1, t0);
  d = 0.0;
  if (pred_fp64_safe<T>(xa) && pred_fp64_safe<T>(xb)) return xa >= -0.25 && xb >= -0.25 ? kNonNeg : kSigned;
  if constexpr (sizeof(T) == 8) {
    constexpr double kLo = 2251799813685248.0, kHi = 4611686018427387904.0, kNear = 1125899906842624.0;
    if (xa >= kLo && xa <= kHi && xb >= kLo && xb <= kHi) {
      d = trunc(xa);
      if (fabs(xa - d) <= kNear && fabs(xb - d) <= kNear) return kOffset;
    }
  }
  return kExact;
}

// Max |residual| of the line over values vs[0, len) (len a multiple of 128), by one warp: every lane
// returns it.  LIMITED: any result above lim only says that a residual is above lim (the scan stops
// there).  Residuals are tracked as 32-bit integers (no 64-bit compare or FP64 maximum per value),
// each the exact difference to the prediction, an integer of the form's bit patterns, modulo 2^64;
// fits = false when one does not fit 32 bits (so does every difference that saturates or wraps: the
// prediction is below 2^63).
template <typename T, bool SMEM, bool LIMITED, int FORM>
__device__ __forceinline__ uint32_t scan_narrow(const T* __restrict__ vs, int len, double t0, double t1, double d,
                                                uint32_t lim, int lane, bool& fits) {
  constexpr long long kHalf = 1ll << 31;
  // residual + 2^31 = y - (pattern of 1.5 * 2^52 + prediction [- d]) + add
  const long long add = kMagicBits + kHalf - (FORM == kOffset ? (long long)d : 0);
  double od[4];
#pragma unroll
  for (int u = 0; u < 4; u++) od[u] = (double)(lane + 32 * u);
  uint32_t mx = (uint32_t)kHalf, mn = (uint32_t)kHalf, wide = 0;
#pragma unroll 2
  for (int o0 = 0; o0 < len; o0 += 128) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const T y = ld_val<SMEM>(vs + o0 + 32 * u + lane);
      const double x = __fma_rn(t1, od[u], t0);
      od[u] = __dadd_rn(od[u], 128.0);
      const double m = FORM == kNonNeg ? __dadd_rz(__dadd_rn(x, 0x1.fffffffffffffp-2), kMagic)  // + 0.5 - 2^-54
                                       : __dadd_rd(__dadd_rn(__dsub_rn(x, d), 0.5), kMagic);
      const unsigned long long r = (unsigned long long)(long long)y - (unsigned long long)__double_as_longlong(m) +
                                   (unsigned long long)add;
      wide |= (uint32_t)(r >> 32);
      mx = max(mx, (uint32_t)r);
      mn = min(mn, (uint32_t)r);
    }
    if (LIMITED && __any_sync(FULL_MASK, max(mx - (uint32_t)kHalf, (uint32_t)kHalf - mn) > lim || wide != 0)) break;
  }
  fits = !__any_sync(FULL_MASK, wide != 0);
  return __reduce_max_sync(FULL_MASK, max(mx - (uint32_t)kHalf, (uint32_t)kHalf - mn));
}

// The same with residuals of any size (FP64 forms, or the format's own arithmetic).
template <typename T, bool SMEM, bool LIMITED, int FORM>
__device__ __noinline__ long long scan_wide(const T* __restrict__ vs, int len, double t0, double t1, double d,
                                            long long lim, int lane, bool& ok) {
  if constexpr (FORM == kExact) {
    long long m = 0;
    for (int o0 = 0; o0 < len; o0 += 128) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int o = o0 + 32 * u + lane;
        const long long r = abs_ref(calc_delta<T>(ld_val<SMEM>(vs + o), predict<T>(t0, t1, o)));
        m = r > m ? r : m;
      }
      if (LIMITED && __any_sync(FULL_MASK, m > lim)) break;
    }
    ok = true;
    return warp_max_ll(m);
  } else {
    const long long c = FORM == kOffset ? (long long)d : 0;
    const double limd = __ll2double_rn(lim);  // only a limit below 2^53 can be exceeded here
    double md = 0.0, od = (double)lane;
    uint32_t high = 0;
    for (int o0 = 0; o0 < len; o0 += 128) {
#pragma unroll
      for (int u = 0; u < 4; u++, od += 32.0) {
        const T y = ld_val<SMEM>(vs + o0 + 32 * u + lane);
        const double x = __fma_rn(t1, od, t0);
        if constexpr (FORM == kOffset) {
          const long long dy = (long long)((uint64_t)y - (uint64_t)c);
          high |= high_bits(dy);
          md = fmax(md, fabs(__dsub_rn(magic_plus(dy), __dadd_rd(__dadd_rn(__dsub_rn(x, d), 0.5), kMagic))));
        } else {
          if (sizeof(T) == 8) high |= TypeTraits<T>::is_signed ? high_bits((long long)y) : (uint32_t)((uint64_t)y >> 32);
          md = fmax(md, abs_resid_fp64(__dsub_rn(magic_plus((long long)y), kMagic), x));
        }
      }
      if (LIMITED && __any_sync(FULL_MASK, md > limd)) break;  // (also when ok fails: measured again then)
    }
    ok = !__any_sync(FULL_MASK, high >= (FORM == kOffset ? 1u << 18 : 1u << 19));
    return warp_max_ll((long long)md);
  }
}

template <typename T, bool SMEM, bool LIMITED>
__device__ __forceinline__ long long scan_line(const T* __restrict__ vs, int len, double t0, double t1, long long lim,
                                               int lane) {
  double d;
  const int form = line_form<T>(t0, t1, 0, len - 1, d);
  if ((form == kNonNeg || (sizeof(T) == 8 && form == kOffset)) && (!LIMITED || lim < 0x7fffffffll)) {
    bool fits;
    const uint32_t m = form == kNonNeg
                           ? scan_narrow<T, SMEM, LIMITED, kNonNeg>(vs, len, t0, t1, d, (uint32_t)lim, lane, fits)
                           : scan_narrow<T, SMEM, LIMITED, kOffset>(vs, len, t0, t1, d, (uint32_t)lim, lane, fits);
    if (fits) return (long long)m;
    if (LIMITED) return lim + 1;  // a residual of 2^31 or more
  }
  bool ok = false;
  long long m = 0;
  if (form == kNonNeg || form == kSigned) m = scan_wide<T, SMEM, LIMITED, kSigned>(vs, len, t0, t1, d, lim, lane, ok);
  else if (sizeof(T) == 8 && form == kOffset) m = scan_wide<T, SMEM, LIMITED, kOffset>(vs, len, t0, t1, d, lim, lane, ok);
  if (!ok) m = scan_wide<T, SMEM, LIMITED, kExact>(vs, len, t0, t1, d, lim, lane, ok);
  return m;
}

// Field bits by which a smaller candidate of `small` values must undercut one of `big` values to
// cost no more per value: 80 / small + b / 8 <= 80 / big + b' / 8, that is b <= b' - 640 (1 / small -
// 1 / big), rounded up.  The computed costs compare as these numbers do: away from equality the two
// sides differ by more than 1 / (8 small big), far above the costs' rounding, and the only equality
// among these sizes, 128 values against 640, is between costs that are exact in FP64.
constexpr int undercut_bits(int small, int big) {
  return (int)((640ll * (big - small) + (long long)small * big - 1) / ((long long)small * big));
}
struct UndercutTable {
  uint8_t q[kNumSizes][kNumSizes];
};
constexpr UndercutTable make_undercut() {
  UndercutTable t{};
  for (int b = 0; b < kNumSizes; b++)
    for (int s = 0; s < kNumSizes; s++) t.q[b][s] = s < b ? (uint8_t)undercut_bits(split_size(s), split_size(b)) : 0;
  return t;
}
__constant__ UndercutTable c_undercut = make_undercut();

// Best end (as a block index; nb for the end of the column) of the start at block j: the candidate
// size with the lowest cost per value, the first of equals.  One warp: every lane takes part and
// returns the same result; th is the warp's own table of lines.  SMEM: the start's reach (up to
// 3712 values) is first copied to win (the warp's own buffer) with all copies in flight at once.
//
// Only the largest candidate's residuals are always taken in full (one pass over the reach instead
// of 14 lines per value: 20.7 K -> 3.7 K value-line evaluations).  A smaller one wins only with
// narrower fields (undercut_bits), so one residual above that limit rules it out: 32 spread samples
// do for most, and a scan that stops at the first such residual for the rest.  200M piecewise uint64
// values: the walks take 645 + 168 us (2017 + 332 with 14 lines measured per value, 763 ranges).
// What is left is instruction latency: seven warps per SM (their reaches fill shared memory), about
// 3.5 K warp instructions per start.  Reading the reach from L1 instead (16 or 32 warps per SM, as
// many shorter ranges) measured 627 + 289 and 629 + 350 us: the second walks of more ranges take
// what the first ones save.
template <typename T, bool SMEM>
__device__ __forceinline__ int32_t split_best_block(const T* __restrict__ v, const RangeSums& rs, int64_t j, int lane,
                                                    double (*th)[2], T* win, long long& best_err) {
  const int64_t s = j * kMinPart;
  const int64_t max_size = (rs.n - s < kMinPart * 32) ? rs.n - s : kMinPart * 32;
  int ncand = 0;
#pragma unroll
  for (int k = 0; k < kNumSizes; k++) ncand += (c_sizes[k] <= max_size) ? 1 : 0;
  best_err = -1;  // not measured
  if (ncand == 0) return (int32_t)rs.nb;  // fewer than 128 values left: the rest is one partition
  __syncwarp();  // the previous start's lines and values are no longer read
  const T* vs = v + s;
  if constexpr (SMEM) {
    stage_reach<T>(v + s, win, c_sizes[ncand - 1], lane);
    vs = win;
  }
  if (lane < ncand) {  // solve_line for lengths whose denominators are exact in FP64
    const int len = c_sizes[lane];
    i128 sy, sxy;
    rs.get(s, s + len, sy, sxy);
    const i128 num = (i128)2 * sxy - (i128)(len - 1) * sy;
    const double t1 = __ddiv_rn(i128_to_double(num), (double)((int64_t)len * ((int64_t)len * len - 1) / 6));
    const double diff = __dsub_rn(i128_to_double(sy), __dmul_rn(t1, (double)(len * (len - 1) / 2)));
    th[lane][0] = __ddiv_rn(diff, (double)len);
    th[lane][1] = t1;
  }
  if constexpr (SMEM) cp_async_wait_all();
  __syncwarp();
  int best = ncand - 1;
  best_err = scan_line<T, SMEM, false>(vs, c_sizes[best], th[best][0], th[best][1], 0, lane);
  unsigned alive = (1u << best) - 1u;  // smaller candidates not ruled out
  while (alive) {
    // the largest residual with which candidate `lane` costs no more than the best one (-1: none)
    const int b = lane < best ? bits_for(best_err) - (int)c_undercut.q[best][lane] : -1;
    const long long lim = b < 0 ? -1 : b < 2 ? 0 : (1ll << (b - 1)) - 1;
    alive &= __ballot_sync(FULL_MASK, lim >= 0);
    if (!alive) break;
    unsigned over = 0;  // (no branch per candidate: the samples' chains overlap)
#pragma unroll
    for (int k = 0; k < kNumSizes - 1; k++) {
      const int o = lane * (split_size(k) / 32) + split_size(k) / 64;
      const double2 t = *reinterpret_cast<const double2*>(th[k]);
      if (k < best) {
        const long long r = abs_ref(calc_delta<T>(ld_val<SMEM>(vs + o), predict<T>(t.x, t.y, o)));
        over |= __any_sync(FULL_MASK, r > __shfl_sync(FULL_MASK, lim, k)) ? 1u << k : 0u;
      }
    }
    alive &= ~over;
    while (alive) {
      const int k = 31 - __clz((int)alive);
      alive &= ~(1u << k);
      const long long limk = __shfl_sync(FULL_MASK, lim, k);
      const long long m = scan_line<T, SMEM, true>(vs, c_sizes[k], th[k][0], th[k][1], limk, lane);
      if (m <= limk) {  // scanned to its end: the best so far, and tighter limits for the rest
        best = k;
        best_err = m;
        break;
      }
    }
  }
  const int64_t e = s + c_sizes[best];
  return (int32_t)(e >= rs.n ? rs.nb : e / kMinPart);
}

// Best end of every 128-aligned start not evaluated yet (one warp per start, the values from L1: the
// reaches of a CTA's eight starts overlap), and the max |delta| of the partition it makes (nb_err:
// -1 where not measured).
template <typename T> __global__ void __launch_bounds__(256)
split_kernel(const T* __restrict__ v, RangeSums rs, int32_t* __restrict__ nb_next, long long* __restrict__ nb_err) {
  __shared__ __align__(16) double s_th[8][kNumSizes][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * 8 + warp;
  if (j >= rs.nb || nb_next[j] != kUnknown) return;
  long long err;
  const int32_t e = split_best_block<T, false>(v, rs, j, lane, s_th[warp], nullptr, err);
  if (lane == 0) {
    nb_next[j] = e;
    nb_err[j] = err;
  }
}

// ---- walk from 0 ---------------------------------------------------------------------------
constexpr int32_t kEnd = -1;

// Ranges of the walk: rb blocks each, a multiple of 29, so that a walk that always takes the
// largest size (data with one slope) leaves a range at the first block of the next.
struct Ranges {
  int64_t nb, nr;
  int rb;
};

// ---- lazy walk: evaluate only the starts a walk can reach --------------------------------------
// The walk from 0 visits one start in ~25 on piecewise-linear data.  Each range is walked from its
// first block, and again from the block where the previous range's first walk leaves it (the
// walk from 0 usually enters there: walks from nearby starts meet where the data changes
// slope).  The ranges are then chained through the exits of the starts these walks visited; if
// the walk from 0 enters a range at a start no walk visited, every start is evaluated instead.
//
// One warp (one CTA) per range.  Of each start a walk visited it keeps where the walk leaves the
// range (cexit, an absolute block) and how many partitions it makes on the way (ccnt); visit: the
// range's own stretch of scratch, the starts in order.
struct WalkOut {
  int32_t* nb_next;
  long long* nb_err;
  int32_t* cexit;
  int32_t* ccnt;
  int32_t* visit;
  int32_t* exit_first;
};

// Walks from `node` to the end of the range, or (MEET) to a start evaluated before.
template <typename T, bool MEET>
__device__ __forceinline__ void walk_range(const T* __restrict__ v, const RangeSums& rs, const Ranges& rg,
                                           const WalkOut& w, int64_t r, int64_t node, int lane, double (*th)[2], T* win) {
  const int64_t lim = (r + 1) * rg.rb < rg.nb ? (r + 1) * rg.rb : rg.nb;
  int32_t* visit = w.visit + r * rg.rb;
  int hops = 0;
  while (node < lim) {
    if (MEET) {
      const int32_t nx = lane == 0 ? w.nb_next[node] : 0;
      if (__shfl_sync(FULL_MASK, nx, 0) != kUnknown) break;
    }
    long long err;
    const int32_t nx = split_best_block<T, true>(v, rs, node, lane, th, win, err);
    if (lane == 0) {
      w.nb_next[node] = nx;
      w.nb_err[node] = err;
      visit[hops] = (int32_t)node;
    }
    hops++;
    node = nx;
  }
  // where the walk ends: the range's exit, or the rest of the walk it met
  int32_t out = (int32_t)node, more = 0;
  if (MEET && node < lim) {
    out = w.cexit[node];
    more = w.ccnt[node];
  }
  __threadfence_block();
  __syncwarp();
  for (int h = lane; h < hops; h += 32) {
    const int32_t p = *(const volatile int32_t*)(visit + h);
    w.cexit[p] = out;
    w.ccnt[p] = hops - h + more;
  }
  if (!MEET && lane == 0) w.exit_first[r] = (int32_t)node;
}

template <typename T, bool FIRST> __global__ void __launch_bounds__(32, kWalksPerSM)
walk_kernel(const T* __restrict__ v, RangeSums rs, Ranges rg, WalkOut w) {
  __shared__ __align__(16) double s_th[kNumSizes][2];
  __shared__ __align__(16) T s_win[kMinPart * kMaxJumpBlocks];
  const int64_t r = blockIdx.x;
  if (FIRST) {
    walk_range<T, false>(v, rs, rg, w, r, r * rg.rb, threadIdx.x, s_th, s_win);
  } else if (r > 0) {
    walk_range<T, true>(v, rs, rg, w, r, w.exit_first[r - 1], threadIdx.x, s_th, s_win);
  }
}

// All starts evaluated: the exit (relative to the next range) and the number of partitions from
// every one of a range's 29 possible entry blocks.  One warp per range, its nexts in shared memory.
__global__ void __launch_bounds__(32)
chain_exit_kernel(const int32_t* __restrict__ nb_next, Ranges rg, int32_t* __restrict__ exits, int32_t* __restrict__ cnts) {
  extern __shared__ int32_t s_next[];
  const int64_t r = blockIdx.x, lo = r * rg.rb;
  const int count = (int)(rg.nb - lo < rg.rb ? rg.nb - lo : rg.rb);
  for (int i = threadIdx.x; i < count; i += 32) s_next[i] = nb_next[lo + i];
  __syncwarp();
  if (threadIdx.x >= kMaxJumpBlocks) return;
  int64_t node = lo + threadIdx.x;
  int c = 0;
  while (node < lo + count) {
    const int64_t next = s_next[node - lo];
    node = next > node ? next : rg.nb;
    c++;
  }
  exits[r * kMaxJumpBlocks + threadIdx.x] = node >= rg.nb ? kEnd : (int32_t)(node - lo - rg.rb);
  cnts[r * kMaxJumpBlocks + threadIdx.x] = c;
}

// Chains the ranges: entries[r] = the block offset at which the walk from 0 enters range r (kEnd past
// the end of the column) and base[r] = the partitions before it; out[0] = all partitions.  LAZY: exits
// from cexit (absolute blocks, kUnknown where no walk passed; out[2] = the first range entered at
// such a start, or -1); otherwise from the table of every entry offset.
//
// One CTA, 1024 ranges at a time: their maps (entry offset -> exit offset, partitions) in shared
// memory; each warp composes the maps of 32 ranges for all 29 entry offsets at once (a lane each), one
// thread chains the 32 composed maps, and each warp walks its ranges again from the entry found (two
// times 32 dependent shared-memory steps instead of 1024).
constexpr int kLinkRanges = 1024;
constexpr uint32_t kLinkEnd = 30, kLinkUnknown = 31;  // exit codes beside the offsets 0..28
constexpr size_t kLinkSmem = sizeof(uint32_t) * kLinkRanges * 32;

template <bool LAZY> __global__ void __launch_bounds__(1024)
chain_link_kernel(const int32_t* __restrict__ exits, const int32_t* __restrict__ cnts, Ranges rg,
                  int32_t* __restrict__ entries, int32_t* __restrict__ base, int64_t* __restrict__ out) {
  extern __shared__ uint32_t s_map[];      // [range][32]: exit code | partitions << 5
  __shared__ uint32_t s_group[32][32];     // composed: exit code of 32 ranges
  __shared__ int32_t s_gcnt[32][32];
  __shared__ int32_t s_gentry[32], s_gbase[32];
  __shared__ long long s_fail;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_fail = -1;
  int32_t carry_e = 0, carry_base = 0;
  for (int64_t r0 = 0; r0 < rg.nr; r0 += kLinkRanges) {
    for (int q = 0; q < 32; q++) {
      const int64_t r = r0 + warp * 32 + q;
      uint32_t code = kLinkUnknown, cnt = 0;
      if (r < rg.nr) {
        if (lane == (int)kLinkEnd) code = kLinkEnd;  // past the end it stays there
        const int64_t b = LAZY ? r * rg.rb + lane : r * kMaxJumpBlocks + lane;
        if (lane < kMaxJumpBlocks && (!LAZY || b < rg.nb)) {
          const int32_t ex = exits[b];
          if (LAZY) {
            code = ex == kUnknown ? kLinkUnknown : (int64_t)ex >= rg.nb ? kLinkEnd : (uint32_t)(ex - (r + 1) * rg.rb);
            cnt = ex == kUnknown ? 0u : (uint32_t)cnts[b];
          } else {
            code = ex == kEnd ? kLinkEnd : (uint32_t)ex;
            cnt = (uint32_t)cnts[b];
          }
        }
      } else {
        code = (uint32_t)lane;  // no such range: the identity
      }
      s_map[(warp * 32 + q) * 32 + lane] = code | cnt << 5;
    }
    __syncwarp();
    uint32_t e = lane;
    int32_t total = 0;
    for (int q = 0; q < 32; q++) {
      const uint32_t w = s_map[(warp * 32 + q) * 32 + e];
      e = w & 31u;
      total += (int32_t)(w >> 5);
    }
    s_group[warp][lane] = e;
    s_gcnt[warp][lane] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t ge = carry_e == kEnd ? kLinkEnd : (uint32_t)carry_e;
      int32_t gb = carry_base;
      for (int g = 0; g < 32; g++) {
        s_gentry[g] = (int32_t)ge;
        s_gbase[g] = gb;
        gb += s_gcnt[g][ge];
        ge = s_group[g][ge];
      }
      carry_e = ge == kLinkEnd ? kEnd : (int32_t)ge;
      carry_base = gb;
    }
    __syncthreads();
    if (lane == 0) {
      uint32_t ge = (uint32_t)s_gentry[warp];
      int32_t gb = s_gbase[warp];
      for (int q = 0; q < 32; q++) {
        const int64_t r = r0 + warp * 32 + q;
        if (r >= rg.nr) break;
        const uint32_t w = s_map[(warp * 32 + q) * 32 + ge];
        const bool unknown = (w & 31u) == kLinkUnknown;  // no walk passed this entry (or an earlier range's)
        entries[r] = ge >= kLinkEnd || unknown ? kEnd : (int32_t)ge;
        base[r] = gb;
        if (LAZY && unknown && ge != kLinkUnknown) s_fail = r;  // the first such range
        ge = w & 31u;
        gb += (int32_t)(w >> 5);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = carry_base;
    out[2] = s_fail;
  }
}

// The walk's partitions in order, with the max |delta| their start's evaluation measured for them
// (-1 for a last partition of fewer than 128 values, which no evaluation measured).  One warp per
// range: lane 0 follows the walk through the range's nexts in shared memory.
__global__ void __launch_bounds__(32)
chain_emit_kernel(const int32_t* __restrict__ nb_next, const long long* __restrict__ nb_err,
                  const int32_t* __restrict__ entries, const int32_t* __restrict__ base, Ranges rg, int64_t n,
                  int32_t* __restrict__ ps, int32_t* __restrict__ pe, long long* __restrict__ kerr) {
  extern __shared__ int32_t s_next[];
  __shared__ int s_hops;
  const int64_t r = blockIdx.x, lo = r * rg.rb;
  const int32_t e = entries[r];
  if (e == kEnd) return;
  const int count = (int)(rg.nb - lo < rg.rb ? rg.nb - lo : rg.rb);
  uint16_t* s_path = reinterpret_cast<uint16_t*>(s_next + rg.rb);
  for (int i = threadIdx.x; i < count; i += 32) s_next[i] = nb_next[lo + i];
  __syncwarp();
  if (threadIdx.x == 0) {
    int node = e, h = 0;
    while (node >= 0 && node < count) {  // (every start on the walk was evaluated: its next lies ahead)
      s_path[h++] = (uint16_t)node;
      const int next = (int)(s_next[node] - lo);
      node = next > node ? next : count;
    }
    s_hops = h;
  }
  __syncwarp();
  for (int h = threadIdx.x; h < s_hops; h += 32) {
    const int node = s_path[h];
    const int64_t k = base[r] + h, end = (int64_t)s_next[node] * kMinPart;
    ps[k] = (int32_t)((lo + node) * kMinPart);
    pe[k] = (int32_t)(end > n ? n : end);
    kerr[k] = nb_err[lo + node];
  }
}

// ---- merge rounds ------------------------------------------------------------------------
// Max |residual| of the line over offsets [o0, o1) of the values at vs, by one warp (every lane returns
// it); above lim it only says so.  Any length; kDeep loads per lane in flight.
template <typename T, int FORM>
__device__ __forceinline__ uint32_t range_narrow(const T* __restrict__ vs, int64_t o0, int64_t o1, double t0, double t1,
                                                 double d, uint32_t lim, int lane, bool& fits) {
  constexpr long long kHalf = 1ll << 31;
  constexpr int kDeep = 16;
  const long long add = kMagicBits + kHalf - (FORM == kOffset ? (long long)d : 0);
  uint32_t mx = (uint32_t)kHalf, mn = (uint32_t)kHalf, wide = 0;
  double od = (double)(o0 + lane);
  auto take = [&](T y, double o) {  // as in scan_narrow
    const double x = __fma_rn(t1, o, t0);
    const double m = FORM == kNonNeg ? __dadd_rz(__dadd_rn(x, 0x1.fffffffffffffp-2), kMagic)
                                     : __dadd_rd(__dadd_rn(__dsub_rn(x, d), 0.5), kMagic);
    const unsigned long long r = (unsigned long long)(long long)y - (unsigned long long)__double_as_longlong(m) +
                                 (unsigned long long)add;
    wide |= (uint32_t)(r >> 32);
    mx = max(mx, (uint32_t)r);
    mn = min(mn, (uint32_t)r);
  };
  const T* p = vs + o0 + lane;
  int64_t left = o1 - o0;
  for (; left >= 32 * kDeep; left -= 32 * kDeep, p += 32 * kDeep) {
    T y[kDeep];
#pragma unroll
    for (int u = 0; u < kDeep; u++) y[u] = __ldg(p + 32 * u);
#pragma unroll
    for (int u = 0; u < kDeep; u++, od = __dadd_rn(od, 32.0)) take(y[u], od);
    if (__any_sync(FULL_MASK, max(mx - (uint32_t)kHalf, (uint32_t)kHalf - mn) > lim || wide != 0)) {
      left = 0;
      break;
    }
  }
  for (int64_t o = lane; o < left; o += 32, p += 32, od = __dadd_rn(od, 32.0)) take(__ldg(p), od);
  fits = !__any_sync(FULL_MASK, wide != 0);
  return __reduce_max_sync(FULL_MASK, max(mx - (uint32_t)kHalf, (uint32_t)kHalf - mn));
}

// The same in the format's own arithmetic, or in FP64 where every quantity is an exact integer.
template <typename T>
__device__ __noinline__ long long range_exact(const T* __restrict__ vs, int64_t o0, int64_t o1, double t0, double t1,
                                              long long lim, int lane) {
  long long m = 0;
  for (int64_t b = o0; b < o1; b += 256) {
    const int64_t e = b + 256 < o1 ? b + 256 : o1;
    if (line_fp64_safe<T>(t0, t1, b, e - 1)) {
      double md = 0.0;
      bool ok = true;
      for (int64_t o = b + lane; o < e; o += 32) {
        const T y = __ldg(vs + o);
        ok &= value_fp64_safe<T>(y);
        md = fmax(md, abs_resid_fp64((double)(long long)y, __fma_rn(t1, (double)o, t0)));
      }
      if (__all_sync(FULL_MASK, ok)) {
        m = max(m, (long long)md);
        if (__any_sync(FULL_MASK, m > lim)) break;
        continue;
      }
    }
    for (int64_t o = b + lane; o < e; o += 32)
      m = max(m, abs_ref(calc_delta<T>(__ldg(vs + o), predict<T>(t0, t1, o))));
    if (__any_sync(FULL_MASK, m > lim)) break;
  }
  return warp_max_ll(m);
}

template <typename T>
__device__ __forceinline__ long long range_line(const T* __restrict__ vs, int64_t o0, int64_t o1, double t0, double t1,
                                                long long lim, int lane) {
  double d;
  const int form = line_form<T>(t0, t1, o0, o1 - 1, d);
  if (form == kNonNeg || (sizeof(T) == 8 && form == kOffset)) {
    bool fits;
    const uint32_t l32 = lim < 0x7fffffffll ? (uint32_t)lim : 0x7fffffffu;
    const uint32_t m = form == kNonNeg ? range_narrow<T, kNonNeg>(vs, o0, o1, t0, t1, d, l32, lane, fits)
                                       : range_narrow<T, kOffset>(vs, o0, o1, t0, t1, d, l32, lane, fits);
    if (fits && m <= 0x7fffffffu) return (long long)m;
    if (lim < 0x7fffffffll) return lim + 1;
  }
  return range_exact<T>(vs, o0, o1, t0, t1, lim, lane);
}

// The largest max |delta| with which a partition of len values costs less than `sum` (-1: none).
__device__ __forceinline__ long long err_below_cost(int64_t len, double sum) {
  int b = 64;
  const double est = (sum - kModelBytes) * 8.0 / (double)len;  // real number of bits at equality
  if (est < 64.0) b = est < 0.0 ? 0 : (int)est + 1;
  while (b >= 0 && !(part_cost(len, b) < sum)) b--;
  return b < 0 ? -1 : b < 2 ? 0 : b >= 64 ? 0x7fffffffffffffffll : (1ll << (b - 1)) - 1;
}

// One version of the partition list.
struct PartList {
  int32_t* start;
  int32_t* end;
  double* cost;
  long long* err;     // max |delta| of the partition's line, bit 63 set when a value is above 2^53
  uint8_t* rejected;  // the pair (this, next) was scored and is not worth merging
};
constexpr long long kOverflowBit = (long long)0x8000000000000000ull;

struct MergeArgs {
  PartList a, b;         // a holds the split's partitions (cost and rejected not set)
  const uint8_t* ovf;    // per block (uint64)
  int64_t n;
  int32_t m;             // partitions in a
  int32_t unit;          // values of a pair that one warp scans
  uint8_t* selected;     // pair (k, k + 1) merges this round
  long long* pair_err;
  double* pair_t;        // line of a pair in the unit queue
  long long* pair_lim;
  uint2* queue;          // (left part, unit) of pairs longer than one unit
  int32_t* cta_heads;    // per CTA
  unsigned* counters;    // kMergeCounters, zero
  int64_t* out;          // [0] partitions left, [1] 1 when they are in b, [2] DEVERR_*
  unsigned absent;       // arrivals that the barriers wait for in vain (0; 1 lets the first one run out)
  uint64_t wait_ns;      // limit of a barrier's wait
};
constexpr int kMaxMergeRounds = 64;
constexpr int kMergeThreads = 512;
constexpr int kMergeShort = 16384;    // partitions of a list that every CTA counts for itself
constexpr int kMergeUnitMost = 4096;  // values of a pair that one warp scans, at most
// counters: [0] grid barrier, then per round: pairs taken, queue length, pairs rejected
constexpr int kMergeCounters = 4 + 4 * kMaxMergeRounds;

// Barrier of all CTAs of a cooperative launch (a counter that only grows); false when the bounded wait
// gave up.  A CTA that gave up arrives no more: the others' next wait runs out too.  The limit is longer
// than kWaitLimitNs: the last CTAs may first have to wait for a kernel of another stream to leave their SMs.
constexpr uint64_t kGridWaitNs = 20000000000ull;
__device__ __forceinline__ bool grid_barrier(const MergeArgs& a, unsigned& arrived) {
  __shared__ int s_ok;
  __syncthreads();
  arrived += gridDim.x;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.counters, 1u);
    const uint64_t t0 = global_ns();
    bool ok = false;
    for (long long spins = 0; spins < kSpinLimit; spins++) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(a.counters) : "memory");
      ok = (int)(seen - (arrived + a.absent)) >= 0;
      if (ok || ((spins & 255) == 255 && global_ns() - t0 > a.wait_ns)) break;
    }
    s_ok = ok;
    if (!ok) atomicExch((unsigned long long*)(a.out + 2), (unsigned long long)DEVERR_TIMEOUT);
  }
  __syncthreads();
  return s_ok != 0;
}

// All merge rounds in one cooperative launch (one CTA per SM; nine launches and a host round trip per
// round before: 15 rounds on 200M piecewise values).  In round r the pairs (k, k + 1) with k + r even
// can merge, so only those are scored, every value read once per round (scoring all pairs read it
// twice).  A pair that is not worth merging stays so until one of its partitions changes (rejected).
// A warp scores a pair: lines of up to four pairs at once by its lanes, 32 spread residuals, then the
// values in order until one residual is above what the merge allows.  Pairs longer than a unit put
// their further units in a queue that all warps empty together after the others.
//
// 200M piecewise uint64 values: 3343 us of error passes and ~450 us of bookkeeping launches -> 1320 us;
// 3M int64 timestamps: 57 + ~170 -> 86 us (95 with a third barrier per round for the counts of a short
// list).  Bound by the values read (about four passes at 5 TB/s) and,
// on short columns, by the barriers.  Units of 32,768 values measured 1829 us (the last warps of a
// round scan alone), 8192: 1420, 4096: 1346; 1024 threads with eight loads in flight per lane 1925
// (64 registers: spills).
template <typename T> __global__ void __launch_bounds__(kMergeThreads)
merge_kernel(const T* __restrict__ v, RangeSums rs, MergeArgs a) {
  __shared__ int32_t s_scan[kMergeThreads / 32];
  __shared__ int32_t s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tid = (int64_t)blockIdx.x * kMergeThreads + threadIdx.x, nthreads = (int64_t)gridDim.x * kMergeThreads;
  const int nwarps = (int)(nthreads >> 5), gwarp = (int)(tid >> 5);
  unsigned arrived = 0;
  PartList cur = a.a, nxt = a.b;
  int m = a.m;
  // costs of the split's partitions: their max |delta| came with the split (-1: fewer than 128 values)
  for (int64_t k = tid; k < m; k += nthreads) {
    const int64_t s = cur.start[k], e = cur.end[k];
    long long err = cur.err[k];
    if (err < 0) {
      double t0, t1;
      rs.line(s, e, t0, t1);
      err = 0;
      for (int64_t o = 0; o < e - s; o++) err = max(err, abs_ref(calc_delta<T>(v[s + o], predict<T>(t0, t1, o))));
    }
    cur.cost[k] = part_cost(e - s, bits_for(err));
    cur.rejected[k] = 0;
    if (!TypeTraits<T>::is_signed && sizeof(T) == 8) {
      bool over = false;
      for (int64_t b = s / kMinPart; b * kMinPart < e; b++) over |= a.ovf[b] != 0;
      if (over) err |= kOverflowBit;
    }
    cur.err[k] = err;
  }
  if (!grid_barrier(a, arrived)) return;
  bool flipped = false;
  for (int round = 0; round < kMaxMergeRounds && m >= 2; round++) {
    unsigned* taken = a.counters + 4 + 4 * round;
    unsigned* queued = taken + 1;
    unsigned* nrej = taken + 2;
    const int odd = round & 1, pairs = (m - odd) / 2;  // k = 2 q + odd, k + 1 < m
    // ---- score ----
    int per = pairs / (nwarps * 8);
    per = per < 1 ? 1 : per > 4 ? 4 : per;
    for (;;) {
      unsigned q0 = lane == 0 ? atomicAdd(taken, (unsigned)per) : 0u;
      q0 = __shfl_sync(FULL_MASK, q0, 0);
      if (q0 >= (unsigned)pairs) break;
      const int mine = (int)q0 + lane;
      const bool have = lane < per && mine < pairs;
      const int kk = 2 * mine + odd;
      int64_t s = 0, e = 0;
      double t0 = 0.0, t1 = 0.0;
      long long lim = -1;
      bool todo = false;
      if (have) {
        a.selected[kk] = 0;
        todo = cur.rejected[kk] == 0;
        if (todo) {
          s = cur.start[kk];
          e = cur.end[kk + 1];
          rs.line(s, e, t0, t1);
          lim = err_below_cost(e - s, __dadd_rn(cur.cost[kk], cur.cost[kk + 1]));
          if (lim < 0) {
            cur.rejected[kk] = 1;
            todo = false;
          }
        }
      }
      unsigned work = __ballot_sync(FULL_MASK, todo);
      while (work) {
        const int src = __ffs((int)work) - 1;
        work &= work - 1;
        const int k = __shfl_sync(FULL_MASK, kk, src);
        const int64_t ps = __shfl_sync(FULL_MASK, s, src), len = __shfl_sync(FULL_MASK, e, src) - ps;
        const double u0 = __shfl_sync(FULL_MASK, t0, src), u1 = __shfl_sync(FULL_MASK, t1, src);
        const long long lk = __shfl_sync(FULL_MASK, lim, src);
        const T* vs = v + ps;
        const int64_t o = len >= 64 ? lane * (len >> 5) + (len >> 6) : lane < len ? lane : 0;
        long long err = warp_max_ll(abs_ref(calc_delta<T>(__ldg(vs + o), predict<T>(u0, u1, o))));
        const bool longer = len > a.unit;
        if (err <= lk) err = range_line<T>(vs, 0, longer ? a.unit : len, u0, u1, lk, lane);
        if (longer && err <= lk) {  // the rest of it by all warps
          const unsigned units = (unsigned)((len + a.unit - 1) / a.unit) - 1;
          unsigned at = lane == 0 ? atomicAdd(queued, units) : 0u;
          at = __shfl_sync(FULL_MASK, at, 0);
          for (unsigned u = lane; u < units; u += 32) a.queue[at + u] = make_uint2((unsigned)k, u + 1);
          if (lane == 0) {
            a.pair_t[2 * k] = u0;
            a.pair_t[2 * k + 1] = u1;
            a.pair_lim[k] = lk;
          }
        }
        if (lane == 0) {
          a.pair_err[k] = err;
          const bool merge = err <= lk;
          a.selected[k] = merge;
          if (!merge) cur.rejected[k] = 1;
        }
      }
    }
    if (!grid_barrier(a, arrived)) return;
    const unsigned nq = *(volatile unsigned*)queued;
    if (nq) {
      for (unsigned i = gwarp; i < nq; i += nwarps) {
        const uint2 w = a.queue[i];
        const int k = (int)w.x;
        const long long lk = a.pair_lim[k];
        long long seen = lane == 0 ? *(volatile long long*)(a.pair_err + k) : 0;
        if (__shfl_sync(FULL_MASK, seen, 0) > lk) continue;  // settled by another unit
        const int64_t ps = cur.start[k], len = cur.end[k + 1] - ps;
        const int64_t o0 = (int64_t)w.y * a.unit, o1 = o0 + a.unit < len ? o0 + a.unit : len;
        const long long err = range_line<T>(v + ps, o0, o1, a.pair_t[2 * k], a.pair_t[2 * k + 1], lk, lane);
        if (lane == 0) {
          atomicMax(a.pair_err + k, err);
          if (err > lk) {
            a.selected[k] = 0;
            cur.rejected[k] = 1;
          }
        }
      }
      if (!grid_barrier(a, arrived)) return;
    }
    // ---- compact: a CTA takes a stretch of the list ----
    const int seg = (m + gridDim.x - 1) / gridDim.x, k0 = min(m, (int)blockIdx.x * seg), k1 = min(m, k0 + seg);
    auto merges = [&](int k) { return k >= odd && ((k + round) & 1) == 0 && k + 1 < m && a.selected[k]; };
    // heads before this CTA, and all of them: counted by every CTA for itself where the list is short
    // (a barrier costs more than m / 512 loads per thread), else by the CTAs' own counts
    int before = 0, all = 0;
    if (m <= kMergeShort) {
#pragma unroll 4
      for (int k = threadIdx.x; k < m; k += kMergeThreads) {
        const int h = !merges(k - 1);
        all += h;
        before += k < k0 ? h : 0;
      }
    } else {
      int heads = 0;
      for (int k = k0 + threadIdx.x; k < k1; k += kMergeThreads) heads += !merges(k - 1);
      heads = __reduce_add_sync(FULL_MASK, heads);
      if (lane == 0) s_scan[warp] = heads;
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < kMergeThreads / 32; w++) t += s_scan[w];
        a.cta_heads[blockIdx.x] = t;
      }
      if (!grid_barrier(a, arrived)) return;
      for (int c = threadIdx.x; c < (int)gridDim.x; c += kMergeThreads) {
        const int h = *(volatile int32_t*)(a.cta_heads + c);
        all += h;
        if (c < (int)blockIdx.x) before += h;
      }
    }
    before = __reduce_add_sync(FULL_MASK, before);
    all = __reduce_add_sync(FULL_MASK, all);
    __shared__ int32_t s_before[kMergeThreads / 32], s_all[kMergeThreads / 32];
    if (lane == 0) {
      s_before[warp] = before;
      s_all[warp] = all;
    }
    __syncthreads();
    before = all = 0;
    for (int w = 0; w < kMergeThreads / 32; w++) {
      before += s_before[w];
      all += s_all[w];
    }
    if (threadIdx.x == 0) s_base = before;
    int rej = 0;
    for (int kb = k0; kb < k1; kb += kMergeThreads) {
      const int k = kb + (int)threadIdx.x;
      const bool head = k < k1 && !merges(k - 1);
      const unsigned bal = __ballot_sync(FULL_MASK, head);
      __syncthreads();  // s_base set; the last step's s_scan read
      if (lane == 0) s_scan[warp] = __popc(bal);
      __syncthreads();
      int d = s_base + __popc(bal & ((1u << lane) - 1u)), total = 0;
      for (int w = 0; w < kMergeThreads / 32; w++) {
        const int c = s_scan[w];
        d += w < warp ? c : 0;
        total += c;
      }
      if (head) {
        const bool sel = merges(k);
        nxt.start[d] = cur.start[k];
        const int32_t end = cur.end[sel ? k + 1 : k];
        nxt.end[d] = end;
        long long err = cur.err[k];
        double cost = cur.cost[k];
        if (sel) {
          const long long pe = a.pair_err[k];
          cost = part_cost((int64_t)end - cur.start[k], bits_for(pe));
          err = pe | ((err | cur.err[k + 1]) & kOverflowBit);
        }
        nxt.err[d] = err;
        nxt.cost[d] = cost;
        const bool r = !sel && k + 1 < m && cur.rejected[k] && !merges(k + 1);
        nxt.rejected[d] = r;
        rej += r;
      }
      __syncthreads();  // everyone has read s_base and s_scan
      if (threadIdx.x == 0) s_base += total;
    }
    rej = __reduce_add_sync(FULL_MASK, rej);
    if (lane == 0 && rej) atomicAdd(nrej, (unsigned)rej);
    if (!grid_barrier(a, arrived)) return;
    const PartList t = cur;
    cur = nxt;
    nxt = t;
    flipped = !flipped;
    m = all;
    if (*(volatile unsigned*)nrej == (unsigned)(m - 1)) break;  // no pair is worth merging
  }
  if (tid == 0) {
    a.out[0] = m;
    a.out[1] = flipped;
  }
}

// ---- the fit of the final partitions ----------------------------------------------------------
// Line, model, max |delta| and width of each partition, all from the partitioner's exact sums and
// errors: no pass over the values (the fit's own pass took 307 us on 200M values).
template <typename T> __global__ void __launch_bounds__(128)
part_fit_kernel(PartList l, RangeSums rs, int32_t P, int32_t* __restrict__ starts, int32_t* __restrict__ ends,
                int32_t* __restrict__ types, double* __restrict__ params, int32_t* __restrict__ bits,
                int64_t* __restrict__ errb, int64_t* __restrict__ widths, unsigned long long* __restrict__ max_bits,
                unsigned long long* __restrict__ per_tile) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int b = 0;
  unsigned k = 0;
  if (p < P) {
    const int64_t s = l.start[p], e = l.end[p];
    const bool copy = l.err[p] < 0;
    double t0 = 0.0, t1 = 0.0;
    if (!copy) rs.line(s, e, t0, t1);
    const long long err = copy ? 0 : l.err[p];
    b = copy ? (int)sizeof(T) * 8 : bits_for(err);
    starts[p] = (int32_t)s;
    ends[p] = (int32_t)e;
    types[p] = copy ? MODEL_DIRECT_COPY : MODEL_LINEAR;
    double2* q = reinterpret_cast<double2*>(params + 4 * (int64_t)p);
    q[0] = make_double2(t0, t1);
    q[1] = make_double2(0.0, 0.0);
    bits[p] = b;
    errb[p] = err;
    widths[p] = (e - s) * b;
    if (p < P - 1) k = (unsigned)((kDecodeTile + e - s - 1) / (e - s));
  }
  b = (int)__reduce_max_sync(FULL_MASK, (unsigned)b);
  k = __reduce_max_sync(FULL_MASK, k);
  if ((threadIdx.x & 31) == 0) {
    if (b > 0) atomicMax(max_bits, (unsigned long long)b);
    if (k > 0) atomicMax(per_tile, (unsigned long long)k);
  }
}

static inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

// Two allocations: the split's arrays by the column's blocks, the lists by the partitions it made.
struct PoolBuf {
  cudaStream_t s;
  char* p = nullptr;
  size_t used = 0;
  explicit PoolBuf(cudaStream_t st) : s(st) {}
  ~PoolBuf() {
    if (p) cudaFreeAsync(p, s);
  }
  template <typename V> void want(V** at, size_t count) { fields.push_back({(void**)at, al(sizeof(V) * count)}); }
  cudaError_t get(glc_ctx* ctx) {
    for (auto& f : fields) used += f.second;
    cudaError_t e = pool_alloc(ctx, &p, used, s);
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    char* q = p;
    for (auto& f : fields) {
      *f.first = q;
      q += f.second;
    }
    return cudaSuccess;
  }
  std::vector<std::pair<void**, size_t>> fields;
};

template <typename T>
static cudaError_t partition_typed(glc_ctx* ctx, const T* v, int64_t n, const PartOut& out, cudaStream_t s, std::string* err) {
  cudaError_t e;
  const int64_t nb = (n + kMinPart - 1) / kMinPart;
  const bool all_starts = nb <= kAllStartsBlocks;
  // all starts: short ranges keep the chains through each short; walks: one wave of ranges (seven
  // reaches fit an SM's shared memory), none shorter than 464 blocks (walks need room to meet)
  int64_t per = 8;
  if (!all_starts) {
    const int64_t wave = (int64_t)kMaxJumpBlocks * kWalksPerSM * ctx->num_sms;
    per = std::min<int64_t>(std::max<int64_t>((nb + wave - 1) / wave, 16), kMaxRangeBlocks / kMaxJumpBlocks);
  }
  const int rb = (int)per * kMaxJumpBlocks;
  const int64_t nr = (nb + rb - 1) / rb;
  const Ranges rg{nb, nr, rb};
  PoolBuf split(s), lists(s);
  SumPair *pre, *ptiles;
  int32_t *nb_next, *exits, *cnts, *entries, *base, *exit_first, *cexit = nullptr, *ccnt = nullptr, *visit = nullptr;
  long long* nb_err;
  uint8_t* ovf;
  int64_t* dsc;        // [1] partitions of the split, [3] first range the walks did not cover (-1: none);
                       // [4] partitions left, [5] list, [6] DEVERR_*
  unsigned* counters;  // right after dsc: cleared together
  split.want(&pre, nb + 1);
  split.want(&ptiles, scan_num_tiles<SumPair>(nb) + 1);
  split.want(&nb_next, nb);
  split.want(&nb_err, nb);
  split.want(&ovf, sizeof(T) == 8 && !TypeTraits<T>::is_signed ? nb : 1);
  split.want(&exits, nr * kMaxJumpBlocks);
  split.want(&cnts, nr * kMaxJumpBlocks);
  split.want(&entries, nr);
  split.want(&base, nr);
  split.want(&exit_first, nr);
  if (!all_starts) {
    split.want(&cexit, nb);
    split.want(&ccnt, nb);
    split.want(&visit, nb);
  }
  split.want(&dsc, 32);
  split.want(&counters, kMergeCounters);
  if ((e = split.get(ctx)) != cudaSuccess) return e;
  RangeSums rs{pre, n, nb};
  static PerDeviceFlag attrs;
  if (const int dev = current_device(); !attrs.test(dev)) {
    if ((e = cudaFuncSetAttribute(chain_link_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLinkSmem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(chain_link_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLinkSmem)) != cudaSuccess)
      return e;
    attrs.set(dev);
  }
  auto grid = [](int64_t x, int b) { return (unsigned)((x + b - 1) / b); };

  if ((e = cudaMemsetAsync(dsc, 0, (size_t)((char*)(counters + kMergeCounters) - (char*)dsc), s)) != cudaSuccess) return e;
  block_sums_kernel<T><<<grid(nb * 8, 256), 256, 0, s>>>(v, n, nb, pre, ovf);
  if ((e = exclusive_scan<SumPair>(pre, pre, nb, pre + nb, ptiles, s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(nb_next, 0xff, sizeof(int32_t) * nb, s)) != cudaSuccess) return e;
  auto linked = [&]() -> cudaError_t {
    cudaError_t ee = cudaGetLastError();
    if (ee == cudaSuccess) ee = cudaMemcpyAsync(ctx->h_stats, dsc + 1, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    return ee == cudaSuccess ? cudaStreamSynchronize(s) : ee;
  };
  auto every_start = [&]() -> cudaError_t {
    split_kernel<T><<<grid(nb, 8), 256, 0, s>>>(v, rs, nb_next, nb_err);
    chain_exit_kernel<<<(unsigned)nr, 32, sizeof(int32_t) * rb, s>>>(nb_next, rg, exits, cnts);
    chain_link_kernel<false><<<1, 1024, kLinkSmem, s>>>(exits, cnts, rg, entries, base, dsc + 1);
    return linked();
  };
  if (all_starts) {
    if ((e = every_start()) != cudaSuccess) return e;
  } else {  // the walk from 0: first only the starts that the walks of the ranges visit
    if ((e = cudaMemsetAsync(cexit, 0xff, sizeof(int32_t) * nb, s)) != cudaSuccess) return e;
    const WalkOut w{nb_next, nb_err, cexit, ccnt, visit, exit_first};
    walk_kernel<T, true><<<(unsigned)nr, 32, 0, s>>>(v, rs, rg, w);
    walk_kernel<T, false><<<(unsigned)nr, 32, 0, s>>>(v, rs, rg, w);
    chain_link_kernel<true><<<1, 1024, kLinkSmem, s>>>(cexit, ccnt, rg, entries, base, dsc + 1);
    if ((e = linked()) != cudaSuccess) return e;
    if (ctx->h_stats[2] >= 0 && (e = every_start()) != cudaSuccess) return e;  // it left the visited starts
  }
  const int64_t m = ctx->h_stats[0];
  if (m <= 0 || m > nb) {
    if (err) *err = "partitioner produced an invalid split";
    return cudaErrorUnknown;
  }

  MergeArgs ma;
  for (PartList* l : {&ma.a, &ma.b}) {
    lists.want(&l->start, m);
    lists.want(&l->end, m);
    lists.want(&l->cost, m);
    lists.want(&l->err, m);
    lists.want(&l->rejected, m);
  }
  lists.want(&ma.selected, m);
  lists.want(&ma.pair_err, m);
  lists.want(&ma.pair_t, 2 * m);
  lists.want(&ma.pair_lim, m);
  // units small enough that a short column's pairs reach every warp
  ma.unit = 512;
  while (ma.unit < kMergeUnitMost && n / ma.unit > 2ll * ctx->num_sms * (kMergeThreads / 32)) ma.unit *= 2;
  lists.want(&ma.queue, n / ma.unit + m + 1);
  lists.want(&ma.cta_heads, ctx->num_sms);
  int64_t *widths, *wtiles;
  lists.want(&widths, m + 1);
  lists.want(&wtiles, scan_num_tiles(m) + 1);
  if ((e = lists.get(ctx)) != cudaSuccess) return e;
  ma.ovf = ovf;
  ma.n = n;
  ma.m = (int32_t)m;
  ma.counters = counters;
  ma.out = dsc + 4;
  ma.absent = 0;
  ma.wait_ns = kGridWaitNs;
  if (ctx->expire_next_merge.load() > 0 && ctx->expire_next_merge.exchange(0) > 0) {
    ma.absent = 1;
    ma.wait_ns = 1000000;
  }
  chain_emit_kernel<<<(unsigned)nr, 32, (sizeof(int32_t) + sizeof(uint16_t)) * rb, s>>>(nb_next, nb_err, entries, base, rg, n,
                                                                                         ma.a.start, ma.a.end, ma.a.err);
  // one CTA per SM, all resident; fewer when the list is short (a cheaper barrier)
  const int64_t ctas = std::min<int64_t>(ctx->num_sms, std::max<int64_t>(1, (m + 15) / 16));
  void* kargs[] = {(void*)&v, (void*)&rs, (void*)&ma};
  if ((e = cudaLaunchCooperativeKernel((const void*)merge_kernel<T>, dim3((unsigned)ctas), dim3(kMergeThreads), kargs, 0, s)) !=
          cudaSuccess ||
      (e = cudaMemcpyAsync(ctx->h_stats, dsc + 4, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return e;
  const int64_t P = ctx->h_stats[0];
  if (ctx->h_stats[2] == DEVERR_TIMEOUT) {
    if (err) *err = "a device-side wait of the partitioner gave up";
    return cudaErrorLaunchTimeout;
  }
  if (ctx->h_stats[2] != DEVERR_NONE || P <= 0 || P > m) {
    if (err) *err = "partitioner produced an invalid merge";
    return cudaErrorUnknown;
  }
  const PartList fin = ctx->h_stats[1] ? ma.b : ma.a;

  if (out.column) {  // the column's arrays, fitted
    glc_column* c = out.column;
    c->P = P;
    if ((e = out.alloc(c, s)) != cudaSuccess || (e = cudaMemsetAsync(out.stats, 0, 4 * sizeof(int64_t), s)) != cudaSuccess) return e;
    part_fit_kernel<T><<<grid(P, 128), 128, 0, s>>>(fin, rs, (int32_t)P, c->d_start, c->d_end, c->d_types, c->d_params,
                                                    c->d_bits, c->d_err, widths, (unsigned long long*)(out.stats + 1),
                                                    (unsigned long long*)(out.stats + 3));
    return exclusive_scan<int64_t>(widths, c->d_offs, P, out.stats, wtiles, s);
  }
  *out.P = P;
  if ((e = pool_alloc(ctx, out.starts, sizeof(int32_t) * P, s)) != cudaSuccess) return e;
  if ((e = pool_alloc(ctx, out.ends, sizeof(int32_t) * P, s)) == cudaSuccess &&
      (e = cudaMemcpyAsync(*out.starts, fin.start, sizeof(int32_t) * P, cudaMemcpyDeviceToDevice, s)) == cudaSuccess)
    e = cudaMemcpyAsync(*out.ends, fin.end, sizeof(int32_t) * P, cudaMemcpyDeviceToDevice, s);
  return e;
}

cudaError_t launch_partition_variable(glc_ctx* ctx, glc_dtype dt, const void* values, int64_t n, const PartOut& out,
                                      cudaStream_t s, std::string* err) {
  switch (dt) {
    case GLC_I32: return partition_typed<int32_t>(ctx, (const int32_t*)values, n, out, s, err);
    case GLC_I64: return partition_typed<int64_t>(ctx, (const int64_t*)values, n, out, s, err);
    case GLC_U64: return partition_typed<uint64_t>(ctx, (const uint64_t*)values, n, out, s, err);
    case GLC_U32: return partition_typed<uint32_t>(ctx, (const uint32_t*)values, n, out, s, err);
  }
  return cudaErrorInvalidValue;
}

}  // namespace glc
