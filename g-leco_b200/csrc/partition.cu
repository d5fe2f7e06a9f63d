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
// (CpuPartitioner.cuh:198-242).  Here merging runs in rounds: every adjacent pair is scored,
// and the profitable pairs with (index + round) even merge, so the chosen pairs never overlap;
// rounds stop when no pair is profitable (at most 64 rounds).  A pair whose two partitions did
// not change keeps its score from the previous round.
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
// 200M values would take 26 times the evaluations of the walks.
constexpr int64_t kAllStartsBlocks = 65536;
constexpr int kMaxMergeRounds = 64;
constexpr int kPairChunk = 4096;
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
template <typename T> __global__ void block_sums_kernel(const T* __restrict__ v, int64_t n, int64_t nb, SumPair* __restrict__ out) {
  const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= nb) return;
  i128 sy = 0, siy = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int64_t i = j * kMinPart + k * 32 + lane;
    if (i < n) {
      const i128 y = (i128)__ldg(v + i);
      sy += y;
      siy += (i128)i * y;
    }
  }
  sy = warp_sum_i128(sy);
  siy = warp_sum_i128(siy);
  if (lane == 0) {
    SumPair s;
    s.y = sy;
    s.iy = siy;
    out[j] = s;
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

template <typename T> __device__ __forceinline__ int line_form(double t0, double t1, int len, double& d) {
  const double xa = __fma_rn(t1, 0.0, t0), xb = __fma_rn(t1, (double)(len - 1), t0);  // monotone between
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
  const int form = line_form<T>(t0, t1, len, d);
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

// ---- costs of partitions ---------------------------------------------------------------
struct LineJob {  // one range whose max |delta| is needed
  int32_t a, b;
  double t0, t1;
  double sum;  // pairs: the two partitions' costs (a merge must cost less); partitions: +inf
};

// chunks of each job (0 for jobs that are cached)
// known (partitions only): a max |delta| already measured (the split evaluation of the
// partition's start, same line and values), or -1.  A pair kept from the previous round (cached)
// keeps its max |delta| too (cached_err).
__global__ void job_setup_kernel(const int32_t* __restrict__ ps, const int32_t* __restrict__ pe, int64_t m, int pairs,
                                 const uint8_t* __restrict__ cached, const long long* __restrict__ cached_err,
                                 const long long* __restrict__ known, const double* __restrict__ pc, RangeSums rs,
                                 LineJob* __restrict__ jobs, int64_t* __restrict__ nch, long long* __restrict__ err) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t njobs = pairs ? m - 1 : m;
  if (k >= njobs) return;
  LineJob jb;
  jb.a = ps[k];
  jb.b = pairs ? pe[k + 1] : pe[k];
  rs.line(jb.a, jb.b, jb.t0, jb.t1);
  jb.sum = pairs ? __dadd_rn(pc[k], pc[k + 1]) : __longlong_as_double(0x7ff0000000000000ll);
  jobs[k] = jb;
  const long long kn = known ? known[k] : -1;
  const bool kept = cached && cached[k];
  err[k] = kn >= 0 ? kn : (kept ? cached_err[k] : 0);
  const bool skip = kept || kn >= 0;
  nch[k] = skip ? 0 : ((int64_t)jb.b - jb.a + kPairChunk - 1) / kPairChunk;
}

// Max |delta| of a job's line over chunk q of the job (256 threads, no CTA barrier: warps may
// skip a chunk independently), folded into *errk by each warp.
template <typename T>
__device__ __forceinline__ void job_chunk(const T* __restrict__ v, const LineJob& jb, int64_t q, long long* errk) {
  const int64_t off0 = q * kPairChunk;
  const int64_t len = (int64_t)jb.b - jb.a;
  const int64_t off1 = off0 + kPairChunk < len ? off0 + kPairChunk : len;
  long long mm = 0;
  bool exact = true;
  if (off1 > off0 && line_fp64_safe<T>(jb.t0, jb.t1, off0, off1 - 1)) {  // exact in FP64 (glc_device.cuh)
    static_assert(kPairChunk == 16 * 256, "16 values per thread");
    T ys[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {  // all loads in flight before the arithmetic
      const int64_t o = off0 + threadIdx.x + u * 256;
      ys[u] = o < off1 ? __ldg(v + jb.a + o) : (T)0;
    }
    double md = 0.0;
    bool ok = true;
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int64_t o = off0 + threadIdx.x + u * 256;
      if (o < off1) {
        ok &= value_fp64_safe<T>(ys[u]);
        md = fmax(md, abs_resid_fp64((double)(long long)ys[u], __fma_rn(jb.t1, (double)o, jb.t0)));
      }
    }
    if (ok) {  // this thread's values were all inside the exact range
      mm = (long long)md;
      exact = false;
    }
  }
  if (exact)
    for (int64_t o = off0 + threadIdx.x; o < off1; o += 256) {
      const long long d = abs_ref(calc_delta<T>(__ldg(v + jb.a + o), predict<T>(jb.t0, jb.t1, o)));
      mm = d > mm ? d : mm;
    }
  mm = warp_max_ll(mm);
  if ((threadIdx.x & 31) == 0 && mm > 0) atomicMax(errk, mm);
}

// A pair whose partial max |delta| already makes the merge cost at least the two partitions'
// costs is not merged whatever the rest of it holds (the score stays unprofitable, also when it
// is kept for the next round), so its remaining chunks are skipped.  One warp decides.
__device__ __forceinline__ bool job_settled(const LineJob& jb, const long long* errk) {
  long long e = 0;
  if ((threadIdx.x & 31) == 0) e = *(const volatile long long*)errk;
  e = __shfl_sync(FULL_MASK, e, 0);
  return !(part_cost((int64_t)jb.b - jb.a, bits_for(e)) < jb.sum);
}

// Max |delta| of every job still to measure: persistent CTAs, one job at a time, its chunks in
// order (each warp stops at the first chunk after which the pair is settled).
template <typename T> __global__ void __launch_bounds__(256, 4)
job_err_kernel(const T* __restrict__ v, const LineJob* __restrict__ jobs, const int64_t* __restrict__ nch,
               int64_t njobs, long long* __restrict__ err) {
  for (int64_t k = blockIdx.x; k < njobs; k += gridDim.x) {
    const int64_t nc = nch[k];  // 0: kept from the previous round
    if (nc == 0) continue;
    const LineJob jb = jobs[k];
    for (int64_t q = 0; q < nc; q++) {
      if (q > 0 && job_settled(jb, err + k)) break;
      job_chunk<T>(v, jb, q, err + k);
    }
  }
}

// Initial part costs.
__global__ void part_cost_kernel(const LineJob* __restrict__ jobs, const long long* __restrict__ err, int64_t m,
                                 double* __restrict__ pc) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  pc[k] = part_cost((int64_t)jobs[k].b - jobs[k].a, bits_for(err[k]));
}

// Pair scores: merged cost (fresh or cached) and profitability; any profitable -> *any = 1.
__global__ void pair_score_kernel(const LineJob* __restrict__ jobs, const long long* __restrict__ err,
                                  const uint8_t* __restrict__ cached, const double* __restrict__ cached_mc,
                                  const double* __restrict__ pc, int64_t m, double* __restrict__ mc,
                                  uint8_t* __restrict__ prof, int* __restrict__ any) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m - 1) return;
  double c;
  if (cached && cached[k]) c = cached_mc[k];
  else c = part_cost((int64_t)jobs[k].b - jobs[k].a, bits_for(err[k]));
  mc[k] = c;
  const bool p = c < __dadd_rn(pc[k], pc[k + 1]);
  prof[k] = p ? 1 : 0;
  if (p) atomicOr(any, 1);
}

// heads: part k starts a new part unless pair k-1 merges.
__global__ void merge_heads_kernel(const uint8_t* __restrict__ prof, int64_t m, int round, int64_t* __restrict__ head) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const bool absorbed = k > 0 && prof[k - 1] && (((k - 1) + round) % 2 == 0);
  head[k] = absorbed ? 0 : 1;
}

__device__ __forceinline__ bool selected(const uint8_t* prof, int64_t m, int64_t k, int round) {
  return k >= 0 && k < m - 1 && prof[k] && ((k + round) % 2 == 0);
}

__global__ void merge_scatter_kernel(const int32_t* __restrict__ ps, const int32_t* __restrict__ pe,
                                     const double* __restrict__ pc, const double* __restrict__ mc,
                                     const uint8_t* __restrict__ prof, const int64_t* __restrict__ head,
                                     const int64_t* __restrict__ idx, int64_t m, int round,
                                     int32_t* __restrict__ ps2, int32_t* __restrict__ pe2, double* __restrict__ pc2,
                                     uint8_t* __restrict__ cached2, double* __restrict__ cmc2,
                                     const long long* __restrict__ pair_err, const long long* __restrict__ part_err,
                                     long long* __restrict__ part_err2, long long* __restrict__ cerr2) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m || !head[k]) return;
  const int64_t d = idx[k];
  const bool sel = selected(prof, m, k, round);
  ps2[d] = ps[k];
  pe2[d] = sel ? pe[k + 1] : pe[k];
  pc2[d] = sel ? mc[k] : pc[k];
  part_err2[d] = sel ? pair_err[k] : part_err[k];  // a merged pair was measured in full (never settled early)
  // the score of (this part, next part) survives when neither changed
  const int64_t nxt = sel ? k + 2 : k + 1;  // old index of the next head
  const bool keep = !sel && nxt < m && !selected(prof, m, nxt, round);
  cached2[d] = keep ? 1 : 0;
  cmc2[d] = keep ? mc[k] : 0.0;
  cerr2[d] = keep ? pair_err[k] : 0;
}

static inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

template <typename T>
static cudaError_t partition_typed(glc_ctx* ctx, const T* v, int64_t n, int32_t** out_s, int32_t** out_e, int64_t* outP,
                                   cudaStream_t s, std::string* err, long long** out_err) {
  cudaError_t e;
  *out_s = nullptr;
  *out_e = nullptr;
  *outP = 0;
  if (out_err) *out_err = nullptr;
  if (n <= 0) return cudaSuccess;
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
  const int64_t mmax = nb;  // split partitions are >= 128 values except the last
  size_t bytes = 0;
  bytes += al(sizeof(SumPair) * (nb + 1));                     // prefix
  bytes += al(sizeof(SumPair) * (scan_num_tiles(nb) + 1));     // scan tiles (pair)
  bytes += al(sizeof(int32_t) * nb);                           // nb_next
  bytes += al(sizeof(int32_t) * nr * kMaxJumpBlocks) * 2;      // exits, counts
  bytes += al(sizeof(int32_t) * nr) * 3;                       // entries, base, exit_first
  bytes += al(sizeof(int32_t) * nb) * 3;                       // cexit, ccnt, visit
  bytes += al(sizeof(long long) * nb);                         // nb_err
  bytes += al(sizeof(long long) * mmax);                       // kerr
  bytes += al(sizeof(long long) * mmax) * 4;                   // part_err, part_err2, cerr, cerr2
  bytes += al(sizeof(int64_t) * (nb + 1)) * 2;                 // flags, idx
  bytes += al(sizeof(int64_t) * (scan_num_tiles(nb) + 1));     // scan tiles (i64)
  bytes += al(sizeof(int32_t) * mmax) * 4;                     // ps, pe, ps2, pe2
  bytes += al(sizeof(double) * mmax) * 5;                      // pc, pc2, mc, cmc, cmc2
  bytes += al(sizeof(uint8_t) * mmax) * 3;                     // prof, cached, cached2
  bytes += al(sizeof(LineJob) * mmax);                         // jobs
  bytes += al(sizeof(int64_t) * (mmax + 1));                   // nch
  bytes += al(sizeof(long long) * mmax);                       // err
  bytes += al(sizeof(int64_t) * 4);                            // device scalars
  char* buf = nullptr;
  if ((e = pool_alloc(ctx, &buf, bytes, s)) != cudaSuccess) return e;
  char* sp = buf;
  auto take = [&](size_t b) { char* r = sp; sp += al(b); return (void*)r; };
  SumPair* pre = (SumPair*)take(sizeof(SumPair) * (nb + 1));
  SumPair* ptiles = (SumPair*)take(sizeof(SumPair) * (scan_num_tiles(nb) + 1));
  int32_t* nb_next = (int32_t*)take(sizeof(int32_t) * nb);
  int32_t* exits = (int32_t*)take(sizeof(int32_t) * nr * kMaxJumpBlocks);
  int32_t* cnts = (int32_t*)take(sizeof(int32_t) * nr * kMaxJumpBlocks);
  int32_t* entries = (int32_t*)take(sizeof(int32_t) * nr);
  int32_t* base = (int32_t*)take(sizeof(int32_t) * nr);
  int32_t* exit_first = (int32_t*)take(sizeof(int32_t) * nr);
  int32_t* cexit = (int32_t*)take(sizeof(int32_t) * nb);
  int32_t* ccnt = (int32_t*)take(sizeof(int32_t) * nb);
  int32_t* visit = (int32_t*)take(sizeof(int32_t) * nb);
  long long* nb_err = (long long*)take(sizeof(long long) * nb);
  long long* kerr = (long long*)take(sizeof(long long) * mmax);
  long long* part_err = (long long*)take(sizeof(long long) * mmax);
  long long* part_err2 = (long long*)take(sizeof(long long) * mmax);
  long long* cerr = (long long*)take(sizeof(long long) * mmax);
  long long* cerr2 = (long long*)take(sizeof(long long) * mmax);
  int64_t* flags = (int64_t*)take(sizeof(int64_t) * (nb + 1));
  int64_t* idx = (int64_t*)take(sizeof(int64_t) * (nb + 1));
  int64_t* itiles = (int64_t*)take(sizeof(int64_t) * (scan_num_tiles(nb) + 1));
  int32_t* ps = (int32_t*)take(sizeof(int32_t) * mmax);
  int32_t* pe = (int32_t*)take(sizeof(int32_t) * mmax);
  int32_t* ps2 = (int32_t*)take(sizeof(int32_t) * mmax);
  int32_t* pe2 = (int32_t*)take(sizeof(int32_t) * mmax);
  double* pc = (double*)take(sizeof(double) * mmax);
  double* pc2 = (double*)take(sizeof(double) * mmax);
  double* mc = (double*)take(sizeof(double) * mmax);
  double* cmc = (double*)take(sizeof(double) * mmax);
  double* cmc2 = (double*)take(sizeof(double) * mmax);
  uint8_t* prof = (uint8_t*)take(mmax);
  uint8_t* cached = (uint8_t*)take(mmax);
  uint8_t* cached2 = (uint8_t*)take(mmax);
  LineJob* jobs = (LineJob*)take(sizeof(LineJob) * mmax);
  int64_t* nch = (int64_t*)take(sizeof(int64_t) * (mmax + 1));
  long long* perr = (long long*)take(sizeof(long long) * mmax);
  int64_t* dsc = (int64_t*)take(sizeof(int64_t) * 4);  // [0] unused, [1] m, [2] any (int), [3] walk fail
  RangeSums rs{pre, n, nb};

  auto fail = [&](cudaError_t ee) { cudaFreeAsync(buf, s); return ee; };
  static PerDeviceFlag link_attr;
  if (const int dev = current_device(); !link_attr.test(dev)) {
    if ((e = cudaFuncSetAttribute(chain_link_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLinkSmem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(chain_link_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLinkSmem)) != cudaSuccess)
      return fail(e);
    link_attr.set(dev);
  }
  auto grid = [](int64_t x, int b) { return (unsigned)((x + b - 1) / b); };

  block_sums_kernel<T><<<grid(nb * 32, 256), 256, 0, s>>>(v, n, nb, pre);
  if ((e = exclusive_scan<SumPair>(pre, pre, nb, pre + nb, ptiles, s)) != cudaSuccess) return fail(e);
  if ((e = cudaMemsetAsync(nb_next, 0xff, sizeof(int32_t) * nb, s)) != cudaSuccess) return fail(e);
  // dsc[1] = partitions, dsc[3] = first range the walks did not cover (-1: none)
  auto emit = [&]() -> cudaError_t {
    chain_emit_kernel<<<(unsigned)nr, 32, (sizeof(int32_t) + sizeof(uint16_t)) * rb, s>>>(nb_next, nb_err, entries, base,
                                                                                           rg, n, ps, pe, kerr);
    cudaError_t ee = cudaGetLastError();
    if (ee == cudaSuccess)
      ee = cudaMemcpyAsync(ctx->h_stats, dsc + 1, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    return ee == cudaSuccess ? cudaStreamSynchronize(s) : ee;
  };
  auto every_start = [&]() -> cudaError_t {
    split_kernel<T><<<grid(nb, 8), 256, 0, s>>>(v, rs, nb_next, nb_err);
    chain_exit_kernel<<<(unsigned)nr, 32, sizeof(int32_t) * rb, s>>>(nb_next, rg, exits, cnts);
    chain_link_kernel<false><<<1, 1024, kLinkSmem, s>>>(exits, cnts, rg, entries, base, dsc + 1);
    return emit();
  };
  if (all_starts) {
    if ((e = every_start()) != cudaSuccess) return fail(e);
  } else {  // the walk from 0: first only the starts that the walks of the ranges visit
    if ((e = cudaMemsetAsync(cexit, 0xff, sizeof(int32_t) * nb, s)) != cudaSuccess) return fail(e);
    const WalkOut w{nb_next, nb_err, cexit, ccnt, visit, exit_first};
    walk_kernel<T, true><<<(unsigned)nr, 32, 0, s>>>(v, rs, rg, w);
    walk_kernel<T, false><<<(unsigned)nr, 32, 0, s>>>(v, rs, rg, w);
    chain_link_kernel<true><<<1, 1024, kLinkSmem, s>>>(cexit, ccnt, rg, entries, base, dsc + 1);
    if ((e = emit()) != cudaSuccess) return fail(e);
    if (ctx->h_stats[2] >= 0 && (e = every_start()) != cudaSuccess) return fail(e);  // it left the visited starts
  }
  int64_t m = ctx->h_stats[0];
  if (m <= 0 || m > mmax) {
    if (err) *err = "partitioner produced an invalid split";
    cudaFreeAsync(buf, s);
    return cudaErrorUnknown;
  }

  // max |delta| of each job's line (partitions, or adjacent pairs of the merge rounds)
  auto run_jobs = [&](int64_t cnt, int pairs, const uint8_t* cache, const long long* known) -> cudaError_t {
    job_setup_kernel<<<grid(cnt, 256), 256, 0, s>>>(ps, pe, m, pairs, cache, cerr, known, pc, rs, jobs, nch, perr);
    const int64_t resident = (int64_t)ctx->num_sms * 4;  // 256-thread CTAs, four per SM
    job_err_kernel<T><<<(unsigned)(cnt < resident ? cnt : resident), 256, 0, s>>>(v, jobs, nch, cnt, perr);
    return cudaGetLastError();
  };
  // costs of the split partitions: their max |delta| came with the split evaluation
  if ((e = run_jobs(m, 0, nullptr, kerr)) != cudaSuccess) return fail(e);
  part_cost_kernel<<<grid(m, 256), 256, 0, s>>>(jobs, perr, m, pc);
  // each partition's max |delta| travels with it through the merge rounds (for the fit)
  if ((e = cudaMemcpyAsync(part_err, perr, sizeof(long long) * m, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
    return fail(e);
  if ((e = cudaMemsetAsync(cached, 0, mmax, s)) != cudaSuccess) return fail(e);

  for (int round = 0; round < kMaxMergeRounds && m >= 2; round++) {
    if ((e = run_jobs(m - 1, 1, cached, nullptr)) != cudaSuccess) return fail(e);
    if ((e = cudaMemsetAsync(dsc + 2, 0, sizeof(int64_t), s)) != cudaSuccess) return fail(e);
    pair_score_kernel<<<grid(m - 1, 256), 256, 0, s>>>(jobs, perr, cached, cmc, pc, m, mc, prof, (int*)(dsc + 2));
    merge_heads_kernel<<<grid(m, 256), 256, 0, s>>>(prof, m, round, flags);
    if ((e = exclusive_scan<int64_t>(flags, idx, m, dsc + 1, itiles, s)) != cudaSuccess) return fail(e);
    merge_scatter_kernel<<<grid(m, 256), 256, 0, s>>>(ps, pe, pc, mc, prof, flags, idx, m, round, ps2, pe2, pc2,
                                                       cached2, cmc2, perr, part_err, part_err2, cerr2);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
    if ((e = cudaMemcpyAsync(ctx->h_stats, dsc + 1, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return fail(e);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(e);
    const int64_t m2 = ctx->h_stats[0];
    const int any = (int)(ctx->h_stats[1] & 0xffffffff);
    if (!any) break;  // nothing merged: the lists are unchanged
    std::swap(ps, ps2);
    std::swap(pe, pe2);
    std::swap(pc, pc2);
    std::swap(cached, cached2);
    std::swap(cmc, cmc2);
    std::swap(part_err, part_err2);
    std::swap(cerr, cerr2);
    m = m2;
  }

  int32_t* rs_out = nullptr;
  int32_t* re_out = nullptr;
  if ((e = pool_alloc(ctx, &rs_out, sizeof(int32_t) * m, s)) != cudaSuccess) return fail(e);
  if ((e = pool_alloc(ctx, &re_out, sizeof(int32_t) * m, s)) != cudaSuccess) {
    cudaFreeAsync(rs_out, s);
    return fail(e);
  }
  cudaMemcpyAsync(rs_out, ps, sizeof(int32_t) * m, cudaMemcpyDeviceToDevice, s);
  cudaMemcpyAsync(re_out, pe, sizeof(int32_t) * m, cudaMemcpyDeviceToDevice, s);
  if (out_err) {
    long long* er_out = nullptr;
    if ((e = pool_alloc(ctx, &er_out, sizeof(long long) * m, s)) != cudaSuccess) {
      cudaFreeAsync(rs_out, s);
      cudaFreeAsync(re_out, s);
      return fail(e);
    }
    cudaMemcpyAsync(er_out, part_err, sizeof(long long) * m, cudaMemcpyDeviceToDevice, s);
    *out_err = er_out;
  }
  cudaFreeAsync(buf, s);
  *out_s = rs_out;
  *out_e = re_out;
  *outP = m;
  return cudaGetLastError();
}

cudaError_t launch_partition_variable(glc_ctx* ctx, glc_dtype dt, const void* values, int64_t n, int32_t** d_starts,
                                      int32_t** d_ends, int64_t* P, cudaStream_t s, std::string* err,
                                      long long** d_err) {
  switch (dt) {
    case GLC_I32: return partition_typed<int32_t>(ctx, (const int32_t*)values, n, d_starts, d_ends, P, s, err, d_err);
    case GLC_I64: return partition_typed<int64_t>(ctx, (const int64_t*)values, n, d_starts, d_ends, P, s, err, d_err);
    case GLC_U64: return partition_typed<uint64_t>(ctx, (const uint64_t*)values, n, d_starts, d_ends, P, s, err, d_err);
    case GLC_U32: return partition_typed<uint32_t>(ctx, (const uint32_t*)values, n, d_starts, d_ends, P, s, err, d_err);
  }
  return cudaErrorInvalidValue;
}

}  // namespace glc
