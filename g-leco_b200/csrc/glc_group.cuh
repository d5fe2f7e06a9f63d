// glc_group.cuh -- a thread per group of 32 consecutive values.
//
// Where every partition starts at a multiple of 32 values, a group's fields, at its partition's width
// b, are exactly b whole words of the bitstream: a thread keeps the 32 fields of its group in
// registers and appends them to words with one funnel shift each.  Shared by the one-pass fixed
// compress (compress_fixed.cu) and the packer of fitted partitions (pack.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "glc_internal.h"

namespace glc {

// A CTA of 128 threads takes a tile of 4096 values; group G's row starts G * (32 sizeof(T) + 16)
// bytes into the stage, so the lanes of a warp read their rows in 16-byte pieces without bank
// conflicts (rows without the 16 bytes would put every lane on the same banks).
constexpr int kCgThreads = 128;
template <typename T> __host__ __device__ constexpr int cg_row_bytes() { return 32 * (int)sizeof(T) + 16; }
template <typename T> __host__ __device__ constexpr int cg_stage_bytes() { return kCgThreads * cg_row_bytes<T>(); }
static_assert(cg_row_bytes<int32_t>() >= 4 * 32, "the staged words of a segment fit its rows");

// Byte offset in the stage of value j of the tile.
template <typename T> __device__ __forceinline__ int cg_at(int j) { return j * (int)sizeof(T) + (j >> 5) * 16; }

template <int BYTES> __device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int valid) {
  // copies `valid` bytes and zeroes the rest of the BYTES
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(valid) : "memory");
}

// Starts the copies of the tile's values (cnt of them at src, the rest zero) into the rows of the stage;
// cg_load_wait waits for this thread's.
template <typename T> __device__ __forceinline__ void cg_load(uint8_t* stage, const T* src, int cnt, int tid) {
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(stage);
  constexpr int kPer = 16 / (int)sizeof(T);  // values per 16-byte copy
  constexpr int kIters = kDecodeTile / kPer / kCgThreads;
  const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (vec && cnt == kDecodeTile) {  // copies a whole number of rows apart: one address each side, constant steps
    constexpr int kStep = kCgThreads * kPer;
    static_assert(kStep % 32 == 0, "a step is a whole number of rows");
    const T* p = src + tid * kPer;
    const uint32_t d = base + cg_at<T>(tid * kPer);
#pragma unroll
    for (int i = 0; i < kIters; i++) cp_async<16>(d + i * (kStep / 32) * cg_row_bytes<T>(), p + i * kStep, 16);
  } else if (vec) {
#pragma unroll 4
    for (int i = 0; i < kIters; i++) {
      const int j = (i * kCgThreads + tid) * kPer;
      const int left = (cnt - j) * (int)sizeof(T);
      cp_async<16>(base + cg_at<T>(j), left > 0 ? src + j : src, left >= 16 ? 16 : (left > 0 ? left : 0));
    }
  } else {  // values aligned to their own size only
#pragma unroll 8
    for (int i = 0; i < kDecodeTile / kCgThreads; i++) {
      const int j = i * kCgThreads + tid;
      cp_async<(int)sizeof(T)>(base + cg_at<T>(j), j < cnt ? src + j : src, j < cnt ? (int)sizeof(T) : 0);
    }
  }
}
__device__ __forceinline__ void cg_load_wait() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory"); }

// The values of 16 bytes of a row.
template <typename T> struct CgVec {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
  __device__ __forceinline__ explicit CgVec(const uint8_t* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    memcpy(v, &u, 16);
  }
};

constexpr double kMagic = 6755399441055744.0;        // K = 1.5 * 2^52: the bits of K + v are 0x4338... + v, |v| <= 2^51
constexpr double kHalfBias = 0x1.fffffffffffffp-2;    // 0.5 - 2^-54

// How a partition's residuals are computed (uniform per partition, so per thread):
//   CF_DIRECT   direct copy (a uint64 value above 2^53): the field is the value;
//   CF_NONNEG   |y| < 2^51 and predictions in [-0.25, 2^51] (4-byte types: inside the type): in
//               FP64 with K: K + y from the bits, K + pred = (x + (0.5 - 2^-54)) + K rounded toward
//               zero, their difference is y - pred exactly;
//   CF_NONPOS   the mirror for signed types, predictions in [-2^51, 0.25]: K - pred =
//               ((0.5 - 2^-54) - x) + K rounded toward zero;
//   CF_OFFSET   8-byte types with predictions in [2^50, 2^62] within 2^50 of c = trunc(theta0):
//               x - c and x - c + 0.5 are exact, pred = c + floor(x - c + 0.5), y - c by integer
//               arithmetic (a thread whose |y - c| reaches 2^51 recomputes its values in general);
//   CF_GENERAL  predict_from / calc_delta / abs_ref per value.
// Each gives calc_delta<T>(y, predict_from<T>(fma(theta1, i, theta0))) exactly; the field is its
// low 32 bits (the low bits of (y - pred) + K), which is all the packing of a width <= 31 reads.
enum : int { CF_DIRECT = 0, CF_NONNEG = 1, CF_NONPOS = 2, CF_GENERAL = 3, CF_OFFSET = 4 };

// Exact sum over a reduction segment of W lanes (32; 16 where a partition is 16 groups, 8 where it is
// eight): for a whole warp two redux sums of 24-bit limbs.  Any |v| < 2^50 will do: 32 low limbs stay
// below 2^29, 32 high limbs (below 2^26 each) below 2^31.
__device__ __forceinline__ long long seg_sum50(long long v, int W) {
  if (W == 32) {
    const unsigned lo = __reduce_add_sync(FULL_MASK, (unsigned)v & 0xFFFFFFu);
    const int hi = __reduce_add_sync(FULL_MASK, (int)(v >> 24));
    return (long long)hi * 16777216ll + (long long)lo;
  }
  for (int msk = W >> 1; msk > 0; msk >>= 1) v += __shfl_xor_sync(FULL_MASK, v, msk);
  return v;
}
__device__ __forceinline__ unsigned seg_max_u32(unsigned v, int W) {
  if (W == 32) return __reduce_max_sync(FULL_MASK, v);
  for (int msk = W >> 1; msk > 0; msk >>= 1) {
    const unsigned o = __shfl_xor_sync(FULL_MASK, v, msk);
    v = o > v ? o : v;
  }
  return v;
}
__device__ __forceinline__ unsigned seg_or_u32(unsigned v, int W) {
  if (W == 32) return __reduce_or_sync(FULL_MASK, v);
  for (int msk = W >> 1; msk > 0; msk >>= 1) v |= __shfl_xor_sync(FULL_MASK, v, msk);
  return v;
}
__device__ __forceinline__ unsigned long long seg_max_u64(unsigned long long v, int W) {
  const unsigned hi = seg_max_u32((unsigned)(v >> 32), W);
  const unsigned lo = seg_max_u32((unsigned)(v >> 32) == hi ? (unsigned)v : 0u, W);
  return ((unsigned long long)hi << 32) | lo;
}

// The residual mode of a partition from its line and the range test of its values.
template <typename T>
__device__ __forceinline__ int cf_mode(double t0, double t1, int len, bool vsafe, double& c, long long& ci) {
  const double xa = t0, xb = __fma_rn(t1, (double)(len - 1), t0);  // the ends (fma is monotone in i)
  const double lo = fmin(xa, xb), hi = fmax(xa, xb);
  constexpr double kS = 2251799813685248.0;  // 2^51
  const double hi_ok = sizeof(T) == 4 ? (TypeTraits<T>::is_signed ? 2147483646.0 : 4294967294.0) : kS;
  const double lo_ok = sizeof(T) == 4 ? -2147483647.0 : -kS;
  if (vsafe && lo >= -0.25 && hi <= hi_ok) return CF_NONNEG;
  if (TypeTraits<T>::is_signed && vsafe && hi <= 0.25 && lo >= lo_ok) return CF_NONPOS;
  if (sizeof(T) == 8 && lo >= 1125899906842624.0 && hi <= 4611686018427387904.0) {  // [2^50, 2^62]
    c = trunc(t0);
    if (fabs(__dsub_rn(xb, c)) < 562949953421312.0) {  // 2^49
      ci = __double2ll_rz(c);
      return CF_OFFSET;
    }
  }
  return CF_GENERAL;
}

// One value's residual, or the value itself for direct copy, in 64 bits (the slow path).  The fast
// modes' formulas are those of cg_resid, exact modulo 2^64 as calc_delta is for signed types; a
// uint64 partition outside direct copy holds values up to 2^53, where calc_delta does not saturate.
template <typename T>
__device__ __forceinline__ long long cg_field(T y, double xi, int mode, double t0, double t1, double c, long long ci) {
  constexpr long long kBits = 0x4338000000000000ll;
  const uint64_t v = TypeTraits<T>::is_signed ? (uint64_t)(long long)y : (uint64_t)y;
  const double x = __fma_rn(t1, xi, t0);
  if (mode == CF_NONNEG) return (long long)(v - (uint64_t)(__double_as_longlong(__dadd_rz(__dadd_rn(x, kHalfBias), kMagic)) - kBits));
  if (sizeof(T) == 8 && mode == CF_OFFSET)
    return (long long)(v - (uint64_t)ci -
                       (uint64_t)(__double_as_longlong(__dadd_rz(__dadd_rn(__dsub_rn(x, c), 0.5), kMagic)) - kBits));
  if (TypeTraits<T>::is_signed && mode == CF_NONPOS)
    return (long long)(v + (uint64_t)(__double_as_longlong(__dadd_rz(__dsub_rn(kHalfBias, x), kMagic)) - kBits));
  if (mode == CF_DIRECT) return (long long)v;  // the field is the value itself
  return calc_delta<T>(y, predict_from<T>(x));
}

// The slow path's packing: the group's values become its words (width b, 1 to 64) in place.  After
// value f, at most (f + 1) b / 32 words are complete, which end no later than value f does (4-byte
// types, fields of up to 33 bits: the 33rd word lies in the row's padding).
template <typename T>
__device__ __forceinline__ void cg_pack_slow(uint8_t* row, int glen, int i0, int b, int mode, double t0, double t1,
                                             double c, long long ci) {
  uint32_t* words = reinterpret_cast<uint32_t*>(row);
  const uint64_t mask = b >= 64 ? ~0ull : ((1ull << b) - 1ull);
  uint32_t acc = 0u;  // bits not yet stored: `have` (0 to 31) of them
  int have = 0, k = 0;
  double xi = (double)i0;
#pragma unroll 1
  for (int f = 0; f < glen; f++) {
    const T y = *reinterpret_cast<const T*>(row + f * (int)sizeof(T));
    const uint64_t v = (uint64_t)cg_field<T>(y, xi, mode, t0, t1, c, ci) & mask;
    xi = __dadd_rn(xi, 1.0);
    const uint64_t lo = (v << have) | acc;
    const uint32_t over = have ? (uint32_t)(v >> 32 >> (32 - have)) : 0u;  // the bits past 64
    int n = have + b;  // 1 to 95 bits in (over, lo)
    uint32_t w0 = (uint32_t)lo, w1 = (uint32_t)(lo >> 32), w2 = over;
    if (n >= 32) { words[k++] = w0; w0 = w1; w1 = w2; n -= 32; }
    if (n >= 32) { words[k++] = w0; w0 = w1; n -= 32; }
    acc = w0;
    have = n;
  }
  if (have) words[k] = acc;
}

// Packs a group's 32 fields (width B) into its B words at stg.  acc holds the bits so far at its top
// and older bits below them: one funnel shift appends a field (whatever lies above its B bits is
// shifted out), and a word is complete when 32 bits have come in.
template <int B>
__device__ __forceinline__ void cg_pack(const uint32_t (&fl)[32], uint32_t* __restrict__ stg) {
  uint32_t acc = 0u;
#pragma unroll
  for (int f = 0; f < 32; f++) {
    const int sh = (f * B) & 31;  // bits of the open word
    if (sh + B < 32) {
      acc = __funnelshift_r(acc, fl[f], B);
    } else {
      stg[(f * B) >> 5] = __funnelshift_r(acc, fl[f], 32 - sh);
      acc = fl[f] << (32 - B);
    }
  }
}

__device__ __forceinline__ void cg_pack_dispatch(int b, const uint32_t (&fl)[32], uint32_t* __restrict__ stg) {
  switch (b) {
#define GLC_CG_PACK(B) \
  case B: cg_pack<B>(fl, stg); break;
    GLC_CG_PACK(1) GLC_CG_PACK(2) GLC_CG_PACK(3) GLC_CG_PACK(4) GLC_CG_PACK(5) GLC_CG_PACK(6) GLC_CG_PACK(7)
    GLC_CG_PACK(8) GLC_CG_PACK(9) GLC_CG_PACK(10) GLC_CG_PACK(11) GLC_CG_PACK(12) GLC_CG_PACK(13) GLC_CG_PACK(14)
    GLC_CG_PACK(15) GLC_CG_PACK(16) GLC_CG_PACK(17) GLC_CG_PACK(18) GLC_CG_PACK(19) GLC_CG_PACK(20)
    GLC_CG_PACK(21) GLC_CG_PACK(22) GLC_CG_PACK(23) GLC_CG_PACK(24) GLC_CG_PACK(25) GLC_CG_PACK(26)
    GLC_CG_PACK(27) GLC_CG_PACK(28) GLC_CG_PACK(29) GLC_CG_PACK(30) GLC_CG_PACK(31)
#undef GLC_CG_PACK
    default: break;  // width 0: no words
  }
}

// A warp's words from its stage to the column: `nw` words of groups of width bs (1 to 31), which lie
// bs words apart, or bs + 1 for an even bs (so that the lanes' stores fall on different banks).
// VEC: dst is 16-byte aligned.
template <bool VEC>
__device__ __forceinline__ void cg_copy_words(const uint32_t* q, uint32_t* __restrict__ dst, int nw, int bs, int lane) {
  const bool pad = (bs & 1) == 0;
  const uint32_t mb = bs > 1 ? 0xffffffffu / (uint32_t)bs + 1u : 0u;  // w / b by a multiply-high (w < 2^10)
  int w0 = 0;
  if (VEC) {
    for (int w = 4 * lane; w + 3 < nw; w += 128) {
      uint32_t v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = q[w + u + (pad ? (int)__umulhi((uint32_t)(w + u), mb) : 0)];
      *reinterpret_cast<uint4*>(dst + w) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    w0 = nw & ~3;
  }
  for (int w = w0 + lane; w < nw; w += 32) dst[w] = q[w + (pad ? (int)__umulhi((uint32_t)w, mb) : 0)];
}

}  // namespace glc
