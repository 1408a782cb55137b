// leco_seqsum.cuh -- the sums of the reference's fit loop over one run of values, by one warp.
//
// sum y and sum i*y, added one value after the other in FP64 (lr.h:72-77), as leco_rows.cuh
// computes them for rows of 32 values (the reasoning is there): lane j takes the values
// j*c .. j*c + c - 1 and adds them to an approximate start and the three doubles above it;
// what stays in its binade is composed by a scan, the rest is walked over.  The tables are
// in registers and the walk is the same in every lane.
#pragma once
#include "leco_device.cuh"

namespace leco {

// (double)y on the FP64 pipe, rounded once: hi * 2^32 - 2^52 is exact, then + (2^52 + lo).
__device__ __forceinline__ double u64_to_double_fp64(uint64_t y) {
  const double h = __dsub_rn(__hiloint2double(0x45300000, (int)(y >> 32)), 19342813118337666422669312.0);  // 2^84 + 2^52
  return __dadd_rn(h, __hiloint2double(0x43300000, (int)(uint32_t)y));
}

// One sum (S = 0: y, 1: i * y) from the approximate sums before (start) and after (end) each
// lane's values.
template <int S>
__device__ __forceinline__ double warp_seq_sum(const uint64_t *y, uint32_t length, uint32_t c, double start, double end) {
  constexpr int32_t kMax = 1 << 20, kNone = INT32_MIN, kFar = 1 << 26;
  const uint32_t lane = threadIdx.x & 31, first = lane * c;
  const uint32_t cnt = length > first ? min(c, length - first) : 0u;
  const uint64_t base = (uint64_t)__double_as_longlong(start) & ~3ull, next = (uint64_t)__double_as_longlong(end) & ~3ull;
  const uint32_t edge = (((uint32_t)(base >> 52) + 1u) << 20) - 1u;
  double v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = __longlong_as_double((long long)(base + q));
  uint32_t m = (uint32_t)(base >> 32) - edge;
  double k = u32_to_double_fp64(first);
#pragma unroll 2
  for (uint32_t j = 0; j < cnt; ++j) {
    const double yd = u64_to_double_fp64(y[first + j]), t = S == 0 ? yd : __dmul_rn(k, yd);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __dadd_rn(v[q], t);
    m = __viaddmin_u32((uint32_t)__double2hiint(v[0]), 0u - edge, m);
    k = __dadd_rn(k, 1.0);
  }
  const uint32_t h = (uint32_t)__double2hiint(v[0]);
  bool reg = m >= 2 && (base & 0xfffffffffffffull) >= (1ull << 28) && h <= edge + 0x100000u - 1u;
  int32_t r[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t d = (int64_t)((uint64_t)__double_as_longlong(v[q]) - next);
    const bool ok = d > -(int64_t)kMax && d < (int64_t)kMax;
    reg = reg && ok;
    r[q] = ok ? (int32_t)d : kNone;
  }
  const bool walked = !reg || h > edge;
  const uint32_t spec = __ballot_sync(0xffffffffu, walked), irr = __ballot_sync(0xffffffffu, !reg);
  const uint32_t below = spec & (0xffffffffu >> (31 - lane));
  const uint32_t run0 = below ? 32u - (uint32_t)__clz((int)below) : 0u;  // the run's first lane
  int32_t c0 = r[0], c1 = r[1] - 1;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const int32_t p0 = __shfl_up_sync(0xffffffffu, c0, d), p1 = __shfl_up_sync(0xffffffffu, c1, d);
    if (!walked && lane >= run0 + d) {
      const int32_t n0 = p0 + ((p0 & 1) ? c1 : c0), n1 = p1 + ((p1 & 1) ? c0 : c1);
      c0 = n0;
      c1 = n1;
    }
  }
  const uint32_t rows = (length + c - 1) / c;
  int64_t wide = 0;  // the sum's distance from the start of lane `pos`, in ulps
  auto add_lane = [&](uint32_t l) {  // value by value from the exact sum
    const uint64_t b0 = __shfl_sync(0xffffffffu, (unsigned long long)base, l), n0 = __shfl_sync(0xffffffffu, (unsigned long long)next, l);
    double acc = __longlong_as_double((long long)(b0 + (uint64_t)wide)), kk = u32_to_double_fp64(l * c);
    const uint32_t e = min(length, (l + 1) * c);
#pragma unroll 4
    for (uint32_t j = l * c; j < e; ++j) {
      const double yd = u64_to_double_fp64(y[j]);
      acc = __dadd_rn(acc, S == 0 ? yd : __dmul_rn(kk, yd));
      kk = __dadd_rn(kk, 1.0);
    }
    wide = (int64_t)((uint64_t)__double_as_longlong(acc) - n0);
  };
  for (uint32_t pos = 0; pos < rows;) {
    const uint32_t rest = spec >> pos, run = min(rest ? (uint32_t)__ffs((int)rest) - 1u : 32u, rows - pos);
    int32_t delta = wide > kFar ? kFar : wide < -kFar ? -kFar : (int32_t)wide;
    const bool near = delta > -kFar && delta < kFar;
    if (run) {
      if (near) {
        const int32_t x0 = __shfl_sync(0xffffffffu, c0, pos + run - 1), x1 = __shfl_sync(0xffffffffu, c1, pos + run - 1);
        wide = delta + ((delta & 1) ? x1 : x0);
      } else {
        for (uint32_t q = 0; q < run; ++q) add_lane(pos + q);
      }
      pos += run;
      continue;
    }
    const uint32_t a = (uint32_t)delta & 3u;
    const int32_t x = __shfl_sync(0xffffffffu, a == 0 ? r[0] : a == 1 ? r[1] : a == 2 ? r[2] : r[3], pos);
    const bool certain = !((irr >> pos) & 1u);
    if (near && (certain || ((uint32_t)delta < 4u && x != kNone))) wide = certain ? ((delta - (int32_t)a) >> 1) + x : x;
    else add_lane(pos);
    ++pos;
  }
  return __longlong_as_double((long long)(__shfl_sync(0xffffffffu, (unsigned long long)next, rows - 1) + (uint64_t)wide));
}

// Both sums over y[0 .. length) (shared or global memory), length >= 1 and the same in every
// lane of the warp; the results too.
__device__ __forceinline__ void warp_seq_sums(const uint64_t *y, uint32_t length, double &sumy, double &sumxy) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t c = ((length + 31) / 32) | 1u;  // odd: the lanes' reads spread over the banks
  const uint32_t first = lane * c, cnt = length > first ? min(c, length - first) : 0u;
  double a0 = 0.0, a1 = 0.0, k = u32_to_double_fp64(first);
#pragma unroll 4
  for (uint32_t j = 0; j < cnt; ++j) {
    const double yd = u64_to_double_fp64(y[first + j]);
    a0 = __dadd_rn(a0, yd);
    a1 = __dadd_rn(a1, __dmul_rn(k, yd));
    k = __dadd_rn(k, 1.0);
  }
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const double o0 = __shfl_up_sync(0xffffffffu, a0, d), o1 = __shfl_up_sync(0xffffffffu, a1, d);
    if (lane >= d) {
      a0 = __dadd_rn(a0, o0);
      a1 = __dadd_rn(a1, o1);
    }
  }
  double s0 = __shfl_up_sync(0xffffffffu, a0, 1), s1 = __shfl_up_sync(0xffffffffu, a1, 1);
  if (lane == 0) s0 = s1 = 0.0;
  sumy = __shfl_sync(0xffffffffu, a0, 31);
  sumxy = __shfl_sync(0xffffffffu, a1, 31);
  // below 2^53 every partial sum is an exact integer
  if (!(sumy < 9007199254740992.0)) sumy = warp_seq_sum<0>(y, length, c, s0, a0);
  if (!(sumxy < 9007199254740992.0)) sumxy = warp_seq_sum<1>(y, length, c, s1, a1);
}

}  // namespace leco
