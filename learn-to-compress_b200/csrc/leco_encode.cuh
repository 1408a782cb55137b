// leco_encode.cuh -- what the encoders share: look-back over per-block sizes, image writers,
// the fit's model formulas, and the block encoder of the legacy u32 format (the other
// codecs' encoder is leco_rows.cuh).
//
// Reference: Leco_int<T>::encodeArray8_int (piecewise_fix_integer_template.h:27-140),
// FOR_int<T>::encodeArray8_int (FOR_integer_template.h:26-81),
// Delta_int<T>::encodeArray8_int (delta_integer_template.h:26-87),
// Leco_int_poly<T,2>::encodeArray8_int (poly_fix_integer_template.h:28-91),
// packers write_delta_int_T / write_FOR_int_T (bit_write.h:257-390).
#pragma once
#include <type_traits>

#include "leco_device.cuh"
#include "leco_internal.h"

namespace leco {

constexpr uint64_t kFlagAgg = 1ull << 62, kFlagIncl = 2ull << 62, kValMask = (1ull << 62) - 1;
constexpr uint32_t kSpinLimit = 1u << 22;  // x ~32-256 ns backoff: far above any real wait

// Per-block model scratch: the sequential reference fit writes 3 doubles per block.
struct EncodeArgs {
  const void *values;
  uint64_t n;
  uint32_t bs;
  uint64_t nb;
  uint8_t *payload;
  uint64_t payload_cap;
  uint64_t *offsets;
  leco_dir_entry *dir;
  const double *seq_models;  // [nb*3] or null (exact fit in-kernel)
  double polyX[10];          // X sums for full blocks [0..4] and for the tail block [5..9]
  uint64_t *status;          // [nb] look-back words, zeroed
  uint32_t *ticket;          // zeroed: [0] the legacy encoder's ticket, [1..3] the row encoder's left items
  uint32_t *error;           // error word
  uint32_t item_wait;        // row encoder: polls after which an item leaves its place
  bool reversed;             // row encoder: the last CTA takes the first role (tests)
};

// Shared-memory layout helper.
template <typename T>
struct EncSmem {
  T *vals;          // [bs] values, later residual magnitudes (linear / poly2)
  uint32_t *signs;  // [bs/32 + 9] sign bits (one word per 32 values, rounded up to 256)
  u128 *red;        // [66]
  uint8_t *hdr;     // [32] header bytes
  uint64_t *bcast;  // [8]
};

template <typename T>
__device__ __forceinline__ EncSmem<T> enc_smem(uint8_t *base, uint32_t bs) {
  EncSmem<T> s;
  s.red = reinterpret_cast<u128 *>(base);                      // 66 * 16 = 1056
  s.bcast = reinterpret_cast<uint64_t *>(base + 1056);         // 8 * 8 = 64
  s.hdr = base + 1120;                                         // 32
  s.signs = reinterpret_cast<uint32_t *>(base + 1152);         // (bs/32+9)*4
  uint32_t soff = 1152 + ((bs / 32 + 9) * 4 + 15) / 16 * 16;
  s.vals = reinterpret_cast<T *>(base + soff);
  return s;
}
// The value region holds round32(bs) values plus 16 bytes: the u64 LeCo path keeps
// round32(bs) staged words and a packed body of up to round32(bs) + 4 words there.
__host__ __device__ inline uint32_t enc_smem_bytes(uint32_t bs, uint32_t s) {
  return 1152 + ((bs / 32 + 9) * 4 + 15) / 16 * 16 + (bs + 31) / 32 * 32 * s + 16;
}
// Decoupled look-back (single-pass prefix sum over per-block totals), run by one
// full warp.  lookback_excl walks back over the predecessors of block b 32 at a
// time (lane i reads block j - i): it needs every block from the nearest one down
// to the first with an inclusive prefix, and waits only while one of those has
// published nothing.  It needs nothing of block b itself, so it can run while the
// block is still being encoded.  Returns the exclusive prefix; on a wait that
// exceeds the spin limit sets kErrTimeout and returns ~0.  lookback_prefix
// publishes block b's total first and its inclusive prefix last.
__device__ __forceinline__ uint64_t lookback_excl(const uint64_t *status, uint64_t b, uint32_t *error,
                                                  uint32_t spin_limit = kSpinLimit) {
  const int lane = threadIdx.x & 31;
  if (b == 0) return 0;
  uint64_t excl = 0;
  int64_t j = (int64_t)b - 1;
  for (;;) {
    const int64_t idx = j - lane;
    uint64_t v = kFlagIncl;  // lanes before block 0 read as "inclusive 0"
    uint32_t spins = 0, ns = 32;
    uint32_t incl;
    int last;  // the farthest lane this window of predecessors needs
    for (;;) {
      if (idx >= 0) v = ld_relaxed(&status[idx]);
      incl = __ballot_sync(0xffffffffu, (v >> 62) == 2);
      last = incl ? __ffs(incl) - 1 : 31;
      const uint32_t need = last == 31 ? 0xffffffffu : ((2u << last) - 1u);
      if (!(__ballot_sync(0xffffffffu, (v >> 62) == 0) & need)) break;
      if (++spins > spin_limit) {
        if (lane == 0) atomicOr(error, kErrTimeout);
        return ~0ull;
      }
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
    }
    excl += warp_sum_u64(lane <= last ? (v & kValMask) : 0);
    if (incl) break;
    j -= 32;
  }
  return excl;
}
__device__ __forceinline__ uint64_t lookback_prefix(uint64_t *status, uint64_t b, uint64_t my, uint32_t *error,
                                                    uint32_t spin_limit = kSpinLimit) {
  const int lane = threadIdx.x & 31;
  if (b > 0 && lane == 0) st_relaxed(&status[b], kFlagAgg | my);
  const uint64_t excl = lookback_excl(status, b, error, spin_limit);
  if (excl != ~0ull && lane == 0) st_relaxed(&status[b], kFlagIncl | (excl + my));
  return excl;
}

// Prefix publisher, one warp.  A block's own look-back ends at the nearest inclusive
// prefix, but those lag: a block publishes its inclusive prefix only when its own
// look-back is done, so with ~900 blocks in flight each look-back sums long runs of
// totals.  This warp walks the status words in block order (128 per step, lane i
// holding blocks j + 4i .. j + 4i + 3) and turns every published total into an
// inclusive prefix as soon as it and all blocks before it have published, so the blocks
// find one among their nearest predecessors.  Every value it writes is the one the
// block's own look-back would publish.  Block 0's inclusive prefix must be published
// (by this warp) before the call.  Returns after block nb - 1, or sets kErrTimeout on a
// wait that exceeds the spin limit.
__device__ __forceinline__ void publish_prefixes(uint64_t *status, uint64_t nb, uint32_t *error,
                                                 uint32_t spin_limit = kSpinLimit) {
  constexpr int K = 4;
  const int lane = threadIdx.x & 31;
  __syncwarp();
  uint64_t run = ld_relaxed(&status[0]) & kValMask;  // inclusive prefix before block j
  uint64_t j = 1;
  uint32_t spins = 0, ns = 32;
  while (j < nb) {
    uint64_t v[K];
    int first = K * 32;  // this lane's first unpublished position
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint64_t idx = j + K * lane + k;
      v[k] = idx < nb ? ld_relaxed(&status[idx]) : 0;
    }
#pragma unroll
    for (int k = K - 1; k >= 0; --k)
      if ((v[k] >> 62) == 0) first = K * lane + k;
    const int n = __reduce_min_sync(0xffffffffu, first);  // published run j .. j + n - 1
    if (n == 0) {
      if (++spins > spin_limit) {
        if (lane == 0) atomicOr(error, kErrTimeout);
        return;
      }
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
      continue;
    }
    spins = 0;
    ns = 32;
    // Segmented inclusive scan: an inclusive prefix restarts the sum.  Lane-local first...
    uint64_t p[K];
    bool f[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint64_t val = v[k] & kValMask;
      const bool fl = (v[k] >> 62) == 2;
      p[k] = (k == 0 || fl) ? val : p[k - 1] + val;
      f[k] = fl || (k > 0 && f[k - 1]);
    }
    // ... then over the lanes' totals
    uint64_t tp = p[K - 1];
    int tf = f[K - 1];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t q = __shfl_up_sync(0xffffffffu, tp, d);
      const int fq = __shfl_up_sync(0xffffffffu, tf, d);
      if (lane >= d && !tf) {
        tp += q;
        tf = fq;
      }
    }
    uint64_t ep = __shfl_up_sync(0xffffffffu, tp, 1);
    int ef = __shfl_up_sync(0xffffffffu, tf, 1);
    if (lane == 0) {
      ep = 0;
      ef = 0;
    }
    if (!ef) ep += run;
    uint64_t last = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint64_t fin = f[k] ? p[k] : ep + p[k];
      const int pos = K * lane + k;
      if (pos < n && (v[k] >> 62) == 1) st_relaxed(&status[j + pos], kFlagIncl | fin);
      if (pos == n - 1) last = fin;
    }
    run = __shfl_sync(0xffffffffu, last, (n - 1) / K);
    j += n;
  }
}

// True when every prediction of a len-value block with model (a0, a1, a2) is a
// finite double inside (-2^62, 2^62): the x86 out-of-range rule cannot apply.
__device__ __forceinline__ bool model_in_range(double a0, double a1, double a2, uint32_t len) {
  const double L = __uint2double_rn(len ? len - 1 : 0);
  return fabs(a0) + fabs(a1) * L + fabs(a2) * L * L < 4611686018427387904.0;
}

// Image writer: writes image bytes [0, size) of a block to payload[goff...].
// Image byte i < H is hdr[i]; byte i >= H is byte (i-H) of the LSB-first
// concatenation of fields 0..n-1 (l bits each), zero past the last field.
template <typename FieldFn>
__device__ __forceinline__ uint64_t gather_bits(uint32_t p, uint32_t nbits, uint32_t l, uint32_t n, FieldFn field) {
  uint32_t k = p / l, o = p - k * l;
  u128 acc = k < n ? (u128)(field(k) >> o) : (u128)0;
  uint32_t have = l - o;
  ++k;
  while (have < nbits) {
    if (k < n) acc |= (u128)field(k) << have;
    have += l;
    ++k;
  }
  return (uint64_t)acc & lowmask(nbits);
}

// 128 bits of the body starting at body bit p, for fields of at most 32 bits:
// 32-bit output words assembled in a 64-bit accumulator; k0 = p / l through a
// reciprocal (exact for p < 2^21 and l <= 64).
template <typename FieldFn>
__device__ __forceinline__ uint4 gather128_narrow(uint32_t p, uint32_t l, uint32_t rcp, uint32_t n, FieldFn field) {
  uint32_t k = l == 1 ? p : __umulhi(p, rcp);
  const uint32_t o = p - k * l;
  uint64_t acc = k < n ? ((uint64_t)field(k) >> o) : 0;
  uint32_t have = l - o;
  ++k;
  uint32_t w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    while (have < 32) {
      if (k < n) acc |= (uint64_t)field(k) << have;
      have += l;
      ++k;
    }
    w[q] = (uint32_t)acc;
    acc >>= 32;
    have -= 32;
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename FieldFn>
__device__ __forceinline__ void write_image(uint8_t *payload, uint64_t goff, uint64_t size, uint32_t H,
                                            const uint8_t *hdr, uint32_t l, uint32_t nfields, FieldFn field,
                                            uint32_t rank, uint32_t nthreads) {
  const uint64_t gend = goff + size;
  const uint64_t c0 = goff >> 4, c1 = (gend + 15) >> 4;
  const uint64_t body0 = goff + H;  // first body byte (global)
  const uint32_t rcp = l > 1 ? (uint32_t)((0x100000000ull + l - 1) / l) : 0;  // ceil(2^32 / l); l == 1 divides trivially
  for (uint64_t c = c0 + rank; c < c1; c += nthreads) {
    const uint64_t cb = c << 4;
    if (cb >= body0 && cb + 16 <= gend && l) {
      uint32_t p = (uint32_t)((cb - body0) * 8);
      if (l <= 32) {
        *reinterpret_cast<uint4 *>(payload + cb) = gather128_narrow(p, l, rcp, nfields, field);
      } else {
        uint64_t lo = gather_bits(p, 64, l, nfields, field);
        uint64_t hi = gather_bits(p + 64, 64, l, nfields, field);
        *reinterpret_cast<ulonglong2 *>(payload + cb) = make_ulonglong2(lo, hi);
      }
    } else {
      for (int j = 0; j < 16; ++j) {
        uint64_t g = cb + j;
        if (g < goff || g >= gend) continue;
        uint64_t i = g - goff;
        uint8_t byte;
        if (i < H) byte = hdr[i];
        else if (!l) byte = 0;
        else byte = (uint8_t)gather_bits((uint32_t)((i - H) * 8), 8, l, nfields, field);
        payload[g] = byte;
      }
    }
  }
}

// (int64_t)(m0 + m1*i) under conversion rule R: 0 = every prediction of the block
// lies in [0, 2^51), both conversions on the FP64 pipe (exact); 1 = in range, plain
// truncation; 2 = the x86 out-of-range rule (f2i_x86).
template <int R>
__device__ __forceinline__ int64_t lin_pred(double m0, double m1, uint32_t i) {
  if (R == 0) return trunc_nonneg_fp64(pred_linear_fp64(m0, m1, i));
  const double p = pred_linear(m0, m1, i);
  return R == 1 ? __double2ll_rz(p) : f2i_x86(p);
}
// Calls fn(std::integral_constant<int, R>) with the cheapest rule valid for the
// block's len predictions, so the loops inside fn carry no per-value test.
template <typename Fn>
__device__ __forceinline__ void with_pred_rule(double m0, double m1, uint32_t len, Fn fn) {
  if (preds_nonneg(m0, m1, len)) fn(std::integral_constant<int, 0>{});
  else if (model_in_range(m0, m1, 0.0, len)) fn(std::integral_constant<int, 1>{});
  else fn(std::integral_constant<int, 2>{});
}

// ---- shared-memory access ------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds_v2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_v2(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y));
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Field of signed residual r (|r| < 2^(L-1)): the magnitude with the sign bit
// (r > 0, "data[i] > pred") at bit L-1 (write_delta_int_T, bit_write.h:257-323).
template <int L>
__device__ __forceinline__ uint32_t lin_field(uint32_t r) {
  return (int32_t)r > 0 ? (r | (1u << (L - 1))) : (uint32_t)(-(int32_t)r);
}
// Adds field f of row position j (bits [j*L, j*L + L) of the row's bit stream) to the
// row's words; fields are disjoint and come in increasing j, so adding is or-ing.
template <int L>
__device__ __forceinline__ void place_field(uint32_t (&w)[L], uint32_t f, int j) {
  const int p = j * L, q = p >> 5, s = p & 31;
  w[q] += f << s;
  if (s + L > 32) w[q + 1] += f >> (32 - s);
}
// Stores bytes [lo, hi) of the 16-byte chunk (w0..w3, little-endian) at dst (16-byte
// aligned) with the fewest aligned stores: the chunk's other bytes belong to the
// neighbouring block's image, written by another CTA.
__device__ __forceinline__ void store_chunk_bytes(uint8_t *dst, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                                                  uint32_t lo, uint32_t hi) {
  for (uint32_t pos = lo; pos < hi;) {
    const uint32_t rem = hi - pos, wi = pos >> 2, sh = (pos & 3u) * 8u;
    const uint32_t w = wi == 0 ? w0 : wi == 1 ? w1 : wi == 2 ? w2 : w3;
    if ((pos & 7u) == 0 && rem >= 8) {
      const uint32_t wn = wi == 0 ? w1 : w3;
      *reinterpret_cast<uint64_t *>(dst + pos) = ((uint64_t)wn << 32) | w;
      pos += 8;
    } else if ((pos & 3u) == 0 && rem >= 4) {
      *reinterpret_cast<uint32_t *>(dst + pos) = w;
      pos += 4;
    } else if ((pos & 1u) == 0 && rem >= 2) {
      *reinterpret_cast<uint16_t *>(dst + pos) = (uint16_t)(w >> sh);
      pos += 2;
    } else {
      dst[pos] = (uint8_t)(w >> sh);
      pos += 1;
    }
  }
}

// Legacy u32 format, piecewise_fix_op_max::encodeArray8
// (piecewise_fix_op_minimize_maxerror.h:45-95): the slope is rounded to float,
// residuals are ints against (long long)(theta0 + theta1*i), the midpoint shift
// is taken in int arithmetic, and the width is bits(max |r|) + 1 where a
// residual of -2^31 does not count (the reference's abs() leaves it negative).
// On return vals holds |r| (2^31 for -2^31), signs the bits r > 0, m1 the
// float slope as a double; returns the width.
template <int G, typename T>
__device__ __forceinline__ uint32_t legacy_residuals(const EncSmem<T> &sm, double &m0, double &m1, uint32_t len,
                                                     uint32_t tid, uint32_t nt) {
  m1 = (double)__double2float_rn(m1);
  bool fast = model_in_range(m0, m1, 0.0, len);
  auto resid = [&](uint32_t i) -> int32_t {
    const double p = pred_linear(m0, m1, i);
    return (int32_t)((int64_t)(uint64_t)sm.vals[i] - (fast ? __double2ll_rz(p) : f2i_x86(p)));
  };
  int32_t dmax = INT32_MIN, dmin = INT32_MAX;
  for (uint32_t i = tid; i < len; i += nt) {
    const int32_t d = resid(i);
    dmax = d > dmax ? d : dmax;
    dmin = d < dmin ? d : dmin;
  }
  u128 rmx = (u128)(uint64_t)(int64_t)dmax, rmn = (u128)(uint64_t)(int64_t)dmin;
  group_reduce2<3, 4, G>(rmx, rmn, sm.red);
  const int32_t mid = (int32_t)((uint32_t)(uint64_t)rmx + (uint32_t)(uint64_t)rmn);
  m0 = __dadd_rn(m0, __dmul_rn(__int2double_rn(mid), 0.5));  // x * 0.5 rounds exactly as x / 2.0
  fast = model_in_range(m0, m1, 0.0, len);
  uint32_t emax = 0;
  for (uint32_t i0 = 0; i0 < len; i0 += nt) {
    const uint32_t i = i0 + tid;
    bool pos = false;
    if (i < len) {
      const int32_t d = resid(i);
      pos = d > 0;
      const uint32_t mag = d < 0 ? 0u - (uint32_t)d : (uint32_t)d;
      sm.vals[i] = (T)mag;
      if (d != INT32_MIN && mag > emax) emax = mag;
    }
    const uint32_t ballot = __ballot_sync(0xffffffffu, pos);
    if ((tid & 31) == 0) sm.signs[i0 / 32 + tid / 32] = ballot;
  }
  emax = (uint32_t)(uint64_t)group_reduce<1, G>((u128)emax, sm.red);
  return emax ? bits_of(emax) + 1 : 0;
}

// ---- sequential reference fits (LECO_FIT_REFERENCE) ---------------------------
// One lane per block adds the block's values in the reference's own order and FP64
// operations, so the model is bit-identical to lr_int_T::caltheta (lr.h:66-85) or to
// the Y sums of polynomial_regression_iter (polynomial_regression_internals.hpp:129-137)
// (the kernels: seq_fit_tiled_kernel and seq_fit_ring_kernel in leco_encode.cu; the row
// encoder computes the same sums in parallel, leco_rows.cuh).
struct PolyX {
  double x[10];
};

// The model of a len-value block from the sums of the reference's fit loop (linear:
// sum y, sum i*y; poly: the three Y sums): lr_int_T::caltheta (lr.h:79-83) with the
// x sums in closed form -- sum i and sum i*i are exact integers below 2^53 at every
// step of the reference's loop (i < 16384), so these are the same doubles -- or the
// degree-2 solve with the column's X sums (polyX: full block [0..4], tail block [5..9]).
template <int CODEC>
__device__ __forceinline__ void store_seq_model(double *m, double s0, double s1, double s2, uint32_t len, uint32_t bs,
                                                const double *polyX) {
  if (CODEC != kPoly2) {
    const double md = __uint2double_rn(len);
    const uint64_t ml = len;
    const double sumx = __ull2double_rn(ml * (ml - 1) / 2), sumxx = __ull2double_rn((ml - 1) * ml * (2 * ml - 1) / 6);
    const double ccc = __dsub_rn(__dmul_rn(s1, md), __dmul_rn(sumx, s0));
    const double xxx = __dsub_rn(__dmul_rn(sumxx, md), __dmul_rn(sumx, sumx));
    const double t1 = __ddiv_rn(ccc, xxx);
    m[0] = __ddiv_rn(__dsub_rn(s0, __dmul_rn(t1, sumx)), md);
    m[1] = t1;
    m[2] = 0.0;
  } else {
    const double *X = polyX + (len == bs ? 0 : 5);
    double Y[3] = {s0, s1, s2}, c[3];
    poly2_solve(X, Y, c);
    m[0] = c[0];
    m[1] = c[1];
    m[2] = c[2];
  }
}

// Encodes block b of a legacy u32 column with one thread group: the whole CTA (G = 256) or
// one warp (G = 32).  The caller guarantees that every block of the column with a smaller
// index was handed to a group that has already started (ticket order), which makes the
// look-back wait finite.  smem_raw: enc_smem_bytes(a.bs, 4) bytes owned by this group.
template <int G>
__device__ __forceinline__ void encode_legacy_block(const EncodeArgs &a, uint64_t b, uint8_t *smem_raw) {
  EncSmem<uint32_t> sm = enc_smem<uint32_t>(smem_raw, a.bs);
  const uint32_t tid = group_rank<G>(), nt = group_size<G>();
  const uint64_t base = b * a.bs;
  const uint32_t len = (uint32_t)umin64((uint64_t)a.bs, a.n - base);
  const uint32_t *src = reinterpret_cast<const uint32_t *>(a.values) + base;

  // ---- stage the block ------------------------------------------------------
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const uint32_t nvec = len / 4;
    for (uint32_t i = tid; i < nvec; i += nt)
      reinterpret_cast<uint4 *>(sm.vals)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
    for (uint32_t i = nvec * 4 + tid; i < len; i += nt) sm.vals[i] = __ldg(src + i);
  } else {
    for (uint32_t i = tid; i < len; i += nt) sm.vals[i] = __ldg(src + i);
  }
  group_sync<G>();

  // ---- fit -----------------------------------------------------------------
  double m0, m1;
  if (a.seq_models) {
    m0 = a.seq_models[b * 3 + 0];
    m1 = a.seq_models[b * 3 + 1];
  } else {
    u128 sy = 0, siy = 0;
    for (uint32_t i = tid; i < len; i += nt) {
      const uint64_t y = (uint64_t)sm.vals[i];
      sy += y;
      siy += (u128)y * i;
    }
    group_reduce2<0, 0, G>(sy, siy, sm.red);
    // lr_int (lr.h:89-111), the same as lr_int_T::caltheta (lr.h:79-83), on exact moments
    double model[3];
    store_seq_model<kLinear>(model, u128_to_double(sy), u128_to_double(siy), 0.0, len, a.bs, nullptr);
    m0 = model[0];
    m1 = model[1];
  }
  const uint32_t l = legacy_residuals<G>(sm, m0, m1, len, tid, nt);
  // the legacy format stores widths of 31 and up as raw u32 values after its full header
  // (piecewise_fix_op_minimize_maxerror.h:104-108)
  const bool raw = l >= 31;
  if (raw) {  // residuals overwrote the values: restage them
    group_sync<G>();
    for (uint32_t i = tid; i < len; i += nt) sm.vals[i] = __ldg(src + i);
  }
  const uint64_t size = block_bytes<kLegacy, 4>(l, len);

  // ---- offset by look-back ----------------------------------------------------
  if (tid < 32) {
    const uint64_t excl = lookback_prefix(a.status, b, size, a.error);
    if (tid == 0) sm.bcast[1] = excl;
  }
  // ---- header bytes: [u8 l][f64 theta0][f32 theta1], raw blocks included ---------
  constexpr uint32_t H = Hdr<kLegacy, 4>::bytes;
  if (tid == 0) {
    sm.hdr[0] = (uint8_t)l;
    const uint64_t w0 = (uint64_t)__double_as_longlong(m0);
    const uint32_t w1 = __float_as_uint(__double2float_rn(m1));
    for (int j = 0; j < 8; ++j) sm.hdr[1 + j] = (uint8_t)(w0 >> (8 * j));
    for (int j = 0; j < 4; ++j) sm.hdr[9 + j] = (uint8_t)(w1 >> (8 * j));
  }
  group_sync<G>();
  const uint64_t goff = sm.bcast[1];
  if (goff == ~0ull) return;                       // look-back gave up (error word set)
  if (goff + size + LECO_PAYLOAD_SLACK > a.payload_cap) {  // never write past the buffer
    if (tid == 0) atomicOr(a.error, kErrCapacity);
    return;
  }

  // ---- body: |r| below the sign bit (write_delta_T, bit_write.h:186-245) ----------
  const uint32_t *vals = sm.vals, *signs = sm.signs;
  if (raw) {
    write_image(a.payload, goff, size, H, sm.hdr, 32, len, [&](uint32_t k) -> uint64_t { return (uint64_t)vals[k]; }, tid, nt);
  } else {
    const uint32_t sb = l ? l - 1 : 0;
    const uint32_t mm = (1u << sb) - 1u;
    write_image(a.payload, goff, size, H, sm.hdr, l, len, [&](uint32_t k) -> uint64_t {
      return (uint64_t)((vals[k] & mm) | (((signs[k >> 5] >> (k & 31)) & 1u) << sb));
    }, tid, nt);
  }

  // ---- offsets and directory -------------------------------------------------------
  if (tid == 0) {
    a.offsets[b] = goff;
    if (b == a.nb - 1) a.offsets[a.nb] = goff + size;
    if (a.dir) {
      leco_dir_entry e;
      const uint32_t dl = raw ? 32u : l;  // as the decoder's directory records it
      e.word0 = ((goff + H) * 8) | ((uint64_t)dl << 56) | ((uint64_t)kLegacy << 48);
      e.a0 = m0; e.a1 = m1; e.a2 = 0.0;
      a.dir[b] = e;
    }
  }
}

}  // namespace leco
