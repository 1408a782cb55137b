// leco_rows.cuh -- the row encoder: one thread per row of 32 consecutive values.
//
// A block of bs values is handled by R threads (R >= bs / 32, 8 .. 512: a power of two in the
// batch engine and for blocks that share a CTA, else as many warps as the rows need);
// thread t takes values 32t .. 32t+31, its row of shared memory, in every pass.  A row's
// fields pack into whole 32-bit words (32 fields of l bits are l words) without any sharing
// between threads, residuals replace the values they came from, and nothing but running
// maxima and sums stays in registers, so that six CTAs of four warps (u64) fit an SM.  A CTA of NT
// threads encodes NT / R consecutive blocks (an item) and takes one offset for all of them.
// Used by the single-column kernels (leco_rows_kernel.cuh) and the batch engine
// (leco_batch_encode.cu); blocks are the reference's images byte for byte.
//
// The reference's fit adds a block's values (and i * value, i * i * value) one after the
// other in FP64 (lr.h:72-77, polynomial_regression_internals.hpp:129-137).  rows_fit
// computes the same doubles in parallel:
//  * every term is >= 0, so the running sum grows; while it stays in one binade it is a
//    multiple of that binade's ulp u, and adding a term rounds the term to a multiple of u,
//    a tie going by the parity of the sum.  A row of 32 terms therefore adds a constant that
//    depends on the parity of the sum alone, and if the sum passes into the next binade
//    inside the row (ulp 2u), on its two lowest bits;
//  * each thread takes an approximate sum of the values before its row (a scan in any
//    order), clears its two lowest bits, and adds its row to that start and to the starts
//    1, 2 and 3 ulps above it with real FP64 additions, one after the other.  These give the
//    row's effect on every sum that differs from the start by a few thousand ulps;
//  * the rows' effects are small integers (ulps relative to the next row's start); rows that
//    stay in their binade are composed by a segmented scan, and one lane per sum walks over
//    the remaining rows (about two for each doubling of the sum).
// A row whose effect is not certain that way (a partial sum within 2^32 ulps of a binade's
// end, two binades passed in one row, a start that is too far off) is added term by term
// from the exact sum before it, unless that sum is one of the starts tried.  When the total
// of a sum is below 2^53 every partial sum is an exact integer and the scan's total is it.
//
// What bounds it: instructions (4096-value blocks, warp instructions per block: u32 FOR 4.0K,
// u64 Delta 6.3K, u64 LeCo with the fit's chains 13K; issue slots 48-56 % busy, the rest
// barriers within the block and the wait for the item's offset).  Against the encoder
// with one CTA per block that gathered each output chunk field by field, or staged twice:
// one 4096-value u64 block 82 -> 13 us (host-bound), 1M u32 LeCo in blocks of 1000 34.8 -> 15.4 us,
// 30M u32 FOR 130 -> 57 us, 20M u64 Delta in blocks of 2048 176 -> 66 us, 100M u64 LeCo (fits
// from the fit kernel, leco_encode.cu) 557 -> 460 us.
#pragma once
#include "leco_encode.cuh"

namespace leco {

constexpr double kExactSum = 9007199254740992.0;  // 2^53
constexpr int32_t kNoEffect = -32768;

// Threads per block where blocks share a CTA: a power of two >= the block's rows.
__host__ __device__ inline uint32_t rows_threads(uint32_t bs) {
  const uint32_t rows = (bs + 31) / 32;
  uint32_t r = 8;
  while (r < rows) r <<= 1;
  return r;
}
// The same for a column of its own: a block of more than 64 rows has its CTA for itself, of as
// many warps as its rows need where that lets more CTAs onto an SM than the next power of two
// (of 224 threads there are as few as of 256; of 416 and 448 two fit where the fit is not in the
// encoder, if the codec needs no more than 72 registers).  60M u64 values, power of two / this,
// us: FOR in blocks of 9000 (283 rows) 418 / 217, LeCo with the exact fit in blocks of 5000
// 472 / 376, of 9000 658 / 356.
__host__ __device__ inline uint32_t column_rows_threads(int codec, uint32_t bs) {
  const uint32_t rows = (bs + 31) / 32, r = (rows + 31) / 32 * 32, most = codec == kPoly2 ? 384u : 448u;
  return rows <= 64 ? rows_threads(bs) : r == 224 ? 256u : r > most ? 512u : r;
}
constexpr uint32_t kWholeCta = 0xffffffffu;  // RT of a block's group that is the CTA, of any number of warps
__host__ __device__ constexpr int rows_sums(int codec) { return codec == kLinear ? 2 : codec == kPoly2 ? 3 : 0; }

// Shared memory of one CTA of nt threads in groups of R; from tab on for the reference's fit
// in the encoder only (`total` with it, `tab` without).
struct RowsLayout {
  uint32_t wtot, red, hdr, model, size, goff, count, next, tab, base, mask, total;
};
__host__ __device__ constexpr RowsLayout rows_layout(uint32_t nt, uint32_t R, uint32_t s, uint32_t ns) {
  RowsLayout L{};
  const uint32_t ng = nt / R, nw = nt / 32;
  uint32_t o = nt * 32 * s;                 // rows of 32 values
  L.wtot = o;  o += 3 * nw * 8;             // double [3][warps]
  L.red = o;   o += 2 * 2 * nw * 8;         // u64 [2][2][warps]
  L.hdr = o;   o += ng * 32;                // u64 [groups][4]: header bytes
  L.model = L.hdr;                          // double [groups][4]: read before the header is made
  L.size = o;  o += ng * 8;                 // u64 [groups]
  L.goff = o;  o += ng * 8;                 // u64 [groups]
  L.count = o; o += 4;                      // u32: groups whose size is known
  L.next = o;  o += 4;                      // u32: the next item that had left its place
  L.tab = o;   o += ns * nt * 8;            // [ns][nt]: a row's effect (four int16) or its run's (two int32)
  L.base = o;  o += ns * (nt + ng) * 8;     // u64 [ns][groups * (R + 1)]: the rows' approximate starts
  L.mask = o;  o += ns * nw * 8;            // uint2 [ns][warps]: rows to walk, uncertain rows
  L.total = o;
  return L;
}

// A thread's place: `rank` in its group of R threads (= its row of the block).  RT: the group
// size when it is fixed at compile time, kWholeCta when it is the CTA's, else 0 (a power of two).
template <uint32_t RT>
struct RowGroup {
  uint32_t nt, Rd, gi, rank, row;  // row: the row's place in shared memory (threadIdx.x)
  uint32_t lane, gl;               // lane, lane among the group's lanes of this warp
  uint32_t warp, w0;               // this warp, the group's first warp
  static constexpr bool whole = RT == kWholeCta;
  __device__ __forceinline__ uint32_t R() const { return RT && !whole ? RT : Rd; }
  __device__ __forceinline__ uint32_t rl() const { return RT >= 32 ? 32u : RT ? RT : (Rd < 32 ? Rd : 32u); }
  __device__ __forceinline__ uint32_t nw() const { return whole ? Rd / 32 : RT >= 32 ? RT / 32 : RT ? 1u : (Rd < 32 ? 1u : Rd / 32); }
  __device__ __forceinline__ explicit RowGroup(uint32_t R) {
    Rd = R;
    nt = blockDim.x;
    row = threadIdx.x;
    rank = whole ? threadIdx.x : threadIdx.x & (this->R() - 1);
    gi = RT ? threadIdx.x / (RT ? RT : 1u) : threadIdx.x >> (31 - __clz((int)R));
    lane = threadIdx.x & 31;
    gl = lane & (rl() - 1);
    warp = threadIdx.x >> 5;
    w0 = whole ? 0u : nw() == 1 ? warp : gi * nw();
  }
  __device__ __forceinline__ void sync() const {
    // Barriers by constant numbers: the warps of a group may wait at different places of the
    // code, and a number in a register would reserve all 16 barriers of every CTA, of which an
    // SM has 64.
    if (nw() == 1) __syncwarp();
    else if (RT >= 128 || R() == nt) asm volatile("bar.sync 0;" ::: "memory");
    else if (gi == 0) asm volatile("bar.sync 1, %0;" ::"r"(R()) : "memory");
    else if (gi == 1) asm volatile("bar.sync 2, %0;" ::"r"(R()) : "memory");
    else if (gi == 2) asm volatile("bar.sync 3, %0;" ::"r"(R()) : "memory");
    else asm volatile("bar.sync 4, %0;" ::"r"(R()) : "memory");
  }
  // the same when the groups of one warp may have taken different ways here
  __device__ __forceinline__ void sync_apart() const {
    if (rl() < 32) __syncwarp(((1u << rl()) - 1u) << (lane - gl));
    else sync();
  }
};

// Max, min and (OR) or of 32-bit values over the group; `slots`: u64 [2][warps] that no
// thread still reads (successive reductions alternate between two sets).  (64-bit reductions
// go by shuffles: as two redux.sync on the halves, the second on a selected operand, they gave
// wrong maxima in one kernel, and the cause was not found.)
template <bool OR, uint32_t RT>
__device__ __forceinline__ void rg_reduce3(const RowGroup<RT> &g, int32_t &mx, int32_t &mn, uint32_t &ov, uint64_t *slots) {
  if (g.rl() == 32) {
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = __reduce_min_sync(0xffffffffu, mn);
    if (OR) ov = __reduce_or_sync(0xffffffffu, ov);
  } else {
    for (uint32_t m = 1; m < g.rl(); m <<= 1) {
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, m));
      mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, m));
      if (OR) ov |= __shfl_xor_sync(0xffffffffu, ov, m);
    }
  }
  if (g.nw() == 1) {
    __syncwarp();
    return;
  }
  const uint32_t nws = g.nt >> 5;
  if (g.lane == 0) {
    slots[g.warp] = ((uint64_t)(uint32_t)mn << 32) | (uint32_t)mx;
    if (OR) slots[nws + g.warp] = ov;
  }
  g.sync();
  for (uint32_t w = g.w0; w < g.w0 + g.nw(); ++w) {
    const uint64_t v = slots[w];
    mx = max(mx, (int32_t)(uint32_t)v);
    mn = min(mn, (int32_t)(uint32_t)(v >> 32));
    if (OR) ov |= (uint32_t)slots[nws + w];
  }
}
// The maxima of one or (TWO) two 64-bit values over the group (minima: of the complements).
template <bool TWO, uint32_t RT>
__device__ __forceinline__ void rg_max(const RowGroup<RT> &g, uint64_t &a, uint64_t &b, uint64_t *slots) {
  for (uint32_t m = 1; m < g.rl(); m <<= 1) {
    const uint64_t o = shfl_xor_u64(a, m);
    a = o > a ? o : a;
    if (TWO) {
      const uint64_t p = shfl_xor_u64(b, m);
      b = p > b ? p : b;
    }
  }
  if (g.nw() == 1) {
    __syncwarp();
    return;
  }
  const uint32_t nws = g.nt >> 5;
  if (g.lane == 0) {
    slots[g.warp] = a;
    if (TWO) slots[nws + g.warp] = b;
  }
  g.sync();
  for (uint32_t w = g.w0; w < g.w0 + g.nw(); ++w) {
    const uint64_t x = slots[w];
    a = x > a ? x : a;
    if (TWO) {
      const uint64_t y = slots[nws + w];
      b = y > b ? y : b;
    }
  }
}
// Sums of N 128-bit values over the group; `slots`: 2 * N u64 [warps] rows that may still be
// read.  The callers' next use of them must come after a group barrier.
template <int N, uint32_t RT>
__device__ __forceinline__ void rg_sums128(const RowGroup<RT> &g, u128 (&v)[N], uint64_t *slots) {
#pragma unroll
  for (int s = 0; s < N; ++s)
    for (uint32_t m = 1; m < g.rl(); m <<= 1) {
      const uint64_t lo = shfl_xor_u64((uint64_t)v[s], m), hi = shfl_xor_u64((uint64_t)(v[s] >> 64), m);
      v[s] += ((u128)hi << 64) | lo;
    }
  if (g.nw() == 1) return;
  const uint32_t nws = g.nt >> 5;
  g.sync();
  if (g.lane == 0) {
#pragma unroll
    for (int s = 0; s < N; ++s) {
      slots[2 * s * nws + g.warp] = (uint64_t)v[s];
      slots[(2 * s + 1) * nws + g.warp] = (uint64_t)(v[s] >> 64);
    }
  }
  g.sync();
#pragma unroll
  for (int s = 0; s < N; ++s) {
    v[s] = 0;
    for (uint32_t w = g.w0; w < g.w0 + g.nw(); ++w) v[s] += ((u128)slots[(2 * s + 1) * nws + w] << 64) | slots[2 * s * nws + w];
  }
}

// ---- rows in shared memory -------------------------------------------------------
// 16-byte slot j of row t sits at slot j ^ (t mod 16) (u64, 16 slots) or j ^ (t mod 8)
// (u32, 8 slots): the copies (consecutive slots of a row) and a warp reading the same slot
// of 32 rows both spread over the banks.  Shared memory starts on 256 bytes, so a row's slot
// j is at (row's slot 0) xor 16 j.
template <typename T>
__device__ __forceinline__ uint32_t row_at(uint32_t sb, uint32_t row) {
  return sb + row * (32u * sizeof(T)) + ((row & (sizeof(T) == 8 ? 15u : 7u)) << 4);
}
template <typename T>
__device__ __forceinline__ T staged_value(uint32_t rowa, uint32_t j) {
  constexpr uint32_t V = 16 / sizeof(T);
  const uint32_t at = (rowa ^ ((j / V) << 4)) + (j % V) * (uint32_t)sizeof(T);
  if constexpr (sizeof(T) == 8) {
    const uint2 v = lds_v2(at);
    return (T)(((uint64_t)v.y << 32) | v.x);
  } else {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return (T)v;
  }
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// Copies the group's len values into its rows.
template <typename T, uint32_t RT>
__device__ __forceinline__ void stage_rows(const RowGroup<RT> &g, uint32_t sb, const T *src, uint32_t len) {
  constexpr uint32_t V = 16 / sizeof(T), SL = 32 / V;  // values per slot, slots per row
  const uint32_t r0 = g.gi * g.R();
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const uint32_t nc = len / V;
    if (RT >= 64 && nc == g.R() * SL) {  // a block of R full rows
#pragma unroll
      for (uint32_t i = 0; i < SL; ++i) {
        const uint32_t q = g.rank + i * g.R();
        cp_async16(row_at<T>(sb, r0 + q / SL) ^ ((q % SL) << 4), src + (size_t)q * V);
      }
    } else {
      for (uint32_t q = g.rank; q < nc; q += g.R()) cp_async16(row_at<T>(sb, r0 + q / SL) ^ ((q % SL) << 4), src + (size_t)q * V);
      const uint32_t i = nc * V + g.rank;
      if (i < len) {
        const uint32_t at = (row_at<T>(sb, r0 + i / 32) ^ (((i % 32) / V) << 4)) + (i % V) * (uint32_t)sizeof(T);
        if constexpr (sizeof(T) == 8) cp_async8(at, src + i);
        else cp_async4(at, src + i);
      }
    }
  } else {
    for (uint32_t i = g.rank; i < len; i += g.R()) {
      const uint32_t at = (row_at<T>(sb, r0 + i / 32) ^ (((i % 32) / V) << 4)) + (i % V) * (uint32_t)sizeof(T);
      if constexpr (sizeof(T) == 8) cp_async8(at, src + i);
      else cp_async4(at, src + i);
    }
  }
  cp_async_wait_all();
}
// Slot i of the row; with FULL false, values from cnt on read as 0.
template <typename T, bool FULL>
__device__ __forceinline__ void load_slot(uint32_t rowa, uint32_t cnt, uint32_t i, T *y) {
  constexpr uint32_t V = 16 / sizeof(T);
  const uint4 v = lds_v4(rowa ^ (i << 4));
  if constexpr (sizeof(T) == 8) {
    y[0] = ((uint64_t)v.y << 32) | v.x;
    y[1] = ((uint64_t)v.w << 32) | v.z;
  } else {
    y[0] = v.x;
    y[1] = v.y;
    y[2] = v.z;
    y[3] = v.w;
  }
  if (!FULL) {
#pragma unroll
    for (uint32_t k = 0; k < V; ++k)
      if (V * i + k >= cnt) y[k] = 0;
  }
}
// Calls slot(i, y) for the row's slots i = 0, 1, ... in order, y[] the slot's values; with
// FULL false, values from cnt on read as 0.
template <typename T, bool FULL, int UNROLL, typename Fn>
__device__ __forceinline__ void for_slots(uint32_t rowa, uint32_t cnt, Fn slot) {
  constexpr uint32_t V = 16 / sizeof(T), SL = 32 / V;
#pragma unroll UNROLL
  for (uint32_t i = 0; i < SL; ++i) {
    T y[V];
    load_slot<T, FULL>(rowa, cnt, i, y);
    slot(i, y);
  }
}
// Writes four 32-bit words over slot i of the row.
__device__ __forceinline__ void put_slot(uint32_t rowa, uint32_t i, const int32_t *r) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(rowa ^ (i << 4)), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}

// (double)y on the FP64 pipe, rounded once.  SMALL: y < 2^52, one addition; else
// hi * 2^32 - 2^52 is exact, then + (2^52 + lo).
template <bool SMALL, typename T>
__device__ __forceinline__ double row_double(T y) {
  if constexpr (sizeof(T) == 4) {
    return u32_to_double_fp64(y);
  } else if constexpr (SMALL) {
    return __dsub_rn(__longlong_as_double((long long)(y + 0x4330000000000000ull)), 4503599627370496.0);
  } else {
    const double h = __dsub_rn(__hiloint2double(0x45300000, (int)(y >> 32)), 19342813118337666422669312.0);  // 2^84 + 2^52
    return __dadd_rn(h, __hiloint2double(0x43300000, (int)(uint32_t)y));
  }
}

// ---- the fit ------------------------------------------------------------------------
// Term s of value y (as a double) at position k (as a double).
__device__ __forceinline__ double fit_term(int s, double y, double k) {
  return s == 0 ? y : s == 1 ? __dmul_rn(k, y) : __dmul_rn(__dmul_rn(k, k), y);
}

// Runs a row's terms of sums S0 .. NS-1 through NV starts each (start + v ulps); c: the sums
// after the row; m: per sum, the smallest distance of a partial sum's high word above the
// word `edge` just below the binade's end, modulo 2^32 (below it reads as large).
template <typename T, int S0, int NS, int NV, bool SMALL, bool FULL>
__device__ __forceinline__ void row_chains(uint32_t rowa, uint32_t cnt, double k0, const uint64_t *base, double (&c)[NS][NV],
                                           uint32_t *m) {
  constexpr uint32_t V = 16 / sizeof(T);
  uint32_t edge[NS];
#pragma unroll
  for (int s = S0; s < NS; ++s) {
    edge[s] = (((uint32_t)(base[s] >> 52) + 1u) << 20) - 1u;
    m[s] = (uint32_t)(base[s] >> 32) - edge[s];
#pragma unroll
    for (int v = 0; v < NV; ++v) c[s][v] = __longlong_as_double((long long)(base[s] + v));
  }
  double ks = k0;
  for_slots<T, FULL, 8 / V>(rowa, cnt, [&](uint32_t, const T *y) {
#pragma unroll
    for (uint32_t j = 0; j < V; ++j) {
      const double yd = row_double<SMALL>(y[j]), k = j ? __dadd_rn(ks, (double)j) : ks;
#pragma unroll
      for (int s = S0; s < NS; ++s) {
        const double t = fit_term(s, yd, k);
#pragma unroll
        for (int v = 0; v < NV; ++v) c[s][v] = __dadd_rn(c[s][v], t);
        m[s] = __viaddmin_u32((uint32_t)__double2hiint(c[s][0]), 0u - edge[s], m[s]);
      }
    }
    ks = __dadd_rn(ks, (double)V);
  });
}

// Effects of the rows' terms of sums S0 .. NS-1 into the tables: walked rows hold r[0..3]
// (the sum after the row from start + v ulps, in ulps above the next row's start), the others
// the effect of their run (from the last walked row below them in the warp) on an even and an
// odd sum.
constexpr int32_t kMaxEffect = 1 << 14;  // effects are stored in 16 bits
template <typename T, int S0, int NS, int NV, bool SMALL, bool FULL, uint32_t RT>
__device__ __forceinline__ void fit_tables(const RowGroup<RT> &g, uint32_t rowa, uint32_t cnt, double k0, const uint64_t *base,
                                           const uint64_t *next, uint8_t *smem, const RowsLayout &L) {
  double c[NS][NV];
  uint32_t m[NS];
  row_chains<T, S0, NS, NV, SMALL, FULL>(rowa, cnt, k0, base, c, m);
#pragma unroll
  for (int s = S0; s < NS; ++s) {
    const uint32_t edge = (((uint32_t)(base[s] >> 52) + 1u) << 20) - 1u, h = (uint32_t)__double2hiint(c[s][0]);
    bool reg = m[s] >= 2 && (base[s] & 0xfffffffffffffull) >= (1ull << 28) && h <= edge + 0x100000u - 1u;
    int32_t r[4];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int64_t d = (int64_t)((uint64_t)__double_as_longlong(c[s][v]) - next[s]);
      const bool ok = d > -(int64_t)kMaxEffect && d < (int64_t)kMaxEffect;
      reg = reg && ok;
      r[v] = ok ? (int32_t)d : kNoEffect;
    }
    if (NV == 2) {
      r[2] = reg ? r[0] + 2 : kNoEffect;
      r[3] = reg ? r[1] + 2 : kNoEffect;
    }
    const bool walked = !reg || h > edge;
    const uint32_t spec = __ballot_sync(0xffffffffu, walked), irr = __ballot_sync(0xffffffffu, !reg);
    const uint32_t g0 = g.lane - g.gl;
    const uint32_t below = spec & (0xffffffffu >> (31 - g.lane)) & ~((1u << g0) - 1u);
    const uint32_t first = below ? 32u - (uint32_t)__clz((int)below) : g0;  // the run's first lane
    int32_t c0 = r[0], c1 = r[1] - 1;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const int32_t p0 = __shfl_up_sync(0xffffffffu, c0, d), p1 = __shfl_up_sync(0xffffffffu, c1, d);
      if (!walked && g.lane >= first + d) {
        const int32_t n0 = p0 + ((p0 & 1) ? c1 : c0), n1 = p1 + ((p1 & 1) ? c0 : c1);
        c0 = n0;
        c1 = n1;
      }
    }
    uint2 e;
    e.x = walked ? ((uint32_t)r[0] & 0xffffu) | ((uint32_t)r[1] << 16) : (uint32_t)c0;
    e.y = walked ? ((uint32_t)r[2] & 0xffffu) | ((uint32_t)r[3] << 16) : (uint32_t)c1;
    reinterpret_cast<uint2 *>(smem + L.tab)[s * g.nt + g.row] = e;
    if (g.lane == 0) reinterpret_cast<uint2 *>(smem + L.mask)[s * (g.nt >> 5) + g.warp] = make_uint2(spec, irr);
  }
}

// One lane per sum follows the running sum over the block's rows: delta = the sum's distance
// from the approximate start of the next row, in ulps.
template <typename T, uint32_t RT>
__device__ __forceinline__ double fit_walk(const RowGroup<RT> &g, uint32_t s, uint32_t len, uint32_t sb, const uint8_t *smem,
                                           const RowsLayout &L) {
  const uint32_t r0 = g.gi * g.R(), g0 = g.lane - g.gl, rl = g.rl();
  const uint64_t *bs = reinterpret_cast<const uint64_t *>(smem + L.base) + s * (g.nt + g.nt / g.R()) + g.gi * (g.R() + 1);
  const uint2 *tab = reinterpret_cast<const uint2 *>(smem + L.tab) + s * g.nt + r0;
  const uint2 *mask = reinterpret_cast<const uint2 *>(smem + L.mask) + s * (g.nt >> 5) + g.w0;
  constexpr int32_t kFar = 1 << 26;
  const uint32_t rows = (len + 31) / 32;
  int64_t wide = 0;    // delta
  int32_t delta = 0;   // the same while it is small
  auto add_row = [&](uint32_t row) {  // term by term from the exact sum
    double acc = __longlong_as_double((long long)(bs[row] + (uint64_t)wide)), k = u32_to_double_fp64(32 * row);
    const uint32_t cnt = min(32u, len - 32 * row), rowa = row_at<T>(sb, r0 + row);
#pragma unroll 8
    for (uint32_t j = 0; j < 32; ++j) {
      const double y = row_double<false>(j < cnt ? staged_value<T>(rowa, j) : (T)0);
      acc = __dadd_rn(acc, s == 0 ? y : s == 1 ? __dmul_rn(k, y) : __dmul_rn(__dmul_rn(k, k), y));
      k = __dadd_rn(k, 1.0);
    }
    wide = (int64_t)((uint64_t)__double_as_longlong(acc) - bs[row + 1]);
  };
  uint32_t at = 0;  // the row delta belongs to
  for (uint32_t w = 0; w < g.nw() && at < rows; ++w) {
    const uint2 mk = mask[w];
    const uint32_t end = min(rl, rows - 32 * w);  // rows of the block here
    uint32_t spec = mk.x >> g0, pos = 0;
    while (pos < end) {
      const uint32_t rest = spec >> pos;
      const uint32_t run = min(rest ? (uint32_t)__ffs((int)rest) - 1u : 32u, end - pos);
      delta = wide > kFar ? kFar : wide < -kFar ? -kFar : (int32_t)wide;
      const bool near = delta > -kFar && delta < kFar;
      if (run) {
        if (near) {
          const uint2 e = tab[32 * w + pos + run - 1];
          delta += (int32_t)((delta & 1) ? e.y : e.x);
          wide = delta;
        } else {
          for (uint32_t q = 0; q < run; ++q) add_row(32 * w + pos + q);
        }
        pos += run;
        if (pos >= end) break;
        if (!near) continue;
      }
      const uint32_t row = 32 * w + pos;
      const uint2 e = tab[row];
      const uint32_t v = (uint32_t)delta & 3u, h = v & 2u ? e.y : e.x;
      const int32_t r = (int32_t)(int16_t)(v & 1u ? h >> 16 : h);
      const bool certain = !((mk.y >> (g0 + pos)) & 1u);
      if (near && (certain || ((uint32_t)delta < 4u && r != kNoEffect))) {
        delta = certain ? ((delta - (int32_t)v) >> 1) + r : r;
        wide = delta;
      } else {
        add_row(row);
      }
      ++pos;
    }
    at = 32 * w + pos;
  }
  return __longlong_as_double((long long)(bs[at] + (uint64_t)wide));
}

// The block's sums in the reference's order (ref) or exactly (128-bit integers rounded
// once), and the model from them, left in the group's model slot for every thread.
template <typename T, int CODEC, bool FULL, uint32_t RT>
__device__ __forceinline__ void rows_fit(const RowGroup<RT> &g, uint32_t len, uint32_t cnt, bool ref, uint32_t sb, uint32_t rowa,
                                         uint8_t *smem, const RowsLayout &L, uint32_t bs, const double *polyX) {
  constexpr int NS = rows_sums(CODEC);
  constexpr uint32_t V = 16 / sizeof(T);
  double *model = reinterpret_cast<double *>(smem + L.model) + 4 * g.gi;
  double *wtot = reinterpret_cast<double *>(smem + L.wtot);
  const uint32_t nws = g.nt >> 5;
  const double k0 = u32_to_double_fp64(32 * g.rank);
  // ---- sums of the row's terms in any order: of y, j * y and j * j * y (j < 32) as integers
  // (exact while y < 2^50) ----
  uint64_t t0 = 0, t1 = 0, t2 = 0;
  uint32_t high = 0;
  for_slots<T, FULL, 16 / V>(rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
    for (uint32_t j = 0; j < V; ++j) {
      const uint32_t p = V * i + j, yl = (uint32_t)y[j], yh = sizeof(T) == 8 ? (uint32_t)((uint64_t)y[j] >> 32) : 0u;
      t0 += y[j];
      t1 += (uint64_t)yl * p;
      if (sizeof(T) == 8) t1 += (uint64_t)(yh * p) << 32;
      if (NS == 3) {
        t2 += (uint64_t)yl * (p * p);
        if (sizeof(T) == 8) t2 += (uint64_t)(yh * (p * p)) << 32;
      }
      high |= yh;
    }
  });
  double a[NS];
  if (high < (1u << 18)) {
    a[0] = __ull2double_rn(t0);
    a[1] = __dadd_rn(__dmul_rn(k0, a[0]), __ull2double_rn(t1));
    if (NS == 3)
      a[NS - 1] = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(k0, k0), a[0]), __dmul_rn(__dadd_rn(k0, k0), __ull2double_rn(t1))),
                            __ull2double_rn(t2));
  } else {
#pragma unroll
    for (int s = 0; s < NS; ++s) a[s] = 0.0;
    double k = k0;
    for_slots<T, FULL, 1>(rowa, cnt, [&](uint32_t, const T *y) {
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        const double yd = row_double<false>(y[j]);
#pragma unroll
        for (int s = 0; s < NS; ++s) a[s] = __dadd_rn(a[s], fit_term(s, yd, k));
        k = __dadd_rn(k, 1.0);
      }
    });
  }
  // ---- approximate sums before and after the row ----
  double start[NS], total[NS];
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double o = __shfl_up_sync(0xffffffffu, a[s], d);
      if (g.gl >= d) a[s] = __dadd_rn(a[s], o);
    }
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double o = __shfl_up_sync(0xffffffffu, a[s], 1);
    start[s] = g.gl ? o : 0.0;
  }
  if (g.nw() == 1) {
#pragma unroll
    for (int s = 0; s < NS; ++s) total[s] = __shfl_sync(0xffffffffu, a[s], g.lane | (g.rl() - 1));
  } else {
    if (g.lane == 31) {
#pragma unroll
      for (int s = 0; s < NS; ++s) wtot[s * nws + g.warp] = a[s];
    }
    g.sync();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      double before = 0.0;
      total[s] = 0.0;
      for (uint32_t w = g.w0; w < g.w0 + g.nw(); ++w) {
        if (w == g.warp) before = total[s];
        total[s] = __dadd_rn(total[s], wtot[s * nws + w]);
      }
      start[s] = __dadd_rn(before, start[s]);
      a[s] = __dadd_rn(before, a[s]);
    }
  }
  // sums below 2^53: every partial sum is an exact integer, in any order.  The sums grow with
  // their power of i, but for a block whose values past the first are 0.
  bool any = false;
#pragma unroll
  for (int s = 0; s < NS; ++s) any = any || !(total[s] < kExactSum);
  if (!any && g.rank == 0) store_seq_model<CODEC>(model, total[0], total[1], total[NS - 1], len, bs, polyX);
  if (ref && __any_sync(0xffffffffu, any)) {  // (a warp of several blocks takes them all along)
    uint64_t base[NS], next[NS];
    bool passes = false;
    const uint32_t ng1 = g.nt + g.nt / g.R();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      base[s] = (uint64_t)__double_as_longlong(start[s]) & ~3ull;
      next[s] = (uint64_t)__double_as_longlong(a[s]) & ~3ull;
      uint64_t *b = reinterpret_cast<uint64_t *>(smem + L.base) + s * ng1 + g.gi * (g.R() + 1);
      b[g.rank] = base[s];
      if (g.rank == g.R() - 1) b[g.R()] = next[s];
      passes = passes || (base[s] >> 52) != (next[s] >> 52);
    }
    const bool all = __any_sync(0xffffffffu, !(total[0] < kExactSum));  // the sum of y too (else from i * y on)
    if (__any_sync(0xffffffffu, cnt)) {  // (rows past the block's end: the walk ends before them)
      passes = __any_sync(0xffffffffu, passes);
      const bool small = sizeof(T) == 4 || __all_sync(0xffffffffu, high < (1u << 20));
      auto tables = [&](auto s0, auto nv, auto sm) {
        fit_tables<T, decltype(s0)::value, NS, decltype(nv)::value, decltype(sm)::value, FULL>(g, rowa, cnt, k0, base, next, smem, L);
      };
      using C0 = std::integral_constant<int, 0>;
      using C1 = std::integral_constant<int, 1>;
      using C2 = std::integral_constant<int, 2>;
      using C4 = std::integral_constant<int, 4>;
      if (small) {
        if (all) passes ? tables(C0{}, C4{}, std::true_type{}) : tables(C0{}, C2{}, std::true_type{});
        else passes ? tables(C1{}, C4{}, std::true_type{}) : tables(C1{}, C2{}, std::true_type{});
      } else if constexpr (sizeof(T) == 8) {
        passes ? tables(C0{}, C4{}, std::false_type{}) : tables(C0{}, C2{}, std::false_type{});
      }
    }
    g.sync();
    if (g.rank < 32) {
      double sum = 0.0;
      if (g.gl < (uint32_t)NS) {
        const double tot = g.gl == 0 ? total[0] : g.gl == 1 ? total[1] : total[NS - 1];
        sum = tot < kExactSum ? tot : fit_walk<T>(g, g.gl, len, sb, smem, L);
      }
      __syncwarp();
      const uint32_t l0 = g.lane - g.gl;
      const double s1 = __shfl_sync(0xffffffffu, sum, l0 + 1), s2 = __shfl_sync(0xffffffffu, sum, l0 + 2);
      if (g.rank == 0 && any) store_seq_model<CODEC>(model, sum, s1, s2, len, bs, polyX);
    }
  }
  if (!ref && __any_sync(0xffffffffu, any)) {
    // exact moments: a row's sums in 64-bit halves, then 128 bits
    uint64_t slo = 0, shi = 0, tlo = 0, thi = 0, qlo = 0, qhi = 0;
    for_slots<T, FULL, 2>(rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        const uint32_t p = V * i + j, yl = (uint32_t)y[j], yh = sizeof(T) == 8 ? (uint32_t)((uint64_t)y[j] >> 32) : 0u;
        slo += yl;
        shi += yh;
        tlo += (uint64_t)yl * p;
        thi += (uint64_t)yh * p;
        if (NS == 3) {
          qlo += (uint64_t)yl * (p * p);
          qhi += (uint64_t)yh * (p * p);
        }
      }
    });
    const u128 sy = ((u128)shi << 32) + slo, sj = ((u128)thi << 32) + tlo, sq = ((u128)qhi << 32) + qlo;
    const uint64_t i0 = 32ull * g.rank;
    u128 m[NS];
    m[0] = sy;
    m[1] = sy * i0 + sj;
    if constexpr (NS == 3) m[2] = sy * (i0 * i0) + sj * (2 * i0) + sq;
    rg_sums128<NS>(g, m, reinterpret_cast<uint64_t *>(smem + L.wtot));  // (wtot and red together)
    if (g.rank == 0 && any)
      store_seq_model<CODEC>(model, u128_to_double(m[0]), u128_to_double(m[1]), u128_to_double(m[NS - 1]), len, bs, polyX);
  }
  g.sync();
}

// ---- packing ------------------------------------------------------------------------
// The packed body of a block is an array of 32-bit words in the group's part of shared
// memory, word k at k ^ ((k / 32) mod 32): rows of any width then store their words (word
// t * l + q by the thread of row t) over most of the banks.
__device__ __forceinline__ uint32_t body_at(uint32_t k4) { return k4 ^ ((k4 >> 5) & 124u); }  // byte offset of word k4 / 4

// Packs the 32 words of this thread's row (slots 0..7: 32-bit signed residuals, SIGNED, or
// fields) into body words rank * L ... of the group's part (at gb), once every thread of the
// group has read its row.
template <int L, bool SIGNED, uint32_t RT>
__device__ __forceinline__ void pack_row_width(const RowGroup<RT> &g, uint32_t gb, uint32_t rowa) {
  uint32_t w[L];
#pragma unroll
  for (int k = 0; k < L; ++k) w[k] = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint4 v = lds_v4(rowa ^ ((uint32_t)j << 4));
    place_field<L>(w, SIGNED ? lin_field<L>(v.x) : v.x, 4 * j);
    place_field<L>(w, SIGNED ? lin_field<L>(v.y) : v.y, 4 * j + 1);
    place_field<L>(w, SIGNED ? lin_field<L>(v.z) : v.z, 4 * j + 2);
    place_field<L>(w, SIGNED ? lin_field<L>(v.w) : v.w, 4 * j + 3);
  }
  g.sync_apart();
  const uint32_t k4 = g.rank * (4u * L);
#pragma unroll
  for (int k = 0; k < L; ++k) sts_u32(gb + body_at(k4 + 4u * k), w[k]);
}
template <bool SIGNED, uint32_t RT>
static __device__ __noinline__ void pack_row_dispatch(uint32_t l, uint32_t Rd, uint32_t gb, uint32_t rowa) {
  const RowGroup<RT> g(Rd);
  switch (l) {
#define LECO_ROW_CASE(L) \
  case L: pack_row_width<L, SIGNED>(g, gb, rowa); break;
    LECO_ROW_CASE(1) LECO_ROW_CASE(2) LECO_ROW_CASE(3) LECO_ROW_CASE(4) LECO_ROW_CASE(5) LECO_ROW_CASE(6)
    LECO_ROW_CASE(7) LECO_ROW_CASE(8) LECO_ROW_CASE(9) LECO_ROW_CASE(10) LECO_ROW_CASE(11) LECO_ROW_CASE(12)
    LECO_ROW_CASE(13) LECO_ROW_CASE(14) LECO_ROW_CASE(15) LECO_ROW_CASE(16) LECO_ROW_CASE(17) LECO_ROW_CASE(18)
    LECO_ROW_CASE(19) LECO_ROW_CASE(20) LECO_ROW_CASE(21) LECO_ROW_CASE(22) LECO_ROW_CASE(23) LECO_ROW_CASE(24)
    LECO_ROW_CASE(25) LECO_ROW_CASE(26) LECO_ROW_CASE(27) LECO_ROW_CASE(28) LECO_ROW_CASE(29) LECO_ROW_CASE(30)
    LECO_ROW_CASE(31) LECO_ROW_CASE(32)
#undef LECO_ROW_CASE
    default: break;
  }
}
// Packs fields of 33..64 bits one after the other into the words of this row's own slots
// (word q in slot q / 4), each written after the values there have been read: after 2s + 2
// fields at most 4s + 4 words are complete.
struct WidePacker {
  uint32_t rowa, l, w0 = 0, have = 0, q = 0;  // `have` < 32 bits pending in w0
  __device__ __forceinline__ void put_word(uint32_t w) {
    sts_u32((rowa ^ ((q >> 2) << 4)) + (q & 3u) * 4u, w);
    ++q;
  }
  __device__ __forceinline__ void put(uint64_t f) {
    const uint32_t lo = (uint32_t)f, hi = (uint32_t)(f >> 32);
    w0 |= lo << have;
    const uint32_t w1 = __funnelshift_l(lo, hi, have), w2 = have ? hi >> (32 - have) : 0u;
    put_word(w0);
    have += l - 32;
    w0 = w1;
    if (have >= 32) {
      put_word(w1);
      have -= 32;
      w0 = w2;
    }
  }
};

// Writes the image [goff, goff + size) of a block whose header (H bytes, H mod 4 == 1, zeros
// after them) is hw and whose body has nw words, word k read by `word` for k < nw, zeros
// after them (the image's tail).  The 16-byte chunks wholly inside the body's words are
// funnel-shifted from five of them, all by the same shift.
template <typename Word>
__device__ __forceinline__ void write_rows_image(uint8_t *payload, uint64_t goff, uint64_t size, uint32_t H,
                                                 const uint32_t *hw, uint32_t nw, uint32_t rank, uint32_t nthreads, Word word) {
  const uint32_t h4 = H >> 2;
  const uint32_t lead = (uint32_t)goff & 15u;                      // image offset of chunk c: 16 c - lead
  const uint32_t chunks = (uint32_t)((lead + size + 15) >> 4);
  const uint32_t sh = ((0u - lead - H) & 3u) * 8u;                  // body bytes of a chunk start at byte sh / 8 of a word
  uint8_t *out = payload + (goff - lead);
  auto word0 = [&](uint32_t k) -> uint32_t { return k < nw ? word(k) : 0u; };
  // image word m: image bytes 4m .. 4m+3 (m < 0: before the image, never stored)
  auto img = [&](int32_t m) -> uint32_t {
    if (m < 0) return 0u;
    if ((uint32_t)m < h4) return hw[m];
    if ((uint32_t)m == h4) return hw[m] | (word0(0) << 8);
    return __funnelshift_r(word0((uint32_t)m - h4 - 1u), word0((uint32_t)m - h4), 24);
  };
  for (uint32_t c = rank; c < chunks; c += nthreads) {
    const int32_t e = (int32_t)(16 * c) - (int32_t)lead;  // image offset of the chunk (>= -15)
    const int32_t q = e - (int32_t)H;                     // body offset
    const uint32_t k = (uint32_t)q >> 2;
    if (q >= 0 && k + 4 < nw && e + 16 <= (int32_t)size) {  // (a last row may hold words past the image)
      const uint32_t w0 = word(k), w1 = word(k + 1), w2 = word(k + 2), w3 = word(k + 3), w4 = word(k + 4);
      *reinterpret_cast<uint4 *>(out + 16 * (size_t)c) = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                                                                    __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
    } else {
      const int32_t m0 = e >> 2;  // floor(e / 4)
      const uint32_t es = (uint32_t)(e & 3) * 8u;
      const uint32_t i0 = img(m0), i1 = img(m0 + 1), i2 = img(m0 + 2), i3 = img(m0 + 3), i4 = img(m0 + 4);
      const uint32_t lo = e < 0 ? (uint32_t)-e : 0u;
      const int64_t left = (int64_t)size - e;
      const uint32_t hi = left < 16 ? (uint32_t)left : 16u;
      const uint32_t x0 = __funnelshift_r(i0, i1, es), x1 = __funnelshift_r(i1, i2, es), x2 = __funnelshift_r(i2, i3, es),
                     x3 = __funnelshift_r(i3, i4, es);
      if (lo == 0 && hi == 16) *reinterpret_cast<uint4 *>(out + 16 * (size_t)c) = make_uint4(x0, x1, x2, x3);
      else store_chunk_bytes(out + 16 * (size_t)c, x0, x1, x2, x3, lo, hi);
    }
  }
}

// ---- the passes over a row ---------------------------------------------------------
// Everything a pass needs to know about its row.
template <typename T, uint32_t RT>
struct RowPass {
  const RowGroup<RT> &g;
  uint32_t rowa, cnt, len;
  uint64_t *slots[2];  // reduction scratch, two sets in turn
  double k0;           // position of the row's first value
};

// LeCo, values and predictions in [0, 2^51): y - trunc(p) = ceil(y - p), which the FP64 pipe
// gives as the low word of (2^52 * 1.5 + y) - p rounded up (the sum on the left is y added to
// the constant's bits; the difference has ulp 1).
__device__ __forceinline__ double ceil_diff(uint64_t y, double p) {
  return __dsub_ru(__longlong_as_double((long long)(y + 0x4338000000000000ull)), p);
}
// Extremes of y - pred over the block in 32 bits; bad: nonzero when one does not fit, or a
// value is 2^51 or more.
template <typename T, bool FULL, uint32_t RT>
__device__ __forceinline__ void lin_extremes(const RowPass<T, RT> &P, double m0, double m1, int32_t &mx, int32_t &mn, uint32_t &bad) {
  constexpr uint32_t V = 16 / sizeof(T);
  mx = INT32_MIN;
  mn = INT32_MAX;
  bad = 0;
  uint32_t high = 0;
  double ks = P.k0;
  constexpr uint32_t SL = 32 / V, CH = 8 / V;  // slots of a row, slots of eight values
#pragma unroll 1
  for (uint32_t c = 0; c < SL; c += CH) {
#pragma unroll
    for (uint32_t q = 0; q < CH; ++q) {
      T y[V];
      load_slot<T, FULL>(P.rowa, P.cnt, c + q, y);
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        const double k = j ? __dadd_rn(ks, (double)j) : ks;
        const double e = ceil_diff((uint64_t)y[j], __dadd_rn(m0, __dmul_rn(m1, k)));
        const int32_t d = __double2loint(e);
        const uint32_t fit = ((uint32_t)__double2hiint(e) + ((uint32_t)d >> 31)) ^ 0x43380000u;
        if (sizeof(T) == 8) high |= (uint32_t)((uint64_t)y[j] >> 32);
        if (FULL || V * (c + q) + j < P.cnt) {
          bad |= fit;
          mx = max(mx, d);
          mn = min(mn, d);
        }
      }
      ks = __dadd_rn(ks, (double)V);
    }
    // a warp in which every row has failed leaves the block to the 64-bit pass
    if (c == 0 && __all_sync(0xffffffffu, bad != 0 || high >> 19)) break;
  }
  bad |= high >> 19;
  rg_reduce3<true>(P.g, mx, mn, bad, P.slots[0]);
}
// Residuals (all below 2^31 in magnitude) over the values' place; returns the largest magnitude.
template <typename T, bool FULL, uint32_t RT>
__device__ __forceinline__ uint32_t lin_residuals(const RowPass<T, RT> &P, double m0, double m1) {
  constexpr uint32_t V = 16 / sizeof(T);
  int32_t mx = 0, mn = 0, r[4];
  double ks = P.k0;
  for_slots<T, FULL, 8 / V>(P.rowa, P.cnt, [&](uint32_t i, const T *y) {
#pragma unroll
    for (uint32_t j = 0; j < V; ++j) {
      const double k = j ? __dadd_rn(ks, (double)j) : ks;
      int32_t d = __double2loint(ceil_diff((uint64_t)y[j], __dadd_rn(m0, __dmul_rn(m1, k))));
      if (!FULL && V * i + j >= P.cnt) d = 0;
      mx = max(mx, d);
      mn = min(mn, d);
      r[(V * i + j) & 3u] = d;
    }
    if (V == 4 || (i & 1u)) put_slot(P.rowa, V == 4 ? i : i >> 1, r);
    ks = __dadd_rn(ks, (double)V);
  });
  uint32_t none = 0;
  rg_reduce3<false>(P.g, mx, mn, none, P.slots[1]);
  return max((uint32_t)mx, (uint32_t)(-mn));
}

// The general residual passes: diff(y, j) gives a value's magnitude and sign (above: true)
// at row position j.  wide_residuals puts signed 32-bit residuals over the values' place and
// returns 0 when all fit, else kWide and, unless every warp saw that from its rows' first values
// and left them alone, kGone: the values have been written over.  wide_extreme gives the
// largest magnitude, wide_fields by the width the 32-bit fields or the packed fields of a
// wide row.
constexpr uint32_t kWide = 1, kGone = 2;
template <typename T, bool FULL, uint32_t RT, typename Diff>
__device__ __forceinline__ uint32_t wide_residuals(const RowPass<T, RT> &P, uint64_t *slots, uint32_t &rm, Diff diff) {
  constexpr uint32_t V = 16 / sizeof(T);
  int32_t mx = 0, mn = 0, r[4];
  uint32_t bad = 0;
  bool up0;
  const uint64_t d0 = diff(staged_value<T>(P.rowa, 0), 0, up0);
  if (__all_sync(0xffffffffu, d0 >> 31 && (FULL || P.cnt))) {
    bad = kWide;
  } else {
    for_slots<T, FULL, 8 / V>(P.rowa, P.cnt, [&](uint32_t i, const T *y) {
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        bool up;
        uint64_t d = diff(y[j], V * i + j, up);
        if (!FULL && V * i + j >= P.cnt) d = 0;
        bad |= (uint32_t)(d >> 32) | ((uint32_t)d & 0x80000000u);
        if (sizeof(T) == 4) bad |= (uint32_t)(up && d == 0);  // a magnitude that is 0 mod 2^32 keeps its sign bit
        const int32_t v = up ? (int32_t)(uint32_t)d : -(int32_t)(uint32_t)d;
        mx = max(mx, v);
        mn = min(mn, v);
        r[(V * i + j) & 3u] = v;
      }
      if (V == 4 || (i & 1u)) put_slot(P.rowa, V == 4 ? i : i >> 1, r);
    });
    bad = kGone | (bad ? kWide : 0u);
  }
  rg_reduce3<true>(P.g, mx, mn, bad, slots);
  rm = max((uint32_t)mx, (uint32_t)(-mn));
  return bad & kWide ? bad : 0u;
}
template <typename T, bool FULL, uint32_t RT, typename Diff>
__device__ __forceinline__ uint64_t wide_extreme(const RowPass<T, RT> &P, Diff diff) {
  constexpr uint32_t V = 16 / sizeof(T);
  uint64_t rmax = 0;
  for_slots<T, FULL, 2>(P.rowa, P.cnt, [&](uint32_t i, const T *y) {
#pragma unroll
    for (uint32_t j = 0; j < V; ++j) {
      bool up;
      const uint64_t d = diff(y[j], V * i + j, up);
      if (FULL || V * i + j < P.cnt) rmax = d > rmax ? d : rmax;
    }
  });
  return rmax;
}
template <typename T, bool FULL, uint32_t RT, typename Diff>
__device__ __forceinline__ void wide_fields(const RowPass<T, RT> &P, uint32_t l, Diff diff) {
  constexpr uint32_t V = 16 / sizeof(T);
  if (l <= 32) {
    int32_t r[4];
    for_slots<T, FULL, 2>(P.rowa, P.cnt, [&](uint32_t i, const T *y) {
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        bool up;
        const uint32_t d = (uint32_t)diff(y[j], V * i + j, up);
        r[(V * i + j) & 3u] = !FULL && V * i + j >= P.cnt ? 0 : (int32_t)(d | (up && l ? 1u << (l - 1) : 0u));
      }
      if (V == 4 || (i & 1u)) put_slot(P.rowa, V == 4 ? i : i >> 1, r);
    });
  } else if constexpr (sizeof(T) == 8) {
    WidePacker pk{P.rowa, l};
    for_slots<T, FULL, 1>(P.rowa, P.cnt, [&](uint32_t i, const T *y) {
      uint64_t f[V];
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        bool up;
        f[j] = diff(y[j], V * i + j, up);
        if (up) f[j] |= 1ull << (l - 1);
        if (!FULL && V * i + j >= P.cnt) f[j] = 0;
      }
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) pk.put(f[j]);
    });
  }
}

// What a block's passes leave: the width, the model or frame, and whether the row's slots
// hold 32-bit words to pack (widths up to 32) or packed fields already.
template <int CODEC, int S>
__device__ __forceinline__ uint64_t image_size(uint32_t l, uint32_t len) { return len ? block_bytes<CODEC, S>(l, len) : 0; }
struct RowCoded {
  uint32_t l;
  double m0, m1, m2;
  uint64_t fbase, fmax;
  bool fields;  // the slots hold fields, else signed residuals (a raw block's values are fields)
};

template <typename T, int CODEC, bool FULL, uint32_t RT>
__device__ __forceinline__ void encode_rows_passes(const EncodeArgs &a, const RowPass<T, RT> &P, bool ref, uint32_t sb, uint8_t *smem,
                                                   const RowsLayout &L, uint64_t b, RowCoded &C, uint64_t *status) {
  uint64_t *sizes = reinterpret_cast<uint64_t *>(smem + L.size);
  uint32_t *count = reinterpret_cast<uint32_t *>(smem + L.count);
  constexpr uint32_t S = sizeof(T), TB = 8 * S, V = 16 / S;
  const RowGroup<RT> &g = P.g;
  const uint32_t len = P.len, cnt = P.cnt, p0 = 32 * g.rank;
  // The values once more, after residuals have taken their place (every thread of the group).
  auto restage = [&]() {
    stage_rows<T>(g, sb, reinterpret_cast<const T *>(a.values) + b * a.bs, len);
    g.sync_apart();
  };
  auto finish_width = [&](uint32_t l) {  // the width a block of this codec is written with
    if (l > TB) l = TB;
    // A width of 8*sizeof(T)-1 is written raw: the reference's bulk decoders treat
    // l >= 8*sizeof(T)-1 as raw (piecewise_fix_integer_template.h:171,
    // FOR_integer_template.h:89, poly_fix_integer_template.h:121), so a packed block of
    // that width would not decode there.  Delta has no such rule.
    if (CODEC != kDelta && l == TB - 1) l = TB;
    // The item's total goes out when its last block has its width, before the fields are made.
    if (g.rank == 0) {
      const uint32_t NB = g.nt / g.R();
      sizes[g.gi] = image_size<CODEC, S>(l, len);
      if (status) {
        __threadfence_block();
        if (NB == 1 || atomicAdd(count, 1u) == NB - 1) {
          __threadfence_block();
          uint64_t total = 0;
          for (uint32_t k = 0; k < NB; ++k) total += reinterpret_cast<volatile uint64_t *>(sizes)[k];
          st_relaxed(status, kFlagAgg | total);
        }
      }
    }
    return l;
  };
  if constexpr (CODEC == kLinear || CODEC == kPoly2) {
    const double *model = reinterpret_cast<const double *>(smem + L.model) + 4 * g.gi;
    if (a.seq_models) model = a.seq_models + (len ? b : 0) * 3;
    else rows_fit<T, CODEC, FULL>(g, len, cnt, ref, sb, P.rowa, smem, L, a.bs, a.polyX);
    C.m0 = model[0];
    C.m1 = model[1];
    C.m2 = model[2];
    bool coded = false, wide = false;
    uint64_t *wide_slots = P.slots[1];
    if constexpr (CODEC == kLinear) {
      // ---- midpoint shift (piecewise_fix_integer_template.h:36-46) ----
      bool done = false, small = false;
      const bool nonneg = preds_nonneg(C.m0, C.m1, len);
      if (__any_sync(0xffffffffu, nonneg)) {  // (a warp may hold several blocks)
        int32_t mx, mn;
        uint32_t bad;
        lin_extremes<T, FULL>(P, C.m0, C.m1, mx, mn, bad);
        if (nonneg && !bad) {
          C.m0 = __dadd_rn(C.m0, __dmul_rn(__ll2double_rn((int64_t)mx + (int64_t)mn), 0.5));  // x * 0.5 rounds exactly as x / 2.0
          small = (int64_t)mx - (int64_t)mn < (1ll << 30);
          done = true;
        }
      }
      if (!__all_sync(0xffffffffu, done)) {
        int64_t dmax = (int64_t)0x8000000000000000ull, dmin = 0x7fffffffffffffffll;
        if (!done)
          with_pred_rule(C.m0, C.m1, len, [&](auto rule) {
            for_slots<T, FULL, 2>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
              for (uint32_t j = 0; j < V; ++j) {
                const int64_t d = (int64_t)((uint64_t)y[j] - (uint64_t)lin_pred<decltype(rule)::value>(C.m0, C.m1, p0 + V * i + j));
                if (FULL || V * i + j < cnt) {
                  dmax = d > dmax ? d : dmax;
                  dmin = d < dmin ? d : dmin;
                }
              }
            });
          });
        __syncwarp();
        uint64_t ux = (uint64_t)dmax ^ (1ull << 63), un = ~((uint64_t)dmin ^ (1ull << 63));
        rg_max<true>(g, ux, un, P.slots[1]);
        wide_slots = P.slots[0];
        if (!done) {
          dmax = (int64_t)(ux ^ (1ull << 63));
          dmin = (int64_t)(~un ^ (1ull << 63));
          small = dmax >= dmin && (uint64_t)(dmax - dmin) < (1ull << 30);
          // half of a span this large has no 32-bit residual (u64), or makes the block raw (u32)
          wide = dmax >= dmin && (uint64_t)dmax - (uint64_t)dmin >= (S == 8 ? (1ull << 32) : (1ull << 31)) + 16;
          const int64_t mid = (int64_t)((uint64_t)dmax + (uint64_t)dmin);
          C.m0 = __dadd_rn(C.m0, __dmul_rn(__ll2double_rn(mid), 0.5));
        }
      }
      // ---- residuals (:51-72) and width (:108-117) ----
      // Differences before the shift that span less than 2^30 leave residuals below 2^31:
      // their low 32 bits are the whole of them.  (After the 64-bit pass the reductions' two
      // sets have been used in the other order, so that way takes the general passes.)
      const bool narrow = small && done && preds_nonneg(C.m0, C.m1, len);
      if (__all_sync(0xffffffffu, narrow)) {
        const uint32_t rm = lin_residuals<T, FULL>(P, C.m0, C.m1);
        C.l = finish_width(rm ? bits_of(rm) + 1 : 0);
        coded = true;
        if (S == 4 && C.l == TB) restage();
      }
    }
    if (!coded) {
      auto general = [&](auto pred) {
        auto diff = [&](T y, uint32_t j, bool &up) -> uint64_t {
          const int64_t p = pred(p0 + j);
          const uint64_t v = (uint64_t)y;
          up = S == 8 && CODEC == kLinear ? v > (uint64_t)p : (int64_t)v > p;
          const uint64_t d = up ? v - (uint64_t)p : (uint64_t)p - v;
          return S == 4 ? d & 0xffffffffull : d;
        };
        uint32_t rm = 0, state = kWide;
        // (a warp of blocks known to be wide does not try; their values are still there)
        const bool known = __all_sync(0xffffffffu, wide);
        if (!known) state = wide_residuals<T, FULL>(P, wide_slots, rm, diff);
        const bool fits = !state;
        if (fits) {
          C.l = finish_width(rm ? bits_of(rm) + 1 : 0);
          if (S == 4 && C.l == TB) restage();
        }
        if (!__all_sync(0xffffffffu, fits)) {  // the same again, from the values
          uint64_t rmax = 0, none = 0;
          if (!fits) {
            if (state & kGone) restage();
            rmax = wide_extreme<T, FULL>(P, diff);
          }
          __syncwarp();
          rg_max<false>(g, rmax, none, known ? wide_slots : wide_slots == P.slots[1] ? P.slots[0] : P.slots[1]);
          if (!fits) {
            C.l = finish_width(rmax ? bits_of(rmax) + 1 : 0);
            if (C.l < TB) wide_fields<T, FULL>(P, C.l, diff);
            C.fields = true;
          }
        }
      };
      if constexpr (CODEC == kLinear) {
        const bool fast = model_in_range(C.m0, C.m1, 0.0, len);
        general([&](uint32_t k) -> int64_t {
          const double p = pred_linear_fp64(C.m0, C.m1, k);
          return fast ? __double2ll_rz(p) : f2i_x86(p);
        });
      } else {
        const bool fast = model_in_range(C.m0, C.m1, C.m2, len);
        general([&](uint32_t k) -> int64_t {
          const double p = pred_poly2(C.m0, C.m1, C.m2, u32_to_double_fp64(k));
          return fast ? __double2ll_rz(p) : f2i_x86(p);
        });
      }
    }
  } else if constexpr (CODEC == kFor) {
    // ---- frame of reference (FOR_integer_template.h:26-52) ----
    if constexpr (S == 8) {
      uint64_t mx = 0, un = 0;  // un: the complement of the minimum
      for_slots<T, FULL, 4>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
        for (uint32_t j = 0; j < V; ++j) {
          if (FULL || V * i + j < cnt) {
            mx = y[j] > mx ? (uint64_t)y[j] : mx;
            un = ~(uint64_t)y[j] > un ? ~(uint64_t)y[j] : un;
          }
        }
      });
      rg_max<true>(g, mx, un, P.slots[0]);
      C.fbase = ~un;
      C.fmax = mx;
    } else {
      uint32_t mx = 0, mn = 0xffffffffu;
      for_slots<T, FULL, 4>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
        for (uint32_t j = 0; j < V; ++j) {
          if (FULL || V * i + j < cnt) {
            mx = max(mx, (uint32_t)y[j]);
            mn = min(mn, (uint32_t)y[j]);
          }
        }
      });
      int32_t ix = (int32_t)(mx ^ 0x80000000u), in = (int32_t)(mn ^ 0x80000000u);
      uint32_t none = 0;
      rg_reduce3<false>(g, ix, in, none, P.slots[0]);
      C.fbase = (uint32_t)in ^ 0x80000000u;
      C.fmax = (uint32_t)ix ^ 0x80000000u;
    }
    if (!len) C.fbase = C.fmax = 0;
    C.fields = true;
    C.l = finish_width(bits_of(C.fmax - C.fbase));
    if (C.l < TB) {
      if (C.l <= 32) {
        int32_t r[4];
        for_slots<T, FULL, 4>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
          for (uint32_t j = 0; j < V; ++j)
            r[(V * i + j) & 3u] = !FULL && V * i + j >= cnt ? 0 : (int32_t)((uint32_t)y[j] - (uint32_t)C.fbase);
          if (V == 4 || (i & 1u)) put_slot(P.rowa, V == 4 ? i : i >> 1, r);
        });
      } else {
        wide_fields<T, FULL>(P, C.l, [&](T y, uint32_t, bool &up) -> uint64_t {
          up = false;
          return (uint64_t)y - C.fbase;
        });
      }
    }
  } else {  // kDelta (delta_integer_template.h:34-66): field k is value k+1 minus value k; the last field is 0
    const uint32_t nd = len > p0 + 1 ? min(32u, len - 1 - p0) : 0u;  // this row's differences
    const T after = nd == 32 ? staged_value<T>(row_at<T>(sb, g.row + 1), 0) : (T)0;  // the next row's first value
    if (len) C.fbase = (uint64_t)staged_value<T>(row_at<T>(sb, g.gi * g.R()), 0);
    // Values below 2^(TB-1) whose differences fit in 32 bits: the unsigned comparison of the
    // reference is the difference's sign.
    int32_t mx = 0, mn = 0;
    uint32_t bad = 0;
    T x0 = 0;
    auto visit = [&](uint32_t k, T x1) {  // difference k of the row: x1 - x0
      const T d = x1 - x0;
      const int32_t dl = (int32_t)(uint32_t)d;
      if (FULL ? (k < 31 || nd == 32) : k < nd) {
        if (S == 8) bad |= (uint32_t)((uint64_t)d >> 32) ^ (uint32_t)(dl >> 31);
        mx = max(mx, dl);
        mn = min(mn, dl);
      }
    };
    for_slots<T, FULL, 8 / V>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
      for (uint32_t j = 0; j < V; ++j) {
        if (i + j) visit(V * i + j - 1, y[j]);
        bad |= (uint32_t)((uint64_t)y[j] >> (TB - 1));
        x0 = y[j];
      }
    });
    visit(31, after);
    bad |= (uint32_t)(mn == INT32_MIN);
    rg_reduce3<true>(g, mx, mn, bad, P.slots[0]);
    const bool narrow = !bad;
    if (narrow) {
      const uint32_t rm = max((uint32_t)mx, (uint32_t)(-mn));
      C.l = finish_width(rm ? bits_of(rm) + 1 : 0);
    }
    if (!__all_sync(0xffffffffu, narrow)) {
      uint64_t rmax = 0, none = 0;
      if (!narrow) {
        auto widen = [&](uint32_t k, T x1) {
          const T d = x1 > x0 ? x1 - x0 : x0 - x1;
          if (k < nd) rmax = (uint64_t)d > rmax ? (uint64_t)d : rmax;
        };
        for_slots<T, FULL, 2>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
          for (uint32_t j = 0; j < V; ++j) {
            if (i + j) widen(V * i + j - 1, y[j]);
            x0 = y[j];
          }
        });
        widen(31, after);
      }
      __syncwarp();
      rg_max<false>(g, rmax, none, P.slots[1]);
      if (!narrow) C.l = finish_width(rmax ? bits_of(rmax) + 1 : 0);
    }
    // Fields: difference k needs value k + 1, the next slot's first for a slot's last, so each
    // slot's differences are completed when the next one has been read.
    if (C.l < TB && C.l <= 32) {
      int32_t r[4];
      auto field = [&](T x1, uint32_t k) -> int32_t {  // signed: mod 2^32 that is the difference itself
        const uint32_t d = (uint32_t)x1 - (uint32_t)x0;
        return k < nd ? (int32_t)d : 0;
      };
      for_slots<T, FULL, 8 / V>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
        for (uint32_t j = 0; j < V; ++j) {
          if (i + j) {
            const uint32_t k = V * i + j - 1;
            r[k & 3u] = field(y[j], k);
            if ((k & 3u) == 3) put_slot(P.rowa, k >> 2, r);
          }
          x0 = y[j];
        }
      });
      r[3] = field(after, 31);
      put_slot(P.rowa, 7, r);
    } else if constexpr (S == 8) {
      if (C.l < TB) {
        WidePacker pk{P.rowa, C.l};
        auto field = [&](T x1, uint32_t k) {
          const bool up = x1 > x0;
          uint64_t d = up ? x1 - x0 : x0 - x1;
          if (up) d |= 1ull << (C.l - 1);
          pk.put(k < nd ? d : 0);
        };
        for_slots<T, FULL, 1>(P.rowa, cnt, [&](uint32_t i, const T *y) {
#pragma unroll
          for (uint32_t j = 0; j < V; ++j) {
            if (i + j) field(y[j], V * i + j - 1);
            x0 = y[j];
          }
        });
        field(after, 31);
      }
    }
  }
}

// ---- offsets of a column's items ------------------------------------------------------
// A single column's items take their byte offsets from a publisher CTA: it walks the status
// words in item order, up to kPubWindow of them a step, and turns every published total into an
// inclusive prefix once all the items before it have published theirs.  An item publishes
// its total, packs, and then polls its own word alone.
// Roles go by blockIdx, the publisher first.  CTAs do start in that order as far as anyone has
// seen, but CUDA does not promise it, and if an item that has not started were kept from starting
// by items that wait for it, none would end.  So an item that has polled `item_wait` times leaves
// its place: it puts itself on a list and ends without its image, so that other CTAs can start,
// and the publisher encodes the items of the list again when every prefix is out.  (Tickets, taken
// as the CTAs start, would order them too, but 1500 CTAs asking one word at once wait 6 us for it:
// 10M u32 Delta values in blocks of 4096 21 us by index, 26 by ticket; 30M u32 FOR 55.1 / 58.3;
// 100M u64 LeCo 454 / 469; CTAs that stay and ask for their next ticket ahead: 71 and 574.)
// Leaving and publishing meet in the item's word.  The item counts itself (left[0]), fences,
// and exchanges its total for the same with kLeft, which fails if the prefix is there; the
// publisher writes the prefixes, fences, and reads left[0].  Whichever word came first, either the
// exchange fails or the publisher sees the count; it then waits until all that are counted
// have gone on or are on the list (left[1]).  All waits are bounded: on the publisher's expiry the
// error word is set and items may be left unwritten.
// The items in flight (~900 to 1500) wait for the step, and a step is a read of L2 and two
// barriers, so its width matters both ways: 24.6M u32 FOR / Delta values, us: windows of 128
// words 47 / 48, 256 42 / 44, 512 41 / 44, 1024 50 / 51; one warp stepping over 256 words 47 / 50.
constexpr uint64_t kLeft = 1ull << 61, kSizeMask = kLeft - 1;
constexpr uint32_t kItemWait = 1u << 16;  // some 40 ms; an item waits for tens of microseconds
__device__ __forceinline__ uint32_t ld_relaxed32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
constexpr uint32_t kPubWindow = 512;
// Returns the head of the list of left items (item + 1; 0: none), the same in every thread.
template <uint32_t NT, bool FIXED>  // NT threads, or at most NT
__device__ __forceinline__ uint32_t publish_items(uint64_t *status, uint64_t items, uint32_t *left, uint32_t *error, uint8_t *smem,
                                                  uint32_t spin_limit = kSpinLimit) {
  constexpr uint32_t NW = NT / 32, kPubWords = kPubWindow / NT;
  uint64_t *wsum = reinterpret_cast<uint64_t *>(smem);                // [2][NW]
  uint32_t *wfirst = reinterpret_cast<uint32_t *>(smem + 2 * NW * 8);  // [2][NW]
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = FIXED ? NW : blockDim.x >> 5, window = kPubWords * 32 * nw;
  uint64_t run = 0, j = 0;  // inclusive prefix before item j
  uint32_t spins = 0, par = 0;
  while (j < items) {
    uint64_t v[kPubWords];
    uint32_t first = window;  // this thread's first unpublished place
#pragma unroll
    for (uint32_t k = 0; k < kPubWords; ++k) {
      const uint64_t idx = j + kPubWords * t + k;
      v[k] = idx < items ? ld_relaxed(&status[idx]) : 0;
    }
    uint64_t own = 0;
#pragma unroll
    for (int k = (int)kPubWords - 1; k >= 0; --k)
      if ((v[k] >> 62) == 0) first = kPubWords * t + k;
#pragma unroll
    for (uint32_t k = 0; k < kPubWords; ++k)
      if (kPubWords * t + k < first) own += v[k] & kSizeMask;
    first = __reduce_min_sync(0xffffffffu, first);
    uint64_t incl = own;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint64_t o = __shfl_up_sync(0xffffffffu, (unsigned long long)incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) wsum[par * NW + warp] = incl;
    if (lane == 0) wfirst[par * NW + warp] = first;
    __syncthreads();  // (the two halves of the scratch alternate, so one barrier a step is enough)
    uint32_t n = window;
    uint64_t before = run + incl - own;
#pragma unroll
    for (uint32_t w = 0; w < NW; ++w)
      if (w < nw) {
        n = min(n, wfirst[par * NW + w]);
        if (w < warp) before += wsum[par * NW + w];
      }
    // the published run is items j .. j + n - 1: words past n (in any thread) are left
    uint64_t last = 0;
    bool has_last = false;
#pragma unroll
    for (uint32_t k = 0; k < kPubWords; ++k) {
      const uint32_t place = kPubWords * t + k;
      if (place < n) {
        before += v[k] & kSizeMask;
        st_relaxed(&status[j + place], kFlagIncl | before);
        if (place == n - 1) {
          last = before;
          has_last = true;
        }
      }
    }
    uint64_t *carry = reinterpret_cast<uint64_t *>(smem + 2 * NW * 12);
    if (has_last) carry[par] = last;
    if (n == 0) {
      if (++spins > spin_limit) {
        if (t == 0) atomicOr(error, kErrTimeout);
        return 0;
      }
      __nanosleep(32);
    } else {
      spins = 0;
    }
    __syncthreads();
    if (n) run = carry[par];
    j += n;
    par ^= 1;
  }
  __threadfence();
  __syncthreads();
  uint32_t *head = reinterpret_cast<uint32_t *>(smem);
  if (t == 0) {
    __threadfence();
    uint32_t h = 0;
    if (ld_relaxed32(left)) {
      // (what is done is read before what is counted: equal, they are all done)
      for (spins = 0;;) {
        const uint32_t done = ld_relaxed32(left + 1);
        __threadfence();
        if (done == ld_relaxed32(left)) {
          h = ld_relaxed32(left + 2);
          break;
        }
        if (++spins > spin_limit) {
          atomicOr(error, kErrTimeout);
          break;
        }
        __nanosleep(64);
      }
    }
    *head = h;
  }
  __syncthreads();
  const uint32_t h = *head;
  __syncthreads();
  return h;
}
// One lane: the item's exclusive prefix, once the publisher has replaced its total by the
// inclusive prefix; ~0 when the item has left its place (link: the word of the list's next).
__device__ __forceinline__ uint64_t await_prefix(uint64_t *status, uint64_t item, uint64_t total, uint32_t *left, uint64_t *link,
                                                 uint32_t wait) {
  for (uint32_t polls = 0;; ++polls) {
    const uint64_t v = ld_relaxed(&status[item]);
    if ((v >> 62) == 2) return (v & kSizeMask) - total;
    if (polls >= wait) break;
    __nanosleep(64);
  }
  atomicAdd(left, 1u);
  __threadfence();
  const unsigned long long mine = kFlagAgg | total;
  const uint64_t was = atomicCAS(reinterpret_cast<unsigned long long *>(&status[item]), mine, mine | kLeft);
  if (was == mine) {
    *link = atomicExch(left + 2, (uint32_t)item + 1u);
    __threadfence();
  }
  atomicAdd(left + 1, 1u);
  return was == mine ? ~0ull : (was & kSizeMask) - total;
}

// ---- one item: the NT / R blocks from item * (NT / R) on ------------------------------
// Every thread of the CTA calls it.  ref: the reference's sequential fit (else the exact
// moments).  a.status has one word per item; PUB: a publisher CTA turns them into prefixes,
// else the item looks back itself (alone: the column's only item; again: an item that had left
// its place).  smem: rows_layout's bytes, 256-byte aligned.
template <typename T, int CODEC, uint32_t RT, bool PUB>
__device__ __forceinline__ void encode_rows_item(const EncodeArgs &a, uint64_t item, uint32_t Rd, bool ref, bool alone, bool again,
                                                 uint8_t *smem) {
  constexpr uint32_t S = sizeof(T), TB = 8 * S;
  const RowGroup<RT> g(Rd);
  const uint32_t R = g.R(), NB = g.nt / R;
  const RowsLayout L = rows_layout(g.nt, R, S, rows_sums(CODEC));
  const uint32_t sb = smem_u32(smem);
  const uint64_t b = item * NB + g.gi;
  RowPass<T, RT> P{g, row_at<T>(sb, g.row), 0, 0, {}, u32_to_double_fp64(32 * g.rank)};
  P.len = b < a.nb ? (uint32_t)umin64(a.bs, a.n - b * a.bs) : 0u;
  P.cnt = P.len > 32 * g.rank ? min(32u, P.len - 32 * g.rank) : 0u;  // values of this row
  P.slots[0] = reinterpret_cast<uint64_t *>(smem + L.red);
  P.slots[1] = P.slots[0] + 2 * (g.nt >> 5);
  const uint32_t len = P.len;
  uint64_t *hdr = reinterpret_cast<uint64_t *>(smem + L.hdr) + 4 * g.gi;
  uint64_t *sizes = reinterpret_cast<uint64_t *>(smem + L.size), *goffs = reinterpret_cast<uint64_t *>(smem + L.goff);

  if (g.row == 0) *reinterpret_cast<uint32_t *>(smem + L.count) = 0;
  stage_rows<T>(g, sb, reinterpret_cast<const T *>(a.values) + b * a.bs, len);
  __syncthreads();
  RowCoded C{};
  // (the two ways meet at the same barriers: the warps of a block may differ.  With a model they
  // do not: the last rows' warp then held up all others, and both forms of the passes in use at
  // once cost more than the masks of the one -- 60M u64, exact fit, blocks of 3000: LeCo 439 us,
  // 390 so; poly2 671, 518.  FOR and Delta are faster with both.)
  uint64_t *status = alone || again ? nullptr : a.status + item;
  constexpr bool kModel = CODEC == kLinear || CODEC == kPoly2;
  if (__all_sync(0xffffffffu, kModel ? len == 32 * R : P.cnt == 32)) encode_rows_passes<T, CODEC, true>(a, P, ref, sb, smem, L, b, C, status);
  else encode_rows_passes<T, CODEC, false>(a, P, ref, sb, smem, L, b, C, status);
  const uint32_t l = C.l;
  const bool raw = l == TB;
  const uint32_t H = raw ? 1u : Hdr<CODEC, S>::bytes;
  const uint64_t size = image_size<CODEC, S>(l, len);
  if (g.rank == 0) {
    uint64_t v0 = 0, v1 = 0, v2 = 0;
    if (!raw) {
      if (CODEC == kLinear || CODEC == kPoly2) {
        v0 = (uint64_t)__double_as_longlong(C.m0);
        v1 = (uint64_t)__double_as_longlong(C.m1);
        if (CODEC == kPoly2) v2 = (uint64_t)__double_as_longlong(C.m2);
      } else if (CODEC == kFor) {
        v0 = S == 8 ? C.fbase : (C.fbase | (C.fmax << 32));
        v1 = S == 8 ? C.fmax : 0;
      } else {
        v0 = C.fbase;
      }
    }
    hdr[0] = (uint64_t)l | (v0 << 8);
    hdr[1] = (v0 >> 56) | (v1 << 8);
    hdr[2] = (v1 >> 56) | (v2 << 8);
    hdr[3] = v2 >> 56;
  }
  __syncthreads();  // every size is known
  uint64_t incl = 0, total = 0, mine = 0;
  if (g.warp == 0) {
    incl = mine = g.lane < NB ? sizes[g.lane] : 0;
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t o = __shfl_up_sync(0xffffffffu, (unsigned long long)incl, d);
      if (g.lane >= d) incl += o;
    }
    total = __shfl_sync(0xffffffffu, (unsigned long long)incl, 31);
  }
  // ---- pack this row ----
  const uint32_t gb = sb + g.gi * R * (32 * S);
  if (len && l && l <= 32) {
    if (C.fields || raw) pack_row_dispatch<false, RT>(l, Rd, gb, P.rowa);
    else pack_row_dispatch<true, RT>(l, Rd, gb, P.rowa);
  }
  // ---- the item's offset ----
  if (g.warp == 0) {
    __syncwarp();
    uint64_t excl;
    if (PUB) {
      excl = g.lane == 0 && !alone ? await_prefix(a.status, item, total, a.ticket + 1, a.offsets + item * NB, a.item_wait) : 0;
      excl = __shfl_sync(0xffffffffu, (unsigned long long)excl, 0);
    } else {
      excl = lookback_excl(a.status, item, a.error);
      if (excl != ~0ull && g.lane == 0) st_relaxed(&a.status[item], kFlagIncl | (excl + total));
    }
    if (g.lane < NB) goffs[g.lane] = excl == ~0ull ? ~0ull : excl + (incl - mine);
  }
  __syncthreads();
  const uint64_t goff = goffs[g.gi];
  if (!len || goff == ~0ull) return;  // (the item has left its place, or the look-back gave up: error word set)
  if (goff + size + LECO_PAYLOAD_SLACK > a.payload_cap) {  // never write past the buffer
    if (g.rank == 0) atomicOr(a.error, kErrCapacity);
    return;
  }
  const uint32_t *hw = reinterpret_cast<const uint32_t *>(hdr);
  const uint32_t nw = (len + 31) / 32 * l;
  if (S == 4 || l <= 32) {
    write_rows_image(a.payload, goff, size, H, hw, nw, g.rank, R, [&](uint32_t k) -> uint32_t {
      uint32_t v;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(gb + body_at(4 * k)));
      return v;
    });
  } else {  // words in their own rows: k / l through a multiply-high, exact for k < 2^16
    const uint32_t M = 0xffffffffu / l + 1u, r0 = g.gi * R;
    write_rows_image(a.payload, goff, size, H, hw, nw, g.rank, R, [&](uint32_t k) -> uint32_t {
      const uint32_t t = __umulhi(k, M), q = k - t * l;
      uint32_t v;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"((row_at<T>(sb, r0 + t) ^ ((q >> 2) << 4)) + (q & 3u) * 4u));
      return v;
    });
  }
  if (g.rank == 0) {
    a.offsets[b] = goff;
    if (b == a.nb - 1) a.offsets[a.nb] = goff + size;
    if (a.dir) {
      leco_dir_entry e;
      e.word0 = ((goff + H) * 8) | ((uint64_t)l << 56) | ((uint64_t)CODEC << 48);
      if (CODEC == kLinear || CODEC == kPoly2) {
        e.a0 = C.m0; e.a1 = C.m1; e.a2 = C.m2;
      } else {
        e.a0 = __longlong_as_double((long long)C.fbase);
        e.a1 = 0; e.a2 = 0;
      }
      a.dir[b] = e;
    }
  }
}

}  // namespace leco
