// leco_partition_gpu.cu -- the variable-length segmentation of
// Leco_cost_merge_double_wo_round<uint64_t>::encodeArray8_int on the GPU.
//
// Same segmentation as the host partitioner (leco_partition.cpp) and the
// reference (headers/piecewise_cost_merge_integer_template_double_wo_round.h:283-570,
// cost model newsegment_size :68-131, cal_bits :274-281, fit lr.h:66-85): coarse
// blocks cut as the reference driver does (experiments/leco_double_int_template_wo_round.cpp:85-91),
// inside each
//   1. one-point segments carrying the first difference to their successor and the
//      bit class of the second difference; for each bit class from the smallest up,
//      a segment of that class is merged with its right neighbour when the merged
//      width costs less than `delta` more bits, then grows left and right greedily;
//   2. pairwise merges while the fitted byte size of a pair is below the sum of the
//      two, pass after pass, until a pass saves less than 0.01 % of the coarse
//      block's raw size.
// Every merge changes what the next step sees, but most steps merge nothing: of a
// 2000-value coarse block's ~24,000 list steps ~2,000 are attempts and ~120 merges (the
// variable-length benchmark's column), and a pass of phase 2 decides on pair sizes that
// depend only on the segmentation before the pass.  Coarse blocks of up to kPartCtaMax
// values therefore take one CTA each (partition_cta_kernel): a warp tries 32 segments at
// a time and stops at the first that merges, and the CTA's warps compute a pass's pair
// sizes one per lane, or one by a whole warp when the pair is long.  Larger ones take one thread per
// coarse block (partition_kernel), persistent threads taking blocks by ticket, each with
// a private scratch slot in global memory (the segment list of phase 1, then the segment
// starts and sizes of phase 2, merged in place).  Every FP64 step is the reference's, one
// rounding each (--fmad=false), so the segment starts are the host partitioner's bit for
// bit.
//
// Output: each coarse block's segment starts go to stage[B0 ...] (at most one per
// value) with their count; a scan of the counts and a gather compact them into the
// caller's starts array.
#include <algorithm>
#include <string>

#include "leco_device.cuh"
#include "leco_internal.h"
#include "leco_seqsum.cuh"

namespace leco {

constexpr int kPartThreads = 128;
constexpr int kPartHead = 0;
constexpr int kPartTail = -2;

// A segment of phase 1.  Its successor and bit class live apart, packed in one
// 32-bit word per segment ((next + 2) << 8 | class; class 255 = the reference's
// 10000 sentinel), because the per-class walks read only those: 4 bytes per step
// instead of the whole record.
struct PSeg {
  int32_t start, end, prev, pad;
  int64_t max_delta, min_delta, next_delta;
};
constexpr uint32_t kNoClass = 255;
__device__ __forceinline__ int lk_next(uint32_t w) { return (int)(w >> 8) - 2; }
__device__ __forceinline__ uint32_t lk_class(uint32_t w) { return w & 0xffu; }
__device__ __forceinline__ uint32_t lk_make(int next, uint32_t cls) { return ((uint32_t)(next + 2) << 8) | cls; }

__device__ __forceinline__ uint32_t bits64_d(uint64_t v) { return v ? 64u - (uint32_t)__clzll((long long)v) : 0u; }

// cal_bits(min, max) (…_double_wo_round.h:274-281): bits of ceil(|max - min| / 2) plus one.
__device__ __forceinline__ int cal_bits_d(int64_t mn, int64_t mx) {
  const int64_t diff = (int64_t)((uint64_t)mx - (uint64_t)mn);
  const int64_t ad = diff < 0 ? (int64_t)(0 - (uint64_t)diff) : diff;
  const int64_t range = f2i_x86(ceil(__ddiv_rn(__ll2double_rn(ad), 2.0)));
  return range ? (int)bits64_d((uint64_t)range) + 1 : 0;
}

// newsegment_size (…_double_wo_round.h:68-131) of segment [a, b]: the reference's
// sequential FP64 fit (lr.h:66-85), slope rounded to float, 128-bit prediction.
__device__ uint32_t segment_cost_d(const uint64_t *__restrict__ array, uint32_t a, uint32_t b) {
  if (a == b) return 9;
  if (b == a + 1) return 13;
  const int length = (int)(b - a + 1);
  double sumx = 0, sumy = 0, sumxy = 0, sumxx = 0;
  for (int i = 0; i < length; i++) {
    const double di = (double)i;
    const double y = __ull2double_rn(__ldg(array + a + i));
    sumx = __dadd_rn(sumx, di);
    sumy = __dadd_rn(sumy, y);
    sumxx = __dadd_rn(sumxx, __dmul_rn(di, di));
    sumxy = __dadd_rn(sumxy, __dmul_rn(di, y));
  }
  const double dm = (double)length;
  const double ccc = __dsub_rn(__dmul_rn(sumxy, dm), __dmul_rn(sumx, sumy));
  const double xxx = __dsub_rn(__dmul_rn(sumxx, dm), __dmul_rn(sumx, sumx));
  const double t1 = __ddiv_rn(ccc, xxx);
  const double t0 = __ddiv_rn(__dsub_rn(sumy, __dmul_rn(t1, sumx)), dm);
  const double slope = (double)__double2float_rn(t1);
  uint64_t maxr = 0;
  for (uint32_t j = 0; j < (uint32_t)length; j++) {
    const i128 pred = f2i128(__dadd_rn(t0, __dmul_rn(slope, __uint2double_rn(j))));
    const i128 y = (i128)__ldg(array + a + j);
    const uint64_t r = (uint64_t)(y > pred ? y - pred : pred - y);
    maxr = r > maxr ? r : maxr;
  }
  const uint32_t bits = maxr ? bits64_d(maxr) + 1 : 0;
  if (bits >= 64) return (uint32_t)(5 + 8ull * (uint64_t)length);
  uint64_t overhead = sizeof(float) + sizeof(double) + 5;
  if (bits) overhead += (uint64_t)ceil(__ddiv_rn(__uint2double_rn(bits * (uint32_t)length), 8.0));
  return (uint32_t)overhead;
}

struct PartitionArgs {
  const uint64_t *array;
  uint64_t n;
  uint32_t bs;       // coarse block size
  uint64_t nblocks;  // coarse blocks
  int overhead;      // merge penalty `delta` (bits)
  PSeg *segs;        // per slot: bs + 1 entries
  uint32_t *links;   // per slot: bs + 1 packed (next, class) words
  uint32_t *pidx;    // per slot: bs entries (segment starts, phase 2)
  uint32_t *psz;     // per slot: bs entries (segment sizes, phase 2)
  uint32_t *stage;   // n entries: block b's starts at [b*bs, ...)
  uint32_t *count;   // nblocks entries
  uint32_t *ticket;
};

// Segmentation of coarse block [B0, B0 + len) by one thread.
__device__ void partition_block_d(const PartitionArgs &a, uint32_t B0, uint32_t len, PSeg *s, uint32_t *lk, uint32_t *idx,
                                  uint32_t *sz, uint32_t *out, uint32_t *count) {
  const uint64_t *array = a.array;
  if (len < 2) {  // the reference needs two points per coarse block (it reads array[B0 + 1])
    out[0] = B0;
    *count = 1;
    return;
  }
  // ---- split: linked list of one-point segments (…:286-312) ----
  int ns = 0;
  s[ns] = PSeg{0, 0, -1, 0, 0, 0, 0};  // head
  lk[ns++] = lk_make(-1, kNoClass);
  int min_sb = 10000, max_sb = -1;
  int64_t delta_prev = (int64_t)(__ldg(array + B0 + 1) - __ldg(array + B0));
  int cur = kPartHead;
  for (uint32_t i = B0 + 1; i < B0 + len - 1; i++) {
    const int64_t delta = (int64_t)(__ldg(array + i + 1) - __ldg(array + i));
    const int sdb = cal_bits_d(delta_prev, delta);
    min_sb = min(min_sb, sdb);
    max_sb = max(max_sb, sdb);
    s[ns] = PSeg{(int32_t)i - 1, (int32_t)i - 1, cur, 0, 0, 0, delta_prev};
    lk[ns] = lk_make(-1, (uint32_t)sdb);
    lk[cur] = lk_make(ns, lk_class(lk[cur]));
    cur = ns++;
    delta_prev = delta;
  }
  s[ns] = PSeg{(int32_t)(B0 + len - 2), (int32_t)(B0 + len - 2), cur, 0, 0, 0, delta_prev};
  lk[ns] = lk_make(kPartTail, kNoClass);
  lk[cur] = lk_make(ns, lk_class(lk[cur]));
  ns++;
  const int overhead = a.overhead;

  // ---- merge by bit class (…:326-433) ----
  for (int aim = min_sb; aim <= max_sb; aim++) {
    int c = lk_next(lk[kPartHead]);
    while (c != kPartTail) {
      const uint32_t wc = lk[c];
      int n = lk_next(wc);
      if (n == kPartTail) break;
      if ((int)lk_class(wc) != aim) {
        c = n;
        continue;
      }
      PSeg sc = s[c];
      const PSeg sn = s[n];
      const uint32_t wn = lk[n];
      const int former = sc.start, start = sn.start, now = sn.end;
      const int lbo = cal_bits_d(sc.min_delta, sc.max_delta), rbo = cal_bits_d(sn.min_delta, sn.max_delta);
      const int64_t nmax = max(max(sc.max_delta, sn.max_delta), sc.next_delta);
      const int64_t nmin = min(min(sc.min_delta, sn.min_delta), sc.next_delta);
      const int nb = cal_bits_d(nmin, nmax);
      const int origin_cost = (start - former) * lbo + (now - start + 1) * rbo;
      const int merged_cost = nb * (now - former + 1);
      if (!(merged_cost - origin_cost < overhead)) {
        c = n;
        continue;
      }
      int cnext = lk_next(wn);
      uint32_t ccls = lk_class(wn);
      sc.end = now;
      if (cnext != kPartTail) s[cnext].prev = c;
      sc.next_delta = sn.next_delta;
      sc.max_delta = nmax;
      sc.min_delta = nmin;
      // grow left (never into the first segment of the block)
      int p = sc.prev;
      while (p != kPartHead && s[p].prev != kPartHead) {
        const PSeg sp = s[p];
        const int left = sp.start;
        const int64_t lmax = max(max(sp.max_delta, sc.max_delta), sp.next_delta);
        const int64_t lmin = min(min(sp.min_delta, sc.min_delta), sp.next_delta);
        const int bnew = cal_bits_d(lmin, lmax);
        const int ol = cal_bits_d(sp.min_delta, sp.max_delta), orr = cal_bits_d(sc.min_delta, sc.max_delta);
        const int oc = (sc.start - left) * ol + (sc.end - sc.start + 1) * orr;
        const int mc = bnew * (sc.end - left + 1);
        if (!(mc - oc < overhead)) break;
        sc.start = left;
        sc.prev = sp.prev;
        lk[sp.prev] = lk_make(c, lk_class(lk[sp.prev]));
        sc.min_delta = lmin;
        sc.max_delta = lmax;
        p = sc.prev;
      }
      // grow right (never into the last segment of the block)
      n = cnext;
      while (n != kPartTail) {
        const uint32_t wr = lk[n];
        if (lk_next(wr) == kPartTail) break;
        const PSeg sr = s[n];
        const int right = sr.end;
        const int64_t rmax = max(max(sr.max_delta, sc.max_delta), sc.next_delta);
        const int64_t rmin = min(min(sr.min_delta, sc.min_delta), sc.next_delta);
        const int bnew = cal_bits_d(rmin, rmax);
        const int ol = cal_bits_d(sc.min_delta, sc.max_delta), orr = cal_bits_d(sr.min_delta, sr.max_delta);
        const int oc = (right - sr.start + 1) * orr + (sr.start - sc.start) * ol;
        const int mc = bnew * (right - sc.start + 1);
        if (!(mc - oc < overhead)) break;
        sc.end = right;
        cnext = lk_next(wr);
        ccls = lk_class(wr);
        s[cnext].prev = c;  // cnext is not the tail: the loop stops before the last segment
        sc.max_delta = rmax;
        sc.min_delta = rmin;
        sc.next_delta = sr.next_delta;
        n = cnext;
      }
      s[c] = sc;
      lk[c] = lk_make(cnext, ccls);
      c = cnext;
    }
  }

  // ---- size-driven pairwise merge passes (…:439-483, merge :516-570), in place ----
  uint32_t m = 0;
  for (int c = lk_next(lk[kPartHead]); c != kPartTail; c = lk_next(lk[c])) idx[m++] = (uint32_t)s[c].start;
  const uint32_t endv = B0 + len;
  uint64_t total = 0;
  for (uint32_t i = 0; i < m; i++) {
    sz[i] = segment_cost_d(array, idx[i], (i + 1 < m ? idx[i + 1] : endv) - 1);
    total += sz[i];
  }
  for (;;) {
    const uint64_t before = total;
    uint64_t tnew = 0;
    uint32_t w = 0, k = 0;
    uint32_t start = idx[0];
    while (k < m) {
      if (k == m - 1) {
        const uint32_t z = sz[k];
        idx[w] = idx[k];
        sz[w++] = z;
        tnew += z;
        k++;
        break;
      }
      const uint32_t at2 = k + 2 < m ? idx[k + 2] : endv;
      const uint32_t init_cost = sz[k] + sz[k + 1];
      const uint32_t merge_cost = segment_cost_d(array, start, at2 - 1);
      if (init_cost > merge_cost) {
        idx[w] = start;
        sz[w++] = merge_cost;
        tnew += merge_cost;
        start = at2;
        k += 2;
      } else {
        const uint32_t at1 = idx[k + 1], z = sz[k];
        idx[w] = idx[k];
        sz[w++] = z;
        tnew += z;
        start = at1;
        k++;
      }
    }
    m = w;
    total = tnew;
    const uint64_t decline = before - total;  // unsigned, as in the reference
    const double pct = __ddiv_rn(__dmul_rn(__ull2double_rn(decline), 100.0), __dmul_rn((double)sizeof(uint64_t), (double)a.bs));
    if (!(decline > 0) || pct < 0.01) break;
  }
  for (uint32_t i = 0; i < m; i++) out[i] = idx[i];
  *count = m;
}

__global__ void __launch_bounds__(kPartThreads) partition_kernel(PartitionArgs a) {
  const uint64_t slot = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  PSeg *s = a.segs + slot * (a.bs + 1);
  uint32_t *lk = a.links + slot * (a.bs + 1);
  uint32_t *idx = a.pidx + slot * a.bs, *sz = a.psz + slot * a.bs;
  for (;;) {
    const uint64_t b = atomicAdd(a.ticket, 1u);
    if (b >= a.nblocks) return;
    const uint64_t B0 = b * a.bs;
    const uint32_t len = (uint32_t)(b == a.nblocks - 1 ? a.n - B0 : a.bs);
    partition_block_d(a, (uint32_t)B0, len, s, lk, idx, sz, a.stage + B0, a.count + b);
  }
}

// ---- one CTA per coarse block ---------------------------------------------------------
// Phase 1 needs no list.  Segments tile the positions 0 .. len-2 (position p carries the
// first difference D[p] = y[p+1] - y[p]), so a bitmap of the positions where a segment ends
// is the list; a segment ending at e has the bit class of D[e], D[e+1] and the difference
// D[e] to its successor, whatever it has absorbed, and starts after the bit before e.  Only
// the extremes of the differences inside a merged segment are kept (single points have
// none), for the first kPartPool of them in shared memory, else in global memory.  The positions are sorted by bit class once, so that a
// class's turn visits its own positions only, 32 at a time; a position that has been
// absorbed is skipped.  Phase 2 keeps 16-bit starts, sizes and pair sizes; a pair's size is
// computed again only when one of the two segments has changed.
// Bound by latency: phase 1 is one warp's, phase 2 mostly sums of the fits.  Shared memory:
// 14 bytes a value and 3 KB, seven CTAs per SM for blocks of 2000 values, one for blocks of 8000.  10M values, 5000 blocks of
// 2000, partition and encode: 43.7 ms with a thread per block, 4.47 ms with one warp per
// block that scanned every class over all positions, 1.86 ms now.
// The longest block of a CTA: starts and sizes fit 16 bits (a raw segment takes 8 bytes a value
// and 5).  2M values in blocks of 8000 / 8001: 2.1 ms / 146 ms, so the limit is the form's, not
// the point where the other kernel wins.
constexpr uint32_t kPartCtaMax = 8000;
// A column of many short coarse blocks keeps the thread per block: a CTA's barriers and list
// set-up take about 5 ns a block when all SMs are full, whatever its size, while a thread's
// chain shortens with it.  CTA time over thread time, regime-switching column / random values:
//   blocks:        4000         12000        25000        60000        300000
//   of 4 values    1.1 / 1.2    1.7 / 1.8    2.5 / 2.7    3.5 / 3.8    4.9 / 5.3
//   of 16          0.5 / 0.7    1.0 / 1.1    1.7 / 1.7    2.7 / 2.6    3.5 / 3.3
//   of 32          0.4 / 0.4    0.7 / 0.6    1.1 / 0.9    1.7 / 1.4    2.1 / 1.7
//   of 64          0.2 / 0.2    0.4 / 0.4    0.7 / 0.5    1.1 / 0.7    1.3 / 0.9
//   of 80          0.2 / 0.2    0.4 / 0.3    0.6 / 0.4    1.0 / 0.6    1.2 / 0.8 (200000)
//   of 96          0.2 / 0.1    0.3 / 0.2    0.5 / 0.3    0.8 / 0.5    0.9 / 0.6 (200000)
constexpr uint32_t kPartThreadMax = 80;     // longest block of that kind
constexpr uint32_t kPartThreadBlocks = 750;  // blocks per value of a block from which it is the faster
constexpr uint32_t kPartLaneMax = 48;    // pairs of up to this many values: one lane each
constexpr uint32_t kPartWarps = 4;
constexpr uint32_t kPartPool = 192;      // merged segments whose extremes are in shared memory
constexpr uint16_t kNoSize = 0xffffu, kNoSlot = 0xffffu;

struct PartShared {
  uint64_t *y;
  uint16_t *idx, *sz, *pc;
  uint16_t *order;  // phase 1 (over idx): positions by class
  uint16_t *slot;   // phase 1 (over pc): a merged segment's place in the pool, at its end
  longlong2 *pool;  // (min, max) as I (below), two to an entry
  uint8_t *cls;     // phase 1 (over sz)
  uint32_t *bits;   // phase 1: segment ends
  uint32_t *hist;   // phase 1: [72] where a class's positions end in order; phase 2: [0] long pairs, [1] segments, [2] sizes missing, [3] done
  uint16_t *jobs;   // phase 2 (over bits): pairs that take a warp
};
__host__ __device__ inline uint32_t part_list_bytes(uint32_t bs) { return ((bs + 2) * 2 + 7) / 8 * 8; }
__host__ __device__ inline uint32_t part_jobs_bytes(uint32_t bs) { return (bs / 32 + 2) * 4 + (bs / kPartLaneMax + 4) * 2 * 2; }
__host__ __device__ inline uint32_t part_smem_bytes(uint32_t bs) {
  return kPartPool * 16 + bs * 8 + 3 * part_list_bytes(bs) + 72 * 4 + part_jobs_bytes(bs);
}
__device__ __forceinline__ PartShared part_shared(uint8_t *smem, uint32_t bs) {
  const uint32_t list = part_list_bytes(bs);
  PartShared P;
  P.pool = reinterpret_cast<longlong2 *>(smem);
  P.y = reinterpret_cast<uint64_t *>(smem + kPartPool * 16);
  uint8_t *p = smem + kPartPool * 16 + (size_t)bs * 8;
  P.idx = P.order = reinterpret_cast<uint16_t *>(p);
  P.sz = reinterpret_cast<uint16_t *>(p + list);
  P.pc = P.slot = reinterpret_cast<uint16_t *>(p + 2 * list);
  P.cls = p + list;
  P.hist = reinterpret_cast<uint32_t *>(p + 3 * list);
  P.bits = P.hist + 72;
  P.jobs = reinterpret_cast<uint16_t *>(P.bits);
  return P;
}

// cal_bits on integers where that is exact: bits of ceil(d / 2) plus one is the bits of d + 1.
__device__ __forceinline__ int cal_bits_fast(int64_t mn, int64_t mx) {
  const int64_t diff = (int64_t)((uint64_t)mx - (uint64_t)mn);
  const uint64_t ad = diff < 0 ? 0 - (uint64_t)diff : (uint64_t)diff;
  if (ad >= (1ull << 53)) return cal_bits_d(mn, mx);
  return ad ? (int)bits64_d(ad + 1) : 0;
}
// The same for mn <= mx; I = int32_t: both in (-2^30, 2^30).
template <typename I>
__device__ __forceinline__ int span_bits(I mn, I mx) {
  if constexpr (sizeof(I) == 4) {
    const uint32_t d = (uint32_t)(mx - mn);
    return d ? 32 - __clz((int)(d + 1)) : 0;
  } else {
    return cal_bits_fast(mn, mx);
  }
}
// The segment end before position e (-1: none) and the one after it (one exists).
__device__ __forceinline__ int part_prev(const uint32_t *bits, int e) {
  int w = e >> 5;
  uint32_t v = bits[w] & ((1u << (e & 31)) - 1u);
  while (!v) {
    if (--w < 0) return -1;
    v = bits[w];
  }
  return 32 * w + 31 - __clz((int)v);
}
__device__ __forceinline__ int part_next(const uint32_t *bits, int e) {
  int w = (e + 1) >> 5;
  uint32_t v = bits[w] & (0xffffffffu << ((e + 1) & 31));
  while (!v) v = bits[++w];
  return 32 * w + __ffs((int)v) - 1;
}
// Size of a segment of `length` >= 3 values from its largest residual.
__device__ __forceinline__ uint32_t part_size(uint64_t maxr, uint32_t length) {
  const uint32_t bits = maxr ? bits64_d(maxr) + 1 : 0;
  if (bits >= 64) return 5 + 8 * length;
  return 17 + (bits * length + 7) / 8;
}
__device__ __forceinline__ void part_model(double sumy, double sumxy, uint32_t length, double &t0, double &slope) {
  const uint64_t m = length;
  const double dm = __uint2double_rn(length);
  // sum i and sum i*i are exact integers at every step of the reference's loop
  const double sumx = __ull2double_rn(m * (m - 1) / 2), sumxx = __ull2double_rn((m - 1) * m * (2 * m - 1) / 6);
  const double ccc = __dsub_rn(__dmul_rn(sumxy, dm), __dmul_rn(sumx, sumy));
  const double xxx = __dsub_rn(__dmul_rn(sumxx, dm), __dmul_rn(sumx, sumx));
  const double t1 = __ddiv_rn(ccc, xxx);
  t0 = __ddiv_rn(__dsub_rn(sumy, __dmul_rn(t1, sumx)), dm);
  slope = (double)__double2float_rn(t1);
}
// The largest residual of values first, first + step, ... of a segment (128-bit predictions,
// 64-bit ones where the ends say that every prediction lies in [0, 2^63)).
__device__ __forceinline__ uint64_t part_residual(const uint64_t *y, uint32_t length, uint32_t first, uint32_t step, double t0,
                                                  double slope) {
  const double p0 = __dadd_rn(t0, __dmul_rn(slope, 0.0)), p1 = __dadd_rn(t0, __dmul_rn(slope, __uint2double_rn(length - 1)));
  const bool narrow = p0 >= 0.0 && p1 >= 0.0 && p0 < 9223372036854775808.0 && p1 < 9223372036854775808.0;
  uint64_t maxr = 0;
  if (narrow) {
#pragma unroll 2
    for (uint32_t j = first; j < length; j += step) {
      const uint64_t pred = __double2ull_rz(__dadd_rn(t0, __dmul_rn(slope, u32_to_double_fp64(j)))), v = y[j];
      const uint64_t r = v > pred ? v - pred : pred - v;
      maxr = r > maxr ? r : maxr;
    }
  } else {
    for (uint32_t j = first; j < length; j += step) {
      const i128 pred = f2i128(__dadd_rn(t0, __dmul_rn(slope, u32_to_double_fp64(j)))), v = (i128)y[j];
      const uint64_t r = (uint64_t)(v > pred ? v - pred : pred - v);
      maxr = r > maxr ? r : maxr;
    }
  }
  return maxr;
}
// newsegment_size of y[0 .. length), one lane.
__device__ __forceinline__ uint32_t lane_size(const uint64_t *y, uint32_t length) {
  if (length == 1) return 9;
  if (length == 2) return 13;
  double sumy = 0, sumxy = 0, k = 0;
#pragma unroll 4
  for (uint32_t i = 0; i < length; i++) {
    const double v = u64_to_double_fp64(y[i]);
    sumy = __dadd_rn(sumy, v);
    sumxy = __dadd_rn(sumxy, __dmul_rn(k, v));
    k = __dadd_rn(k, 1.0);
  }
  double t0, slope;
  part_model(sumy, sumxy, length, t0, slope);
  return part_size(part_residual(y, length, 0, 1, t0, slope), length);
}
// The same by the whole warp.
__device__ __noinline__ uint32_t warp_size(const uint64_t *y, uint32_t length) {
  double sumy, sumxy, t0, slope;
  warp_seq_sums(y, length, sumy, sumxy);
  part_model(sumy, sumxy, length, t0, slope);
  return part_size(warp_max_u64(part_residual(y, length, threadIdx.x & 31, 32, t0, slope)), length);
}

// Classes of a coarse block of len >= 2 values, every position a segment; by the whole CTA.
// hist[71]: nonzero when some difference lies outside (-2^30, 2^30).
__device__ __forceinline__ void part_classes(const PartShared &P, uint32_t len) {
  const int last = (int)len - 2;  // the last segment's end
  const uint64_t *y = P.y;
  for (int p = threadIdx.x; p < last; p += blockDim.x) {
    const int64_t d0 = (int64_t)(y[p + 1] - y[p]), d1 = (int64_t)(y[p + 2] - y[p + 1]);
    const int c = cal_bits_fast(d0, d1);
    P.cls[p] = (uint8_t)c;
    atomicAdd(&P.hist[c], 1u);
  }
  for (int p = threadIdx.x; p <= last; p += blockDim.x) {
    const int64_t d = (int64_t)(y[p + 1] - y[p]);
    if (d <= -(1ll << 30) || d >= 1ll << 30) P.hist[71] = 1;
  }
  const int words = (last >> 5) + 1;
  for (int w = threadIdx.x; w < words; w += blockDim.x) P.bits[w] = 32 * w + 31 <= last ? 0xffffffffu : (2u << (last & 31)) - 1u;
}

// Phase 1, by one warp; mm: the (min, max) differences of merged segments that the pool has
// no place for, at their ends.  I: the type of differences, int32_t when all are small.
template <typename I>
__device__ __forceinline__ void part_merge_classes(const PartShared &P, uint32_t len, int overhead, longlong2 *mm) {
  const int lane = threadIdx.x & 31, last = (int)len - 2;
  const uint64_t *y = P.y;
  struct Ext {
    I lo, hi;
  };
  Ext *pool = reinterpret_cast<Ext *>(P.pool), *far = reinterpret_cast<Ext *>(mm);
  // positions by class, in order within a class
  uint32_t carry = 0;
  for (int c0 = 0; c0 < 72; c0 += 32) {
    const int c = c0 + lane;
    const uint32_t own = c < 71 ? P.hist[c] : 0;
    uint32_t incl = own;
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (c < 72) P.hist[c] = carry + incl - own;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  __syncwarp();
  for (int p0 = 0; p0 < last; p0 += 32) {
    const int p = p0 + lane, c = p < last ? P.cls[p] : 71;
    const uint32_t same = __match_any_sync(0xffffffffu, c), before = same & ((1u << lane) - 1u);
    const uint32_t at = P.hist[c];
    __syncwarp();
    if (p < last) {
      P.order[at + __popc(before)] = (uint16_t)p;
      if (!before) P.hist[c] = at + __popc(same);
    }
    __syncwarp();
  }
  auto diff = [&](int p) { return (I)(y[p + 1] - y[p]); };
  auto extremes = [&](int s, int e) {  // of segment [s, e]
    if (s == e) return Ext{0, 0};
    const uint32_t at = P.slot[e];
    return at == kNoSlot ? far[e] : pool[at];
  };
  uint32_t pooled = 0;  // places of the pool handed out; a merge keeps a place of its parts
  uint32_t i = 0;  // hist[c] is now where class c ends
  for (int aim = 0; aim < 71; ++aim) {
    const uint32_t i1 = P.hist[aim];
    int from = 0;  // segments that end before it have had their turn
    while (i < i1) {
      const int e = i + lane < i1 ? P.order[i + lane] : -1;
      // segment c = [s, e] with its right neighbour [e + 1, en]
      int s = 0, en = 0;
      Ext x{0, 0};
      bool merge = false;
      if (e >= from && ((P.bits[e >> 5] >> (e & 31)) & 1u)) {
        s = part_prev(P.bits, e) + 1;
        en = part_next(P.bits, e);
        const Ext c = extremes(s, e), n = extremes(e + 1, en);
        const I d = diff(e);
        x.hi = max(max(c.hi, n.hi), d);
        x.lo = min(min(c.lo, n.lo), d);
        const int origin = (e + 1 - s) * span_bits(c.lo, c.hi) + (en - e) * span_bits(n.lo, n.hi);
        merge = span_bits(x.lo, x.hi) * (en - s + 1) - origin < overhead;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, merge);
      if (!hit) {
        i += 32;
        continue;
      }
      const int f = __ffs((int)hit) - 1;  // the first segment that merges; those before it stay as they are
      uint32_t place = kNoSlot;  // of the merged segment
      auto inherit = [&](int a, int b) {  // segment [a, b] is absorbed
        if (a != b && place == kNoSlot) place = P.slot[b];
      };
      int cs = __shfl_sync(0xffffffffu, s, f), ce = __shfl_sync(0xffffffffu, en, f);
      x.lo = __shfl_sync(0xffffffffu, x.lo, f);
      x.hi = __shfl_sync(0xffffffffu, x.hi, f);
      const int fe = __shfl_sync(0xffffffffu, e, f);
      inherit(cs, fe);
      inherit(fe + 1, ce);
      __syncwarp();  // every lane has read the bits
      if (lane == 0) P.bits[fe >> 5] &= ~(1u << (fe & 31));
      __syncwarp();
      int width = span_bits(x.lo, x.hi);
      // grow left (never into the first segment of the block)
      while (cs > 0) {
        const int pe = cs - 1, ps = part_prev(P.bits, pe) + 1;
        if (ps == 0) break;
        const Ext p = extremes(ps, pe);
        const I d = diff(pe);
        const Ext g{min(min(p.lo, x.lo), d), max(max(p.hi, x.hi), d)};
        const int gw = span_bits(g.lo, g.hi);
        const int oc = (cs - ps) * span_bits(p.lo, p.hi) + (ce - cs + 1) * width;
        if (!(gw * (ce - ps + 1) - oc < overhead)) break;
        inherit(ps, pe);
        __syncwarp();
        if (lane == 0) P.bits[pe >> 5] &= ~(1u << (pe & 31));
        __syncwarp();
        cs = ps;
        x = g;
        width = gw;
      }
      // grow right (never into the last segment of the block)
      while (ce < last) {
        const int ne = part_next(P.bits, ce);
        if (ne == last) break;
        const Ext n = extremes(ce + 1, ne);
        const I d = diff(ce);
        const Ext g{min(min(n.lo, x.lo), d), max(max(n.hi, x.hi), d)};
        const int gw = span_bits(g.lo, g.hi);
        const int oc = (ne - ce) * span_bits(n.lo, n.hi) + (ce + 1 - cs) * width;
        if (!(gw * (ne - cs + 1) - oc < overhead)) break;
        inherit(ce + 1, ne);
        __syncwarp();
        if (lane == 0) P.bits[ce >> 5] &= ~(1u << (ce & 31));
        __syncwarp();
        ce = ne;
        x = g;
        width = gw;
      }
      if (place == kNoSlot && pooled < kPartPool) place = pooled++;
      __syncwarp();
      if (lane == 0) {
        P.slot[ce] = (uint16_t)place;
        if (place != kNoSlot) pool[place] = x;
        else far[ce] = x;
      }
      __syncwarp();
      from = ce + 1;
      i += f + 1;
    }
    i = i1;
  }
}

// Fills out[k] for k < count where it holds kNoSize and take(k) with the size of
// y[idx[k] .. idx[k + span]), by the whole CTA; out is complete after the call's last barrier.
template <typename Take>
__device__ __forceinline__ void part_sizes(const PartShared &P, uint16_t *out, uint32_t first, uint32_t step, uint32_t count,
                                           uint32_t span, Take take) {
  if (threadIdx.x == 0) P.hist[0] = 0;
  __syncthreads();
  for (uint32_t k = first + step * threadIdx.x; k < count; k += step * blockDim.x) {
    if (out[k] != kNoSize || !take(k)) continue;
    const uint32_t s = P.idx[k], length = P.idx[k + span] - s;
    if (length <= kPartLaneMax) out[k] = (uint16_t)lane_size(P.y + s, length);
    else P.jobs[atomicAdd(&P.hist[0], 1u)] = (uint16_t)k;
  }
  __syncthreads();
  const uint32_t jobs = P.hist[0];
  for (uint32_t j = threadIdx.x >> 5; j < jobs; j += blockDim.x >> 5) {
    const uint32_t k = P.jobs[j], s = P.idx[k];
    const uint32_t z = warp_size(P.y + s, P.idx[k + span] - s);
    if ((threadIdx.x & 31) == 0) out[k] = (uint16_t)z;
  }
  __syncthreads();
}
// The groups of 32 pairs of a pass, from the left: a pair whose size is smaller than its
// parts' merges and is passed over, so in a run of such pairs every other one merges, from
// the run's first on.  want: the pairs that would merge; taken: 1 when the group's first
// segment went into the pair before it.  Returns the pairs that merge.
__device__ __forceinline__ uint32_t part_merging(uint32_t want, uint32_t taken) {
  const uint32_t f = want & ~taken, even = 0x55555555u, run0 = f & ~(f << 1);
  const uint32_t from_even = f & ~(f + (run0 & even));  // the runs that begin at an even place
  return (from_even & even) | ((f & ~from_even) & ~even);
}
// True when a pass would come to a pair whose size is not known (one warp).
__device__ __forceinline__ bool part_pairs_missing(const PartShared &P, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t taken = 0;
  for (uint32_t k0 = 0; k0 + 1 < m; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint32_t q = k + 1 < m ? P.pc[k] : kNoSize, z = k + 1 < m ? (uint32_t)P.sz[k] + P.sz[k + 1] : 0;
    const uint32_t merge = part_merging(__ballot_sync(0xffffffffu, z > q), taken);
    const uint32_t unknown = __ballot_sync(0xffffffffu, k + 1 < m && q == kNoSize);
    if (unknown & ~((merge << 1) | taken)) return true;
    taken = merge >> 31;
  }
  return false;
}

// One merge pass by one warp: m segments, their sizes and the pair sizes it comes to known.  Returns the new
// number of segments and, in tnew, the sum of their sizes.
__device__ __forceinline__ uint32_t part_merge_pass(const PartShared &P, uint32_t m, uint32_t len, uint64_t &tnew) {
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  uint32_t w = 0;      // segments of the new list
  uint32_t taken = 0;  // 1: the first segment of this group went into the pair before it
  tnew = 0;
  // (entries of the list are written no further on than they were read: the group's own
  // are in registers, and w <= k0; the next group's first pair flag is taken ahead)
  for (uint32_t k0 = 0; k0 < m; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint32_t z = k < m ? P.sz[k] : 0, q = k + 1 < m ? P.pc[k] : kNoSize;
    const uint32_t z1 = k + 1 < m ? P.sz[k + 1] : 0, i0 = k < m ? P.idx[k] : 0;
    const bool want = k + 1 < m && z + z1 > q;
    const uint32_t merge = part_merging(__ballot_sync(0xffffffffu, want), taken);
    const uint32_t gone = (merge << 1) | taken, in = m - k0 >= 32 ? 0xffffffffu : (1u << (m - k0)) - 1u;
    const uint32_t keep = ~gone & in;
    // the pair (k, k + 1) stays a pair when neither merges (k + 1's flag may be the next group's)
    const uint32_t k1 = k0 + 32;
    uint32_t next_merges = 0;
    if (!(merge >> 31) && k1 + 1 < m) next_merges = (uint32_t)P.sz[k1] + P.sz[k1 + 1] > P.pc[k1];  // segment k1 is free
    const uint32_t after = (merge >> 1) | (next_merges << 31);  // does segment k + 1 merge
    __syncwarp();
    if ((keep >> lane) & 1u) {
      const uint32_t o = w + __popc(keep & below);
      const bool mg = (merge >> lane) & 1u;
      const uint32_t nz = mg ? q : z;
      P.idx[o] = (uint16_t)i0;
      P.sz[o] = (uint16_t)nz;
      P.pc[o] = mg || ((after >> lane) & 1u) ? kNoSize : (uint16_t)q;
      tnew += nz;
    }
    w += __popc(keep);
    taken = merge >> 31;
    __syncwarp();
  }
  if (lane == 0) P.idx[w] = P.idx[w + 1] = (uint16_t)len;  // ends of the last segment and of the last pair
  tnew = warp_sum_u64(tnew);
  return w;
}

// Phase 2, by the whole CTA: the pairwise merge passes; returns the number of segments, their
// starts in P.idx.
__device__ __forceinline__ uint32_t part_merge_pairs(const PartShared &P, uint32_t len, uint32_t bs) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, last = len - 2;
  if (warp == 0) {  // starts: 0 and each end but the last, plus one
    const uint32_t below = (1u << lane) - 1u;
    uint32_t m = 1;
    if (lane == 0) P.idx[0] = 0;
    for (uint32_t w = 0; w <= last >> 5; ++w) {
      uint32_t v = P.bits[w];
      if (w == last >> 5) v &= ~(1u << (last & 31));
      if ((v >> lane) & 1u) P.idx[m + __popc(v & below)] = (uint16_t)(32 * w + lane + 1);
      m += __popc(v);
    }
    __syncwarp();
    if (lane == 0) {
      P.idx[m] = P.idx[m + 1] = (uint16_t)len;
      P.hist[1] = m;
    }
  }
  __syncthreads();
  uint32_t m = P.hist[1];
  for (uint32_t k = threadIdx.x; k < m; k += blockDim.x) P.sz[k] = P.pc[k] = kNoSize;
  part_sizes(P, P.sz, 0, 1, m, 1, [](uint32_t) { return true; });
  uint64_t total = 0;  // warp 0's
  if (warp == 0) {
    for (uint32_t k = lane; k < m; k += 32) total += P.sz[k];
    total = warp_sum_u64(total);
  }
  for (;;) {
    // Most pairs merge while segments are short, and a pair that merges keeps the next one from
    // being looked at: every other pair first, then those after a pair that does not merge,
    // and the rest only if the pass would come to one of them.
    part_sizes(P, P.pc, 0, 2, m - 1, 2, [](uint32_t) { return true; });
    part_sizes(P, P.pc, 1, 2, m - 1, 2, [&](uint32_t k) { return (uint32_t)P.sz[k - 1] + P.sz[k] <= P.pc[k - 1]; });
    if (warp == 0) {
      const bool missing = part_pairs_missing(P, m);
      if (lane == 0) P.hist[2] = missing;
    }
    __syncthreads();
    if (P.hist[2]) part_sizes(P, P.pc, 0, 1, m - 1, 2, [](uint32_t) { return true; });
    if (warp == 0) {
      uint64_t tnew;
      const uint32_t w = part_merge_pass(P, m, len, tnew);
      const uint64_t decline = total - tnew;  // unsigned, as in the reference
      total = tnew;
      const double pct = __ddiv_rn(__dmul_rn(__ull2double_rn(decline), 100.0), __dmul_rn((double)sizeof(uint64_t), (double)bs));
      if (lane == 0) {
        P.hist[1] = w;
        P.hist[3] = !(decline > 0) || pct < 0.01;
      }
    }
    __syncthreads();
    m = P.hist[1];
    if (P.hist[3]) return m;
  }
}

__global__ void __launch_bounds__(32 * kPartWarps) partition_cta_kernel(PartitionArgs a) {
  extern __shared__ __align__(16) uint8_t part_smem[];
  __shared__ uint32_t ticket;
  const uint32_t tid = threadIdx.x;
  const PartShared P = part_shared(part_smem, a.bs);
  longlong2 *mm = reinterpret_cast<longlong2 *>(a.segs) + (size_t)blockIdx.x * a.bs;
  for (;;) {
    __syncthreads();  // the block before has been written out
    if (tid == 0) ticket = atomicAdd(a.ticket, 1u);
    if (tid < 72) P.hist[tid] = 0;
    __syncthreads();
    const uint64_t b = ticket;
    if (b >= a.nblocks) return;
    const uint64_t B0 = b * a.bs;
    const uint32_t len = (uint32_t)(b == a.nblocks - 1 ? a.n - B0 : a.bs);
    if (len < 2) {  // the reference needs two points per coarse block (it reads array[B0 + 1])
      if (tid == 0) {
        a.stage[B0] = (uint32_t)B0;
        a.count[b] = 1;
      }
      continue;
    }
    for (uint32_t i = tid; i < len; i += blockDim.x) P.y[i] = __ldg(a.array + B0 + i);
    __syncthreads();
    part_classes(P, len);
    __syncthreads();
    if (tid < 32) {
      if (P.hist[71]) part_merge_classes<int64_t>(P, len, a.overhead, mm);
      else part_merge_classes<int32_t>(P, len, a.overhead, mm);
    }
    __syncthreads();
    const uint32_t m = part_merge_pairs(P, len, a.bs);
    for (uint32_t k = tid; k < m; k += blockDim.x) a.stage[B0 + k] = (uint32_t)B0 + P.idx[k];
    if (tid == 0) a.count[b] = m;
  }
}

// Exclusive scan of the per-block counts (one CTA, chunks of 1024), then each
// block's starts are copied to their place in the caller's array.
__global__ void __launch_bounds__(1024) count_scan_kernel(const uint32_t *count, uint64_t nb, uint64_t *base, uint64_t *total) {
  __shared__ uint64_t wsum[32];
  __shared__ uint64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t c0 = 0; c0 < nb; c0 += 1024) {
    const uint64_t i = c0 + threadIdx.x;
    const uint64_t x = i < nb ? count[i] : 0;
    uint64_t inc = x;
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const uint64_t v = wsum[lane];
      uint64_t vi = v;
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, vi, d);
        if (lane >= d) vi += y;
      }
      wsum[lane] = vi - v;
    }
    __syncthreads();
    if (i < nb) base[i] = carry + wsum[warp] + inc - x;
    __syncthreads();
    if (threadIdx.x == 1023) carry += wsum[31] + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(256) starts_gather_kernel(const uint32_t *stage, const uint32_t *count, const uint64_t *base,
                                                            uint64_t nb, uint32_t bs, uint64_t *starts, uint64_t cap,
                                                            uint32_t *error) {
  for (uint64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const uint32_t c = count[b];
    const uint64_t o = base[b];
    for (uint32_t j = threadIdx.x; j < c; j += blockDim.x) {
      if (o + j < cap) starts[o + j] = stage[b * bs + j];
      else atomicOr(error, kErrCapacity);
    }
  }
}

static void part_layout(uint64_t n, uint32_t coarse_blocks, uint32_t &bs, uint64_t &nb, uint64_t &slots) {
  uint64_t b = n / coarse_blocks;
  if (!b) b = 1;
  bs = (uint32_t)b;
  nb = n / b;
  if (nb * b < n) nb++;
  slots = std::min<uint64_t>((nb + kPartThreads - 1) / kPartThreads, 148 * 4) * kPartThreads;
}

static uint64_t align256(uint64_t x) { return (x + 255) / 256 * 256; }

}  // namespace leco

using namespace leco;

extern "C" {

uint64_t leco_varlen_partition_workspace_bytes(uint64_t n, uint32_t coarse_blocks) {
  if (!coarse_blocks || n < 2) return 0;
  uint32_t bs;
  uint64_t nb, slots;
  part_layout(n, coarse_blocks, bs, nb, slots);
  return align256(slots * (bs + 1) * sizeof(PSeg)) + align256(slots * (bs + 1) * 4ull) + 2 * align256(slots * bs * 4ull) +
         align256(n * 4) +
         align256(nb * 4) + align256(nb * 8) + 256;
}

int leco_varlen_partition_device(const uint64_t *d_values, uint64_t n, uint32_t coarse_blocks, int64_t delta,
                                 uint64_t *d_starts, uint64_t starts_cap, uint64_t *d_nseg, void *d_ws, uint64_t ws_bytes,
                                 leco_stream_t stream) {
  if (!d_values || !d_starts || !d_nseg || !coarse_blocks || n < 2)
    return record_error(LECO_ERR_ARG, "leco_varlen_partition_device: need values (n >= 2), starts and a block count");
  if (n > 0xffffffffull) return record_error(LECO_ERR_ARG, "leco_varlen_partition_device: segments start at 32-bit indices");
  if (n / coarse_blocks >= (1ull << 24) - 4)
    return record_error(LECO_ERR_ARG, "leco_varlen_partition_device: coarse blocks of at most 2^24 - 5 values");
  if (!d_ws || ws_bytes < leco_varlen_partition_workspace_bytes(n, coarse_blocks) || (reinterpret_cast<uintptr_t>(d_ws) & 255))
    return record_error(LECO_ERR_ARG, "leco_varlen_partition_device: workspace must be leco_varlen_partition_workspace_bytes(), 256-byte aligned");
  uint32_t *err = nullptr;
  int rc = device_error_word(&err);
  if (rc) return rc;
  uint32_t bs;
  uint64_t nb, slots;
  part_layout(n, coarse_blocks, bs, nb, slots);
  uint8_t *w = static_cast<uint8_t *>(d_ws);
  PartitionArgs A;
  A.array = d_values;
  A.n = n;
  A.bs = bs;
  A.nblocks = nb;
  A.overhead = (int)delta;
  A.segs = reinterpret_cast<PSeg *>(w);
  w += align256(slots * (bs + 1) * sizeof(PSeg));
  A.links = reinterpret_cast<uint32_t *>(w);
  w += align256(slots * (bs + 1) * 4ull);
  A.pidx = reinterpret_cast<uint32_t *>(w);
  w += align256(slots * bs * 4ull);
  A.psz = reinterpret_cast<uint32_t *>(w);
  w += align256(slots * bs * 4ull);
  A.stage = reinterpret_cast<uint32_t *>(w);
  w += align256(n * 4);
  A.count = reinterpret_cast<uint32_t *>(w);
  w += align256(nb * 4);
  uint64_t *base = reinterpret_cast<uint64_t *>(w);
  w += align256(nb * 8);
  A.ticket = reinterpret_cast<uint32_t *>(w);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(A.ticket, 0, 4, st) != cudaSuccess) return record_error(LECO_ERR_CUDA, "leco_varlen_partition_device: memset");
  const bool many_short = bs <= kPartThreadMax && nb >= (uint64_t)kPartThreadBlocks * bs;
  if (bs <= kPartCtaMax && !many_short) {
    const uint32_t smem = part_smem_bytes(bs);
    cudaError_t se = cudaSuccess;
    if (smem > 48 * 1024)  // the largest block's limit: it is the kernel's, and another thread may be about to launch one
      se = cudaFuncSetAttribute(partition_cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)part_smem_bytes(kPartCtaMax));
    int dev = 0, sms = 148, per_sm = 1;
    if (se == cudaSuccess) se = cudaGetDevice(&dev);
    if (se == cudaSuccess) se = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (se == cudaSuccess) se = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, partition_cta_kernel, 32 * kPartWarps, smem);
    if (se != cudaSuccess)
      return record_error(LECO_ERR_CUDA, std::string("leco_varlen_partition_device: ") + cudaGetErrorString(se));
    // a CTA's scratch (16 bytes a value) lies in its slot's segment list (40 bytes a value): no more CTAs than slots
    const uint64_t grid = std::min<uint64_t>(std::min<uint64_t>(nb, slots), (uint64_t)sms * (uint64_t)std::max(per_sm, 1));
    partition_cta_kernel<<<(unsigned)grid, 32 * kPartWarps, smem, st>>>(A);
  } else {
    partition_kernel<<<(unsigned)(slots / kPartThreads), kPartThreads, 0, st>>>(A);
  }
  count_scan_kernel<<<1, 1024, 0, st>>>(A.count, nb, base, d_nseg);
  starts_gather_kernel<<<(unsigned)std::min<uint64_t>(nb, 148 * 8), 256, 0, st>>>(A.stage, A.count, base, nb, bs, d_starts,
                                                                                   starts_cap, err);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return record_error(LECO_ERR_CUDA, std::string("leco_varlen_partition_device: ") + cudaGetErrorString(e));
  return LECO_OK;
}

}  // extern "C"
