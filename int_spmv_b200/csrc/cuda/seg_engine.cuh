// seg_engine.cuh - deterministic segmented row reduction for slot streams.
//
// The AXT layouts (and the compacted one's CSR order) lay every row's slots
// out contiguously, so a warp that walks a contiguous range of "units" (an
// AXT tile, a tile column, or one slot) sees each row as one run of equal
// row ids.  A warp owns one segment of units and:
//   - writes every run that starts and ends inside its segment straight to
//     y (such a run is a whole row);
//   - records its first run (head) and last run (tail) - which may continue
//     into a neighbouring segment - as (row, partial) pairs;
// and a fix-up kernel then adds each row's partials in segment order and
// writes y.  y is overwritten (beta = 0) or accumulated (beta = 1, by one
// reduction per row) deterministically: every row is written exactly once.
#pragma once
#include "common.cuh"

namespace ispmv {
namespace seg {

struct State {
  UIN crow;       // row of the run still open at the end of the last batch
  double csum;    // its partial sum
  bool head_done; // the segment's first run has been recorded
};

struct Out {
  FPT *y;
  const UIN *rowmap;  // compressed -> real row (nullptr: identity)
  UIN *rec_row;       // 2 records per segment: [2s] head, [2s+1] tail
  double *rec_sum;
  int beta;
};

__device__ __forceinline__ UIN real_row(const Out &o, UIN r) { return o.rowmap ? o.rowmap[r] : r; }

// The row's value to y.  beta = 1 adds with a reduction at L2 (red.add: y + v
// in FP64, rounded once, as a load and an add give it; every row is written
// once, so the result does not depend on any order): a load of y in the
// middle of a batch stalls its warp.
// FORM: 0 or 1 = beta, known to the compiler; RED or ATOMIC: o.beta decides, and
// the reduction is inline assembly (the compiler keeps loads and row writes in
// their order) or the intrinsic (it may move and predicate them).  RED is the
// faster in stream_wide (power-law n = 4M, beta = 0: 180.0 us, ATOMIC 182.6),
// ATOMIC in the kernels of 4 slots per lane (stream_ldg's variant 2, n = 1M,
// beta = 0: 73.7 us, RED 77.8; 75.2 with a load and an add) but the work-queue
// one (64 FEM blocks, 147M nonzeros: RED 373 us, ATOMIC 400).
enum RowWrite : int { RED = -1, ATOMIC = -2 };
template <int FORM>
__device__ __forceinline__ void write_row(const Out &o, UIN r, double v) {
  FPT *q = o.y + real_row(o, r);
  if (!(FORM < 0 ? o.beta : FORM)) *q = v;
  else if constexpr (FORM == RED) asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(q), "d"(v) : "memory");
  else atomicAdd(q, v);
}

// One batch of 32 units, one per lane: `p` the unit's partial sum, `r` its
// row (NO_ROW when !live).  Live lanes form a prefix of the warp.
__device__ __forceinline__ void batch(double p, UIN r, bool live, State &st, const Out &o, size_t segid) {
  const unsigned lane = threadIdx.x & 31u;
  // a batch past the segment's last unit changes nothing (the open run stays open)
  if (!__any_sync(FULL, live)) return;
  const UIN rprev = __shfl_up_sync(FULL, r, 1);
  const bool head = (lane == 0) ? (r != st.crow) : (r != rprev);
  // Did the carried run end at the previous batch's last lane?
  const bool carry_done = __shfl_sync(FULL, (unsigned)head, 0) && st.crow != NO_ROW;
  if (carry_done) {
    if (!st.head_done) {
      if (lane == 0) { o.rec_row[2 * segid] = st.crow; o.rec_sum[2 * segid] = st.csum; }
      st.head_done = true;
    } else if (lane == 0) {
      write_row<ATOMIC>(o, st.crow, st.csum);
    }
  }
  if (lane == 0 && !head) p += st.csum;
  const double s = warp_seg_scan(p, head);
  const UIN rnext = __shfl_down_sync(FULL, r, 1);
  const bool nlive = __shfl_down_sync(FULL, (unsigned)live, 1) != 0;
  const bool is_end = lane < 31 && live && nlive && r != rnext;
  unsigned ends = __ballot_sync(FULL, is_end);
  if (!st.head_done && ends) {
    const unsigned first = __ffs(ends) - 1;
    if (lane == first) { o.rec_row[2 * segid] = r; o.rec_sum[2 * segid] = s; }
    ends &= ~(1u << first);
    st.head_done = true;
  }
  if ((ends >> lane) & 1u) write_row<ATOMIC>(o, r, s);
  const unsigned lives = __ballot_sync(FULL, live);
  const int last = lives ? 31 - __clz(lives) : 0;
  const UIN lr = __shfl_sync(FULL, r, last);
  const double ls = __shfl_sync(FULL, s, last);
  if (lives) { st.crow = lr; st.csum = ls; }
}

// Records the segment's open run: its head if no run was recorded yet,
// else its tail.
__device__ __forceinline__ void finish(const State &st, const Out &o, size_t segid) {
  if ((threadIdx.x & 31u) != 0) return;
  if (!st.head_done) {
    o.rec_row[2 * segid] = st.crow;
    o.rec_sum[2 * segid] = st.crow == NO_ROW ? 0.0 : st.csum;
    o.rec_row[2 * segid + 1] = NO_ROW;
    o.rec_sum[2 * segid + 1] = 0.0;
  } else {
    o.rec_row[2 * segid + 1] = st.crow;
    o.rec_sum[2 * segid + 1] = st.crow == NO_ROW ? 0.0 : st.csum;
  }
}

// Fix-up: record i writes its row if it is the row's last record, adding the
// row's earlier records (walking back).  Also zeroes (beta = 0) the rows
// that own no slot at all (rows of length 0).  Launched as a programmatic
// dependent of the main kernel where the stream allows it, so its launch
// overlaps the main kernel's last CTAs: griddepcontrol.wait then blocks until
// the main kernel has completed and its records and rows are visible (it
// returns at once for an ordinary launch).
// LONG (a plan with a row of more than FIX_LONG segments): a thread walks
// FIX_WALK records back by itself, and the rest of a longer row's are added by
// its warp, 32 * FIX_U at a time, in an order that depends on the records
// alone.  One row of 1M nonzeros among 10,000 short ones (2,000 segments):
// 492.7 us a product with the records added one by one, 17.5 so.  Without
// such a row the warp's part only costs: 52.0 -> 52.4 us (power-law n = 1M).
constexpr size_t FIX_LONG = 8;
constexpr int FIX_WALK = 4, FIX_U = 8;
template <bool LONG>
__global__ void __launch_bounds__(256) fixup(size_t nrec, const UIN *rec_row_, const double *rec_sum_,
                                             const UIN *__restrict__ rowmap, const UIN *__restrict__ empty,
                                             size_t nempty, FPT *y_, int beta) {
  pdl_trigger();  // the next product's main kernel may launch; it waits for this grid
  pdl_wait();
  const UIN *rec_row = after_wait(rec_row_);
  const double *rec_sum = after_wait(rec_sum_);
  FPT *y = after_wait(y_);
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nempty && !beta) y[empty[i]] = 0.0;
  UIN r = i < nrec ? rec_row[i] : NO_ROW;
  if (!LONG && r == NO_ROW) return;
  if (r != NO_ROW) {
    size_t j = i + 1;
    while (j < nrec && rec_row[j] == NO_ROW) j++;
    if (j < nrec && rec_row[j] == r) r = NO_ROW;  // not the row's last record
  }
  if (!LONG && r == NO_ROW) return;
  double total = 0.0;
  size_t k = i;       // records [0, k) are left
  bool more = false;  // and some of them may be the row's
  if (r != NO_ROW) {
    total = rec_sum[i];
    more = true;
    for (int t = 0; more && (!LONG || t < FIX_WALK); t++) {
      more = false;
      if (!k) break;
      const UIN rk = rec_row[--k];
      more = rk == NO_ROW || rk == r;
      if (rk == r) total += rec_sum[k];
    }
  }
  if constexpr (LONG) {
    const unsigned lane = threadIdx.x & 31u;
    for (unsigned need = __ballot_sync(FULL, more); need; need &= need - 1) {
      const int src = __ffs(need) - 1;
      const UIN rs = __shfl_sync(FULL, r, src);
      unsigned long long e = __shfl_sync(FULL, (unsigned long long)k, src);
      double part = 0.0;
      for (bool go = true; go && e;) {
        UIN rk[FIX_U];
        double v[FIX_U];
#pragma unroll
        for (int u = 0; u < FIX_U; u++) {
          const unsigned long long d = 32u * u + lane + 1u;  // record e - d
          rk[u] = d <= e ? rec_row[e - d] : NO_ROW;
          v[u] = d <= e ? rec_sum[e - d] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < FIX_U; u++) {
          const unsigned other = __ballot_sync(FULL, rk[u] != rs && rk[u] != NO_ROW);
          if (go && rk[u] == rs && lane < (other ? (unsigned)__ffs(other) - 1u : 32u)) part += v[u];
          if (other) go = false;
        }
        e = e > 32u * FIX_U ? e - 32u * FIX_U : 0;
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(FULL, part, d);
      if ((int)lane == src) total += part;
    }
    if (r == NO_ROW) return;
  }
  const UIN rr = rowmap ? rowmap[r] : r;
  y[rr] = beta ? total + y[rr] : total;
}

}  // namespace seg
}  // namespace ispmv
