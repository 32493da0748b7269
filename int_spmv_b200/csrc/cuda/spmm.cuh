// spmm.cuh - multi-RHS SpMM on the slot stream: Y = A X, X and Y row-major
// n x k (FP64), one plan's slot stream read once per block of up to 32
// right-hand sides.
//
// A warp splits into NG = 32/G groups of G lanes; lane jl of a group owns the
// W columns j0 + W*jl .. of the column block (G*W = 8, 16 or 32 columns).
// Each group walks its own contiguous part of the slot stream.  Row starts
// come from the stream's bitmap; a row that ends inside the part is written
// to Y directly.  Rows that cross parts are joined at the CTA's end by the
// group they start in; only the runs open at the CTA's two ends become
// G*W-wide records that spmm_fixup adds per row.  Deterministic, no atomics.
//
// What bounds it: a slot costs G*W*8 bytes of X, gathered through L1 (a tag
// lookup and 64 bytes per SM and cycle) and, past 126 MB of X, from DRAM.  The
// kernel therefore keeps the other users of the L1 pipe small and as many X
// pieces in flight as it can:
//   - values and columns come in by cp.async, 16 bytes per lane, into a
//     double-buffered chunk of 4G slots per group in shared memory, read back
//     as broadcasts of 16 bytes (2 values, 4 columns); loading them slot by
//     slot touched 24 lines per 32 nonzeros, three quarters of what X does;
//   - no registers hold the stream, so 16-24 warps per SM keep 4 to 8 X pieces
//     per lane in flight: four slots of a step are consumed, then the pieces of
//     the same four slots of the next step are loaded into the registers freed
//     (slot by slot, the loads outnumber the barriers a warp waits on, and the
//     two-column form took 175 us where it takes 138 so, the same X each time);
//   - parts are short (spmm_part): the warps resident at a time then work on
//     neighbouring rows, whose columns' X rows stay in L2 (k = 32, 256 MB of
//     X: 323 us at 128 slots, 413 at 512), and the joins inside the CTA keep
//     the records few (records per part cost 12-44 us of fix-up).
// Power-law n = 1M, 14.9M nonzeros, FP64, against one slot's value and column
// per lane and step, three matrices and X in turn (neither in L2 when a product
// starts): k = 8 236 us -> 151, k = 32 450 -> 372.
#pragma once
#include <type_traits>

#include "wide.cuh"

namespace ispmv {
namespace mm {

struct Out {
  FPT *Y;
  const UIN *rowmap;
  double *head;     // G*W per part: the sum of the run open at the part's start
  UIN *rec_row;     // 2 per CTA
  double *rec_sum;  // 2 * G*W per CTA
  UIN k, j0, kb;    // row stride, first column of the block, columns in the block
};

__device__ __forceinline__ UIN real_row(const Out &o, UIN r) { return o.rowmap ? o.rowmap[r] : r; }

// The plan's stream: `lspl` = log2 of the slots per lane of a lane-interleaved
// plan (wide::il_pos), 0 for one in slot order.
struct Stream {
  size_t nslots, nslots_pad, seg_slots;
  const void *val;
  const UIN *col, *heads, *segh;
  unsigned lspl;
};

// Position of the vector of 1 << lv elements that starts at slot s.
__device__ __forceinline__ size_t il_vec(size_t s, unsigned lspl, unsigned lv) {
  if (!lspl) return s;
  const size_t bt = (size_t)32 << lspl;
  const unsigned r = (unsigned)(s & (bt - 1)), l = r >> lspl, k = r & ((1u << lspl) - 1u);
  return (s & ~(bt - 1)) + ((size_t)(k >> lv) << (5 + lv)) + (l << lv);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tma::smem_addr(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// W consecutive doubles of a row of X (or to a row of Y): one access of 8*W
// bytes when VEC (aligned, all W columns live), else those below ncol.
template <int W, bool VEC>
__device__ __forceinline__ void ld_x(const double *p, int ncol, double (&d)[W]) {
  if constexpr (VEC && W == 4) {
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(d[0]), "=d"(d[1]), "=d"(d[2]), "=d"(d[3])
                 : "l"(p));
  } else if constexpr (VEC) {
    static_assert(W == 2, "two or four columns per lane");
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(d[0]), "=d"(d[1]) : "l"(p));
  } else {
#pragma unroll
    for (int w = 0; w < W; w++) d[w] = w < ncol ? __ldg(p + w) : 0.0;
  }
}
template <int W, bool VEC>
__device__ __forceinline__ void st_y(double *p, int ncol, const double (&d)[W]) {
  if constexpr (VEC && W == 4) {
    if (ncol > 0)
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(d[0]), "d"(d[1]), "d"(d[2]), "d"(d[3])
                   : "memory");
  } else if constexpr (VEC) {
    if (ncol > 0) *reinterpret_cast<double2 *>(p) = make_double2(d[0], d[1]);
  } else {
#pragma unroll
    for (int w = 0; w < W; w++)
      if (w < ncol) p[w] = d[w];
  }
}

// One chunk of 4G slots of a group in shared memory, padded so that the
// groups' 16-byte broadcasts fall in different banks.
template <int G, typename VT>
struct alignas(16) Chunk {
  VT v[4 * G + 16 / sizeof(VT)];
  UIN c[4 * G + (G == 2 ? 8 : 4)];
};

template <int G, int W, int T, int MINB, bool VEC, typename VT>
__global__ void __launch_bounds__(256, MINB)
    stream_spmm(Stream st, size_t part, size_t nparts, const FPT *__restrict__ X, Out o) {
  constexpr int NG = 32 / G, CB = G * W, C = 4 * G, NU = C / T, V = 16 / (int)sizeof(VT), LV = V == 2 ? 1 : 2;
  static_assert(T % 4 == 0 && C % T == 0 && (C <= 32 || C == 64), "whole 16-byte pieces, chunks inside bitmap words");
  __shared__ Chunk<G, VT> chunks[8][2][NG];
  pdl_trigger();  // the record fix-up may launch; it waits for this grid
  const unsigned lane = threadIdx.x & 31u, grp = lane / G, jl = lane % G;
  const size_t pid = (((size_t)blockIdx.x * 256 + threadIdx.x) >> 5) * NG + grp;
  Chunk<G, VT> *const mine = &chunks[threadIdx.x >> 5][0][grp];  // and mine + NG
  const bool has = pid < nparts;
  const size_t a = has ? pid * part : 0, b = has ? min(a + part, st.nslots_pad) : 0;
  const int ncol = jl * W < o.kb ? min(W, (int)(o.kb - jl * W)) : 0;  // my live columns
  // lanes past the block's last column load a piece of the block and store nothing
  const FPT *const xb = X + o.j0 + (VEC && !ncol ? o.kb - W : jl * W);
  const UIN kb8 = o.k * 8u;  // row stride in bytes (VEC: k < 2^29)
  auto x_row = [&](UIN c) {
    if constexpr (VEC) return reinterpret_cast<const FPT *>(reinterpret_cast<const char *>(xb) + (uint64_t)c * kb8);
    else return xb + (size_t)c * o.k;
  };
  FPT *const yb = o.Y + o.j0 + jl * W;
  // compressed row of the run open at slot a: row starts before a, minus one
  UIN row = 0;
  bool a_head = false;
  if (has) {
    const size_t sg = a / st.seg_slots;
    for (size_t w = (sg * st.seg_slots >> 5) + jl; w < (a >> 5); w += G) row += __popc(__ldg(st.heads + w));
    if (jl == 0) row += __ldg(st.segh + sg);
    a_head = (__ldg(st.heads + (a >> 5)) & 1u) != 0;
  }
#pragma unroll
  for (int d = 1; d < G; d <<= 1) row += __shfl_xor_sync(FULL, row, d);
  row -= 1u;
  const UIN row_a = a_head ? NO_ROW : row;

  const VT *const val = static_cast<const VT *>(st.val);
  // the group's chunk at c0: each lane copies 4/V value vectors and one
  // column vector, neighbouring lanes neighbouring addresses
  auto issue = [&](size_t c0, Chunk<G, VT> *dst) {
    const unsigned lgl = st.lspl && (C >> st.lspl) > 1 ? 31 - __clz(C >> st.lspl) : 0;  // log2 lanes the chunk spans
#pragma unroll
    for (int r = 0; r < 4 / V; r++) {
      const unsigned rank = r * G + jl;
      const unsigned m = ((rank & ((1u << lgl) - 1u)) << (st.lspl ? st.lspl - LV : 0)) + (rank >> lgl);
      cp_async16(dst->v + V * m, val + il_vec(c0 + V * m, st.lspl, LV));
    }
    const unsigned m = ((jl & ((1u << lgl) - 1u)) << (st.lspl ? st.lspl - 2 : 0)) + (jl >> lgl);
    cp_async16(dst->c + 4 * m, st.col + il_vec(c0 + 4 * m, st.lspl, 2));
  };
  // row-start bits of the chunk at c0
  using Bits = std::conditional_t<C == 64, unsigned long long, unsigned>;
  auto bits_of = [&](size_t c0) {
    Bits h = __ldg(st.heads + (c0 >> 5));
    if constexpr (C == 64) h |= (Bits)__ldg(st.heads + (c0 >> 5) + 1) << 32;
    else h >>= (unsigned)(c0 & 31u);
    return h;
  };

  double xv[T][W], acc[W];
#pragma unroll
  for (int w = 0; w < W; w++) acc[w] = 0.0;
  double *const head = o.head + pid * CB + jl * W;
  double *ydst = head;  // where the open run goes if it ends here: the part's head first
  Bits hs = 0, hnext = 0;
  if (a < b) {
    issue(a, mine);
    hnext = bits_of(a);
  }
  cp_async_wait();
  __syncwarp();
  if (a < b) {
#pragma unroll
    for (int i = 0; i < T; i++) ld_x<W, VEC>(x_row(mine->c[i]), ncol, xv[i]);
  }
  bool first = true;
  const int nch = (int)(part / C);
  for (int q = 0; q < nch; q++) {
    const size_t c0 = a + (size_t)q * C;
    const bool on = c0 < b, next = c0 + C < b;
    const Chunk<G, VT> *cur = mine + (q & 1) * NG, *other = mine + (~q & 1) * NG;
    hs = hnext;
    if (next) {
      issue(c0 + C, const_cast<Chunk<G, VT> *>(other));
      hnext = bits_of(c0 + C);
    }
#pragma unroll 1
    for (int u = 0; u < NU; u++) {
      const UIN *cn = cur->c + (u + 1) * T;
      bool more = on;
      if (u == NU - 1) {  // the next step is the next chunk's first: it must have landed
        cp_async_wait();
        __syncwarp();
        cn = other->c;
        more = next;
      }
      if (on) {
        const size_t s = c0 + u * T;
        if (s + T > st.nslots) {  // the stream's zero padding adds nothing, whatever X holds
#pragma unroll
          for (int i = 0; i < T; i++)
            if (s + i >= st.nslots) {
#pragma unroll
              for (int w = 0; w < W; w++) xv[i][w] = 0.0;
            }
        }
#pragma unroll
        for (int i0 = 0; i0 < T; i0 += 4) {
          VT v[4];
          UIN c[4];
          if constexpr (V == 2) {
            const double2 t0 = *reinterpret_cast<const double2 *>(cur->v + u * T + i0);
            const double2 t1 = *reinterpret_cast<const double2 *>(cur->v + u * T + i0 + 2);
            v[0] = t0.x, v[1] = t0.y, v[2] = t1.x, v[3] = t1.y;
          } else {
            const float4 t = *reinterpret_cast<const float4 *>(cur->v + u * T + i0);
            v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
          }
          {
            const uint4 t = *reinterpret_cast<const uint4 *>(cn + i0);  // stale past the part's end: not used
            c[0] = t.x, c[1] = t.y, c[2] = t.z, c[3] = t.w;
          }
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (hs & 1u) {  // a row starts here: the open run ends (the part's first one, maybe empty, as a record)
              st_y<W, VEC>(ydst, ncol, acc);
              row++;
              first = false;
              ydst = o.rowmap ? yb + (size_t)o.rowmap[row] * o.k : yb + (size_t)row * o.k;
#pragma unroll
              for (int w = 0; w < W; w++) acc[w] = 0.0;
            }
            hs >>= 1;
#pragma unroll
            for (int w = 0; w < W; w++) acc[w] = fma((double)v[i], xv[i0 + i][w], acc[w]);
            if (more && (i % 4) == 3) {
#pragma unroll
              for (int e = 0; e < 4; e++) ld_x<W, VEC>(x_row(c[i - 3 + e]), ncol, xv[i0 + i - 3 + e]);
            }
          }
        }
      }
    }
    __syncwarp();  // the chunk is read: its buffer may be filled again
  }
  // Join the rows that cross parts of this CTA.  flag of a part: it starts
  // with a row (1), no row starts in it (2).
  constexpr int CG = 8 * NG;  // parts of a CTA
  __shared__ unsigned char flag[CG];
  const unsigned gi = (threadIdx.x >> 5) * NG + grp;
  if (has && first) st_y<W, VEC>(head, ncol, acc);
  if (jl == 0) flag[gi] = (a_head ? 1 : 0) | (first ? 2 : 0);
  __syncthreads();  // the CTA's heads and flags are written
  const unsigned live = (unsigned)min((size_t)CG, nparts - (size_t)blockIdx.x * CG);
  // adds to acc what the following parts hold of the row open at part i's
  // end; true if the row ends in this CTA
  auto follow = [&](unsigned i) {
    for (unsigned j = i + 1; j < live; j++) {
      const unsigned char f = flag[j];
      if (f & 1u) return true;
      const double *h = o.head + ((size_t)blockIdx.x * CG + j) * CB + jl * W;
#pragma unroll
      for (int w = 0; w < W; w++)
        if (VEC ? ncol > 0 : w < ncol) acc[w] += h[w];
      if (!(f & 2u)) return true;
    }
    return false;
  };
  if (!has) return;
  const size_t r2 = 2 * (size_t)blockIdx.x;
  bool tail = false;  // the CTA's last run is mine, and goes to its tail record
  if (!first) {
    if (follow(gi)) {
      st_y<W, VEC>(ydst, ncol, acc);
    } else {
      tail = true;
      st_y<W, VEC>(o.rec_sum + (r2 + 1) * CB + jl * W, ncol, acc);
    }
  }
  if (tail && jl == 0) o.rec_row[r2 + 1] = row;
  if (gi == 0) {
    // the CTA's head record: the run open at its start; no tail if that run never ends
    bool whole = false;
    if (!a_head) {
#pragma unroll
      for (int w = 0; w < W; w++) acc[w] = (VEC ? ncol > 0 : w < ncol) ? head[w] : 0.0;
      if (first) whole = !follow(0);
      st_y<W, VEC>(o.rec_sum + r2 * CB + jl * W, ncol, acc);
    }
    if (jl == 0) {
      o.rec_row[r2] = row_a;
      if (whole) o.rec_row[r2 + 1] = NO_ROW;
    }
  }
}

// Record i (of 2 per CTA) writes its row if it is that row's last record,
// adding the row's earlier records; rows with no slot get zeros.  A
// programmatic dependent of the main kernel.
template <int CB>  // columns of one pass
__global__ void spmm_fixup(size_t nrec, const UIN *__restrict__ empty, size_t nempty, Out o) {
  pdl_wait();
  const UIN *rec_row = after_wait((const UIN *)o.rec_row);
  const double *rec_sum = after_wait((const double *)o.rec_sum);
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t i = t / CB;
  const unsigned j = t % CB;
  if (j >= o.kb) return;
  if (i < nempty) o.Y[(size_t)empty[i] * o.k + o.j0 + j] = 0.0;
  if (i >= nrec) return;
  const UIN r = rec_row[i];
  if (r == NO_ROW) return;
  size_t q = i + 1;
  while (q < nrec && rec_row[q] == NO_ROW) q++;
  if (q < nrec && rec_row[q] == r) return;
  double total = rec_sum[i * CB + j];
  for (size_t m = i; m-- > 0;) {
    const UIN rm = rec_row[m];
    if (rm == NO_ROW) continue;
    if (rm != r) break;
    total += rec_sum[m * CB + j];
  }
  o.Y[(size_t)real_row(o, r) * o.k + o.j0 + j] = total;
}

}  // namespace mm
}  // namespace ispmv
