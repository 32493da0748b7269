// plan_kernels.cuh - sm_100a SpMV kernels of the plan layer (fresh x per
// call, gathered through the read-only path / L2; values and columns are
// streamed once with evict-first loads).
//
// VT is the stored value type (double, or float for the reduced-byte form:
// FP32 multiply, FP64 accumulation).
#pragma once
#include "seg_engine.cuh"

namespace ispmv {
namespace pk {

constexpr int TPB = 256;

template <typename VT>
__device__ __forceinline__ double prod(VT v, double x);
template <>
__device__ __forceinline__ double prod<double>(double v, double x) { return v * x; }
template <>
__device__ __forceinline__ double prod<float>(float v, double x) { return (double)(v * __double2float_rn(x)); }

template <typename VT>
__device__ __forceinline__ double fmac(VT v, double x, double acc);
template <>
__device__ __forceinline__ double fmac<double>(double v, double x, double acc) { return fma(v, x, acc); }
template <>
__device__ __forceinline__ double fmac<float>(float v, double x, double acc) {
  return acc + (double)(v * __double2float_rn(x));
}

// ---------------------------------------------------------------- CSR --
// Vector CSR ("naive" CSR on the GPU): L lanes per row, shuffle reduction,
// overwrite / accumulate y.
template <typename VT, int L>
__global__ void __launch_bounds__(TPB) csr_vec(UIN n, const UIN *__restrict__ row, const UIN *__restrict__ col,
                                               const VT *__restrict__ val, const FPT *__restrict__ x,
                                               FPT *__restrict__ y, int beta) {
  const unsigned sub = threadIdx.x & (L - 1);
  const size_t r = ((size_t)blockIdx.x * TPB + threadIdx.x) / L;
  const bool live = r < n;
  double s = 0.0;
  if (live) {
    const UIN b = row[r], e = row[r + 1];
    for (UIN j = b + sub; j < e; j += L) s = fmac<VT>(ld_stream(val + j), ldg(x + ld_stream(col + j)), s);
  }
#pragma unroll
  for (int d = L / 2; d > 0; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
  if (live && sub == 0) y[r] = beta ? s + y[r] : s;
}

// ---------------------------------------------------------------- AXC --
// 8 lanes per row, one 8-value brick per step (the reference's row loop,
// M:711-732, with x gathered from the column companion).
template <typename VT>
__global__ void __launch_bounds__(TPB) axc_rows(UIN n, const UIN *__restrict__ bptr, const UIN *__restrict__ col,
                                                const VT *__restrict__ val, const FPT *__restrict__ x,
                                                FPT *__restrict__ y, int beta) {
  const unsigned k = threadIdx.x & 7u;
  const size_t r = ((size_t)blockIdx.x * TPB + threadIdx.x) >> 3;
  const bool live = r < n;
  double s = 0.0;
  if (live) {
    const size_t b = (size_t)bptr[r] * 8, e = (size_t)bptr[r + 1] * 8;
    for (size_t p = b + k; p < e; p += 8) s = fmac<VT>(ld_stream(val + p), ldg(x + ld_stream(col + p)), s);
  }
  s += __shfl_xor_sync(FULL, s, 4);
  s += __shfl_xor_sync(FULL, s, 2);
  s += __shfl_xor_sync(FULL, s, 1);
  if (live && k == 0) y[r] = beta ? s + y[r] : s;
}

// ----------------------------------------------------------------- K1 --
// K1 orders rows by length (descending), so a chunk's rows are unrelated
// rows of the matrix and nearly every gather misses the lines its
// neighbours touched: the gathers (one L1 tag lookup each) bound the kernel,
// as long as no chunk is one thread group's serial chain.  The chunks' column
// counts nmc never increase, so three prefixes of the chunks get as many
// lanes as their length pays for:
//   chunks [0, ncta), at least K1_CTA columns: a CTA each, its 32 groups of 8
//     lanes take every 32nd column pair, sums joined in shared memory;
//   chunks [ncta, nlong), at least K1_LONG columns: a warp each, 4 groups;
//   the rest: 4 chunks to a warp, one group each.
// A group reads two columns of its chunk at once: lane l holds rows 2(l%4)
// and 2(l%4)+1 of column parity l/4, so a value load is 128 contiguous bytes
// per group (16 B per lane) and touches half the lines one column per load
// would.  Each lane keeps K1_U pairs of loads, then their 2*K1_U gathers, in
// flight, in the remainder of a chunk too (predicated, not one after the
// other).  SCATTER writes y[permi] (K1 with integrated reordering), else res
// in chunk order (then k1_order).  Measured on power-law rows (n = 1M, 14.9M
// nonzeros, longest row 1,100-3,000, FP64, K1p): 147.7 us with the long
// chunks on one warp each and the remainders serial, 64.0 us so; the L1's one
// tag lookup per gather and cycle alone takes 52 us.
constexpr UIN K1_LONG = 64;   // columns from which a chunk gets a warp
constexpr UIN K1_CTA = 256;   // columns from which a chunk gets a CTA
constexpr int K1_U = 4;       // column pairs in flight per lane

__device__ __forceinline__ double2 ld_pair(const double *p) { return ld_stream(reinterpret_cast<const double2 *>(p)); }
__device__ __forceinline__ float2 ld_pair(const float *p) { return ld_stream(reinterpret_cast<const float2 *>(p)); }

// Sums of this lane's two rows over the column pairs kp0, kp0 + stride, ...
// of a chunk of m columns at slot `off`.
template <typename VT, int STRIDE>
__device__ __forceinline__ double2 k1_sum(const VT *__restrict__ val, const UIN *__restrict__ col,
                                          const FPT *x, size_t off, UIN kp0, UIN m, unsigned lane8) {
  using V2 = decltype(ld_pair((const VT *)nullptr));
  double a0[K1_U], a1[K1_U];
#pragma unroll
  for (int u = 0; u < K1_U; u++) a0[u] = a1[u] = 0.0;
  const UIN np = m / 2 + (m & ((lane8 >> 2) ^ 1u));  // pairs whose column of my parity exists
  const size_t base = off + 2u * lane8;
  UIN k = kp0;
  for (; (uint64_t)k + (K1_U - 1) * STRIDE < np; k += K1_U * STRIDE) {
    V2 v[K1_U];
    uint2 c[K1_U];
#pragma unroll
    for (int u = 0; u < K1_U; u++) {
      const size_t p = base + (size_t)16 * (k + (UIN)(u * STRIDE));
      v[u] = ld_pair(val + p);
      c[u] = ld_stream(reinterpret_cast<const uint2 *>(col + p));
    }
    double x0[K1_U], x1[K1_U];
#pragma unroll
    for (int u = 0; u < K1_U; u++) {
      x0[u] = x[c[u].x];
      x1[u] = x[c[u].y];
    }
#pragma unroll
    for (int u = 0; u < K1_U; u++) {
      a0[u] = fmac<VT>(v[u].x, x0[u], a0[u]);
      a1[u] = fmac<VT>(v[u].y, x1[u], a1[u]);
    }
  }
  if (k < np) {  // the remainder: at most K1_U - 1 pairs, in flight together
    V2 v[K1_U - 1];
    uint2 c[K1_U - 1];
    double x0[K1_U - 1], x1[K1_U - 1];
#pragma unroll
    for (int u = 0; u < K1_U - 1; u++) {
      const UIN kk = k + (UIN)(u * STRIDE);
      if (kk < np) {
        const size_t p = base + (size_t)16 * kk;
        v[u] = ld_pair(val + p);
        c[u] = ld_stream(reinterpret_cast<const uint2 *>(col + p));
      }
    }
#pragma unroll
    for (int u = 0; u < K1_U - 1; u++) {
      if (k + (UIN)(u * STRIDE) < np) {
        x0[u] = x[c[u].x];
        x1[u] = x[c[u].y];
      }
    }
#pragma unroll
    for (int u = 0; u < K1_U - 1; u++) {
      if (k + (UIN)(u * STRIDE) < np) {
        a0[u] = fmac<VT>(v[u].x, x0[u], a0[u]);
        a1[u] = fmac<VT>(v[u].y, x1[u], a1[u]);
      }
    }
  }
  return make_double2((a0[0] + a0[1]) + (a0[2] + a0[3]), (a1[0] + a1[1]) + (a1[2] + a1[3]));
}

template <typename VT, bool SCATTER>
__global__ void __launch_bounds__(TPB) k1_chunks(UIN n, UIN chunkNum, UIN ncta, UIN nlong,
                                                 const UIN *__restrict__ chp, const UIN *__restrict__ nmc,
                                                 const UIN *__restrict__ permi, const UIN *__restrict__ col,
                                                 const VT *__restrict__ val, const FPT *x_, FPT *out_, int beta) {
  pdl_trigger();
  pdl_wait();  // the launch before this one wrote x, or still reads or writes out
  const FPT *x = after_wait(x_);
  FPT *out = after_wait(out_);
  __shared__ double2 part[TPB / 32][4];
  const unsigned lane = threadIdx.x & 31u, lane8 = lane & 7u, wib = threadIdx.x >> 5;
  size_t c;
  double2 s;
  if (blockIdx.x < ncta) {  // one CTA per chunk (the whole CTA takes this branch)
    c = blockIdx.x;
    s = k1_sum<VT, TPB / 8>(val, col, x, chp[c], threadIdx.x >> 3, nmc[c], lane8);
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) {  // column parities and groups: lanes of the same rows
      s.x += __shfl_xor_sync(FULL, s.x, d);
      s.y += __shfl_xor_sync(FULL, s.y, d);
    }
    if (lane < 4) part[wib][lane] = s;
    __syncthreads();
    if (threadIdx.x >= 4) return;
    s = part[0][lane];
#pragma unroll
    for (int w = 1; w < TPB / 32; w++) {
      s.x += part[w][lane].x;
      s.y += part[w][lane].y;
    }
  } else {
    const size_t w = (size_t)(blockIdx.x - ncta) * (TPB / 32) + wib;
    if (w < nlong - ncta) {  // one warp per chunk: group g takes pairs g, g + 4, ...
      c = ncta + w;
      s = k1_sum<VT, 4>(val, col, x, chp[c], lane >> 3, nmc[c], lane8);
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) {
        s.x += __shfl_xor_sync(FULL, s.x, d);
        s.y += __shfl_xor_sync(FULL, s.y, d);
      }
      if (lane >= 4) return;
    } else {
      c = nlong + (w - (nlong - ncta)) * 4 + (lane >> 3);
      const bool live = c < chunkNum;
      s = live ? k1_sum<VT, 1>(val, col, x, chp[c], 0, nmc[c], lane8) : make_double2(0.0, 0.0);
      s.x += __shfl_xor_sync(FULL, s.x, 4);
      s.y += __shfl_xor_sync(FULL, s.y, 4);
      if (!live || lane8 >= 4) return;
    }
  }
  const size_t i = c * 8 + 2u * (lane8 & 3u);  // my rows: i, i + 1
  if (SCATTER) {
    if (i < n) {
      const UIN r = permi[i];
      out[r] = beta ? s.x + out[r] : s.x;
    }
    if (i + 1 < n) {
      const UIN r = permi[i + 1];
      out[r] = beta ? s.y + out[r] : s.y;
    }
  } else {
    *reinterpret_cast<double2 *>(out + i) = s;  // chunk-order scratch of chunkNum * 8 entries
  }
}

// CTAs of a K1 launch: one per CTA chunk, then warps: one per long chunk,
// one per 4 other chunks.
inline size_t k1_ctas(UIN chunkNum, UIN ncta, UIN nlong) {
  const size_t warps = (size_t)(nlong - ncta) + ((size_t)(chunkNum - nlong) + 3) / 4;
  return ncta + (warps + TPB / 32 - 1) / (TPB / 32);
}

// K1's reorder (orderArrayK1): y in original row order from the chunk-order
// result; a programmatic dependent launch of k1_chunks where the stream
// allows it, so it first waits for that grid and its writes.
__global__ void k1_order(UIN n, const UIN *__restrict__ permi, const FPT *res_, FPT *y_, int beta) {
  pdl_trigger();
  pdl_wait();
  const FPT *res = after_wait(res_);
  FPT *y = after_wait(y_);
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const UIN r = permi[i];
    y[r] = beta ? res[i] + y[r] : res[i];
  }
}

// ------------------------------------------------------- AXT NOC, th>1 --
// Unit = tile column of th slots (row id: sec[8*T + c]).  th % 4 == 0: each
// step the warp loads 4 consecutive sub-rows of a tile (32 consecutive
// slots), adds them per column, and after th/4 steps reduces the 4 partials
// of each column with 2 shuffles; 4 tiles make a batch of 32 columns.
// Bound by its gathers' latency: 6 CTAs per SM (40 registers); at the 48 the
// compiler takes otherwise 5 fit, and power-law n = 4M takes 413.6 us for 360.1
// (tileH 4; tileH 8 394.3 for 347.5; n = 1M 129 for 133).
template <typename VT>
__global__ void __launch_bounds__(TPB, 6) noc_hn(size_t nunits, size_t nseg, UIN th, UIN useg, const UIN *__restrict__ urow,
                                              const UIN *__restrict__ col, const VT *__restrict__ val,
                                              const FPT *__restrict__ x, seg::Out o) {
  pdl_trigger();
  const unsigned lane = threadIdx.x & 31u;
  const size_t segid = ((size_t)blockIdx.x * TPB + threadIdx.x) >> 5;
  if (segid >= nseg) return;
  const size_t u0 = segid * useg;  // useg is a multiple of 32 (4 tiles)
  const size_t u1 = min(u0 + useg, nunits);
  seg::State st{NO_ROW, 0.0, false};
  const size_t tslots = (size_t)th * 8;
  for (size_t ub = u0; ub < u1; ub += 32) {
    double mine = 0.0;
    for (int tt = 0; tt < 4; tt++) {
      const size_t T = ub / 8 + tt;
      double p = 0.0;
      if (T * 8 < u1) {
        const size_t base = T * tslots + lane;
        if (th % 4 == 0) {
          for (UIN R = 0; R < th; R += 4) {
            const size_t q = base + (size_t)R * 8;
            p = fmac<VT>(ld_stream(val + q), ldg(x + ld_stream(col + q)), p);
          }
        } else {
          // generic tileH: lane = (group g = lane/8, column c): sub-rows g, g+4, ...
          for (UIN R = lane >> 3; R < th; R += 4) {
            const size_t q = T * tslots + (size_t)R * 8 + (lane & 7u);
            p = fmac<VT>(ld_stream(val + q), ldg(x + ld_stream(col + q)), p);
          }
        }
      }
      p += __shfl_xor_sync(FULL, p, 8);
      p += __shfl_xor_sync(FULL, p, 16);
      if ((lane >> 3) == (unsigned)tt) mine = p;
    }
    const size_t u = ub + lane;
    const bool live = u < u1;
    const UIN r = live ? urow[u] : NO_ROW;
    seg::batch(mine, r, live, st, o, segid);
  }
  seg::finish(st, o, segid);
}

}  // namespace pk
}  // namespace ispmv
