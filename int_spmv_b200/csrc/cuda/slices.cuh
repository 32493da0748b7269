// slices.cuh - SpMV over slices of 32 rows, 16-bit column deltas.
//
// For matrices whose neighbouring rows are about equally long (a stencil on a
// grid).  A warp takes 32 consecutive rows, lane = row; element k of the 32
// rows lies side by side (val and d16 at 32*(off + k) + lane, column base +
// d16).  Neighbouring rows' k-th columns are neighbours too, so a gather
// touches two or three lines where the slot stream's (16 slots of a row per
// lane) touches about twelve and is bound by them; there is no row reduction
// and no record, and FP32 values round x as they use it (the same product):
// one launch where the slot stream needs three.
//
// Bound by latency and L1 capacity: of 27 elements a row, U = 9 are loaded
// and then gathered together (14 or 27 hold more lines than L1 keeps: 60-100
// us).  27-point stencil, 101^3: FP32 values 44.5 us by the slot stream, 38.2
// so (28.5 at the copy rate); FP64 values 65.7 and 49.8 (45.0).  At small sizes the
// two launches saved count: 40^3 8.2 us, 5-point 800^2 9.0.  Slices staged by
// bulk copies into shared memory take L1 from the gathers and were no faster.
#pragma once
#include <type_traits>

#include "plan_kernels.cuh"

namespace ispmv {
namespace sl {

// meta[s] = {off, base} of slice s, meta[nslices].x = the end; len: row
// lengths.  U elements of a row at a time: 9, or 5 where no row is longer (the
// loads of a remainder wait on one another's tests).
template <typename VT, int U>
__global__ void __launch_bounds__(pk::TPB, sizeof(VT) == 8 ? 4 : 5)
    slice_rows(UIN n, UIN nslices, const uint2 *__restrict__ meta, const uint8_t *__restrict__ len,
               const uint16_t *__restrict__ d16, const VT *__restrict__ val, const FPT *x, FPT *y_, int beta) {
  pdl_trigger();
  const UIN s = blockIdx.x * (pk::TPB / 32) + (threadIdx.x >> 5);
  if (s >= nslices) return;
  const unsigned lane = threadIdx.x & 31u;
  const uint2 m = __ldg(meta + s);
  const UIN w = __ldg(&meta[s + 1].x) - m.x;
  const UIN r = s * 32u + lane;
  const UIN l = r < n ? (UIN)__ldg(len + r) : 0u;
  const bool full = __all_sync(FULL, l == w);
  pdl_wait();
  const FPT *const xb = after_wait(x + m.y);
  FPT *const y = after_wait(y_);
  size_t p = (size_t)m.x * 32 + lane;
  double acc = 0.0;
  auto elements = [&](UIN k0, auto rest_c) {
    constexpr bool REST = decltype(rest_c)::value;
    VT v[U];
    UIN c[U];
    double xv[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (!REST || k0 + u < w) {
        c[u] = ld_stream(d16 + p + 32 * u);
        v[u] = ld_stream(val + p + 32 * u);
      }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (!REST || k0 + u < w) xv[u] = xb[c[u]];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (!REST || k0 + u < w) {
        if (!full && k0 + u >= l) xv[u] = 0.0;  // padding (the base column) adds nothing, whatever x holds
        acc = pk::fmac<VT>(v[u], xv[u], acc);
      }
  };
  UIN k0 = 0;
  for (; k0 + U <= w; k0 += U, p += U * 32) elements(k0, std::false_type{});
  if (k0 < w) elements(k0, std::true_type{});
  if (r < n) y[r] = beta ? acc + y[r] : acc;
}

}  // namespace sl
}  // namespace ispmv
