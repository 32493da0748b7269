// plan.cu - plans: a format uploaded once to HBM as a value stream and a
// column-index stream plus the format's row structure, then y = A*x +
// beta*y for a fresh x on every call.
//
// Device layouts (slot streams in the reference format's own slot order; the
// x halves of `ax` are dropped and the column companion takes their place):
//   stream  CSR / AXT COM (CSR order), AXT NOC tileH=1 (tile order, rows
//           padded to 8) and AXC (brick order, rows padded to 8): val[S],
//           col[S] zero-padded to a multiple of 512 slots, a row-start bitmap
//           (1 bit per slot), per-segment start counts, and the compressed ->
//           real row map when some rows are empty.  Kernels: sss::stream_ldg,
//           sss::stream_tma; wide::stream_wide reads val/col from a
//           lane-interleaved copy (wide::il_pos) instead of slot order.
//   units   AXT NOC tileH>1 (tile columns): val/col in tile order plus the
//           reference's per-column row array (sec) cut to the used columns.
//           Kernels: pk::noc_hn, tk::nocn_tma.
//   rows    CSR row pointer (pk::csr_vec) and AXC brick pointer
//           (pk::axc_rows): the row-parallel kernels.
//   K1      val/col column-major per chunk, chp, nmc, permi (pk::k1_chunks).
//   slices  16-bit-delta plans of equally long neighbouring rows: 32 rows side
//           by side, values and deltas per element, row lengths
//           (sl::slice_rows).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include <cub/device/device_scan.cuh>

#include "plan_tma.cuh"
#include "slices.cuh"
#include "spmm.cuh"
#include "sss.cuh"
#include "tmem.cuh"
#include "wide.cuh"

using namespace ispmv;

enum PlanFormat { F_CSR = 0, F_AXC = 1, F_K1 = 2, F_K1P = 3, F_AXT_NOC = 4, F_AXT_COM = 5 };
enum PlanPath { P_STREAM = 0, P_UNITS = 1, P_ROWS = 2, P_K1 = 3, P_SLICES = 4 };

struct ispmv_plan_s {
  int fmt = 0;
  int path = P_STREAM;
  ispmv_plan_opts opts{};
  UIN n = 0, nnz = 0, th = 1, bs = 0, lanes = 8;
  size_t slots = 0, slots_pad = 0, nunits = 0;
  bool alone = false;   // ispmv_plan_time_main: launches wait for one another
  bool no_win = false;  // staged variants: empty x windows
  bool chosen = false;  // kernel and variant by AUTO
  bool long_rows = false;  // stream and unit plans: a row of more than seg::FIX_LONG segments (seg::fixup's form)
  uint2 *slices = nullptr;  // P_SLICES: first element column and base column of each slice, and the end
  uint8_t *slen = nullptr;  // P_SLICES: row lengths
  UIN slice_w = 0;          // P_SLICES: the widest slice
  size_t fslots = 0;  // the format's slots, padding included (stream path: slots holds none)
  size_t seg_slots = 0, nseg = 0;
  UIN useg = 0;
  void *val = nullptr;  // double or float
  UIN *col = nullptr;
  UIN *rows = nullptr;  // row / brick pointer, or unit rows
  UIN *heads = nullptr, *segh = nullptr, *rowmap = nullptr, *empty = nullptr;
  size_t nempty = 0;
  size_t nrowmap = 0;   // entries of rowmap (0: no empty rows, no map)
  UIN *chp = nullptr, *nmc = nullptr, *permi = nullptr;
  UIN chunkNum = 0;
  FPT *res = nullptr;  // K1 result in chunk order
  UIN *rec_row = nullptr;
  double *rec_sum = nullptr;
  int *status = nullptr;
  sss::Narrow narrow{};   // D16 / LO side streams (stream path only)
  sss::XWin xw{};         // x bands staged in shared memory (variants >= 8)
  double lo_frac = 0.0;   // fraction of slots carrying a lo-word
  size_t esc_batches = 0; // D16 batches kept as u32 columns
  size_t d16_batch = 128;  // D16 slots per base column (128; 32*slots per lane for stream_wide)
  FPT *hx = nullptr, *hy = nullptr;  // device staging of ispmv_plan_spmv_host
  float *x32 = nullptr;              // FP32 copy of x (FP32-value stream_wide plans)
  cudaTextureObject_t xtex = 0;      // linear texture over x (stream_wide texture-gather variants)
  const void *xtex_src = nullptr;    // the buffer it covers
  size_t xtex_bytes = 0;
  uint32_t *tblocks = nullptr;       // the stream in TMEM-staged blocks (stream_tmem variants)
  unsigned long long *queue = nullptr;  // work-queue counter (variant ISPMV_VARIANT_QUEUE)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  const FPT *g_x = nullptr;
  FPT *g_y = nullptr;
  int g_beta = -1;
  UIN *mm_row = nullptr;             // SpMM records (allocated on first use)
  double *mm_sum = nullptr;
  size_t mm_cap = 0;                 // doubles in mm_sum
  size_t mm_rows_cap = 0;            // entries of mm_row
  UIN k1_cta = 0, k1_long = 0;       // K1: chunks [0, k1_cta) a CTA each, [k1_cta, k1_long) a warp each
  std::vector<void *> owned;
  ispmv_plan_info info{};
  std::vector<cudaEvent_t> tev;      // kernel timing: event pairs around the main kernel (a ring)
  size_t tcap = 0;                   // pairs in the ring (0: timing off)
  size_t tcount = 0;                 // pairs recorded since the last read
  bool capturing = false;            // inside graph capture: no timing events
  const char *kname = "";            // main kernel of the latest product (a static string)
};

namespace {

constexpr size_t SS = sss::SS;      // slots per staged stage; streams pad to it
constexpr size_t SEG_SLOTS = 2048;  // default slots per warp segment

#define TRY(expr)        \
  do {                   \
    int s__ = (expr);    \
    if (s__) return s__; \
  } while (0)

template <typename T>
int dev_upload(ispmv_plan_s *p, const T *h, size_t n, T **d) {
  void *ptr = nullptr;
  TRY(pool_alloc(&ptr, (n ? n : 1) * sizeof(T)));
  p->owned.push_back(ptr);
  if (n && h) ISPMV_TRY(cudaMemcpy(ptr, h, n * sizeof(T), cudaMemcpyHostToDevice));
  *d = static_cast<T *>(ptr);
  return ISPMV_OK;
}
template <typename T>
int dev_alloc(ispmv_plan_s *p, size_t n, T **d) {
  return dev_upload<T>(p, nullptr, n, d);
}

size_t vbytes(const ispmv_plan_s *p) { return p->opts.val_kind == ISPMV_VAL_F64 ? 8 : 4; }

// The reduced-byte side streams exist only on the slot-stream path.
bool narrow_kinds(const ispmv_plan_s *p) {
  return p->opts.val_kind == ISPMV_VAL_F32_LO16 || p->opts.col_kind == ISPMV_COL_D16;
}

uint16_t to_bf16(float f) {  // round to nearest even
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

int upload_values(ispmv_plan_s *p, const std::vector<double> &v) {
  if (p->opts.val_kind == ISPMV_VAL_F64) {
    double *d;
    TRY(dev_upload(p, v.data(), v.size(), &d));
    p->val = d;
    return ISPMV_OK;
  }
  // FP32 (and the hi part of FP32 + lo-word)
  std::vector<float> f(v.size());
  for (size_t i = 0; i < v.size(); i++) f[i] = (float)v[i];
  float *d;
  TRY(dev_upload(p, f.data(), f.size(), &d));
  p->val = d;
  return ISPMV_OK;
}

void finish_info(ispmv_plan_s *p, const char *name) {
  ispmv_plan_info &i = p->info;
  i.nrows = p->n;
  i.nnz = p->nnz;
  i.slots = p->path == P_STREAM || p->path == P_SLICES ? p->fslots : p->slots;
  i.format = p->fmt;
  i.val_kind = p->opts.val_kind;
  i.col_kind = p->opts.col_kind;
  i.kernel = p->opts.kernel;
  i.tile_h = p->th;
  i.bs = p->bs;
  // b_val: 8 | 4 | 4 + 2*(lo-word fraction); b_idx: 4 | 2 + 4*(batch bases + escaped columns)/nnz
  double bv = (double)vbytes(p), bi = 4.0;
  if (p->opts.val_kind == ISPMV_VAL_F32_LO16) bv = 4.0 + 2.0 * p->lo_frac;
  if (p->opts.col_kind == ISPMV_COL_D16 && p->slots_pad) {
    const double B = (double)p->d16_batch, batches = (double)(p->slots_pad / p->d16_batch);
    bi = 2.0 + (4.0 * batches + B * 4.0 * (double)p->esc_batches) / std::max(1.0, (double)p->nnz);
  }
  if (p->path == P_SLICES) bi = 2.0 + (8.0 * ((p->n + 31) / 32) + (double)p->n) / std::max(1.0, (double)p->nnz);
  i.alg_bytes = (double)p->nnz * (bv + bi) + (double)p->n * 16.0 + 4.0 * ((double)p->n + 1.0);
  snprintf(i.name, sizeof i.name, "%s", name);
}

int check_csr(const str_matCSR *csr) {
  if (!csr || !csr->row || csr->nrows == 0) return ISPMV_ERR_ARG;
  if (csr->nnz && (!csr->col || !csr->val)) return ISPMV_ERR_ARG;
  if (csr->row[0] != 0 || csr->row[csr->nrows] != csr->nnz) return ISPMV_ERR_ARG;
  return ISPMV_OK;
}

int begin(const ispmv_plan_opts *o, ispmv_plan_s **out) {
  if (!out) return ISPMV_ERR_ARG;
  *out = nullptr;
  auto *p = new (std::nothrow) ispmv_plan_s();
  if (!p) return ISPMV_ERR_OOM;
  if (o) p->opts = *o;
  else ispmv_plan_opts_default(&p->opts);
  if (p->opts.val_kind < ISPMV_VAL_F64 || p->opts.val_kind > ISPMV_VAL_F32_LO16 || p->opts.col_kind < ISPMV_COL_U32 ||
      p->opts.col_kind > ISPMV_COL_D16 || p->opts.kernel < 0 || p->opts.kernel > ISPMV_KERNEL_WIDE ||
      (p->opts.spmm_kernel != ISPMV_KERNEL_AUTO && p->opts.spmm_kernel != ISPMV_KERNEL_LDG &&
       p->opts.spmm_kernel != ISPMV_KERNEL_WIDE)) {
    delete p;
    return ISPMV_ERR_UNSUPPORTED;
  }
  *out = p;
  return ISPMV_OK;
}

// A host builder's copies are waited for here (a small copy from pageable
// memory may return before it has reached the device): products run on any
// stream, and read the plan's arrays before they wait for the launches before
// them.  `waited`: the builder has waited for its own stream.
int done(ispmv_plan_s *p, int st, ispmv_plan *out, bool waited = false) {
  if (st == ISPMV_OK && !waited) {
    const cudaError_t e = cudaStreamSynchronize(nullptr);
    if (e != cudaSuccess) st = cuda_status(e, "cudaStreamSynchronize");
  }
  if (st != ISPMV_OK) {
    ispmv_plan_destroy(p);
    return st;
  }
  *out = p;
  return ISPMV_OK;
}

// The list of empty rows, and whether a row spans many segments.
int empty_rows(ispmv_plan_s *p, const str_matCSR *csr) {
  std::vector<UIN> e;
  for (UIN r = 0; r < csr->nrows; r++) {
    const UIN l = csr->row[r + 1] - csr->row[r];
    if (!l) e.push_back(r);
    if (l > seg::FIX_LONG * p->seg_slots) p->long_rows = true;
  }
  p->nempty = e.size();
  if (!e.empty()) TRY(dev_upload(p, e.data(), e.size(), &p->empty));
  return ISPMV_OK;
}

// The work areas of a stream or unit plan, set on `s`.
int alloc_records(ispmv_plan_s *p, cudaStream_t s = nullptr) {
  const size_t nrec = std::max<size_t>(1, 2 * p->nseg);
  TRY(dev_alloc(p, nrec, &p->rec_row));
  TRY(dev_alloc(p, nrec, &p->rec_sum));
  TRY(dev_alloc(p, 1, &p->status));
  // no row: a staged kernel that gives up a wait leaves records unwritten,
  // which the fix-up reads all the same
  ISPMV_TRY(cudaMemsetAsync(p->rec_row, 0xFF, nrec * sizeof(UIN), s));
  ISPMV_TRY(cudaMemsetAsync(p->status, 0, sizeof(int), s));
  TRY(dev_alloc(p, 1, &p->queue));
  return ISPMV_OK;
}

size_t seg_slots_of(const ispmv_plan_s *p, size_t upu) {
  if (p->opts.units_per_warp <= 0) return SEG_SLOTS;
  return std::max(SS, ((size_t)p->opts.units_per_warp * upu + SS - 1) / SS * SS);
}

// stream_wide variants, numbered as measured (numbers not listed here were
// measured and retired: x bands in shared memory, per-warp row buffers,
// other segment sizes, stage counts and window sizes):
// slots per lane, per-CTA x window (cap doubles), segment slots (at most:
// wide_seg), CTAs per SM
// the registers are sized for (plain loads), and for the staged form (tma)
// the stages per warp and warps per CTA.
struct WideCfg {
  int spl; UIN cap; size_t seg; int minb; bool tma; int stages; int warps; bool tex = false;
  bool tmem = false;  // stream staged through tensor memory (stream_tmem); stages = TMEM stages,
                      // warps = consumer warps per CTA (4 per column half)
  bool stg = false;   // one x window per CTA (cap doubles), chosen at plan time, copied by one bulk copy
  bool pfc = false;   // the next batch's columns loaded one batch ahead
  bool ok = true;     // a variant this build runs
};
constexpr int WIDE_WARPS = 8;
WideCfg wide_variant(int v) {
  switch (v) {
    case 0: return {16, 0, 4096, 3, false, 0, 8};
    case 4: return {8, 0, 2048, 4, false, 0, 8};
    case 8: return {16, 0, 8192, 3, false, 0, 8};
    case 9: return {16, 0, 2048, 3, false, 0, 8};
    case 11: return {16, 0, 4096, 0, true, 2, 4};                            // bulk-copy staged stream
    case 16: return {8, 0, 2048, 4, false, 0, 8, true};                      // texture gathers
    case 18: return {8, 0, 8192, 0, false, 4, 4, false, true};               // TMEM-staged stream
    case 19: return {16, 0, 8192, 0, false, 2, 4, false, true};
    case 20: return {8, 0, 8192, 0, false, 2, 8, false, true};
    case 21: return {16, 0, 8192, 0, false, 2, 8, false, true};
    case 26: return {8, 3584, 1536, 4, false, 0, 8, false, false, true};     // per-CTA x window, one bulk copy
    case 32: return {8, 0, 2048, 4, false, 0, 8, false, false, false, true}; // next batch's columns ahead
    default: {
      WideCfg c{16, 0, 4096, 3, false, 0, 8};
      c.ok = false;
      return c;
    }
  }
}

// Slots per warp segment of a lane-interleaved plan of `slots` slots: the
// variant's segment at most, and short enough that the warps fill the GPU.  A
// warp works its batches of 32*spl slots one after the other, about 1.5 us
// each when little else runs, so a matrix below one full load of warps (as
// many as the GPU holds at once) takes the time of its longest warp, and one
// a little above a whole number of loads pays for the next one: 1.24 loads of
// 3072 slots take 30.9 us where 0.93 of 4096 take 25.6 and 1.85 of 2048 26.9
// (27-point stencil, 80^3, FP32 values).  The longest segments whose last load
// is at least 0.9 full are taken, else the ones that fill it best; beyond
// three loads the last one hardly shows.  The bulk-copy staged kernel's
// persistent warps take segments in turn, 8 or more each.  Measured against
// the variants' fixed segments: 5-point 512^2 15.2 -> 10.1 us (from 2048
// slots, padding dropped), power-law n = 30,000 17.8 -> 8.4 us, 32 FEM blocks
// of 22M nonzeros in one graph 57.2 -> 54.8 us (staged, from 4096).
size_t wide_seg(const WideCfg &w, size_t slots) {
  if (w.tmem) return w.seg;
  if (w.tma) {
    const size_t s = slots / ((size_t)sm_count() * 4 * w.warps * 8);
    return std::min(w.seg, std::max(SS, (s + SS - 1) / SS * SS));
  }
  const double held = (double)sm_count() * w.minb * WIDE_WARPS;
  size_t best = w.seg;
  double best_fill = 0.0;
  for (size_t s = w.seg; s >= SS; s -= SS) {
    const double loads = std::ceil((double)slots / (double)s) / held;
    const double fill = std::max(loads / std::ceil(loads), loads > 3.0 ? 0.93 : 0.0);
    if (fill > best_fill) {
      best = s;
      best_fill = fill;
    }
    if (fill >= 0.9) break;
  }
  return best;
}

// Fraction of a deterministic sample of the nonzeros whose column lies
// far from the diagonal (|c - r| > 1536, outside a 3072-column window) with
// no column of the next row within 16 of c + 1: gathers with no locality
// between neighbouring rows, which the L1 cache cannot share between the
// lanes of a warp (uniformly scattered columns; not the fixed far offsets
// of a stencil).  Such matrices gain from the staged per-CTA windows.
double random_far_fraction(const str_matCSR *csr) {
  const size_t nnz = csr->nnz, S = std::min<size_t>(nnz, 1u << 16);
  if (!S) return 0.0;
  const double stride = (double)nnz / (double)S;
  size_t far = 0;
  for (size_t i = 0, r = 0; i < S; i++) {
    const size_t j = (size_t)(i * stride);
    while (r < csr->nrows && csr->row[r + 1] <= j) r++;
    if (r >= csr->nrows) break;  // a row pointer that does not cover nnz
    const long long c = csr->col[j];
    if (std::llabs(c - (long long)r) <= 1536) continue;
    bool near_next = false;
    if (r + 1 < csr->nrows)
      for (UIN k = csr->row[r + 1]; k < csr->row[r + 2] && !near_next; k++)
        near_next = std::llabs((long long)csr->col[k] - c - 1) <= 16;
    far += !near_next;
  }
  return (double)far / (double)S;
}

// AUTO's staged plans of fewer nonzeros than this leave the windows empty: a
// window is copied before a CTA's first gather, and where a warp has a batch
// or two that wait shows (n = 30,000: 10.3 us with windows, 8.4 without; n =
// 100,000, 1.5M nonzeros: equal).
constexpr UIN WIN_MIN_NNZ = 1u << 20;

// AUTO on a slot-stream plan: the lane-interleaved kernel (stream_wide) and
// its variant.  8 slots per lane for rows of fewer than 16 nonzeros on
// average, with per-CTA x windows where the columns are scattered (FP64
// values) or the next batch's columns loaded ahead (FP32 values, whose
// kernel has the registers for it); else 16 slots per lane, bulk-copy staged
// for FP64 values with u32 columns that are not scattered (measured fastest
// there), plain loads for scattered columns and for the FP32, lo-word and
// 16-bit-delta forms (FP32 values: 8192-slot segments).  An explicit variant
// is kept.
int auto_variant(const ispmv_plan_s *p, bool long_rows, bool scattered) {
  const bool plain = p->opts.val_kind == ISPMV_VAL_F64 && p->opts.col_kind == ISPMV_COL_U32;
  const bool f32 = p->opts.val_kind == ISPMV_VAL_F32;
  if (!long_rows) return scattered && !narrow_kinds(p) ? (f32 ? 32 : 26) : 4;
  if (plain && !scattered) return 11;
  return f32 ? 8 : 0;  // FP32 values: 8192-slot segments (measured 3% faster on the 27-point stencil)
}
void auto_wide(ispmv_plan_s *p, const str_matCSR *csr) {
  p->opts.kernel = ISPMV_KERNEL_WIDE;
  if (p->opts.variant != 0) return;
  p->opts.variant = auto_variant(p, (double)csr->nnz >= 16.0 * (double)p->n, random_far_fraction(csr) >= 0.05);
  p->no_win = csr->nnz < WIN_MIN_NNZ;
  p->chosen = true;
}

// The per-CTA x windows of the staged stream_wide variants: CTA t walks
// slots [t*T, (t+1)*T), T = WIDE_WARPS*seg_slots; its window is W = cap
// columns of x that hold many of those slots' columns, started at an even
// column inside x[0, n rounded down to even), so the bulk copy starts on a
// 16-byte boundary and moves a multiple of 16 bytes.  Columns outside a CTA's
// window are gathered from x, so the choice costs time only; it is made from
// every eighth group of 8 slots, by counting twice:
//   1. columns per bin of 2^s1 (at most 8192 bins): the l1 neighbouring bins
//      with the most columns, l1 bins being wide enough for any W columns;
//   2. columns per bin of 2^s2 inside those (at most 2048 bins): the W >> s2
//      bins with the most; the first of equals in both.
// The device builder makes the same choice (dcsr_windows).
struct WinGeom {
  UIN W, ne, s1, nb1, l1, s2, nb2, w2;
};
WinGeom win_geom(UIN n, UIN cap) {
  WinGeom g{};
  g.W = cap & ~1u;
  g.ne = n & ~1u;
  for (g.s1 = 10; ((n - 1) >> g.s1) >= 8192u;) g.s1++;
  g.nb1 = ((n - 1) >> g.s1) + 1;
  g.l1 = ((g.W + (1u << g.s1) - 1) >> g.s1) + 1;
  for (g.s2 = 0; (((uint64_t)g.l1 << g.s1) >> g.s2) > 2048u;) g.s2++;
  g.nb2 = (UIN)(((uint64_t)g.l1 << g.s1) >> g.s2);
  g.w2 = std::max<UIN>(1, g.W >> g.s2);
  return g;
}
__host__ __device__ inline bool win_sampled(size_t slot) { return ((slot >> 3) & 7u) == 0; }

// The first start of the `w` neighbouring bins with the most counts.
UIN best_run(const UIN *h, UIN nb, UIN w) {
  uint64_t sum = 0, best = 0;
  UIN at = 0;
  for (UIN i = 0; i < std::min(w, nb); i++) sum += h[i];
  best = sum;
  for (UIN i = 1; i < nb; i++) {
    sum -= h[i - 1];
    if ((uint64_t)i + w - 1 < nb) sum += h[i + w - 1];
    if (sum > best) {
      best = sum;
      at = i;
    }
  }
  return at;
}

int stage_windows(ispmv_plan_s *p, const std::vector<UIN> &c) {
  const WinGeom g = win_geom(p->n, wide_variant(p->opts.variant).cap);
  const size_t T = (size_t)WIDE_WARPS * p->seg_slots, nt = std::max<size_t>(1, (p->nseg + WIDE_WARPS - 1) / WIDE_WARPS);
  std::vector<UIN> lo(nt, 0), len(nt, p->no_win ? 0 : std::min(g.ne, g.W));
  if (!p->no_win && g.ne > g.W) {
#pragma omp parallel
    {
      std::vector<UIN> h1(g.nb1), h2(g.nb2);
#pragma omp for schedule(dynamic, 16)
      for (long long t = 0; t < (long long)nt; t++) {
        const size_t a = (size_t)t * T, e = std::min(p->slots, a + T);
        std::fill(h1.begin(), h1.end(), 0u);
        std::fill(h2.begin(), h2.end(), 0u);
        for (size_t q = a; q < e; q++)
          if (win_sampled(q) && (c[q] >> g.s1) < g.nb1) h1[c[q] >> g.s1]++;
        const UIN r = best_run(h1.data(), g.nb1, g.l1) << g.s1;
        for (size_t q = a; q < e; q++)
          if (win_sampled(q) && c[q] >= r && ((c[q] - r) >> g.s2) < g.nb2) h2[(c[q] - r) >> g.s2]++;
        const uint64_t l = (uint64_t)r + ((uint64_t)best_run(h2.data(), g.nb2, g.w2) << g.s2);
        lo[t] = (UIN)std::min<uint64_t>(l, g.ne - g.W) & ~1u;
      }
    }
  }
  UIN *dlo, *dlen;
  TRY(dev_upload(p, lo.data(), lo.size(), &dlo));
  TRY(dev_upload(p, len.data(), len.size(), &dlen));
  p->xw.tlo = dlo;
  p->xw.tlen = dlen;
  p->xw.cap = p->no_win ? 0 : g.W;
  p->xw.nwin = 1;
  p->xw.n = p->n;
  return ISPMV_OK;
}

// Drops the formats' row padding (AXC bricks, AXT tiles: rows padded to 8
// slots, or to tileH) from the slot streams: the kernels find rows by their
// start bits and need none, and every slot costs its 12 bytes and a gather of
// x[0].  On power-law rows (14.9 nonzeros) tileH = 8 pads 24%, on 5-point rows
// 8 slots hold 5.  The 4-slots-per-lane kernels find fewer row starts per batch
// with the padding, and only the plain one is bound by the slots, on large
// matrices (AXT tileH = 1, padded and packed: staged at power-law n = 200,000 33
// and 37 us, n = 1M 107 and 112; plain at n = 200,000, 3.7M slots, 20.6 and 22.7,
// n = 1M 69.9 and 66.8, n = 4M 230 and 207).
// Leaves the stream as it is, too, where the format is not the CSR's
// (row pointer decreasing, rows past the format's slots, or values outside the
// CSR's rows): the format's own slots are multiplied then.
// In place, row after row: a copy of the stream takes the host as long again as
// the rest of the plan (first touch of its pages).
constexpr size_t PACK_LDG = (size_t)1 << 22;  // slots
void pack_rows(ispmv_plan_s *p, const str_matCSR *csr, std::vector<double> &v, std::vector<UIN> &c,
               std::vector<size_t> &start) {
  const long long n = csr->nrows, slots = (long long)v.size();
  bool fits = true;
  long long values = 0;  // outside the CSR's rows
#pragma omp parallel for schedule(static) reduction(+ : values)
  for (long long q = 0; q < slots; q++) values += v[q] != 0.0;
#pragma omp parallel for schedule(static) reduction(&& : fits) reduction(- : values)
  for (long long r = 0; r < n; r++) {
    const UIN a = csr->row[r], e = csr->row[r + 1];
    const size_t s = start[r], l = e - a;
    // in order, inside the format, and no further left than in the CSR
    const bool ok = e >= a && s >= a && s + l <= (r + 1 < n ? start[r + 1] : v.size()) && s + l <= v.size();
    fits = fits && ok;
    for (size_t k = 0; ok && k < l; k++) values -= v[s + k] != 0.0;
  }
  if (!fits || values) return;
  for (long long r = 0; r < n; r++) {
    const UIN a = csr->row[r], l = csr->row[r + 1] - a;
    if (!l) continue;  // a row without slots: start[r] names no slot of its own
    std::copy_n(v.begin() + start[r], l, v.begin() + a);
    std::copy_n(c.begin() + start[r], l, c.begin() + a);
    start[r] = a;
  }
  v.resize(csr->nnz);
  c.resize(csr->nnz);
  p->slots = csr->nnz;
}

// Slices of 32 rows (sl::slice_rows) for AUTO's 16-bit-delta plans, where the
// rows of a slice are nearly equally long (at most 8% padding: the bytes it
// adds are then less than the kernel saves) and short (a row is one lane's
// work: at most 48 elements), and every slice's columns span less than 65536.
// v, c: the slot stream; it fits only with the CSR's rows back to back.
// Returns false where a slice does not fit.
bool slice_fit(const ispmv_plan_s *p, const str_matCSR *csr, const std::vector<UIN> &c,
               const std::vector<size_t> &start, std::vector<uint2> &meta) {
  for (UIN r = 0; r < p->n; r++)
    if (csr->row[r + 1] < csr->row[r] || (csr->row[r + 1] > csr->row[r] && start[r] != csr->row[r])) return false;
  const UIN ns = (p->n + 31) / 32;
  meta.assign((size_t)ns + 1, uint2{0, 0});
  uint64_t cols = 0;
  for (UIN s = 0; s < ns; s++) {
    const UIN r0 = s * 32, r1 = std::min<UIN>(p->n, r0 + 32);
    UIN w = 0;
    for (UIN r = r0; r < r1; r++) w = std::max(w, csr->row[r + 1] - csr->row[r]);
    if (w > 48) return false;
    UIN lo = 0xFFFFFFFFu, hi = 0;
    for (UIN q = csr->row[r0]; q < csr->row[r1]; q++) {
      lo = std::min(lo, c[q]);
      hi = std::max(hi, c[q]);
    }
    if (w && hi - lo > 0xFFFFu) return false;
    meta[s] = {(UIN)cols, w ? lo : 0};
    cols += w;
  }
  meta[ns] = {(UIN)cols, 0};
  return cols * 32 <= csr->nnz + csr->nnz / 12 + 1024 && cols * 32 <= 0xFFFFFFFFull;
}

int setup_slices(ispmv_plan_s *p, const str_matCSR *csr, const std::vector<double> &v, const std::vector<UIN> &c,
                 const std::vector<uint2> &meta) {
  p->path = P_SLICES;
  p->slots_pad = (size_t)meta.back().x * 32;
  std::vector<double> sv(p->slots_pad, 0.0);
  std::vector<uint16_t> sd(p->slots_pad, 0);
  std::vector<uint8_t> len(p->n);
#pragma omp parallel for schedule(static)
  for (long long r = 0; r < (long long)p->n; r++) {
    const uint2 m = meta[r / 32];
    const UIN a = csr->row[r], l = csr->row[r + 1] - a;
    len[r] = (uint8_t)l;
    for (UIN k = 0; k < l; k++) {
      const size_t q = ((size_t)m.x + k) * 32 + r % 32;
      sv[q] = v[a + k];
      sd[q] = (uint16_t)(c[a + k] - m.y);
    }
  }
  uint16_t *d;
  TRY(upload_values(p, sv));
  TRY(dev_upload(p, sd.data(), sd.size(), &d));
  TRY(dev_upload(p, meta.data(), meta.size(), &p->slices));
  TRY(dev_upload(p, len.data(), len.size(), &p->slen));
  p->narrow.col16 = d;
  p->info.device_bytes = (uint64_t)p->slots_pad * (vbytes(p) + 2) + meta.size() * 8 + p->n;
  for (size_t s = 0; s + 1 < meta.size(); s++) p->slice_w = std::max(p->slice_w, meta[s + 1].x - meta[s].x);
  return ISPMV_OK;
}

// The stream path: `v`/`c` the slot streams (length p->slots), `start[r]`
// the first slot of row r (rows with no slot are skipped).
int setup_stream(ispmv_plan_s *p, const str_matCSR *csr, std::vector<double> &v, std::vector<UIN> &c,
                 std::vector<size_t> &start) {
  p->path = P_STREAM;
  p->fslots = p->slots;
  if (p->slots != csr->nnz && (p->opts.kernel == ISPMV_KERNEL_WIDE ||
                               (p->opts.kernel == ISPMV_KERNEL_LDG && p->slots >= PACK_LDG)))
    pack_rows(p, csr, v, c, start);
  if (p->chosen && p->opts.col_kind == ISPMV_COL_D16 && p->opts.val_kind != ISPMV_VAL_F32_LO16 &&
      p->opts.units_per_warp <= 0 && p->slots && p->slots == csr->nnz) {
    std::vector<uint2> meta;
    if (slice_fit(p, csr, c, start, meta)) return setup_slices(p, csr, v, c, meta);
  }
  p->slots_pad = std::max(SS, (p->slots + SS - 1) / SS * SS);
  if (p->opts.kernel == ISPMV_KERNEL_WIDE && wide_variant(p->opts.variant).tmem) {
    // whole CTAs: every consumer warp of stream_tmem walks a full segment
    const size_t unit = (size_t)wide_variant(p->opts.variant).warps * wide_variant(p->opts.variant).seg;
    p->slots_pad = std::max(unit, (p->slots + unit - 1) / unit * unit);
  }
  v.resize(p->slots_pad, 0.0);
  c.resize(p->slots_pad, 0);
  std::vector<UIN> heads(p->slots_pad / 32, 0), rowmap;
  bool any_empty = false;
  for (UIN r = 0; r < p->n; r++) {
    if (csr->row[r + 1] == csr->row[r]) {
      any_empty = true;
      continue;
    }
    const size_t q = start[r];
    heads[q >> 5] |= 1u << (q & 31);
    rowmap.push_back(r);
  }
  const bool wide = p->opts.kernel == ISPMV_KERNEL_WIDE;
  if (wide) {
    const WideCfg wc = wide_variant(p->opts.variant);
    const bool lo16 = p->opts.val_kind == ISPMV_VAL_F32_LO16;
    if (!wc.ok) return fail(ISPMV_ERR_UNSUPPORTED, "stream_wide: no such variant");
    if ((narrow_kinds(p) && (wc.tma || wc.tmem || wc.stg || wc.pfc)) || (lo16 && wc.tex))
      return fail(ISPMV_ERR_UNSUPPORTED,
                  "stream_wide: 16-bit column deltas and BF16 lo-words on the plain-load variants "
                  "(lo-words: not the texture-gather variants)");
  }
  p->seg_slots = seg_slots_of(p, 1);
  if (wide && (p->opts.units_per_warp <= 0 || wide_variant(p->opts.variant).tmem))
    p->seg_slots = wide_seg(wide_variant(p->opts.variant), p->slots_pad);
  p->nseg = (p->slots_pad + p->seg_slots - 1) / p->seg_slots;
  std::vector<UIN> segh(std::max<size_t>(1, p->nseg), 0);
  UIN acc = 0;
  for (size_t sg = 0, w = 0; sg < p->nseg; sg++) {
    const size_t wend = std::min(heads.size(), (sg * p->seg_slots) >> 5);
    for (; w < wend; w++) acc += __builtin_popcount(heads[w]);
    segh[sg] = acc;
  }
  if (wide && wide_variant(p->opts.variant).tmem) {
    // TMEM-staged blocks: block j of CTA c holds batch j of segments
    // nw*c..nw*c+nw-1, one half-block per 4 of them; in half-block h,
    // lane-row r = 32q + l (segment nw*c + 4h + q, lane l) with its SPL values
    // then its SPL columns, in the copy's canonical layout (tmemk::blk_word)
    const unsigned spl = (unsigned)wide_variant(p->opts.variant).spl, BT = 32u * spl;
    const unsigned nw = (unsigned)wide_variant(p->opts.variant).warps;  // 4 per column half
    const bool f64 = p->opts.val_kind == ISPMV_VAL_F64;
    const unsigned vw = f64 ? 2u : 1u, W = vw * spl + spl, BW = W / 8u * 1024u;  // words per half-block
    const size_t nbat = p->seg_slots / BT, nctas = p->nseg / nw;
    std::vector<uint32_t> blk(nctas * nbat * BW * (nw / 4u), 0u);
    for (size_t cta = 0; cta < nctas; cta++)
      for (size_t j = 0; j < nbat; j++)
        for (unsigned w = 0; w < nw; w++) {
          uint32_t *B = blk.data() + ((cta * nbat + j) * (nw / 4u) + w / 4u) * BW;
          const unsigned q = w % 4u;
          for (unsigned l = 0; l < 32u; l++)
            for (unsigned k = 0; k < spl; k++) {
              const size_t sl = (cta * nw + w) * p->seg_slots + j * BT + (size_t)spl * l + k;
              const unsigned r = 32u * q + l;
              if (f64) {
                uint64_t u;
                std::memcpy(&u, &v[sl], 8);
                B[tmemk::blk_word(r, 2u * k)] = (uint32_t)u;
                B[tmemk::blk_word(r, 2u * k + 1u)] = (uint32_t)(u >> 32);
              } else {
                const float f = (float)v[sl];
                std::memcpy(&B[tmemk::blk_word(r, k)], &f, 4);
              }
              B[tmemk::blk_word(r, vw * spl + k)] = c[sl];
            }
      }
    TRY(dev_upload(p, blk.data(), blk.size(), &p->tblocks));
  } else if (wide) {
    // the lane-interleaved copy: batches of 32*spl slots, one 16-byte vector per lane and step
    const unsigned spl = (unsigned)wide_variant(p->opts.variant).spl;
    std::vector<double> vi(p->slots_pad);
    std::vector<UIN> ci(p->slots_pad);
    const unsigned vv = p->opts.val_kind == ISPMV_VAL_F64 ? 2u : 4u;
    for (size_t q = 0; q < p->slots_pad; q++) {
      vi[wide::il_pos(q, spl, vv)] = v[q];
      ci[wide::il_pos(q, spl, 4u)] = c[q];
    }
    TRY(upload_values(p, vi));
    if (p->opts.col_kind == ISPMV_COL_U32) {
      TRY(dev_upload(p, ci.data(), ci.size(), &p->col));
    } else {
      // per batch of 32*spl slots: base = the smallest column among nonzero
      // values, deltas to it in 16 bits (lane-interleaved, 8 per vector), or
      // the batch's interleaved u32 columns when the span is wider
      const size_t BT = 32u * spl, nb = p->slots_pad / BT;
      p->d16_batch = BT;
      std::vector<UIN> cmeta(nb), esc;
      std::vector<uint16_t> c16(p->slots_pad, 0);
      for (size_t b = 0; b < nb; b++) {
        UIN lo = 0xFFFFFFFFu, hi = 0;
        for (size_t q = b * BT; q < b * BT + BT; q++)
          if (v[q] != 0.0) { lo = std::min(lo, c[q]); hi = std::max(hi, c[q]); }
        if (lo == 0xFFFFFFFFu) lo = hi = 0;
        if (hi - lo <= 0xFFFFu && lo < sss::ESCAPE) {
          cmeta[b] = lo;
          for (size_t q = b * BT; q < b * BT + BT; q++)
            c16[wide::il_pos(q, spl, 8u)] = v[q] != 0.0 ? (uint16_t)(c[q] - lo) : 0;
        } else {
          cmeta[b] = sss::ESCAPE | (UIN)p->esc_batches++;
          esc.insert(esc.end(), ci.begin() + b * BT, ci.begin() + b * BT + BT);  // interleaved already
        }
      }
      uint16_t *d16; UIN *dm, *de;
      TRY(dev_upload(p, c16.data(), c16.size(), &d16));
      TRY(dev_upload(p, cmeta.data(), cmeta.size(), &dm));
      TRY(dev_upload(p, esc.data(), esc.size(), &de));
      p->narrow.col16 = d16; p->narrow.cmeta = dm; p->narrow.esc = de;
    }
  } else {
    TRY(upload_values(p, v));
    if (p->opts.col_kind == ISPMV_COL_U32) TRY(dev_upload(p, c.data(), c.size(), &p->col));
  }
  if (p->opts.col_kind == ISPMV_COL_D16 && !wide) {
    // per 128-slot batch: base = the smallest column among nonzero values;
    // deltas to it in 16 bits, or the batch's u32 columns when the span is wider
    const size_t nb = p->slots_pad / 128;
    std::vector<UIN> cmeta(nb), esc;
    std::vector<uint16_t> c16(p->slots_pad, 0);
    for (size_t b = 0; b < nb; b++) {
      UIN lo = 0xFFFFFFFFu, hi = 0;
      for (size_t q = b * 128; q < b * 128 + 128; q++)
        if (v[q] != 0.0) { lo = std::min(lo, c[q]); hi = std::max(hi, c[q]); }
      if (lo == 0xFFFFFFFFu) lo = hi = 0;
      if (hi - lo <= 0xFFFFu && lo < sss::ESCAPE) {
        cmeta[b] = lo;
        for (size_t q = b * 128; q < b * 128 + 128; q++) c16[q] = v[q] != 0.0 ? (uint16_t)(c[q] - lo) : 0;
      } else {
        cmeta[b] = sss::ESCAPE | (UIN)p->esc_batches++;
        esc.insert(esc.end(), c.begin() + b * 128, c.begin() + b * 128 + 128);
      }
    }
    uint16_t *d16; UIN *dm, *de;
    TRY(dev_upload(p, c16.data(), c16.size(), &d16));
    TRY(dev_upload(p, cmeta.data(), cmeta.size(), &dm));
    TRY(dev_upload(p, esc.data(), esc.size(), &de));
    p->narrow.col16 = d16; p->narrow.cmeta = dm; p->narrow.esc = de;
  }
  if (p->opts.val_kind == ISPMV_VAL_F32_LO16) {
    // rows whose FP32 rounding error, relative to their row sum, exceeds
    // lo_tol get a BF16 residual; it is stored for every segment they touch
    const double tol = p->opts.lo_tol > 0 ? p->opts.lo_tol : 1e-6;
    std::vector<char> segflag(p->nseg, 0);
    for (UIN r = 0; r < p->n; r++) {
      double err = 0.0, sum = 0.0;
      for (UIN j = csr->row[r]; j < csr->row[r + 1]; j++) {
        err += std::fabs(csr->val[j] - (double)(float)csr->val[j]);
        sum += csr->val[j];
      }
      if (csr->row[r + 1] == csr->row[r] || err <= tol * std::fabs(sum)) continue;
      const size_t a = start[r], e = start[r] + (csr->row[r + 1] - csr->row[r]);
      for (size_t sg = a / p->seg_slots; sg <= (e - 1) / p->seg_slots && sg < p->nseg; sg++) segflag[sg] = 1;
    }
    // a flagged segment's residuals in slot order, or lane-interleaved like
    // the 16-bit deltas (8 per vector) for the lane-interleaved kernel; its
    // slot count is a multiple of the batch, so batches stay whole
    const unsigned ilspl = wide ? (unsigned)wide_variant(p->opts.variant).spl : 0u;
    std::vector<UIN> off(p->nseg, NO_ROW);
    std::vector<uint16_t> lo;
    for (size_t sg = 0; sg < p->nseg; sg++) {
      if (!segflag[sg]) continue;
      const size_t base = lo.size();
      off[sg] = (UIN)base;
      const size_t a = sg * p->seg_slots, e = std::min(p->slots_pad, a + p->seg_slots);
      lo.resize(base + (e - a));
      for (size_t q = a; q < e; q++)
        lo[base + (ilspl ? wide::il_pos(q - a, ilspl, 8u) : q - a)] = to_bf16((float)(v[q] - (double)(float)v[q]));
    }
    p->lo_frac = p->slots ? (double)lo.size() / (double)p->slots_pad : 0.0;
    uint16_t *dl; UIN *dof;
    TRY(dev_upload(p, lo.data(), lo.size(), &dl));
    TRY(dev_upload(p, off.data(), off.size(), &dof));
    p->narrow.lo16 = dl; p->narrow.lo_off = dof;
  }
  TRY(dev_upload(p, heads.data(), heads.size(), &p->heads));
  TRY(dev_upload(p, segh.data(), segh.size(), &p->segh));
  if (any_empty) TRY(dev_upload(p, rowmap.data(), rowmap.size(), &p->rowmap));
  p->nrowmap = any_empty ? rowmap.size() : 0;
  const bool stg = wide && wide_variant(p->opts.variant).stg;
  if (stg) TRY(stage_windows(p, c));
  TRY(empty_rows(p, csr));
  TRY(alloc_records(p));
  if (stg) p->xw.status = p->status;
  p->info.device_bytes = (uint64_t)(stg ? 8 * ((p->nseg + WIDE_WARPS - 1) / WIDE_WARPS) : 0) +
                         (uint64_t)p->slots_pad * vbytes(p) + p->slots_pad / 8 +
                         (p->opts.col_kind == ISPMV_COL_D16 ? p->slots_pad * 2 + p->slots_pad / p->d16_batch * 4 +
                                                                 p->esc_batches * p->d16_batch * 4
                                                           : p->slots_pad * 4) +
                         (uint64_t)(p->lo_frac * (double)p->slots_pad * 2.0);
  return ISPMV_OK;
}

}  // namespace

ISPMV_API void ispmv_plan_opts_default(ispmv_plan_opts *o) {
  if (!o) return;
  std::memset(o, 0, sizeof *o);
  o->val_kind = ISPMV_VAL_F64;
  o->col_kind = ISPMV_COL_U32;
  o->kernel = ISPMV_KERNEL_AUTO;
}

ISPMV_API int ispmv_plan_destroy(ispmv_plan p) {
  if (!p) return ISPMV_OK;
  for (cudaEvent_t e : p->tev) cudaEventDestroy(e);
  if (p->xtex) cudaDestroyTextureObject(p->xtex);
  if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  pool_free(p->owned.data(), p->owned.size(), false);
  delete p;
  return ISPMV_OK;
}

// ---------------------------------------------------------------- CSR --
ISPMV_API int ispmv_plan_csr(const str_matCSR *csr, const ispmv_plan_opts *o, ispmv_plan *out) {
  TRY(check_csr(csr));
  ispmv_plan_s *p;
  TRY(begin(o, &p));
  p->fmt = F_CSR;
  p->n = csr->nrows;
  p->nnz = csr->nnz;
  p->slots = csr->nnz;
  int st = ISPMV_OK;
  if (p->opts.kernel == ISPMV_KERNEL_AUTO) auto_wide(p, csr);  // the CSR-order slot stream
  if (p->opts.kernel == ISPMV_KERNEL_ROWS) {
    // the naive CSR product on the GPU: L lanes per row
    if (narrow_kinds(p)) { ispmv_plan_destroy(p); return ISPMV_ERR_UNSUPPORTED; }
    p->opts.kernel = ISPMV_KERNEL_ROWS;
    p->path = P_ROWS;
    const double mean = (double)csr->nnz / csr->nrows;
    p->lanes = mean <= 2.5 ? 2 : mean <= 5 ? 4 : mean <= 12 ? 8 : mean <= 24 ? 16 : 32;
    std::vector<double> v(csr->val, csr->val + csr->nnz);
    st = upload_values(p, v);
    if (!st) st = dev_upload(p, csr->col, csr->nnz, &p->col);
    if (!st) st = dev_upload(p, csr->row, (size_t)csr->nrows + 1, &p->rows);
    p->info.device_bytes = (uint64_t)csr->nnz * (vbytes(p) + 4) + 4ull * (csr->nrows + 1);
  } else {
    std::vector<double> v(csr->val, csr->val + csr->nnz);
    std::vector<UIN> c(csr->col, csr->col + csr->nnz);
    std::vector<size_t> start(csr->row, csr->row + csr->nrows);
    st = setup_stream(p, csr, v, c, start);
  }
  finish_info(p, "CSR");
  return done(p, st, out);
}

// ------------------------------------------ plans from a device CSR --
// The CSR-order slot stream (the compacted AXT's stream) built on the GPU
// from d_row / d_col / d_val, with the arrays setup_stream builds on the host
// for a lane-interleaved plan: values and columns interleaved per batch of
// 32*spl slots (wide::il_pos), zero padding to the stream length, the
// row-start bitmap, per-segment start counts, the compressed -> real row map
// (when rows are empty) and the empty-row list.  Row starts are set with
// atomicOr, so the bitmap does not depend on the order of the writes.
namespace {

// *bad = 1 if the row pointer decreases, row[0] != 0 or row[n] != nnz;
// flag[r] = 1 for a row with elements, flag[n] = 0, so the exclusive prefix
// at n is the count of non-empty rows.
__global__ void dcsr_check_rows(UIN n, UIN nnz, const UIN *__restrict__ row, UIN *__restrict__ flag,
                                int *__restrict__ bad) {
  const size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r > n) return;
  if (r == n) {
    flag[n] = 0;
    if (row[0] != 0 || row[n] != nnz) *bad = 1;
    return;
  }
  const UIN a = row[r], e = row[r + 1];
  flag[r] = e > a;
  if (e < a) *bad = 1;
}

// Row-start bits, the compressed -> real map and the empty-row list from the
// prefix `pos` of the non-empty flags; and segh[g] = row starts at slots
// below g*seg = pos[first r with row[r] >= g*seg], written by that r's thread
// (n's, past the last row); *long_rows = 1 for a row of more than
// seg::FIX_LONG segments.
__global__ void dcsr_rows(UIN n, const UIN *__restrict__ row, const UIN *__restrict__ pos, UIN *__restrict__ heads,
                          UIN *__restrict__ rowmap, UIN *__restrict__ empty, size_t nseg, UIN seg,
                          UIN *__restrict__ segh, int *__restrict__ long_rows) {
  const size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r > n) return;
  const UIN a = row[r], q = pos[r];
  const size_t g1 = r == n ? nseg : min((size_t)(a / seg) + 1, nseg);
  for (size_t g = r == 0 ? 0 : (size_t)(row[r - 1] / seg) + 1; g < g1; g++) segh[g] = q;
  if (r == n) return;
  const UIN e = row[r + 1];
  if (e > a) {
    if (e - a > seg::FIX_LONG * seg) *long_rows = 1;
    atomicOr(&heads[a >> 5], 1u << (a & 31u));
    if (rowmap) rowmap[q] = (UIN)r;
  } else if (empty) {
    empty[r - q] = (UIN)r;
  }
}

// The lane-interleaved value and column copies, zero beyond nnz; *bad = 1 for
// a column >= n (no pass before this one indexes by a column).
template <typename VT, int SPL>
__global__ void dcsr_interleave(UIN n, size_t nnz, size_t spad, const UIN *__restrict__ col,
                                const FPT *__restrict__ val, VT *__restrict__ vi, UIN *__restrict__ ci,
                                int *__restrict__ bad) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < spad; q += stride) {
    const bool in = q < nnz;
    vi[wide::il_pos_c<SPL, 16u / sizeof(VT)>(q)] = (VT)(in ? val[q] : 0.0);
    const UIN c = in ? col[q] : 0u;
    if (c >= n) *bad = 1;
    ci[wide::il_pos_c<SPL, 4u>(q)] = c;
  }
}

// Builder scratch, given back on every exit; the stream it was used on is
// synchronised first.
struct DevTmp {
  cudaStream_t s;
  std::vector<void *> v;
  explicit DevTmp(cudaStream_t st) : s(st) {}
  ~DevTmp() {
    if (v.empty()) return;
    const bool idle = cudaStreamSynchronize(s) == cudaSuccess;
    if (!idle) (void)cudaGetLastError();
    pool_free(v.data(), v.size(), idle);
  }
  template <typename T>
  int alloc(size_t n, T **d) {
    void *q = nullptr;
    TRY(pool_alloc(&q, (n ? n : 1) * sizeof(T)));
    v.push_back(q);
    *d = static_cast<T *>(q);
    return ISPMV_OK;
  }
};

// random_far_fraction on a device CSR: the same sample (nonzero
// j = (size_t)(i * stride)), its row the r with row[r] <= j < row[r+1], the
// same test; *far counts the hits.  8 lanes per sample: a 9-way search for
// the row (7 steps at a million rows, where a thread's binary search takes 20
// dependent loads), then the next row's columns 8 at a time.  Does nothing
// when the row pointer is malformed (*bad).
__global__ void __launch_bounds__(256) dcsr_far(size_t S, double stride, UIN n, const UIN *__restrict__ row,
                                                const UIN *__restrict__ col, const int *__restrict__ bad,
                                                unsigned long long *__restrict__ far) {
  if (*bad) return;
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const unsigned g = threadIdx.x & 7u, sh = threadIdx.x & 24u, gm = 0xFFu << sh;
  if (i >= S) return;
  const size_t j = (size_t)(i * stride);
  UIN a = 1, b = n;  // first k in [a, b] with row[k] > j (row[n] = nnz > j)
  while (b - a >= 8u) {
    const UIN step = (b - a) / 9u + 1u, k = a + min((g + 1u) * step, b - a);
    const unsigned m = (__ballot_sync(gm, row[k] > j) & gm) >> sh;  // a suffix of the lanes, or none
    const unsigned f = m ? __ffs(m) - 1u : 8u;
    const UIN na = f ? a + min(f * step, b - a) + 1u : a;
    if (f < 8u) b = a + min((f + 1u) * step, b - a);
    a = min(na, b);
  }
  {
    const UIN k = a + min(g, b - a);
    const unsigned m = (__ballot_sync(gm, row[k] > j) & gm) >> sh;
    a = m ? a + min((UIN)__ffs(m) - 1u, b - a) : b;
  }
  const size_t r = a - 1;
  const long long c = col[j];
  if (llabs(c - (long long)r) <= 1536) return;
  bool near_next = false;
  if (r + 1 < n)
    for (UIN k = row[r + 1] + g; k < row[r + 2]; k += 8u) near_next |= llabs((long long)col[k] - c - 1) <= 16;
  if (!(__ballot_sync(gm, near_next) & gm) && g == 0) atomicAdd(far, 1ull);
}

// best_run by one CTA of 256 threads: h holds the counts of nb bins (bin i
// at WH(i): a word of padding per 32 keeps the threads' runs of bins in
// different banks) and becomes their exclusive prefix.
__device__ __forceinline__ UIN WH(UIN i) { return i + (i >> 5); }
__device__ UIN cta_best_run(UIN *h, UIN nb, UIN w, unsigned long long *red) {
  const unsigned t = threadIdx.x, lane = t & 31u, wid = t >> 5;
  const UIN per = (nb + 255u) / 256u, i0 = min(nb, t * per), i1 = min(nb, i0 + per);
  UIN sum = 0;
  for (UIN i = i0; i < i1; i++) sum += h[WH(i)];
  UIN incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const UIN u = __shfl_up_sync(FULL, incl, d);
    if ((int)lane >= d) incl += u;
  }
  if (lane == 31) red[wid] = incl;
  __syncthreads();
  UIN run = incl - sum;
  for (unsigned k = 0; k < wid; k++) run += (UIN)red[k];
  for (UIN i = i0; i < i1; i++) {
    const UIN c = h[WH(i)];
    h[WH(i)] = run;
    run += c;
  }
  if (t == 255) h[WH(nb)] = run;  // the total
  __syncthreads();
  unsigned long long best = 0;  // count, then the smallest start
  for (UIN i = i0; i < i1; i++) {
    const UIN cnt = h[WH(w < nb - i ? i + w : nb)] - h[WH(i)];
    const unsigned long long k = ((unsigned long long)cnt << 32) | (0xFFFFFFFFu - i);
    best = k > best ? k : best;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long o = __shfl_xor_sync(FULL, best, d);
    best = o > best ? o : best;
  }
  if (lane == 0) red[wid] = best;
  __syncthreads();
  best = red[0];
#pragma unroll
  for (unsigned k = 1; k < 8; k++) best = red[k] > best ? red[k] : best;
  __syncthreads();  // red and h are free again
  return 0xFFFFFFFFu - (UIN)best;
}

// One CTA per plan CTA tile: stage_windows' choice.  Reads an eighth of the
// columns (twice, the second time from L2); a sort of every tile's columns
// and a search for the densest interval took 690 us of the 860 a plan's
// kernels did at n = 1M, 14.9M nonzeros.
__global__ void __launch_bounds__(256) dcsr_windows(WinGeom g, size_t T, size_t nnz, const UIN *__restrict__ col,
                                                    UIN *__restrict__ tlo, UIN *__restrict__ tlen) {
  __shared__ UIN h[8192 + 256 + 1];
  __shared__ unsigned long long red[8];
  const size_t a = blockIdx.x * T, e = min(nnz, a + T);
  auto count = [&](UIN nb, UIN lo, UIN s) {
    for (UIN i = threadIdx.x; i < WH(nb) + 1; i += 256) h[i] = 0;
    __syncthreads();
    // groups of 8 slots 0, 8, 16, ... of the tile (T is a multiple of 64)
    for (size_t k = threadIdx.x;; k += 256) {
      const size_t q = a + (k >> 3) * 64 + (k & 7u);
      if (q >= e) break;
      const UIN c = col[q];
      if (c >= lo && ((c - lo) >> s) < nb) atomicAdd(&h[WH((c - lo) >> s)], 1u);
    }
    __syncthreads();
  };
  count(g.nb1, 0u, g.s1);
  const UIN r = cta_best_run(h, g.nb1, g.l1, red) << g.s1;
  count(g.nb2, r, g.s2);
  const unsigned long long l = r + ((unsigned long long)cta_best_run(h, g.nb2, g.w2, red) << g.s2);
  if (threadIdx.x == 0) {
    tlo[blockIdx.x] = (UIN)min(l, (unsigned long long)(g.ne - g.W)) & ~1u;
    tlen[blockIdx.x] = g.W;
  }
}

__global__ void fill_u32(size_t n, UIN v, UIN *__restrict__ a) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

int dev_csr_stream(ispmv_plan_s *p, UIN n, UIN nnz, const UIN *row, const UIN *col, const FPT *val, cudaStream_t s) {
  if (p->opts.kernel != ISPMV_KERNEL_AUTO && p->opts.kernel != ISPMV_KERNEL_WIDE)
    return fail(ISPMV_ERR_UNSUPPORTED, "plan from a device CSR: the lane-interleaved kernel");
  if (p->opts.val_kind == ISPMV_VAL_F32_LO16 || p->opts.col_kind != ISPMV_COL_U32)
    return fail(ISPMV_ERR_UNSUPPORTED, "plan from a device CSR: FP64/FP32 values, u32 columns");
  // the row pointer is checked before any pass indexes through it, the
  // columns by the pass that copies them
  struct Found {
    unsigned long long far;
    UIN nonempty;
    int bad, long_rows;
  } *found, hf{};
  DevTmp tmp(s);
  p->n = n;
  p->nnz = nnz;
  UIN *flag, *pos;
  TRY(tmp.alloc(1, &found));
  TRY(tmp.alloc((size_t)n + 1, &flag));
  TRY(tmp.alloc((size_t)n + 1, &pos));
  int *const bad = &found->bad;
  ISPMV_TRY(cudaMemsetAsync(found, 0, sizeof *found, s));
  dcsr_check_rows<<<(unsigned)(((size_t)n + 1 + 255) / 256), 256, 0, s>>>(n, nnz, row, flag, bad);
  TRY(check_launch("dcsr_check_rows"));
  size_t tb = 0;
  ISPMV_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, flag, pos, (int)n + 1, s));
  void *tst;
  TRY(tmp.alloc(tb, reinterpret_cast<unsigned char **>(&tst)));
  ISPMV_TRY(cub::DeviceScan::ExclusiveSum(tst, tb, flag, pos, (int)n + 1, s));
  const size_t S = std::min<size_t>(nnz, 1u << 16);
  const bool choose = p->opts.kernel == ISPMV_KERNEL_AUTO && p->opts.variant == 0;
  if (choose && S) {
    dcsr_far<<<(unsigned)((S * 8 + 255) / 256), 256, 0, s>>>(S, (double)nnz / (double)S, n, row, col, bad,
                                                               &found->far);
    TRY(check_launch("dcsr_far"));
  }
  ISPMV_TRY(cudaMemcpyAsync(&found->nonempty, pos + n, sizeof(UIN), cudaMemcpyDeviceToDevice, s));
  ISPMV_TRY(cudaMemcpyAsync(&hf, found, sizeof hf, cudaMemcpyDeviceToHost, s));
  ISPMV_TRY(cudaStreamSynchronize(s));
  const char *malformed = "plan from a device CSR: malformed row pointer or a column >= n";
  if (hf.bad) return fail(ISPMV_ERR_ARG, malformed);
  const UIN nonempty = hf.nonempty;
  if (p->opts.kernel == ISPMV_KERNEL_AUTO) {
    // the compacted AXT's default (ispmv_plan_axt), with the scatter test
    // run on the device sample
    p->opts.kernel = ISPMV_KERNEL_WIDE;
    if (choose) {
      p->opts.variant = auto_variant(p, (double)nnz >= 16.0 * (double)n, S && (double)hf.far / (double)S >= 0.05);
      p->no_win = nnz < WIN_MIN_NNZ;
    }
  }
  const WideCfg wc = wide_variant(p->opts.variant);
  if (!wc.ok || wc.tmem)
    return fail(ISPMV_ERR_UNSUPPORTED, "plan from a device CSR: the lane-interleaved kernel without TMEM staging");
  if (wc.stg && nnz > 0x7FFFFFFFu)
    return fail(ISPMV_ERR_UNSUPPORTED, "plan from a device CSR: per-CTA x windows up to 2^31 - 1 nonzeros");
  p->fmt = F_CSR;
  p->path = P_STREAM;
  p->slots = p->fslots = nnz;
  p->slots_pad = std::max(SS, (p->slots + SS - 1) / SS * SS);
  p->seg_slots = p->opts.units_per_warp <= 0 ? wide_seg(wc, p->slots_pad) : seg_slots_of(p, 1);
  p->nseg = (p->slots_pad + p->seg_slots - 1) / p->seg_slots;
  void *vi;
  if (p->opts.val_kind == ISPMV_VAL_F64) TRY(dev_alloc(p, p->slots_pad, reinterpret_cast<double **>(&vi)));
  else TRY(dev_alloc(p, p->slots_pad, reinterpret_cast<float **>(&vi)));
  p->val = vi;
  TRY(dev_alloc(p, p->slots_pad, &p->col));
  TRY(dev_alloc(p, p->slots_pad / 32, &p->heads));
  TRY(dev_alloc(p, std::max<size_t>(1, p->nseg), &p->segh));
  p->nempty = n - nonempty;
  p->nrowmap = p->nempty ? nonempty : 0;
  if (p->nempty) {
    TRY(dev_alloc(p, p->nrowmap, &p->rowmap));
    TRY(dev_alloc(p, p->nempty, &p->empty));
  }
  ISPMV_TRY(cudaMemsetAsync(p->heads, 0, p->slots_pad / 32 * sizeof(UIN), s));
  const unsigned gi = (unsigned)std::min<size_t>((p->slots_pad + 255) / 256, (size_t)sm_count() * 32);
  auto interleave = [&](auto *v, auto spl_c) {
    dcsr_interleave<std::remove_pointer_t<decltype(v)>, decltype(spl_c)::value>
        <<<gi, 256, 0, s>>>(n, nnz, p->slots_pad, col, val, v, p->col, bad);
  };
  using S8 = std::integral_constant<int, 8>;
  using S16 = std::integral_constant<int, 16>;
  if (p->opts.val_kind == ISPMV_VAL_F64) {
    if (wc.spl == 8) interleave(static_cast<double *>(vi), S8{});
    else interleave(static_cast<double *>(vi), S16{});
  } else {
    if (wc.spl == 8) interleave(static_cast<float *>(vi), S8{});
    else interleave(static_cast<float *>(vi), S16{});
  }
  TRY(check_launch("dcsr_interleave"));
  dcsr_rows<<<(unsigned)(((size_t)n + 1 + 255) / 256), 256, 0, s>>>(n, row, pos, p->heads, p->rowmap, p->empty,
                                                                      p->nseg, (UIN)p->seg_slots, p->segh,
                                                                      &found->long_rows);
  TRY(check_launch("dcsr_rows"));
  size_t nt = 0;
  if (wc.stg) {
    // per-CTA x windows, as stage_windows picks them on the host
    const WinGeom g = win_geom(n, wc.cap);
    nt = std::max<size_t>(1, (p->nseg + WIDE_WARPS - 1) / WIDE_WARPS);
    UIN *tlo, *tlen;
    TRY(dev_alloc(p, nt, &tlo));
    TRY(dev_alloc(p, nt, &tlen));
    if (!p->no_win && g.ne > g.W) {
      dcsr_windows<<<(unsigned)nt, 256, 0, s>>>(g, (size_t)WIDE_WARPS * p->seg_slots, nnz, col, tlo, tlen);
      TRY(check_launch("dcsr_windows"));
    } else {  // no window, or all of x (but an odd last element)
      ISPMV_TRY(cudaMemsetAsync(tlo, 0, nt * sizeof(UIN), s));
      fill_u32<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(nt, p->no_win ? 0u : g.ne, tlen);
      TRY(check_launch("fill_u32"));
    }
    p->xw.tlo = tlo;
    p->xw.tlen = tlen;
    p->xw.cap = p->no_win ? 0 : g.W;
    p->xw.nwin = 1;
    p->xw.n = p->n;
  }
  TRY(alloc_records(p, s));
  if (wc.stg) p->xw.status = p->status;
  ISPMV_TRY(cudaMemcpyAsync(&hf, found, sizeof hf, cudaMemcpyDeviceToHost, s));
  ISPMV_TRY(cudaStreamSynchronize(s));
  if (hf.bad) return fail(ISPMV_ERR_ARG, malformed);
  p->long_rows = hf.long_rows != 0;
  p->info.device_bytes = (uint64_t)(8 * nt) + (uint64_t)p->slots_pad * (vbytes(p) + 4) + p->slots_pad / 8;
  return ISPMV_OK;
}

}  // namespace

ISPMV_API int ispmv_plan_dev_csr(UIN n, UIN nnz, const UIN *d_row, const UIN *d_col, const FPT *d_val,
                                 const ispmv_plan_opts *o, ispmv_plan *out, void *stream) {
  if (!out || !d_row || n == 0 || (nnz && (!d_col || !d_val))) return ISPMV_ERR_ARG;
  if ((uint64_t)nnz + sss::SS > 0xFFFFFFFFull) return ISPMV_ERR_OVERFLOW;  // slot ids stay in 32 bits
  ispmv_plan_s *p;
  TRY(begin(o, &p));
  const int st = dev_csr_stream(p, n, nnz, d_row, d_col, d_val, as_stream(stream));
  finish_info(p, "CSR");
  return done(p, st, out, true);
}

ISPMV_API int ispmv_plan_get_layout(ispmv_plan p, ispmv_plan_layout *l) {
  if (!p || !l) return ISPMV_ERR_ARG;
  if (p->path != P_STREAM || p->opts.col_kind != ISPMV_COL_U32 ||
      (p->opts.kernel == ISPMV_KERNEL_WIDE && wide_variant(p->opts.variant).tmem))
    return ISPMV_ERR_UNSUPPORTED;
  std::memset(l, 0, sizeof *l);
  l->slots = p->slots;
  l->slots_pad = p->slots_pad;
  l->seg_slots = p->seg_slots;
  l->nseg = p->nseg;
  l->nrowmap = p->nrowmap;
  l->nempty = p->nempty;
  l->val_bytes = (UIN)vbytes(p);
  l->spl = p->opts.kernel == ISPMV_KERNEL_WIDE ? (UIN)wide_variant(p->opts.variant).spl : 0u;
  l->nwin = p->opts.kernel == ISPMV_KERNEL_WIDE && wide_variant(p->opts.variant).stg
                ? std::max<size_t>(1, (p->nseg + WIDE_WARPS - 1) / WIDE_WARPS)
                : 0;
  return ISPMV_OK;
}

ISPMV_API int ispmv_plan_export_windows(ispmv_plan p, UIN *lo, UIN *len, void *stream) {
  ispmv_plan_layout l;
  TRY(ispmv_plan_get_layout(p, &l));
  cudaStream_t s = as_stream(stream);
  if (l.nwin && lo) ISPMV_TRY(cudaMemcpyAsync(lo, p->xw.tlo, l.nwin * sizeof(UIN), cudaMemcpyDefault, s));
  if (l.nwin && len) ISPMV_TRY(cudaMemcpyAsync(len, p->xw.tlen, l.nwin * sizeof(UIN), cudaMemcpyDefault, s));
  ISPMV_TRY(cudaStreamSynchronize(s));
  return ISPMV_OK;
}

ISPMV_API int ispmv_plan_export_stream(ispmv_plan p, void *val, UIN *col, UIN *heads, UIN *segh, UIN *rowmap,
                                       UIN *empty, void *stream) {
  ispmv_plan_layout l;
  TRY(ispmv_plan_get_layout(p, &l));
  cudaStream_t s = as_stream(stream);
  auto cp = [&](void *dst, const void *src, size_t bytes) -> int {
    if (dst && src && bytes) ISPMV_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, s));
    return ISPMV_OK;
  };
  TRY(cp(val, p->val, l.slots_pad * l.val_bytes));
  TRY(cp(col, p->col, l.slots_pad * sizeof(UIN)));
  TRY(cp(heads, p->heads, l.slots_pad / 32 * sizeof(UIN)));
  TRY(cp(segh, p->segh, l.nseg * sizeof(UIN)));
  TRY(cp(rowmap, p->rowmap, l.nrowmap * sizeof(UIN)));
  TRY(cp(empty, p->empty, l.nempty * sizeof(UIN)));
  ISPMV_TRY(cudaStreamSynchronize(s));
  return ISPMV_OK;
}

// ---------------------------------------------------------------- AXC --
ISPMV_API int ispmv_plan_axc(const str_matCSR *csr, const str_matAXC *axc, const UIN *axi,
                             const ispmv_plan_opts *o, ispmv_plan *out) {
  TRY(check_csr(csr));
  if (!axc || !axi || !axc->ax || !axc->brp || axc->nrows != csr->nrows) return ISPMV_ERR_ARG;
  ispmv_plan_s *p;
  TRY(begin(o, &p));
  p->fmt = F_AXC;
  p->n = csr->nrows;
  p->nnz = csr->nnz;
  p->slots = axc->lenAX / 2;
  std::vector<double> v(p->slots);
  std::vector<UIN> c(axi, axi + p->slots);
  for (size_t s = 0; s < p->slots; s++) v[s] = axc->ax[(s / 8) * 16 + s % 8];
  int st = ISPMV_OK;
  if (p->opts.kernel == ISPMV_KERNEL_AUTO) auto_wide(p, csr);  // the brick stream
  if (p->opts.kernel == ISPMV_KERNEL_ROWS) {
    // the reference's row loop (M:711-732): 8 lanes per row over its bricks
    if (narrow_kinds(p)) { ispmv_plan_destroy(p); return ISPMV_ERR_UNSUPPORTED; }
    p->opts.kernel = ISPMV_KERNEL_ROWS;
    p->path = P_ROWS;
    std::vector<UIN> bptr((size_t)p->n + 1);
    for (size_t r = 0; r <= p->n; r++) bptr[r] = axc->brp[r] / 16;
    st = upload_values(p, v);
    if (!st) st = dev_upload(p, c.data(), c.size(), &p->col);
    if (!st) st = dev_upload(p, bptr.data(), bptr.size(), &p->rows);
    p->info.device_bytes = (uint64_t)p->slots * (vbytes(p) + 4) + 4ull * (p->n + 1);
  } else {
    std::vector<size_t> start(p->n);
    for (UIN r = 0; r < p->n; r++) start[r] = axc->brp[r] / 2;
    st = setup_stream(p, csr, v, c, start);
  }
  finish_info(p, "AXC");
  return done(p, st, out);
}

// ----------------------------------------------------------------- K1 --
ISPMV_API int ispmv_plan_k1(const str_matCSR *csr, const str_matK1 *k1, int reorder, const ispmv_plan_opts *o,
                            ispmv_plan *out) {
  TRY(check_csr(csr));
  if (!k1 || !k1->val || !k1->col || !k1->chp || !k1->nmc || !k1->permi || k1->nrows != csr->nrows)
    return ISPMV_ERR_ARG;
  ispmv_plan_s *p;
  TRY(begin(o, &p));
  if (narrow_kinds(p)) {
    delete p;
    return ISPMV_ERR_UNSUPPORTED;
  }
  p->fmt = reorder ? F_K1P : F_K1;
  p->path = P_K1;
  p->opts.kernel = ISPMV_KERNEL_ROWS;
  p->n = csr->nrows;
  p->nnz = csr->nnz;
  p->slots = k1->lenVC;
  p->chunkNum = k1->chunkNum;
  // the long chunks (a CTA or a warp each): prefixes of the chunks, whose
  // column counts never increase (rows are sorted by length)
  while (p->k1_long < k1->chunkNum && k1->nmc[p->k1_long] >= pk::K1_LONG) p->k1_long++;
  while (p->k1_cta < p->k1_long && k1->nmc[p->k1_cta] >= pk::K1_CTA) p->k1_cta++;
  std::vector<double> v;
  const UIN *kc = k1->col, *chp = k1->chp;
  size_t lenVC = k1->lenVC;
  std::vector<UIN> c2, o2;
  // the kernel reads pairs of slots: if a chunk is at an odd offset (the
  // builders make none), the chunks are moved to even ones
  if (std::any_of(chp, chp + k1->chunkNum, [](UIN o) { return o & 1u; })) {
    for (UIN c = 0; c < k1->chunkNum; c++) {
      const size_t a = chp[c], e = a + (size_t)8 * k1->nmc[c];
      o2.push_back((UIN)v.size());
      v.insert(v.end(), k1->val + a, k1->val + e);
      c2.insert(c2.end(), kc + a, kc + e);
    }
    kc = c2.data();
    chp = o2.data();
    lenVC = v.size();
  } else {
    v.assign(k1->val, k1->val + lenVC);
  }
  int st = upload_values(p, v);
  if (!st) st = dev_upload(p, kc, lenVC, &p->col);
  if (!st) st = dev_upload(p, chp, k1->chunkNum, &p->chp);
  if (!st) st = dev_upload(p, k1->nmc, k1->chunkNum, &p->nmc);
  if (!st) st = dev_upload(p, k1->permi, (size_t)k1->chunkNum * 8, &p->permi);
  if (!st && !reorder) st = dev_alloc(p, (size_t)k1->chunkNum * 8, &p->res);
  finish_info(p, reorder ? "K1P" : "K1");
  p->info.device_bytes = (uint64_t)p->slots * (vbytes(p) + 4) + 8ull * k1->chunkNum + 32ull * k1->chunkNum;
  return done(p, st, out);
}

// ---------------------------------------------------------------- AXT --
ISPMV_API int ispmv_plan_axt(const str_matCSR *csr, const str_matAXT *axt, const UIN *axi, const ispmv_plan_opts *o,
                             ispmv_plan *out) {
  TRY(check_csr(csr));
  if (!axt || !axi || !axt->ax || !axt->sec || !axt->con || axt->nrows != csr->nrows) return ISPMV_ERR_ARG;
  if (axt->tileHW != 8 || axt->tileH == 0) return ISPMV_ERR_UNSUPPORTED;
  const bool com = std::strncmp(axt->mode, "COM", 3) == 0;
  const bool noc = std::strncmp(axt->mode, "NOC", 3) == 0;
  if (!com && !noc) return ISPMV_ERR_ARG;
  if (com && axt->tileH != 1) return ISPMV_ERR_UNSUPPORTED;
  ispmv_plan_s *p;
  TRY(begin(o, &p));
  if (p->opts.kernel == ISPMV_KERNEL_ROWS) {
    delete p;
    return ISPMV_ERR_UNSUPPORTED;
  }
  p->n = csr->nrows;
  p->nnz = csr->nnz;
  p->th = axt->tileH;
  p->fmt = com ? F_AXT_COM : F_AXT_NOC;
  char name[32];
  int st = ISPMV_OK;
  const UIN th = axt->tileH;
  if (com) {
    p->bs = 1u << axt->log;
    snprintf(name, sizeof name, "AXT_COM_BS%u", p->bs);
  } else {
    snprintf(name, sizeof name, "AXT_NOC_H%u", th);
  }
  // tileH > 1 on the slot-stream kernels: the tiles' slots in tile-column
  // order (tile, column, sub-row), where each row is one contiguous run
  const bool noc_stream = !com && th > 1 && (p->opts.kernel == ISPMV_KERNEL_AUTO || p->opts.kernel == ISPMV_KERNEL_WIDE);
  if (com || th == 1 || noc_stream) {
    // the tileH=1 tile stream and the packed compacted stream: every row is
    // a contiguous run of slots starting at the slot its con[] names; a
    // tileH > 1 tile (th sub-rows of 8 columns, a row filling columns top to
    // bottom, M:1188-1221) read column by column is such a stream too
    p->slots = com ? csr->nnz : (size_t)axt->lenAX / 2;
    std::vector<double> v(p->slots);
    std::vector<UIN> c(p->slots);
    std::vector<size_t> start(p->n);
    if (th == 1) {
      std::copy(axi, axi + p->slots, c.begin());
      for (size_t q = 0; q < p->slots; q++) v[q] = axt->ax[(q / 8) * 16 + q % 8];
      for (UIN r = 0; r < p->n; r++) start[r] = (size_t)(axt->con[r] / 16) * 8 + axt->con[r] % 16;
    } else {
      const size_t tile = (size_t)8 * th;  // value slots per tile
      for (size_t q = 0; q < p->slots; q++) {  // q: slot in ax order (tile, sub-row, column)
        const size_t T = q / tile, R = (q % tile) / 8, C = q % 8;
        const size_t sc = T * tile + C * th + R;  // the same slot in column order
        v[sc] = axt->ax[(q / 8) * 16 + q % 8];
        c[sc] = axi[q];
      }
      for (UIN r = 0; r < p->n; r++) {  // con = T*16*th + R*16 + C (M:1118-1148)
        const size_t T = axt->con[r] / (16 * th), rem = axt->con[r] % (16 * th);
        start[r] = T * tile + (rem % 16) * th + rem / 16;
      }
    }
    if (p->opts.kernel == ISPMV_KERNEL_AUTO) {
      // the lane-interleaved kernel: 8 slots per lane for rows of fewer than
      // 16 nonzeros on average, where the columns are scattered with per-CTA
      // x windows (FP64 values) or the next batch's columns loaded ahead
      // (FP32 values, whose kernel has the registers for it); else 16,
      // bulk-copy staged for FP64 values with u32 columns that are not
      // scattered (measured fastest there), plain loads for scattered columns
      // and for the FP32, lo-word and 16-bit-delta forms
      auto_wide(p, csr);
    }
    st = setup_stream(p, csr, v, c, start);
  } else {
    // tile columns: the unit engine on the reference's per-column rows
    p->path = P_UNITS;
    if (narrow_kinds(p)) st = ISPMV_ERR_UNSUPPORTED;
    size_t used = 0;
    for (UIN r = 0; r < p->n; r++) used += ((size_t)csr->rl[r] + th - 1) / th * th;
    p->slots = (size_t)axt->lenAX / 2;
    p->nunits = used / th;
    p->slots_pad = std::max(SS, (p->slots + SS - 1) / SS * SS);
    const bool regular = th == 4 || th == 8 || th == 16;
    if (p->opts.kernel == ISPMV_KERNEL_TMA && !regular) st = ISPMV_ERR_UNSUPPORTED;
    if (p->opts.kernel == ISPMV_KERNEL_AUTO) p->opts.kernel = ISPMV_KERNEL_LDG;
    if (regular) {
      p->seg_slots = seg_slots_of(p, th);
      p->useg = (UIN)(p->seg_slots / th);
      p->nseg = (p->slots_pad + p->seg_slots - 1) / p->seg_slots;
    } else {
      UIN u = p->opts.units_per_warp > 0 ? (UIN)p->opts.units_per_warp : std::max<UIN>(32u, (2048u / th) & ~31u);
      p->useg = std::max<UIN>(32u, u & ~31u);
      p->seg_slots = (size_t)p->useg * th;
      p->nseg = (p->nunits + p->useg - 1) / p->useg;
    }
    std::vector<double> v(p->slots_pad, 0.0);
    std::vector<UIN> c(p->slots_pad, 0);
    for (size_t q = 0; q < p->slots; q++) {
      v[q] = axt->ax[(q / 8) * 16 + q % 8];
      c[q] = axi[q];
    }
    if (!st) st = upload_values(p, v);
    if (!st) st = dev_upload(p, c.data(), c.size(), &p->col);
    std::vector<UIN> ur(std::max<size_t>(p->slots_pad / th, p->nunits) + 32, NO_ROW);
    std::copy(axt->sec, axt->sec + p->nunits, ur.begin());
    if (!st) st = dev_upload(p, ur.data(), ur.size(), &p->rows);
    if (!st) st = empty_rows(p, csr);
    if (!st) st = alloc_records(p);
    p->info.device_bytes = (uint64_t)p->slots_pad * (vbytes(p) + 4) + 4ull * p->nunits;
  }
  finish_info(p, name);
  return done(p, st, out);
}

ISPMV_API int ispmv_plan_get_info(ispmv_plan p, ispmv_plan_info *info) {
  if (!p || !info) return ISPMV_ERR_ARG;
  *info = p->info;
  return ISPMV_OK;
}

// ------------------------------------------------------------ execute --
namespace {

constexpr int TW = 4;  // warps per CTA of the staged kernels
constexpr int TS = 4;  // stages per warp

template <typename K>
int launch_staged(K kernel, size_t smem, size_t nseg, int ctas_per_sm, cudaStream_t s, const char *what,
                  void **args) {
  const size_t want = (nseg + TW - 1) / TW;
  const size_t cap = (size_t)sm_count() * (size_t)(ctas_per_sm > 0 ? ctas_per_sm : 2);
  const unsigned g = (unsigned)std::max<size_t>(1, std::min(want, cap));
  ISPMV_TRY(cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ISPMV_TRY(cudaLaunchKernel((const void *)kernel, dim3(g), dim3(TW * 32), args, smem, s));
  return check_launch(what);
}

template <int W, typename K>
int launch_staged_w(K kernel, size_t smem, size_t nseg, int ctas_per_sm, cudaStream_t s, const char *what,
                    void **args) {
  const size_t want = (nseg + W - 1) / W;
  const size_t cap = (size_t)sm_count() * (size_t)ctas_per_sm;
  const unsigned g = (unsigned)std::max<size_t>(1, std::min(want, cap));
  ISPMV_TRY(cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ISPMV_TRY(cudaLaunchKernel((const void *)kernel, dim3(g), dim3(W * 32), args, smem, s));
  return check_launch(what);
}

// Whether a product's first kernel may start while the launch before the
// product finishes: not where a timing event sits between them, nor where the
// kernel is timed by itself.
bool overlaps(const ispmv_plan_s *p) { return !p->alone && (!p->tcap || p->capturing); }

// A launch; `early`: it may start while the launches before it in the stream
// finish (its kernel waits for them before it touches anything but the plan's
// constant arrays).
template <typename... KA, typename... A>
int launch_dependent(const char *name, void (*k)(KA...), size_t grid, unsigned block, size_t smem, cudaStream_t s,
                     bool early, A... a) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  ISPMV_TRY(cudaLaunchKernelEx(&cfg, k, static_cast<KA>(a)...));
  return check_launch(name);
}

// A linear texture over `src` (bytes long, FP64 read as int2 or FP32),
// cached on the plan for the same buffer; 0 when the buffer does not meet
// the texture alignment or size limits (the caller then gathers with loads).
// Not inside graph capture: a later product with another x replaces the
// texture, which a captured graph would still name.
cudaTextureObject_t x_texture(ispmv_plan_s *p, const void *src, size_t bytes, bool f32) {
  if (p->capturing) return 0;
  if (p->xtex && p->xtex_src == src && p->xtex_bytes == bytes) return p->xtex;
  if (p->xtex) cudaDestroyTextureObject(p->xtex);
  p->xtex = 0;
  p->xtex_src = nullptr;
  int dev = 0, align = 0, maxw = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&align, cudaDevAttrTextureAlignment, dev) ||
      cudaDeviceGetAttribute(&maxw, cudaDevAttrMaxTexture1DLinearWidth, dev))
    return 0;
  const size_t elems = bytes / (f32 ? 4 : 8);
  if (align <= 0 || reinterpret_cast<uintptr_t>(src) % (uintptr_t)align || elems > (size_t)maxw || elems >= (1u << 31))
    return 0;
  cudaResourceDesc rd{};
  rd.resType = cudaResourceTypeLinear;
  rd.res.linear.devPtr = const_cast<void *>(src);
  rd.res.linear.desc = f32 ? cudaCreateChannelDesc<float>() : cudaCreateChannelDesc<int2>();
  rd.res.linear.sizeInBytes = bytes;
  cudaTextureDesc td{};
  td.readMode = cudaReadModeElementType;
  if (cudaCreateTextureObject(&p->xtex, &rd, &td, nullptr) != cudaSuccess) {
    cudaGetLastError();
    p->xtex = 0;
    return 0;
  }
  p->xtex_src = src;
  p->xtex_bytes = bytes;
  return p->xtex;
}

template <typename VT, int SPL, int MINB, bool D16 = false, bool TEX = false, bool STG = false, bool LO = false,
          bool PFC = false>
int launch_wide(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s, const char *name) {
  constexpr int NW = STG ? 1 : 0;
  const size_t ctas = (p->nseg + WIDE_WARPS - 1) / WIDE_WARPS;
  // one load of CTAs: stream_wide's DEP form; never with texture gathers.  Not
  // with a caller's segment length either: a few long CTAs started early pile
  // up on the SMs that are free first (power-law n = 200,000, 2048-slot
  // segments: 22-26 us, 20.9 late; the automatic lengths 17.4 and 21.0)
  const bool early =
      STG || (!TEX && p->opts.units_per_warp <= 0 && ctas <= (size_t)sm_count() * MINB);
  if constexpr (sizeof(VT) == 4 && !STG && !LO) {
    // FP32 values: gather from an FP32 copy of x (the value the FP32 multiply uses)
    if (!p->x32) TRY(dev_alloc(p, p->n, &p->x32));
    const unsigned gc = (unsigned)std::min<size_t>(((size_t)p->n / 2 + 255) / 256, (size_t)sm_count() * 8) + 1;
    auto *kx = (reinterpret_cast<uintptr_t>(x) & 15u) == 0 ? wide::x_to_f32<true> : wide::x_to_f32<false>;
    TRY(launch_dependent("x_to_f32", kx, gc, 256, 0, s, overlaps(p), p->n, x, p->x32));
    const cudaTextureObject_t tx = TEX ? x_texture(p, p->x32, (size_t)p->n * 4, true) : 0;
    if (TEX && !tx) return launch_wide<VT, SPL, MINB, D16, false>(p, x, o, s, "stream_wide<tex: x gathered with loads>");
    auto *k = early ? wide::stream_wide<VT, float, SPL, 0, WIDE_WARPS, MINB, D16, TEX, false, false, PFC, !TEX>
                    : wide::stream_wide<VT, float, SPL, 0, WIDE_WARPS, MINB, D16, TEX, false, false, PFC, false>;
    return launch_dependent(name, k, ctas, WIDE_WARPS * 32, 0, s, early, p->slots, p->slots_pad, p->seg_slots, p->nseg,
                            static_cast<const VT *>(p->val), p->col, p->heads, p->segh, p->xw, p->x32, o, p->narrow, tx);
  } else {
    const cudaTextureObject_t tx = TEX ? x_texture(p, x, (size_t)p->n * 8, false) : 0;
    if (TEX && !tx) return launch_wide<VT, SPL, MINB, D16, false>(p, x, o, s, "stream_wide<tex: x gathered with loads>");
    auto *k = early ? wide::stream_wide<VT, double, SPL, NW, WIDE_WARPS, MINB, D16, TEX, STG, LO, PFC, !TEX>
                    : wide::stream_wide<VT, double, SPL, NW, WIDE_WARPS, MINB, D16, TEX, STG, LO, PFC, STG>;
    const size_t smem = STG ? (size_t)p->xw.cap * sizeof(double) : 0;
    if (smem) ISPMV_TRY(cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_dependent(name, k, ctas, WIDE_WARPS * 32, smem, s, early && overlaps(p), p->slots, p->slots_pad,
                            p->seg_slots, p->nseg, static_cast<const VT *>(p->val), p->col, p->heads, p->segh, p->xw, x,
                            o, p->narrow, tx);
  }
}

// The staged form: persistent, as many CTAs as fit on the SMs (at most one
// warp per segment).
template <typename VT, int SPL, int STAGES, int W>
int launch_wide_tma(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s, const char *name) {
  auto *k = wide::stream_wide_tma<VT, SPL, STAGES, W>;
  const size_t smem = wide::tma_smem_bytes<VT, SPL, STAGES, W>();
  ISPMV_TRY(cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  ISPMV_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, W * 32, smem));
  if (p->opts.ctas_per_sm > 0) per_sm = std::min(per_sm, p->opts.ctas_per_sm);
  const size_t want = (p->nseg + W - 1) / W;
  const unsigned g = (unsigned)std::max<size_t>(1, std::min(want, (size_t)sm_count() * (size_t)std::max(1, per_sm)));
  // an ordinary launch: starting before the launch before it ends gave
  // nothing here (32 FEM blocks 54.8 / 54.6 us) and 1% away at 160^3
  k<<<g, W * 32, smem, s>>>(p->slots, p->slots_pad, p->seg_slots, p->nseg, static_cast<const VT *>(p->val), p->col,
                            p->heads, p->segh, x, o, p->status);
  return check_launch(name);
}

// The TMEM-staged form: one CTA of 4 consumer warps + 1 producer warp per 4
// segments.
template <typename VT, int SPL, int S, int H>
int launch_tmem(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s, const char *name) {
  const void *xs = x;
  if constexpr (sizeof(VT) == 4) {  // FP32 values: gather the FP32 copy of x
    if (!p->x32) TRY(dev_alloc(p, p->n, &p->x32));
    const unsigned gc = (unsigned)std::min<size_t>(((size_t)p->n / 2 + 255) / 256, (size_t)sm_count() * 8) + 1;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) wide::x_to_f32<true><<<gc, 256, 0, s>>>(p->n, x, p->x32);
    else wide::x_to_f32<false><<<gc, 256, 0, s>>>(p->n, x, p->x32);
    TRY(check_launch("x_to_f32"));
    xs = p->x32;
  }
  using XT = typename std::conditional<sizeof(VT) == 4, float, double>::type;
  constexpr int B0 = SPL == 8 ? 0 : (int)seg::RED, B1 = SPL == 8 ? 1 : (int)seg::RED;
  auto *k = o.beta ? tmemk::stream_tmem<VT, XT, SPL, S, H, B1> : tmemk::stream_tmem<VT, XT, SPL, S, H, B0>;
  const size_t smem = tmemk::smem_bytes<VT, SPL, S, H>();
  ISPMV_TRY(cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const unsigned g = (unsigned)(p->nseg / (tmemk::CW * H));
  k<<<g, (tmemk::CW * H + 1) * 32, smem, s>>>(p->slots, p->seg_slots, p->tblocks, p->heads, p->segh,
                                               static_cast<const XT *>(xs), o, p->status);
  return check_launch(name);
}

template <typename VT>
int run_wide(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s) {
  const WideCfg wc = wide_variant(p->opts.variant);
  if (wc.tmem) {
    switch (p->opts.variant) {
      case 18: return launch_tmem<VT, 8, 4, 1>(p, x, o, s, "stream_tmem<8,s4,w4>");
      case 19: return launch_tmem<VT, 16, 2, 1>(p, x, o, s, "stream_tmem<16,s2,w4>");
      case 20: return launch_tmem<VT, 8, 2, 2>(p, x, o, s, "stream_tmem<8,s2,w8>");
      default: return launch_tmem<VT, 16, 2, 2>(p, x, o, s, "stream_tmem<16,s2,w8>");
    }
  }
  if (wc.tma) return launch_wide_tma<VT, 16, 2, 4>(p, x, o, s, "stream_wide_tma<16,s2,w4>");
  const bool d = p->opts.col_kind == ISPMV_COL_D16;
  if constexpr (sizeof(VT) == 4) {
    if (p->opts.val_kind == ISPMV_VAL_F32_LO16) {  // plain loads, FP64 x (setup checks)
      if (wc.spl == 8)
        return d ? launch_wide<VT, 8, 4, true, false, false, true>(p, x, o, s, "stream_wide<8,w0,b4,d16,lo>")
                 : launch_wide<VT, 8, 4, false, false, false, true>(p, x, o, s, "stream_wide<8,w0,b4,lo>");
      return d ? launch_wide<VT, 16, 3, true, false, false, true>(p, x, o, s, "stream_wide<16,w0,b3,d16,lo>")
               : launch_wide<VT, 16, 3, false, false, false, true>(p, x, o, s, "stream_wide<16,w0,b3,lo>");
    }
  }
  if (wc.pfc)  // u32 columns (setup checks)
    return launch_wide<VT, 8, 4, false, false, false, false, true>(p, x, o, s, "stream_wide<8,w0,b4,pfc>");
  if (wc.stg) {
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0)
      return launch_wide<VT, 8, 4, false, false, true>(p, x, o, s, "stream_wide<8,stg,b4>");
    // x not 16-byte aligned (no bulk copy): plain loads over the same stream
    return launch_wide<VT, 8, 4>(p, x, o, s, "stream_wide<8,w0,b4>");
  }
  if (wc.tex)  // texture gathers (loads where x does not fit a texture)
    return d ? launch_wide<VT, 8, 4, true, true>(p, x, o, s, "stream_wide<8,w0,b4,d16,tex>")
             : launch_wide<VT, 8, 4, false, true>(p, x, o, s, "stream_wide<8,w0,b4,tex>");
  if (wc.spl == 8)
    return d ? launch_wide<VT, 8, 4, true>(p, x, o, s, "stream_wide<8,w0,b4,d16>")
             : launch_wide<VT, 8, 4>(p, x, o, s, "stream_wide<8,w0,b4>");
  return d ? launch_wide<VT, 16, 3, true>(p, x, o, s, "stream_wide<16,w0,b3,d16>")
           : launch_wide<VT, 16, 3>(p, x, o, s, "stream_wide<16,w0,b3>");
}

template <typename VT>
int run_stream(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s) {
  if (p->opts.kernel == ISPMV_KERNEL_WIDE) return run_wide<VT>(p, x, o, s);
  const VT *val = static_cast<const VT *>(p->val);
  size_t nslots = p->slots, spad = p->slots_pad, sslots = p->seg_slots, nseg = p->nseg;
  const UIN *col = p->col, *heads = p->heads, *segh = p->segh;
  if (narrow_kinds(p)) {
    const unsigned g = (unsigned)((nseg * 32 + 255) / 256);
    const bool lo = p->opts.val_kind == ISPMV_VAL_F32_LO16, d16 = p->opts.col_kind == ISPMV_COL_D16;
    if (lo && d16)
      sss::stream_narrow<VT, true, true><<<g, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, p->narrow, x, o);
    else if (lo)
      sss::stream_narrow<VT, true, false><<<g, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, p->narrow, x, o);
    else
      sss::stream_narrow<VT, false, true><<<g, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, p->narrow, x, o);
    return check_launch("stream_narrow");
  }
  if (p->opts.kernel == ISPMV_KERNEL_TMA) {
    int *status = p->status;
    void *args[] = {&nslots, &spad, &sslots, &nseg, &val, &col, &heads, &segh, (void *)&x, &o, &status};
    const int cps = p->opts.ctas_per_sm;
    // 8 warps per CTA, 2 stages of 256 slots per warp; CTAs per SM from shared memory
    return launch_staged_w<8>(sss::stream_tma<VT, 8, 2, 256>, sss::smem_bytes<8, 2, VT, 256>(), nseg,
                              cps ? cps : 4, s, "stream_tma<8,2,256>", args);
  }
  if (p->opts.variant == ISPMV_VARIANT_QUEUE) {
    ISPMV_TRY(cudaMemsetAsync(p->queue, 0, sizeof(unsigned long long), s));
    const size_t warps = std::min<size_t>(nseg, (size_t)sm_count() * 6 * 8);
    const unsigned gq = (unsigned)std::max<size_t>(1, (warps + 7) / 8);
    sss::stream_queue<VT><<<gq, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, x, p->queue, o);
    return check_launch("stream_queue");
  }
  const unsigned g = (unsigned)((nseg * 32 + 255) / 256);
  // variants: slots per lane x prefetch depth (batches in flight) x CTAs per
  // SM the register budget allows; the default (variant 0) is (4, 0, 5)
  const char *nm = "stream_ldg";
#define ISPMV_SSS(SPL, PD, MINB)                                                                              \
  sss::stream_ldg<VT, SPL, PD, MINB><<<g, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, x, o); \
  nm = "stream_ldg<" #SPL "," #PD "," #MINB ">";                                                                \
  break
#define ISPMV_SSS_PF(SPL, PD, MINB, PF)                                                              \
  sss::stream_ldg<VT, SPL, PD, MINB, PF><<<g, 256, 0, s>>>(nslots, spad, sslots, nseg, val, col, heads, segh, x, \
                                                           o);                                                   \
  nm = "stream_ldg<" #SPL "," #PD "," #MINB ",pf" #PF ">";                                                      \
  break
  switch (p->opts.variant) {
    case 2: ISPMV_SSS(4, 0, 6);
    case 12: ISPMV_SSS_PF(4, 0, 6, 2);
    default: ISPMV_SSS(4, 0, 5);
  }
#undef ISPMV_SSS
#undef ISPMV_SSS_PF
  return check_launch(nm);
}

template <typename VT>
int run_units(ispmv_plan_s *p, const FPT *x, seg::Out &o, cudaStream_t s) {
  const VT *val = static_cast<const VT *>(p->val);
  if (p->opts.kernel == ISPMV_KERNEL_TMA) {
    using L = tk::StageLayout<VT>;
    size_t nunits = p->nunits, spad = p->slots_pad, nseg = p->nseg, sslots = p->seg_slots;
    const UIN *col = p->col, *urow = p->rows;
    int *status = p->status;
    void *args[] = {&nunits, &spad, &nseg, &sslots, &val, &col, &urow, (void *)&x, &o, &status};
    const int cps = p->opts.ctas_per_sm;
    switch (p->th) {
      case 4:
        return launch_staged(tk::nocn_tma<VT, 4, TW, TS>, tk::smem_bytes<TW, TS>(L::VB + L::CB + (tk::SS / 4) * 4),
                             nseg, cps, s, "nocn_tma<4>", args);
      case 8:
        return launch_staged(tk::nocn_tma<VT, 8, TW, TS>, tk::smem_bytes<TW, TS>(L::VB + L::CB + (tk::SS / 8) * 4),
                             nseg, cps, s, "nocn_tma<8>", args);
      case 16:
        return launch_staged(tk::nocn_tma<VT, 16, TW, TS>,
                             tk::smem_bytes<TW, TS>(L::VB + L::CB + (tk::SS / 16) * 4), nseg, cps, s, "nocn_tma<16>",
                             args);
      default:
        return ISPMV_ERR_UNSUPPORTED;
    }
  }
  const unsigned g = (unsigned)((p->nseg * 32 + pk::TPB - 1) / pk::TPB);
  pk::noc_hn<VT><<<g, pk::TPB, 0, s>>>(p->nunits, p->nseg, p->th, p->useg, p->rows, p->col, val, x, o);
  return check_launch("noc_hn");
}

// Kernel timing marks: `which` 0 before the main kernel of a product, 1 after it.
int tmark(ispmv_plan_s *p, cudaStream_t s, int which) {
  if (!p->tcap || p->capturing) return ISPMV_OK;
  const size_t i = p->tcount % p->tcap;
  ISPMV_TRY(cudaEventRecord(p->tev[2 * i + which], s));
  if (which) p->tcount++;
  return ISPMV_OK;
}

template <typename VT>
int run_main(ispmv_plan_s *p, const FPT *x, FPT *y, int beta, cudaStream_t s);

template <typename VT>
int run(ispmv_plan_s *p, const FPT *x, FPT *y, int beta, cudaStream_t s) {
  TRY(tmark(p, s, 0));
  const int st = run_main<VT>(p, x, y, beta, s);
  if (st) return st;
  p->kname = last_launch();
  // the kernel after the main one (the row fix-up, K1's reorder) is a
  // programmatic dependent launch when nothing (a timing event) sits between
  // the two in the stream
  const bool pdl = !p->tcap || p->capturing;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  if (p->path == P_STREAM || p->path == P_UNITS) {
    TRY(tmark(p, s, 1));
    const size_t nrec = p->slots ? 2 * p->nseg : 0;
    const size_t work = std::max(nrec, p->nempty);
    if (work) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)((work + 255) / 256));
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = 0;
      cfg.stream = s;
      cfg.attrs = at;
      cfg.numAttrs = pdl ? 1 : 0;
      ISPMV_TRY(cudaLaunchKernelEx(&cfg, p->long_rows ? seg::fixup<true> : seg::fixup<false>, nrec, (const UIN *)p->rec_row, (const double *)p->rec_sum,
                                   (const UIN *)p->rowmap, (const UIN *)p->empty, p->nempty, y, beta));
      return check_launch("fixup");
    }
    return ISPMV_OK;
  }
  if (p->path == P_K1 && p->fmt != F_K1P) {
    TRY(tmark(p, s, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((p->n + 255) / 256));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    ISPMV_TRY(cudaLaunchKernelEx(&cfg, pk::k1_order, p->n, (const UIN *)p->permi, (const FPT *)p->res, y, beta));
    return check_launch("k1_order");
  }
  return tmark(p, s, 1);
}

// The main kernel of one product.
template <typename VT>
int run_main(ispmv_plan_s *p, const FPT *x, FPT *y, int beta, cudaStream_t s) {
  const VT *val = static_cast<const VT *>(p->val);
  switch (p->path) {
    case P_ROWS: {
      if (p->fmt == F_AXC) {
        const unsigned g = (unsigned)(((size_t)p->n * 8 + pk::TPB - 1) / pk::TPB);
        pk::axc_rows<VT><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta);
        return check_launch("axc_rows");
      }
      const size_t thr = (size_t)p->n * p->lanes;
      const unsigned g = (unsigned)((thr + pk::TPB - 1) / pk::TPB);
      switch (p->lanes) {
        case 2: pk::csr_vec<VT, 2><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta); break;
        case 4: pk::csr_vec<VT, 4><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta); break;
        case 8: pk::csr_vec<VT, 8><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta); break;
        case 16: pk::csr_vec<VT, 16><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta); break;
        default: pk::csr_vec<VT, 32><<<g, pk::TPB, 0, s>>>(p->n, p->rows, p->col, val, x, y, beta); break;
      }
      return check_launch("csr_vec");
    }
    case P_SLICES: {
      const UIN ns = (p->n + 31) / 32;
      auto *k = p->slice_w <= 5 ? sl::slice_rows<VT, 5> : sl::slice_rows<VT, 9>;
      return launch_dependent("slice_rows<rows32,d16>", k, (ns + pk::TPB / 32 - 1) / (pk::TPB / 32), pk::TPB, 0, s,
                              overlaps(p), p->n, ns, p->slices, p->slen, p->narrow.col16, val, x, y, beta);
    }
    case P_K1: {
      const unsigned g = (unsigned)pk::k1_ctas(p->chunkNum, p->k1_cta, p->k1_long);
      if (p->fmt == F_K1P)
        return launch_dependent("k1_chunks<scatter>", pk::k1_chunks<VT, true>, g, pk::TPB, 0, s, overlaps(p), p->n,
                                p->chunkNum, p->k1_cta, p->k1_long, p->chp, p->nmc, p->permi, p->col, val, x, y, beta);
      return launch_dependent("k1_chunks", pk::k1_chunks<VT, false>, g, pk::TPB, 0, s, overlaps(p), p->n, p->chunkNum,
                              p->k1_cta, p->k1_long, p->chp, p->nmc, p->permi, p->col, val, x, p->res, beta);
    }
    case P_STREAM:
    case P_UNITS: {
      seg::Out o{y, p->rowmap, p->rec_row, p->rec_sum, beta};
      if (p->slots) TRY(p->path == P_STREAM ? run_stream<VT>(p, x, o, s) : run_units<VT>(p, x, o, s));
      return ISPMV_OK;
    }
    default:
      return ISPMV_ERR_ARG;
  }
}

}  // namespace

ISPMV_API int ispmv_plan_spmv(ispmv_plan p, const FPT *x, FPT *y, int beta, void *stream) {
  if (!p || !x || !y || (beta != 0 && beta != 1)) return ISPMV_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (p->opts.val_kind == ISPMV_VAL_F64) return run<double>(p, x, y, beta, s);
  return run<float>(p, x, y, beta, s);
}

// Streams to capture graph products on, kept between captures: a stream made
// for a plan and destroyed with it took 65-100 us of the plan's first graph
// product, and the driver then keeps less for the graphs (50,000 FEM rows, a
// new plan's first graph product 330 -> 113 us, a new x on the same plan 148 ->
// 36).  A capture has its stream for itself; those of other contexts are left
// alone.
namespace {
struct CaptureStream {
  static constexpr size_t MOST = 4;  // kept
  struct Idle {
    std::mutex mu;
    std::vector<std::pair<unsigned long long, cudaStream_t>> v;  // context, stream
  };
  static Idle &idle() {
    static Idle *i = new Idle();  // never destroyed: plans may outlive static objects
    return *i;
  }
  cudaStream_t s = nullptr;
  int open() {
    const unsigned long long ctx = current_ctx_id();
    {
      std::lock_guard<std::mutex> g(idle().mu);
      auto &v = idle().v;
      for (size_t i = 0; i < v.size() && !s; i++)
        if (ctx && v[i].first == ctx) {
          s = v[i].second;
          v.erase(v.begin() + i);
        }
    }
    if (!s) ISPMV_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    return ISPMV_OK;
  }
  ~CaptureStream() {
    if (!s) return;
    const unsigned long long ctx = current_ctx_id();
    {
      std::lock_guard<std::mutex> g(idle().mu);
      if (ctx && idle().v.size() < MOST) {
        idle().v.emplace_back(ctx, s);
        return;
      }
    }
    cudaStreamDestroy(s);
  }
};
}  // namespace

ISPMV_API int ispmv_plan_spmv_graph(ispmv_plan p, const FPT *x, FPT *y, int beta, void *stream) {
  if (!p || !x || !y || (beta != 0 && beta != 1)) return ISPMV_ERR_ARG;
  if (!p->graph_exec || p->g_x != x || p->g_y != y || p->g_beta != beta) {
    if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    p->graph_exec = nullptr;
    p->graph = nullptr;
    CaptureStream cap;
    TRY(cap.open());
    // work areas a product allocates on first use, allocated before the
    // capture (no allocation may happen inside it): the FP32 copy of x of
    // FP32-value plans on the lane-interleaved kernel
    if (p->opts.val_kind != ISPMV_VAL_F64 && p->opts.kernel == ISPMV_KERNEL_WIDE && p->path == P_STREAM && !p->x32)
      TRY(dev_alloc(p, p->n, &p->x32));
    ISPMV_TRY(cudaStreamBeginCapture(cap.s, cudaStreamCaptureModeThreadLocal));
    p->capturing = true;
    const int st = p->opts.val_kind == ISPMV_VAL_F64 ? run<double>(p, x, y, beta, cap.s)
                                                     : run<float>(p, x, y, beta, cap.s);
    p->capturing = false;
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(cap.s, &g);
    if (st || e != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      // a failed capture leaves its error as the runtime's last error: clear
      // it so that it is not reported again by a later, unrelated call
      (void)cudaGetLastError();
      return st ? st : cuda_status(e, "cudaStreamEndCapture");
    }
    p->graph = g;
    ISPMV_TRY(cudaGraphInstantiate(&p->graph_exec, p->graph, 0));
    p->g_x = x;
    p->g_y = y;
    p->g_beta = beta;
  }
  ISPMV_TRY(cudaGraphLaunch(p->graph_exec, as_stream(stream)));
  count_launch();
  return ISPMV_OK;
}

ISPMV_API int ispmv_plan_time_kernels(ispmv_plan p, int pairs) {
  if (!p || pairs < 0) return ISPMV_ERR_ARG;
  for (cudaEvent_t e : p->tev) cudaEventDestroy(e);
  p->tev.clear();
  p->tcap = 0;
  p->tcount = 0;
  for (int i = 0; i < 2 * pairs; i++) {
    cudaEvent_t e;
    ISPMV_TRY(cudaEventCreate(&e));
    p->tev.push_back(e);
  }
  p->tcap = (size_t)pairs;
  return ISPMV_OK;
}

ISPMV_API int ispmv_plan_kernel_ms(ispmv_plan p, double *total_ms, int *launches) {
  if (!p || !total_ms || !launches) return ISPMV_ERR_ARG;
  const size_t m = std::min(p->tcount, p->tcap);
  double sum = 0.0;
  for (size_t i = 0; i < m; i++) {
    float ms = 0.f;
    ISPMV_TRY(cudaEventElapsedTime(&ms, p->tev[2 * i], p->tev[2 * i + 1]));
    sum += ms;
  }
  *total_ms = sum;
  *launches = (int)m;
  p->tcount = 0;
  return ISPMV_OK;
}

ISPMV_API int ispmv_plan_time_main(ispmv_plan p, const FPT *x, FPT *y, int reps, void *stream, double *ms) {
  if (!p || !x || !y || reps < 1 || !ms) return ISPMV_ERR_ARG;
  if (p->capturing) return fail(ISPMV_ERR_ARG, "ispmv_plan_time_main: not inside a graph capture");
  cudaStream_t s = as_stream(stream);
  auto ck = [](cudaError_t e, const char *where) { return e == cudaSuccess ? ISPMV_OK : cuda_status(e, where); };
  cudaEvent_t e[2] = {nullptr, nullptr};
  ISPMV_TRY(cudaEventCreate(&e[0]));
  int st = ck(cudaEventCreate(&e[1]), "cudaEventCreate");
  if (!st) st = ck(cudaEventRecord(e[0], s), "cudaEventRecord");
  p->alone = true;
  for (int i = 0; i < reps && !st; i++)
    st = p->opts.val_kind == ISPMV_VAL_F64 ? run_main<double>(p, x, y, 0, s) : run_main<float>(p, x, y, 0, s);
  p->alone = false;
  if (!st) st = ck(cudaEventRecord(e[1], s), "cudaEventRecord");
  if (!st) st = ck(cudaEventSynchronize(e[1]), "cudaEventSynchronize");
  float t = 0.f;
  if (!st) st = ck(cudaEventElapsedTime(&t, e[0], e[1]), "cudaEventElapsedTime");
  for (cudaEvent_t ev : e)
    if (ev) cudaEventDestroy(ev);
  if (!st) *ms = (double)t / reps;
  return st;
}

ISPMV_API const char *ispmv_plan_kernel_name(ispmv_plan p) { return p ? p->kname : ""; }

ISPMV_API int ispmv_plan_status(ispmv_plan p) {
  if (!p) return ISPMV_ERR_ARG;
  if (!p->status) return ISPMV_OK;
  int v = 0;
  ISPMV_TRY(cudaMemcpy(&v, p->status, sizeof v, cudaMemcpyDeviceToHost));
  return v;
}

ISPMV_API int ispmv_plan_spmv_host(ispmv_plan p, const FPT *h_x, FPT *h_y, void *stream) {
  if (!p || !h_x || !h_y) return ISPMV_ERR_ARG;
  if (!p->hx) {
    TRY(dev_alloc(p, p->n, &p->hx));
    TRY(dev_alloc(p, p->n, &p->hy));
  }
  cudaStream_t s = as_stream(stream);
  ISPMV_TRY(cudaMemcpyAsync(p->hx, h_x, (size_t)p->n * sizeof(FPT), cudaMemcpyHostToDevice, s));
  TRY(ispmv_plan_spmv(p, p->hx, p->hy, 0, stream));
  ISPMV_TRY(cudaMemcpyAsync(h_y, p->hy, (size_t)p->n * sizeof(FPT), cudaMemcpyDeviceToHost, s));
  ISPMV_TRY(cudaStreamSynchronize(s));
  return ispmv_plan_status(p);
}

namespace {
// Slots per lane of a lane-interleaved (stream_wide) plan, 0 for slot order.
unsigned il_spl(const ispmv_plan_s *p) {
  return p->opts.kernel == ISPMV_KERNEL_WIDE ? (unsigned)wide_variant(p->opts.variant).spl : 0u;
}
bool tmem_plan(const ispmv_plan_s *p) {
  return p->opts.kernel == ISPMV_KERNEL_WIDE && wide_variant(p->opts.variant).tmem;
}

// Slots per group of the SpMM kernel, whole chunks (a multiple of 64): an even
// share of as many loads of the GPU's `held` groups as keep it at 192 or less.
// Longer parts spread the resident groups over more of the matrix (less of X
// found in L2), shorter ones pay their start more often: k = 8 / 32 on
// power-law rows 144 / 323 us at 128 slots, 138 / 330 at 192, 149 / 339 at 256
// (the same X each time).
size_t spmm_part(size_t slots, size_t held) {
  const size_t loads = std::max<size_t>(1, (slots + held * 192 - 1) / (held * 192));
  return std::max<size_t>(64, ((slots + loads * held - 1) / (loads * held) + 63) / 64 * 64);
}

// One pass per block of CB = G*W right-hand sides (G lanes per group, W
// columns per lane).
template <int G, int W, int T, int MINB, bool VEC, typename VT>
int spmm_blocks(ispmv_plan_s *p, UIN k, const FPT *X, FPT *Y, cudaStream_t s, const char *name) {
  constexpr int NG = 32 / G, CB = G * W;
  const size_t part = spmm_part(p->slots_pad, (size_t)sm_count() * MINB * 8 * NG);
  const size_t nparts = (p->slots_pad + part - 1) / part, ctas = (nparts + 8 * NG - 1) / (8 * NG), nrec = 2 * ctas;
  if (p->mm_rows_cap < nrec) {
    TRY(dev_alloc(p, nrec, &p->mm_row));
    p->mm_rows_cap = nrec;
  }
  if (p->mm_cap < (nparts + nrec) * CB) {
    TRY(dev_alloc(p, (nparts + nrec) * CB, &p->mm_sum));
    p->mm_cap = (nparts + nrec) * CB;
  }
  const unsigned spl = il_spl(p);
  if (spl != 0 && spl != 8 && spl != 16)
    return fail(ISPMV_ERR_UNSUPPORTED, "ispmv_plan_spmm: lane-interleaved plans of 8 or 16 slots per lane");
  const mm::Stream st{p->slots, p->slots_pad, p->seg_slots, p->val, p->col, p->heads, p->segh,
                      spl == 16 ? 4u : spl == 8 ? 3u : 0u};
  for (UIN j0 = 0; j0 < k; j0 += CB) {
    mm::Out o{Y, p->rowmap, p->mm_sum, p->mm_row, p->mm_sum + nparts * CB, k, j0, std::min<UIN>(CB, k - j0)};
    mm::stream_spmm<G, W, T, MINB, VEC, VT><<<(unsigned)ctas, 256, 0, s>>>(st, part, nparts, X, o);
    TRY(check_launch(name));
    p->kname = last_launch();
    TRY(launch_dependent("spmm_fixup", mm::spmm_fixup<CB>, (std::max(nrec, p->nempty) * CB + 255) / 256, 256, 0, s,
                         true, nrec, p->empty, p->nempty, o));
  }
  return ISPMV_OK;
}

// Two columns per lane: 16-byte X loads where k is even and X and Y are
// 16-byte aligned, else column by column.
template <int G, typename VT>
int spmm_two(ispmv_plan_s *p, UIN k, const FPT *X, FPT *Y, cudaStream_t s) {
  if ((k & 1u) == 0 && k < (1u << 29) && ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 15u) == 0)
    return spmm_blocks<G, 2, 8, 3, true, VT>(p, k, X, Y, s, "stream_spmm");
  return spmm_blocks<G, 2, 8, 3, false, VT>(p, k, X, Y, s, "stream_spmm");
}

// RHS block 8, 16 or 32 columns (ispmv_plan_opts.rhs_block, else by k).
// spmm_kernel: WIDE four columns per lane with 32-byte X loads (k a
// multiple of 4, X and Y 32-byte aligned); LDG two columns per lane (4, 8 or 16
// lanes per group); AUTO the four-column form for blocks of 16 and 32
// columns where it applies, else two (on 8-column blocks the two-column
// form is the faster with FP64 values).
template <typename VT>
int spmm_run(ispmv_plan_s *p, UIN k, const FPT *X, FPT *Y, cudaStream_t s) {
  int g = p->opts.rhs_block;
  if (g != 8 && g != 16 && g != 32) g = k <= 8 ? 8 : k <= 16 ? 16 : 32;
  const bool four_ok = (k & 3u) == 0 && k < (1u << 29) && ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 31u) == 0;
  const int kind = p->opts.spmm_kernel;
  if (kind == ISPMV_KERNEL_WIDE && !four_ok)
    return fail(ISPMV_ERR_UNSUPPORTED,
                "ispmv_plan_spmm: four columns per lane need k a multiple of 4 and X, Y 32-byte aligned");
  if (four_ok && (kind == ISPMV_KERNEL_WIDE || (kind == ISPMV_KERNEL_AUTO && g > 8))) {
    if (g == 8) return spmm_blocks<2, 4, 4, 3, true, VT>(p, k, X, Y, s, "stream_spmm4");
    if (g == 16) return spmm_blocks<4, 4, 8, 2, true, VT>(p, k, X, Y, s, "stream_spmm4");
    return spmm_blocks<8, 4, 8, 2, true, VT>(p, k, X, Y, s, "stream_spmm4");
  }
  if (g == 8) return spmm_two<4, VT>(p, k, X, Y, s);
  if (g == 16) return spmm_two<8, VT>(p, k, X, Y, s);
  return spmm_two<16, VT>(p, k, X, Y, s);
}
}  // namespace

// Y = A X for k right-hand sides (row-major n x k): the slot-stream plans
// (AXT COM, AXT tileH=1, AXC and CSR built with the stream kernels).
ISPMV_API int ispmv_plan_spmm(ispmv_plan p, UIN k, const FPT *X, FPT *Y, void *stream) {
  if (!p || !X || !Y || k == 0) return ISPMV_ERR_ARG;
  if (p->path != P_STREAM || narrow_kinds(p) || tmem_plan(p))
    return fail(ISPMV_ERR_UNSUPPORTED, "ispmv_plan_spmm: needs a slot-stream plan with u32 columns");
  cudaStream_t s = as_stream(stream);
  if (!p->slots) {  // every row empty
    ISPMV_TRY(cudaMemsetAsync(Y, 0, (size_t)p->n * k * sizeof(FPT), s));
    return ISPMV_OK;
  }
  if (p->opts.val_kind == ISPMV_VAL_F64) return spmm_run<double>(p, k, X, Y, s);
  return spmm_run<float>(p, k, X, Y, s);
}
