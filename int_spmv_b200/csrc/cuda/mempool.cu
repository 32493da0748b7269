// mempool.cu - device memory of plans, GPU-built formats and builder scratch.
//
// cudaMalloc and cudaFree map and unmap memory: a plan built from a device
// CSR and dropped again after one product (a matrix assembled anew in every
// step) spent 5-11 ms of its 6-12 on them at n = 1M, 14.9M nonzeros, where
// its kernels take 0.9.  Freed blocks are kept here, by device, and given
// to later requests of nearly their size.
//   - Bounded: at most POOL_MAX bytes are kept; the block kept longest goes
//     first.  ispmv_pool_trim gives them back on demand, and a failing
//     cudaMalloc empties the pool and tries again.
//   - A block is kept only once no work can use it any more: the caller has
//     synchronised the stream it was used on (idle = true), or all work on the
//     device is waited for here with a cudaFree, as dropping a plan always did
//     (wait_for_work).  Where that fails the block itself goes to cudaFree.
//   - Blocks belong to the context they were allocated in: they are given out
//     and freed in it alone; those of a context that was destroyed
//     (cudaDeviceReset) are forgotten.
//   - One lock; the pool lives until the process ends.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace ispmv {
namespace {

constexpr size_t POOL_MAX = (size_t)2 << 30;

// Driver calls through the runtime's entry points, so the library links no
// driver library.  Null when unavailable.
typedef CUresult(CUDAAPI *CtxGetCurrentFn)(CUcontext *);
typedef CUresult(CUDAAPI *CtxGetIdFn)(CUcontext, unsigned long long *);
typedef CUresult(CUDAAPI *CtxPushFn)(CUcontext);
typedef CUresult(CUDAAPI *CtxPopFn)(CUcontext *);
typedef CUresult(CUDAAPI *PtrGetAttrFn)(void *, CUpointer_attribute, CUdeviceptr);
CtxGetCurrentFn g_ctx_current = nullptr;
CtxGetIdFn g_ctx_id = nullptr;
CtxPushFn g_ctx_push = nullptr;
CtxPopFn g_ctx_pop = nullptr;
PtrGetAttrFn g_ptr_attr = nullptr;
std::once_flag g_ctx_fns_once;

template <typename F>
void find_fn(const char *name, F *fn) {
  void *f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
    *fn = reinterpret_cast<F>(f);
}
void find_ctx_fns() {
  find_fn("cuCtxGetCurrent", &g_ctx_current);
  find_fn("cuCtxGetId", &g_ctx_id);
  find_fn("cuCtxPushCurrent", &g_ctx_push);
  find_fn("cuCtxPopCurrent", &g_ctx_pop);
  find_fn("cuPointerGetAttribute", &g_ptr_attr);
  (void)cudaGetLastError();
}

struct Block {
  void *ptr;
  size_t bytes;
  int dev;
  unsigned long long ctx;
};
struct Pool {
  std::mutex mu;
  std::vector<Block> kept;                  // oldest first
  size_t kept_bytes = 0;
  std::unordered_map<void *, Block> live;   // blocks handed out
  std::vector<unsigned long long> anchors;  // contexts that hold wait_for_work's anchor
};
Pool &pool() {
  static Pool *p = new Pool();  // never destroyed: plans may outlive static objects
  return *p;
}

// Requests are rounded up to steps of 1/8 of their power of two (512 bytes at
// least, STEP_MAX at most), so that a matrix of nearly the same size finds the
// same blocks; those too large to be kept are left as they are.
constexpr size_t STEP_MAX = (size_t)8 << 20;
size_t rounded(size_t n) {
  size_t step = 512;
  while (step * 16 <= n && step < STEP_MAX) step *= 2;
  if (n > POOL_MAX) step = 512;
  return std::max<size_t>(1, (n + step - 1) / step) * step;
}

// Waits for all work on the current device, on every stream, by freeing an
// allocation of no use: cudaFree waits for it.  cudaDeviceSynchronize waits
// too, but it is prohibited while any stream of the device is being captured
// and ends that capture, whatever its mode; cudaFree is allowed beside another
// thread's thread-local or relaxed capture.  `anchors` holds one allocation
// per context beside it, so that the small pages stay mapped: 10 us for the
// pair, 700 us where they are mapped and unmapped each time.
bool wait_for_work(Pool &p) {
  const unsigned long long ctx = current_ctx_id();
  void *a = nullptr, *t = nullptr;
  bool ok = true;
  {
    std::lock_guard<std::mutex> g(p.mu);
    if (std::find(p.anchors.begin(), p.anchors.end(), ctx) == p.anchors.end()) {
      ok = cudaMalloc(&a, 512) == cudaSuccess;
      if (ok) p.anchors.push_back(ctx);
    }
  }
  ok = ok && cudaMalloc(&t, 512) == cudaSuccess && cudaFree(t) == cudaSuccess;
  if (!ok) (void)cudaGetLastError();
  return ok;
}

// Gives a kept block back, in the context it was allocated in, whatever the
// calling thread's device and context are.  The driver names the context that
// owns the address now: another one than the block's, or none, means that the
// block's context was destroyed and its memory with it.
void give_back(const Block &b) {
  CUcontext c = nullptr, popped;
  unsigned long long id = 0;
  if (!g_ctx_push || !g_ctx_pop || !g_ptr_attr) {  // no driver entry points: no context to choose
    if (cudaFree(b.ptr) != cudaSuccess) (void)cudaGetLastError();
    return;
  }
  if (g_ptr_attr(&c, CU_POINTER_ATTRIBUTE_CONTEXT, (CUdeviceptr)(uintptr_t)b.ptr) != CUDA_SUCCESS || !c ||
      g_ctx_id(c, &id) != CUDA_SUCCESS || id != b.ctx || g_ctx_push(c) != CUDA_SUCCESS)
    return;
  if (cudaFree(b.ptr) != cudaSuccess) (void)cudaGetLastError();
  (void)g_ctx_pop(&popped);
}

// Gives kept blocks back, oldest first, until at most `keep` bytes are kept.
void trim_locked(Pool &p, size_t keep) {
  size_t k = 0;
  for (; k < p.kept.size() && p.kept_bytes > keep; k++) {
    p.kept_bytes -= p.kept[k].bytes;
    give_back(p.kept[k]);
  }
  p.kept.erase(p.kept.begin(), p.kept.begin() + k);
}

}  // namespace

unsigned long long current_ctx_id() {
  std::call_once(g_ctx_fns_once, find_ctx_fns);
  if (!g_ctx_current || !g_ctx_id) return 0;
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (g_ctx_current(&c) != CUDA_SUCCESS || !c) return 0;
  if (g_ctx_id(c, &id) != CUDA_SUCCESS) return 0;
  return id;
}

int pool_alloc(void **out, size_t bytes) {
  *out = nullptr;
  int dev = 0;
  ISPMV_TRY(cudaGetDevice(&dev));
  Pool &p = pool();
  const size_t want = rounded(bytes);
  {
    const unsigned long long ctx = current_ctx_id();
    std::lock_guard<std::mutex> g(p.mu);
    size_t best = p.kept.size();
    for (size_t i = 0; ctx && i < p.kept.size(); i++) {
      const Block &b = p.kept[i];
      if (b.dev == dev && b.ctx == ctx && b.bytes >= want && b.bytes <= want + want / 4 &&
          (best == p.kept.size() || b.bytes < p.kept[best].bytes))
        best = i;
    }
    if (best < p.kept.size()) {
      const Block b = p.kept[best];
      p.kept.erase(p.kept.begin() + best);
      p.kept_bytes -= b.bytes;
      p.live[b.ptr] = b;
      *out = b.ptr;
      return ISPMV_OK;
    }
  }
  void *ptr = nullptr;
  cudaError_t e = cudaMalloc(&ptr, want);
  if (e == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    {
      std::lock_guard<std::mutex> g(p.mu);
      trim_locked(p, 0);
    }
    e = cudaMalloc(&ptr, want);
  }
  if (e != cudaSuccess) return cuda_status(e, "cudaMalloc");
  const unsigned long long ctx = current_ctx_id();
  std::lock_guard<std::mutex> g(p.mu);
  p.live[ptr] = Block{ptr, want, dev, ctx};
  *out = ptr;
  return ISPMV_OK;
}

void pool_free(void *const *ptrs, size_t count, bool idle) {
  Pool &p = pool();
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) cur = -1;
  unsigned long long ctx = 0;
  int synced = -1;  // the device whose work is known to be done
  for (size_t i = 0; i < count; i++) {
    if (!ptrs[i]) continue;
    Block b{nullptr, 0, -1, 0};
    {
      std::lock_guard<std::mutex> g(p.mu);
      auto it = p.live.find(ptrs[i]);
      if (it != p.live.end()) {
        b = it->second;
        p.live.erase(it);
      }
    }
    bool keep = b.ptr && b.ctx && b.bytes <= POOL_MAX && cur >= 0;
    if (keep && synced != b.dev) {
      keep = (cur == b.dev || cudaSetDevice(b.dev) == cudaSuccess) &&
             (idle || wait_for_work(p));
      ctx = keep ? current_ctx_id() : 0;
      if (keep) synced = b.dev;
      else (void)cudaGetLastError();
      if (cur != b.dev) (void)cudaSetDevice(cur);
    }
    if (keep && ctx == b.ctx) {
      std::lock_guard<std::mutex> g(p.mu);
      p.kept.push_back(b);
      p.kept_bytes += b.bytes;
      trim_locked(p, POOL_MAX);
    } else if (cudaFree(ptrs[i]) != cudaSuccess) {
      (void)cudaGetLastError();
    }
  }
}

}  // namespace ispmv

ISPMV_API int ispmv_pool_trim(uint64_t keep_bytes, uint64_t *kept) {
  using namespace ispmv;
  Pool &p = pool();
  std::lock_guard<std::mutex> g(p.mu);
  trim_locked(p, (size_t)keep_bytes);
  if (kept) *kept = p.kept_bytes;
  return ISPMV_OK;
}
