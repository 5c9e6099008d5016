// ##################################################################
//
// trisolve.cu -- batched 4x4 block-tridiagonal solves on device arrays
//
// The reference's TRISOLVER::blockTridag4 (triSolvers.cpp:769-847) and
// blockTridagPeriodic4 (triSolvers.cpp:850-1046) as a batched entry point:
// two warps per line, factor_line_team and follow_line_team of
// line_solve.cuh, so each line's solution is bit-identical to one reference
// call.  A line is a recurrence over its rows; with the solve (and the periodic
// fill column) behind the factorisation in a second warp a row takes 1.95 us
// open and 2.43 us periodic, against 4.00 and 4.53 in one warp, and 52 FP64
// instructions against 66, so it is the better split from one line to lines that
// fill the GPU: one line of 128 rows 512 -> 251 us open, 583 -> 315 periodic, 400
// lines of 17 rows 70 -> 42 and 81 -> 54, 20,000 lines of 17 rows (FP64 pipe 82%
// busy either way) 1,434 -> 1,198 us.
// ##################################################################
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <string>

#include "../../include/hamstr_gpu.h"
#include "line_solve.cuh"

namespace hamstr {
void set_last_error(const std::string& m);
}

namespace {

using namespace hamstr;

__global__ void __launch_bounds__(64) block_tridag_kernel(int N, int periodic, const double* __restrict__ A,
                                                          const double* __restrict__ B, const double* __restrict__ C,
                                                          double* __restrict__ F, double* __restrict__ scratch)
{
   __shared__ TeamShared ts;
   const size_t line = blockIdx.x;
   const size_t nb = (size_t)N * 16;
   double* fac = scratch + line * ((size_t)kFacRec * N + 16);
   double* facN = fac + (size_t)kFacRec * N;
   const bool per = periodic != 0;
   const int lane = threadIdx.x & 31;
   team_init(&ts);
   __syncthreads();
   bool ok = true;
   if (threadIdx.x < 32)
      factor_line_team(A + line * nb, B + line * nb, C + line * nb, 16, N, per, fac, facN, lane, &ts, &ok);
   else
      follow_line_team(A + line * nb, 16, fac, facN, N, per, F + line * (size_t)N * 4, lane, &ts, &ok);
   // a wait that gave up (never expected, line_solve.cuh) leaves no plausible solution behind
   if (__syncthreads_or(!ok))
      for (int i = threadIdx.x; i < 4 * N; i += 64) F[line * (size_t)N * 4 + i] = __longlong_as_double(-1);
}

}  // namespace

namespace hamstr {

// validation shared by the block-tridiagonal entry points
int block_tridag_check(int nlines, int N, int periodic, const double* A, const double* B, const double* C,
                       const double* F)
{
   if (nlines < 0 || N < 1 || (periodic && N < 2) || (periodic != 0 && periodic != 1)) {
      set_last_error("block_tridag4: need nlines >= 0, N >= 1 (open) or N >= 2 (periodic)");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (nlines > 0 && (!A || !B || !C || !F)) {
      set_last_error("block_tridag4: null array");
      return HAMSTR_GPU_ERR_ARG;
   }
   return HAMSTR_GPU_OK;
}

int block_tridag_launch(int nlines, int N, int periodic, const double* A, const double* B, const double* C,
                        double* F, double* scratch, cudaStream_t st)
{
   if (nlines == 0) return HAMSTR_GPU_OK;
   block_tridag_kernel<<<nlines, 64, 0, st>>>(N, periodic, A, B, C, F, scratch);
   const cudaError_t e = cudaGetLastError();
   if (e != cudaSuccess) {
      set_last_error(std::string("block_tridag4 launch: ") + cudaGetErrorString(e));
      return HAMSTR_GPU_ERR_CUDA;
   }
   return HAMSTR_GPU_OK;
}

}  // namespace hamstr

namespace {

// The allocating entry point's scratch: a stream-ordered pool of its own per
// device, so that a call neither maps fresh memory nor waits for the whole
// device as cudaMalloc and cudaFree do (384 x 96, both directions: about 80 us
// of two calls).  It keeps at most kPoolKept bytes between calls; more goes
// back to the device when the call's stream is synchronised.  The allocator
// orders reuse between streams and threads.
constexpr unsigned long long kPoolKept = 64ull << 20;
//
// cudaDeviceReset ends the device's context and the pool with it, so a pool goes
// by the id of the context it was made in, which is never used again.
constexpr int kMaxDevices = 64;
std::mutex g_pool_mutex;
struct ContextPool {
   unsigned long long context;
   cudaMemPool_t pool;
};
ContextPool g_pool[kMaxDevices] = {};

template <typename F>
F driver_entry(const char* name, unsigned version)
{
   void* p = nullptr;
   cudaDriverEntryPointQueryResult q;
   const bool ok = cudaGetDriverEntryPointByVersion(name, &p, version, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess;
   return ok ? reinterpret_cast<F>(p) : nullptr;
}

// the id of the device's primary context, the one the runtime works in
cudaError_t primary_context_id(int dev, unsigned long long* id)
{
   static const auto retain = driver_entry<PFN_cuDevicePrimaryCtxRetain_v7000>("cuDevicePrimaryCtxRetain", 7000);
   static const auto release = driver_entry<PFN_cuDevicePrimaryCtxRelease_v11000>("cuDevicePrimaryCtxRelease", 11000);
   static const auto state = driver_entry<PFN_cuDevicePrimaryCtxGetState_v7000>("cuDevicePrimaryCtxGetState", 7000);
   static const auto ctx_id = driver_entry<PFN_cuCtxGetId_v12000>("cuCtxGetId", 12000);
   if (!retain || !release || !state || !ctx_id) return cudaErrorNotSupported;
   unsigned flags = 0;
   int active = 0;
   if (state(dev, &flags, &active) != CUDA_SUCCESS) return cudaErrorInitializationError;
   if (!active) {   // the runtime makes and keeps the next one
      const cudaError_t e = cudaSetDevice(dev);
      if (e != cudaSuccess) return e;
   }
   CUcontext c = nullptr;
   if (retain(&c, dev) != CUDA_SUCCESS) return cudaErrorInitializationError;
   const CUresult r = ctx_id(c, id);
   release(dev);
   return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInitializationError;
}

cudaError_t scratch_pool(cudaMemPool_t* out)
{
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
   std::lock_guard<std::mutex> lock(g_pool_mutex);
   ContextPool& have = g_pool[dev];
   unsigned long long context = 0;
   e = primary_context_id(dev, &context);
   if (e != cudaSuccess) return e;
   if (!have.pool || have.context != context) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.handleTypes = cudaMemHandleTypeNone;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      cudaMemPool_t p = nullptr;
      e = cudaMemPoolCreate(&p, &props);
      if (e != cudaSuccess) return e;
      unsigned long long kept = kPoolKept;
      e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &kept);
      if (e != cudaSuccess) {
         cudaMemPoolDestroy(p);
         return e;
      }
      have = {context, p};
   }
   *out = have.pool;
   return cudaSuccess;
}

// Scratch the pool does not keep is mapped and unmapped on every call, and
// cudaMalloc does that faster than a pool does: open lines, pool / cudaMalloc,
// 200,000 of 17 rows (2.2 GB) 16.3 / 13.1 ms, 9,000 of 33 (192 MB) 1.49 / 1.38,
// 5,000 (106 MB) 0.86 / 0.85, 4,099 (87 MB, most of it kept) 0.67 / 0.72, 3,200 (68 MB)
// 0.56 / 0.62.  So the pool serves up to half as much again as it keeps.
constexpr size_t kPoolServes = kPoolKept + kPoolKept / 2;

cudaError_t scratch_alloc(double** p, size_t bytes, cudaStream_t s, bool* pooled)
{
   *pooled = bytes <= kPoolServes;
   if (!*pooled) return cudaMalloc((void**)p, bytes);
   cudaMemPool_t pool = nullptr;
   const cudaError_t e = scratch_pool(&pool);
   return e != cudaSuccess ? e : cudaMallocFromPoolAsync((void**)p, bytes, pool, s);
}

}  // namespace

extern "C" int hamstr_gpu_block_tridag4(int nlines, int N, int periodic, const double* A, const double* B,
                                        const double* C, double* F, void* stream)
{
   int st = block_tridag_check(nlines, N, periodic, A, B, C, F);
   if (st || nlines == 0) return st;
   const cudaStream_t s = (cudaStream_t)stream;
   double* scratch = nullptr;
   bool pooled = false;
   const size_t bytes = (size_t)nlines * ((size_t)kFacRec * N + 16) * sizeof(double);
   cudaError_t e = scratch_alloc(&scratch, bytes, s, &pooled);
   if (e != cudaSuccess) {
      cudaGetLastError();
      set_last_error(std::string("block_tridag4 scratch: ") + cudaGetErrorString(e));
      return e == cudaErrorMemoryAllocation ? HAMSTR_GPU_ERR_NOMEM : HAMSTR_GPU_ERR_CUDA;
   }
   st = block_tridag_launch(nlines, N, periodic, A, B, C, F, scratch, s);
   if (pooled) cudaFreeAsync(scratch, s);
   e = cudaStreamSynchronize(s);
   if (!pooled) cudaFree(scratch);
   if (st) return st;
   if (e != cudaSuccess) {
      set_last_error(std::string("block_tridag4: ") + cudaGetErrorString(e));
      return HAMSTR_GPU_ERR_CUDA;
   }
   return HAMSTR_GPU_OK;
}

// ------------------------------------------------------------------
// Allocation-free variant.
//
// Some callers cannot allocate device memory on every call, or wait for their
// stream in it: code that runs in a loop beside work on other streams, stream
// capture, and hosts whose device memory is owned by their own pool allocator
// with a fixed budget.  This variant runs the same kernel with its scratch in a
// fixed array that the library image places in device memory when it is
// loaded: every GPU that loads the library holds these 8 MiB until the
// process exits, and the call itself allocates nothing.
// ------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocScratchDoubles = size_t(1) << 20;   // 8 MiB
static __device__ __align__(256) double g_tridag_scratch[kNoAllocScratchDoubles];

std::mutex g_scratch_mutex;
struct ContextScratch {
   unsigned long long context;
   double* addr;
};
ContextScratch g_scratch_addr[kMaxDevices] = {};

// Device address of g_tridag_scratch on the current device, looked up once
// per context of the device (host code only sees a host-side stand-in for the
// symbol, and a reset loads the image anew).
int noalloc_scratch(double** out)
{
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) {
      set_last_error(std::string("block_tridag4_noalloc: cudaGetDevice: ") + cudaGetErrorString(e));
      return HAMSTR_GPU_ERR_CUDA;
   }
   if (dev < 0 || dev >= kMaxDevices) {
      set_last_error("block_tridag4_noalloc: device ordinal beyond 63");
      return HAMSTR_GPU_ERR_ARG;
   }
   unsigned long long context = 0;
   e = primary_context_id(dev, &context);
   if (e != cudaSuccess) {
      set_last_error(std::string("block_tridag4_noalloc: context: ") + cudaGetErrorString(e));
      return HAMSTR_GPU_ERR_CUDA;
   }
   std::lock_guard<std::mutex> lock(g_scratch_mutex);
   ContextScratch& have = g_scratch_addr[dev];
   if (!have.addr || have.context != context) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_tridag_scratch);
      if (e != cudaSuccess || !p) {
         set_last_error(std::string("block_tridag4_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
         return HAMSTR_GPU_ERR_CUDA;
      }
      have = {context, static_cast<double*>(p)};
   }
   *out = have.addr;
   return HAMSTR_GPU_OK;
}

}  // namespace

extern "C" int hamstr_gpu_block_tridag4_noalloc(int nlines, int N, int periodic, const double* A, const double* B,
                                                const double* C, double* F, void* stream)
{
   int st = block_tridag_check(nlines, N, periodic, A, B, C, F);
   if (st || nlines == 0) return st;
   // per-line need compared against the per-line share, so no product of
   // two large ints can wrap past the limit
   const size_t per_line = (size_t)kFacRec * N + 16;
   if (per_line > kNoAllocScratchDoubles / (size_t)nlines) {
      set_last_error("block_tridag4_noalloc: nlines*(80*N+16) with nlines = " + std::to_string(nlines) +
                     ", N = " + std::to_string(N) + " exceeds the fixed scratch of " +
                     std::to_string(kNoAllocScratchDoubles) + " doubles");
      return HAMSTR_GPU_ERR_ARG;
   }
   double* scratch = nullptr;
   st = noalloc_scratch(&scratch);
   if (st) return st;
   // every scratch value the kernel reads it has written earlier in the same
   // launch, so nothing needs clearing between calls
   return block_tridag_launch(nlines, N, periodic, A, B, C, F, scratch, (cudaStream_t)stream);
}
