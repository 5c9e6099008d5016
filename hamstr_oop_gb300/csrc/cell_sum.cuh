// ##################################################################
//
// cell_sum.cuh -- what the kernels that sum over a cell's faces share
//
// ##################################################################
#ifndef HAMSTR_GPU_CELL_SUM_CUH
#define HAMSTR_GPU_CELL_SUM_CUH

#include "device_state.h"

namespace hamstr {

// faces of a cell whose loads are issued together (a cell has three or four)
constexpr int kGather = 4;

__device__ __forceinline__ void cell_entries(const DeviceState& d, int e, int e1, int (&ent)[kGather])
{
#pragma unroll
   for (int u = 0; u < kGather; u++) ent[u] = e + u < e1 ? d.cell_ent[e + u] : 0;
}

// the larger of two non-negative numbers by their bits
__device__ __forceinline__ unsigned long long max_bits(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// deterministic block reduction of {sum, max} into norm_part[blockIdx.x]; am
// is an absolute value.  The maximum goes by the bits, off the FP64 pipe; a
// NaN counts for it as nothing, as in fmax
__device__ __forceinline__ void block_norm(const DeviceState& d, double sq, double am)
{
   __shared__ double s_sq[kNormBlock / 32];
   __shared__ unsigned long long s_am[kNormBlock / 32];
   unsigned long long m = (unsigned long long)__double_as_longlong(am);
   if (m > 0x7FF0000000000000ull) m = 0;
#pragma unroll
   for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      m = max_bits(m, __shfl_xor_sync(0xffffffffu, m, o));
   }
   const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
   if (l == 0) { s_sq[w] = sq; s_am[w] = m; }
   __syncthreads();
   if (threadIdx.x == 0) {
      double a = 0.0;
      unsigned long long b = 0;
#pragma unroll
      for (int i = 0; i < kNormBlock / 32; i++) { a += s_sq[i]; b = max_bits(b, s_am[i]); }
      d.norm_part[blockIdx.x] = make_double2(a, __longlong_as_double((long long)b));
   }
}

}  // namespace hamstr
#endif
