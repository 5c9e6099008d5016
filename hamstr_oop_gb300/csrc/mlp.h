// ##################################################################
//
// mlp.h -- kernels of the learned warm start (BF16 tensor cores)
// ##################################################################
#ifndef HAMSTR_GPU_MLP_H
#define HAMSTR_GPU_MLP_H

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/hamstr_gpu.h"

namespace hamstr {
namespace mlp {

// C (+ split * M * N) = A B^T in FP32
struct GemmArgs {
   const __nv_bfloat16* A = nullptr;   // [M][K]
   const __nv_bfloat16* B = nullptr;   // [N][K]
   int M = 0, N = 0, K = 0, splits = 1;
   float* C = nullptr;
   int* err = nullptr;                  // device word: 1 after a timed-out wait
};

int gemm(const GemmArgs& a, cudaStream_t st);

}  // namespace mlp
}  // namespace hamstr
#endif
