// ##################################################################
//
// mlp_gemm.cu -- BF16 tensor-core GEMM for the learned warm start
//
// C[M x N] = A[M x K] * B[N x K]^T, A and B BF16 with K contiguous,
// FP32 accumulation in tensor memory, on the 5th-generation tensor cores:
//   * TMA (cp.async.bulk.tensor) brings 128 x 64 tiles of A and BN x 64
//     tiles of B into shared memory with 128-byte swizzling, STAGES deep,
//     each stage completing an mbarrier by transaction count;
//   * one thread issues tcgen05.mma (kind::f16, M = 128, N = BN, K = 16)
//     per 16-wide slice, accumulating in TMEM, and tcgen05.commit frees
//     the stage for the producer;
//   * all four warps read the accumulator with tcgen05.ld (warp w owns
//     TMEM lanes 32w..32w+31, one output row per thread) and store it.
// The network's own products run in mlp_net.cu, fused over its layers.
// Every wait is bounded (about two seconds); a timeout raises a flag in
// the caller's error word and the CTA still frees its tensor memory.
// ##################################################################
#include <cstdint>
#include <string>

#include "mlp.h"
#include "mlp_tc.cuh"

namespace hamstr {
void set_last_error(const std::string& m);

namespace mlp {

namespace {

constexpr int STAGES = 4;
constexpr int kThreads = 128;

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int M, int N,
                int kb_per_split, int nkb, float* __restrict__ C, int* err)
{
   extern __shared__ __align__(1024) unsigned char smem_raw[];
   // 1024-byte aligned stage buffers (the 128-byte swizzle atom)
   unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
   constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE = A_BYTES + B_BYTES;
   uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);   // full[S], empty[S], done
   __shared__ uint32_t tmem_base;
   __shared__ int failed;

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
   const int kb0 = blockIdx.z * kb_per_split;
   const int kb1 = min(nkb, kb0 + kb_per_split);
   const int nk = kb1 - kb0;

   const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES), done = smem_u32(bars + 2 * STAGES);
   if (threadIdx.x == 0) {
      failed = 0;
      for (int s = 0; s < STAGES; s++) {
         mbar_init(full0 + 8 * s, 1);
         mbar_init(empty0 + 8 * s, 1);
      }
      mbar_init(done, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   constexpr uint32_t kCols = BN < 32 ? 32 : BN;   // TMEM columns: a power of two >= 32
   if (warp == 2) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                   "r"(kCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   const uint32_t tmem = tmem_base;

   if (warp == 0 && lane == 0) {
      // producer: TMA loads of A and B tiles into the stages
      for (int i = 0; i < nk; i++) {
         const int s = i % STAGES, round = i / STAGES;
         if (round > 0 && !mbar_wait(empty0 + 8 * s, (round - 1) & 1)) {
            failed = 1;
            break;
         }
         const uint32_t sa = smem_u32(smem + s * STAGE), sb = sa + A_BYTES;
         mbar_expect_tx(full0 + 8 * s, STAGE);
         tma_load_2d(sa, &mapA, (kb0 + i) * BK, m0, full0 + 8 * s);
         tma_load_2d(sb, &mapB, (kb0 + i) * BK, n0, full0 + 8 * s);
      }
   } else if (warp == 1 && lane == 0) {
      // MMA issuer: four K = 16 slices per 64-wide stage
      const uint32_t idesc = instr_desc(BN);
      for (int i = 0; i < nk; i++) {
         const int s = i % STAGES, round = i / STAGES;
         if (!mbar_wait(full0 + 8 * s, round & 1)) {
            failed = 1;
            break;
         }
         asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
         const uint32_t sa = smem_u32(smem + s * STAGE), sb = sa + A_BYTES;
#pragma unroll
         for (int kk = 0; kk < BK / 16; kk++)
            mma_bf16(tmem, smem_desc(sa + 32 * kk), smem_desc(sb + 32 * kk), idesc, (i > 0 || kk > 0) ? 1u : 0u);
         mma_commit(empty0 + 8 * s);   // the stage is free once these MMAs have read it
      }
      mma_commit(done);                // the accumulator is complete
   }
   __syncwarp();

   // epilogue: every warp waits for the accumulator
   const bool ok = mbar_wait(done, 0);
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   if (!ok || failed) {
      if (threadIdx.x == 0) atomicOr(err, 1);
   } else {
      const int row = 32 * warp + lane, grow = m0 + row;
      const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
         float v[16];
         tmem_ld16(taddr + c, v);
         float* out = C + (size_t)blockIdx.z * M * N + (size_t)grow * N + n0 + c;
#pragma unroll
         for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(out + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   if (warp == 2)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

template <int BN>
int launch(const GemmArgs& a, cudaStream_t st)
{
   CUtensorMap ma, mb;
   if (!make_map(&ma, a.A, a.M, a.K, BM) || !make_map(&mb, a.B, a.N, a.K, BN)) {
      set_last_error("mlp gemm: tensor map encoding failed");
      return HAMSTR_GPU_ERR_CUDA;
   }
   constexpr int smem = STAGES * (BM * BK * 2 + BN * BK * 2) + 1024 + 2 * STAGES * 8 + 8 + 64;
   static bool configured = false;
   if (!configured) {
      if (cudaFuncSetAttribute(gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
         set_last_error("mlp gemm: shared memory request refused");
         return HAMSTR_GPU_ERR_CUDA;
      }
      configured = true;
   }
   const int nkb = a.K / BK;
   const int splits = a.splits < 1 ? 1 : (a.splits > nkb ? nkb : a.splits);
   const int per = (nkb + splits - 1) / splits;
   const int gz = (nkb + per - 1) / per;   // every split has at least one K block
   dim3 grid(a.M / BM, a.N / BN, gz);
   gemm_kernel<BN><<<grid, kThreads, smem, st>>>(ma, mb, a.M, a.N, per, nkb, a.C, a.err);
   const cudaError_t e = cudaGetLastError();
   if (e != cudaSuccess) {
      set_last_error(std::string("mlp gemm launch: ") + cudaGetErrorString(e));
      return HAMSTR_GPU_ERR_CUDA;
   }
   return HAMSTR_GPU_OK;
}

}  // namespace

int gemm(const GemmArgs& a, cudaStream_t st)
{
   if (!a.A || !a.B || !a.err || a.M <= 0 || a.N <= 0 || a.K <= 0 || a.M % BM || a.K % BK ||
       ((uintptr_t)a.A & 15) || ((uintptr_t)a.B & 15)) {
      set_last_error("mlp gemm: need M % 128 == 0, K % 64 == 0, 16-byte aligned operands");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (!a.C || ((uintptr_t)a.C & 15)) {   // stored by float4
      set_last_error("mlp gemm: need a 16-byte aligned C");
      return HAMSTR_GPU_ERR_ARG;
   }
   switch (a.N) {
      case 16: return launch<16>(a, st);
      case 64: return launch<64>(a, st);
      case 128: return launch<128>(a, st);
      case 256: return launch<256>(a, st);
      default:
         if (a.N % 256 == 0) return launch<256>(a, st);
         set_last_error("mlp gemm: N must be 16, 64, 128 or a multiple of 256");
         return HAMSTR_GPU_ERR_ARG;
   }
}

}  // namespace mlp
}  // namespace hamstr
