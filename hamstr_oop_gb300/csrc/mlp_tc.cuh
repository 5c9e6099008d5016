// ##################################################################
//
// mlp_tc.cuh -- the tensor-core building blocks of the warm-start kernels
//
// mbarriers with bounded waits, TMA tile loads, tcgen05.mma on K-major
// BF16 tiles with 128-byte swizzling, and tensor-memory loads, shared by
// the general GEMM (mlp_gemm.cu) and the network's kernels (mlp_net.cu).
// ##################################################################
#ifndef HAMSTR_GPU_MLP_TC_CUH
#define HAMSTR_GPU_MLP_TC_CUH

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

namespace hamstr {
namespace mlp {

constexpr int BM = 128, BK = 64;
constexpr unsigned long long kWaitNs = 2000000000ull;   // bounded waits: 2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns()
{
   unsigned long long t;
   asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
   return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
   asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
   asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// true when phase `parity` of the barrier has completed; false after the
// time limit, or at once when another role has given up (failed, may be null)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* failed = nullptr)
{
   const unsigned long long t0 = global_ns();
   for (;;) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(bar), "r"(parity)
          : "memory");
      if (ok) return true;
      if (global_ns() - t0 > kWaitNs || (failed && *failed)) return false;
   }
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
   asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar)
{
   asm volatile(
       "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
           dst),
       "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar)
       : "memory");
}

// shared-memory matrix descriptor: K-major tile with 128-byte swizzling,
// 8-row atoms of 1024 bytes (stride byte offset), version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr)
{
   uint64_t d = 0;
   d |= (uint64_t)((addr & 0x3FFFF) >> 4);          // start address
   d |= (uint64_t)1 << 16;                           // leading byte offset (unused for swizzled K-major)
   d |= (uint64_t)(1024 >> 4) << 32;                 // stride byte offset
   d |= (uint64_t)1 << 46;                           // descriptor version
   d |= (uint64_t)2 << 61;                           // 128-byte swizzle
   return d;
}

// instruction descriptor: kind::f16 with BF16 A and B, FP32 D, both
// K-major, M = 128, N = BN
__host__ __device__ constexpr uint32_t instr_desc(int bn)
{
   return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
   asm volatile(
       "{\n\t.reg .pred p;\n\t"
       "setp.ne.b32 p, %4, 0;\n\t"
       "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
       "l"(a), "l"(b), "r"(idesc), "r"(accum)
       : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
   asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane: begin the load, and
// wait for every load begun (the registers may be read only then)
__device__ __forceinline__ void tmem_ld16_begin(uint32_t taddr, uint32_t (&r)[16])
{
   asm volatile(
       "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
       "[%16];"
       : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
         "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
       : "r"(taddr));
}

// (the registers pass through, so that no use of them moves above the wait)
__device__ __forceinline__ void tmem_ld16_wait(uint32_t (&r)[16], float (&v)[16])
{
   asm volatile("tcgen05.wait::ld.sync.aligned;"
                : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                  "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                :
                : "memory");
#pragma unroll
   for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
   uint32_t r[16];
   tmem_ld16_begin(taddr, r);
   tmem_ld16_wait(r, v);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link-time dependency on the driver library)
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
   static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
   static std::once_flag once;
   std::call_once(once, [] {
      void* p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
         fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
   });
   return fn;
}

// rows x k BF16 matrix (k contiguous), box of box_rows x 64
inline bool make_map(CUtensorMap* map, const void* base, int rows, int k, int box_rows)
{
   auto fn = encode_fn();
   if (!fn) return false;
   cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
   cuuint64_t strides[1] = {(cuuint64_t)k * 2};
   cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};   // BK <= k
   cuuint32_t estr[2] = {1, 1};
   return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace mlp
}  // namespace hamstr
#endif
