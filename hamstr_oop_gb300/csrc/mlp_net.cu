// ##################################################################
//
// mlp_net.cu -- the warm-start network: 5 -> 256 -> 256 -> 256 -> 4,
// GELU, BF16 weights and activations, FP32 accumulation
//
// One kernel carries a tile of 128 rows through every layer (net_kernel):
// the layer's input sits in shared memory as the A operand, weight tiles
// stream from L2 through a ring of TMA stages, tcgen05.mma accumulates the
// 128 x 256 product in TMEM, and eight warps turn it into the next layer's
// input in shared memory (bias, GELU).  In training the same kernel goes on
// with the loss and the backward pass; what the weight gradients need
// (activations and their gradients, transposed so that both operands of the
// gradient products are K-major) goes to memory, as does GELU'(Z) of the
// forward pass.  wgrad_kernel forms the four weight gradients in one launch,
// split over the batch, and update_kernel sums the splits in order, the bias
// gradients and the loss, and applies Adam (FP32 master weights, BF16 copies
// and transposes).  Three launches and one host round trip a training step,
// one and one for inference.
//
// What bounds it: erff.  A tile has 98,304 GELUs of about 30 FP32
// instructions each, 23,000 cycles of an SM's FP32 lanes, against 5,400 of
// its tensor cores and 4,700 of its L2 port for the weights (296 KB a tile);
// so inference keeps two tiles on an SM, one's products under the other's
// GELUs (63% of the issue slots; a last wave of 512 tiles on 152 SMs costs
// 16%).  Layer by layer, as before, every activation went through memory three
// times, the row-major ones in 2-byte stores 512 bytes apart, with a gather, a
// launch per product and copies between.  Measured, call to call: 65,500 rows
// 1,052 -> 104 us; a training step of 16,384 rows 727 -> 111 us.  Weight gradients
// and hidden biases are summed in the order they were, the loss and the output
// biases (FP64 sums, the biases then rounded) in another; trained networks came
// out the same bit for bit in every run.
//
// Shapes are padded for the tensor cores: the 5 inputs and the 4 outputs to
// one K slice of 16 where they are a K dimension (the weights' rows are 64
// wide), the outputs to 16 where they are N; the padding stays exactly zero
// through training.
// ##################################################################
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "mlp.h"
#include "mlp_tc.cuh"

namespace hamstr {
void set_last_error(const std::string& m);
}

using namespace hamstr;
using namespace hamstr::mlp;
using bf16 = __nv_bfloat16;

namespace {

constexpr int W = 256;       // hidden width
constexpr int NIN = 5, NOUT = 4;
constexpr int KIN = 64;      // stored row length of W1
constexpr int NOP = 16;      // padded outputs (and inputs, where they are N)
constexpr int KOP = 64;      // stored row length of W4^T

// logical parameter layout (host API): W1[256][5] b1 W2[256][256] b2
// W3[256][256] b3 W4[4][256] b4
constexpr int kNParams = W * NIN + W + 2 * (W * W + W) + NOUT * W + NOUT;

__device__ __forceinline__ unsigned long long mix64(unsigned long long x)
{
   // splitmix64 finaliser (Steele, Lea & Flood, 2014)
   x += 0x9E3779B97F4A7C15ull;
   x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
   x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
   return x ^ (x >> 31);
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z)
{
   return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// ------------------------------------------------------------------
// the layers of a tile, forward and backward
// ------------------------------------------------------------------
// EW warps turn the products into the next layer's input, EW/4 threads to a
// row; beside them one warp loads the weights and one issues the products.
// Inference with more tiles than SMs: 8, and two blocks to an SM; otherwise 16
// and one, which halves a tile's time where it has an SM to itself.
constexpr int net_threads(int ew) { return 32 * (ew + 2); }
constexpr int kFwdLayers = 4, kAllLayers = 7;             // W1 W2 W3 W4 | W4^T W3^T W2^T
constexpr int kStageBytes = 128 * BK * 2;                 // a 128 x 64 weight tile
constexpr int kInBytes = 4 * 128 * BK * 2;                // a layer's input, 128 x 256
constexpr int net_stages(int ew) { return ew == 8 ? 2 : 8; }

struct NetMaps {
   CUtensorMap w[kAllLayers];   // boxes of 128 rows, W4's of 16
};

struct NetArgs {
   const float* feat;
   const float* targ;             // training
   long long n_all;
   int n, rows;                   // rows computed (a multiple of 128 in training), valid ones
   unsigned long long seed, step; // minibatch draw (seed 0: rows in order)
   const float *b1, *b2, *b3, *b4;
   float* y;                      // inference: [n][4]
   // training: transposed BF16 activations and gradients, rows ld apart
   bf16 *Xt, *Ht[3], *dZt[3], *dZ4t;
   int ld;
   float* G;                      // GELU'(Z): [tile][layer][column][row]
   double* lpart;                 // per 32 rows: loss, db4[4]
   int* err;                      // 1 after a wait that gave up
   int give_up;                   // self-test: the weight tile at which a block's loader gives up (-1: none)
};

template <int STAGES>
struct NetShared {
   uint64_t full[STAGES], empty[STAGES], acc, input;
   uint32_t tmem;
   int failed;
   float bias[3][W];
};

// weight tiles of a layer: (K blocks) x (halves of N); W4 is one stage of
// four 16-row boxes
__host__ __device__ constexpr int layer_stages(int l) { return l == 3 ? 1 : (l == 0 || l == 4) ? 2 : 8; }

// 16 BF16 values of row `row`, columns col .. col+15, into the K-major
// 128-byte-swizzled layer input
__device__ __forceinline__ void put16(unsigned char* in, int row, int col, const uint32_t (&p)[8])
{
   unsigned char* base = in + (size_t)(col >> 6) * (128 * BK * 2) + row * 128;
   const int q = (col & 63) >> 3;
   *reinterpret_cast<uint4*>(base + ((q ^ (row & 7)) << 4)) = make_uint4(p[0], p[1], p[2], p[3]);
   *reinterpret_cast<uint4*>(base + (((q + 1) ^ (row & 7)) << 4)) = make_uint4(p[4], p[5], p[6], p[7]);
}

__device__ __forceinline__ uint32_t pack2(bf16 a, bf16 b)
{
   return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
__device__ __forceinline__ uint32_t pack2(__nv_bfloat162 h) { return pack2(h.x, h.y); }

template <bool TRAIN, int EW>
__global__ void __launch_bounds__(net_threads(EW), EW == 8 ? 2 : 1)
    net_kernel(const __grid_constant__ NetMaps maps, const __grid_constant__ NetArgs a)
{
   constexpr int STAGES = net_stages(EW), CW = 4 * W / EW;   // CW: a thread's columns
   constexpr int LAYERS = TRAIN ? kAllLayers : kFwdLayers;
   extern __shared__ __align__(1024) unsigned char smem_raw[];
   unsigned char* in = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);   // the layer's input
   unsigned char* ring = in + kInBytes;
   __shared__ NetShared<STAGES> s;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int ntiles = (a.n - 1) / 128 + 1;   // a.n may be the largest int
   const uint32_t full0 = smem_u32(s.full), empty0 = smem_u32(s.empty), acc = smem_u32(&s.acc),
                  input = smem_u32(&s.input);
   if (threadIdx.x == 0) {
      s.failed = 0;
      for (int i = 0; i < STAGES; i++) {
         mbar_init(full0 + 8 * i, 1);
         mbar_init(empty0 + 8 * i, 1);
      }
      mbar_init(acc, 1);
      mbar_init(input, EW);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   for (int t = threadIdx.x; t < 3 * W; t += net_threads(EW))
      s.bias[t / W][t % W] = (t < W ? a.b1 : t < 2 * W ? a.b2 : a.b3)[t % W];
   if (warp == EW + 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem)),
                   "r"((uint32_t)W)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   const uint32_t tmem = s.tmem;
   volatile int* failed = &s.failed;

   if (warp == EW) {
      if (lane == 0) {
         // weight tiles, in the order the products use them
         int it = 0;
         for (int tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x)
            for (int l = 0; l < LAYERS && !*failed; l++)
               for (int st = 0; st < layer_stages(l); st++, it++) {
                  const int slot = it % STAGES, round = it / STAGES;
                  if ((round > 0 && !mbar_wait(empty0 + 8 * slot, (round - 1) & 1, failed)) || it == a.give_up) {
                     *failed = 1;
                     break;
                  }
                  const uint32_t dst = smem_u32(ring + slot * kStageBytes), bar = full0 + 8 * slot;
                  if (l == 3) {
                     mbar_expect_tx(bar, 4 * NOP * BK * 2);
                     for (int kb = 0; kb < 4; kb++) tma_load_2d(dst + kb * NOP * BK * 2, &maps.w[3], kb * BK, 0, bar);
                  } else {
                     mbar_expect_tx(bar, kStageBytes);
                     tma_load_2d(dst, &maps.w[l], (st >> 1) * BK, (st & 1) * 128, bar);
                  }
               }
         if (*failed)   // the copies in flight end before the block does
            for (int k = std::max(0, it - STAGES); k < it; k++) mbar_wait(full0 + 8 * (k % STAGES), (k / STAGES) & 1);
      }
   } else if (warp == EW + 1) {
      if (lane == 0) {
         int it = 0, n = 0;
         for (int tile = blockIdx.x; tile < ntiles && !*failed; tile += gridDim.x)
            for (int l = 0; l < LAYERS && !*failed; l++, n++) {
               // the layer's input is in place and the accumulator has been read
               if (!mbar_wait(input, n & 1, failed)) {
                  *failed = 1;
                  break;
               }
               asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
               const int slices = (l == 0 || l == 4) ? 1 : BK / 16;   // their K is one slice of 16
               for (int st = 0; st < layer_stages(l); st++, it++) {
                  const int slot = it % STAGES;
                  if (!mbar_wait(full0 + 8 * slot, (it / STAGES) & 1, failed)) {
                     *failed = 1;
                     break;
                  }
                  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                  const uint32_t sb = smem_u32(ring + slot * kStageBytes), sa = smem_u32(in);
                  if (l == 3) {
                     for (int kb = 0; kb < 4; kb++)
                        for (int kk = 0; kk < BK / 16; kk++)
                           mma_bf16(tmem, smem_desc(sa + kb * 128 * BK * 2 + 32 * kk),
                                    smem_desc(sb + kb * NOP * BK * 2 + 32 * kk), instr_desc(NOP),
                                    (kb > 0 || kk > 0) ? 1u : 0u);
                  } else {
                     const int kb = st >> 1;
                     for (int kk = 0; kk < slices; kk++)
                        mma_bf16(tmem + (st & 1) * 128, smem_desc(sa + kb * 128 * BK * 2 + 32 * kk),
                                 smem_desc(sb + 32 * kk), instr_desc(128), (kb > 0 || kk > 0) ? 1u : 0u);
                  }
                  mma_commit(empty0 + 8 * slot);
               }
               mma_commit(acc);
            }
         // products in flight end before their tensor memory is given back
         if (*failed && n > 0) mbar_wait(acc, (n - 1) & 1);
      }
   } else {
      const int row = 32 * (warp & 3) + lane, ch = warp >> 2, c0 = CW * ch;   // this thread's row and first column
      const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c0;
      const float scale = 2.f / (float)(a.rows * NOUT);
      int n = 0;
      bool ok = true;
      // the input is written and the accumulator read: the products may go on
      auto next = [&] {
         asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
         asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
         __syncwarp();
         if (lane == 0) mbar_arrive(input);
      };
      auto product = [&] {
         if (ok && !mbar_wait(acc, n & 1, failed)) {
            *failed = 1;
            ok = false;
         }
         n++;
         asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
         __syncwarp();
         ok = __all_sync(0xffffffffu, ok);
      };
      for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
         const int i = 128 * tile + row;   // the batch row
         long long src = -1;
         if (ch == 0) {
            if (i < a.rows)
               src = a.seed ? (long long)(mix64(a.seed ^ mix64(a.step * 0x100000001ull + i)) % (unsigned long long)a.n_all)
                            : i;
            float x[NIN];
#pragma unroll
            for (int k = 0; k < NIN; k++) x[k] = src >= 0 ? a.feat[src * NIN + k] : 0.f;
            bf16 xb[6];
#pragma unroll
            for (int k = 0; k < 6; k++) xb[k] = __float2bfloat16_rn(k < NIN ? x[k] : 0.f);
            const uint32_t p[8] = {pack2(xb[0], xb[1]), pack2(xb[2], xb[3]), pack2(xb[4], xb[5]), 0, 0, 0, 0, 0};
            put16(in, row, 0, p);
            if (TRAIN) {
#pragma unroll
               for (int k = 0; k < NIN; k++) a.Xt[(size_t)k * a.ld + i] = xb[k];
            }
         }
         next();
         // hidden layers
         for (int l = 0; l < 3; l++) {
            product();
            if (!ok) break;
            float* G = TRAIN ? a.G + (((size_t)tile * 3 + l) * W + c0) * 128 + row : nullptr;
            bf16* Ht = TRAIN ? a.Ht[l] + (size_t)c0 * a.ld + i : nullptr;
            const float* bias = s.bias[l] + c0;
            uint32_t r[16];
            tmem_ld16_begin(taddr, r);
#pragma unroll 1
            for (int c = 0; c < CW; c += 16) {
               float v[16];
               tmem_ld16_wait(r, v);
               if (c + 16 < CW) tmem_ld16_begin(taddr + c + 16, r);   // under this group's GELUs
               uint32_t p[8];
#pragma unroll
               for (int j = 0; j < 16; j += 2) {
                  const float z0 = v[j] + bias[c + j], z1 = v[j + 1] + bias[c + j + 1];
                  const __nv_bfloat162 h = __floats2bfloat162_rn(gelu(z0), gelu(z1));
                  if (TRAIN) {
                     G[(size_t)(c + j) * 128] = gelu_grad(z0);
                     G[(size_t)(c + j + 1) * 128] = gelu_grad(z1);
                     Ht[(size_t)(c + j) * a.ld] = h.x;
                     Ht[(size_t)(c + j + 1) * a.ld] = h.y;
                  }
                  p[j / 2] = pack2(h);
               }
               put16(in, row, c0 + c, p);
            }
            next();
         }
         if (!ok) break;
         // output layer
         product();
         if (!ok) break;
         if (ch == 0) {
            float v[16];
            tmem_ld16(taddr, v);
            if (!TRAIN) {
               if (i < a.rows) {
#pragma unroll
                  for (int k = 0; k < NOUT; k++) a.y[(size_t)i * NOUT + k] = v[k] + a.b4[k];
               }
            } else {
               // loss = sum over valid rows of (y - t)^2 / (rows * 4), dY = 2 (y - t) / (rows * 4)
               double part[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
               bf16 d[NOUT];
#pragma unroll
               for (int k = 0; k < NOUT; k++) {
                  float g = 0.f;
                  if (src >= 0) {
                     const float e = (v[k] + a.b4[k]) - a.targ[src * NOUT + k];
                     part[0] += (double)e * e;
                     g = scale * e;
                     part[1 + k] = g;
                  }
                  d[k] = __float2bfloat16_rn(g);
                  a.dZ4t[(size_t)k * a.ld + i] = d[k];
               }
               const uint32_t p[8] = {pack2(d[0], d[1]), pack2(d[2], d[3]), 0, 0, 0, 0, 0, 0};
               put16(in, row, 0, p);
#pragma unroll
               for (int q = 0; q < 5; q++) {
#pragma unroll
                  for (int o = 16; o > 0; o >>= 1) part[q] += __shfl_xor_sync(0xffffffffu, part[q], o);
                  if (lane == 0)
                     a.lpart[5 * (4 * (size_t)tile + warp) + q] = q == 0 ? part[0] / ((double)a.rows * NOUT) : part[q];
               }
            }
         }
         if (TRAIN) {
            next();
            // backward: dZ of hidden layer l = (dZ of the next layer times its weights) * GELU'(Z)
            for (int l = 2; l >= 0; l--) {
               product();
               if (!ok) break;
               const float* G = a.G + (((size_t)tile * 3 + l) * W + c0) * 128 + row;
               bf16* dZt = a.dZt[l] + (size_t)c0 * a.ld + i;
               uint32_t r[16];
               tmem_ld16_begin(taddr, r);
#pragma unroll 1
               for (int c = 0; c < CW; c += 16) {
                  float v[16], g[16];
#pragma unroll
                  for (int j = 0; j < 16; j++) g[j] = G[(size_t)(c + j) * 128];
                  tmem_ld16_wait(r, v);
                  if (c + 16 < CW) tmem_ld16_begin(taddr + c + 16, r);
                  uint32_t p[8];
#pragma unroll
                  for (int j = 0; j < 16; j += 2) {
                     const __nv_bfloat162 d = __floats2bfloat162_rn(v[j] * g[j], v[j + 1] * g[j + 1]);
                     dZt[(size_t)(c + j) * a.ld] = d.x;
                     dZt[(size_t)(c + j + 1) * a.ld] = d.y;
                     p[j / 2] = pack2(d);
                  }
                  if (l > 0) put16(in, row, c0 + c, p);
               }
               if (l > 0) next();
            }
            if (!ok) break;
         }
         // the next tile's input overwrites what the last product has read, and
         // its first product what every warp has read of the accumulator
      }
   }
   __syncwarp();
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   // whichever role gave up: the others may have come to their end, the epilogue
   // with a product that is not complete
   if (threadIdx.x == 0 && *failed) *(volatile int*)a.err = 1;
   if (warp == EW + 1)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)W) : "memory");
}

// ------------------------------------------------------------------
// weight gradients: D [256][N] = A [256][B] * Bm [N][B]^T over a range of the
// batch, stored transposed ([N][256], so that a warp's rows are contiguous)
// ------------------------------------------------------------------
struct WgradMaps {
   CUtensorMap A[4], B[4];   // products: dW2^T (H1, dZ2), dW3^T (H2, dZ3), dW4^T (H3, dZ4), dW1 (dZ1, X)
};
struct WgradArgs {
   int nkb, per, splits;     // 64-wide blocks of the batch, of them to a split
   float* out[4];            // [split][N][256]
   int* err;
};
constexpr int kWgradStages = 2;   // two blocks to an SM
constexpr int kWgradStage = 128 * BK * 2 + W * BK * 2;

__global__ void __launch_bounds__(128, 2)
    wgrad_kernel(const __grid_constant__ WgradMaps maps, const __grid_constant__ WgradArgs a)
{
   extern __shared__ __align__(1024) unsigned char smem_raw[];
   unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
   __shared__ uint64_t full[kWgradStages], empty[kWgradStages], done_bar;
   __shared__ uint32_t tmem_base;
   __shared__ int failed_s;
   volatile int* failed = &failed_s;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   // dW2 and dW3 (N = 256) first, then dW4 and dW1 (N = 16)
   const int job = blockIdx.x / (2 * a.splits), mt = blockIdx.x & 1, split = (blockIdx.x % (2 * a.splits)) >> 1;
   const int N = job < 2 ? W : NOP, per = a.per;
   const int kb0 = split * per, nk = min(a.nkb, kb0 + per) - kb0;
   const uint32_t full0 = smem_u32(full), empty0 = smem_u32(empty), done = smem_u32(&done_bar);
   if (threadIdx.x == 0) {
      failed_s = 0;
      for (int i = 0; i < kWgradStages; i++) {
         mbar_init(full0 + 8 * i, 1);
         mbar_init(empty0 + 8 * i, 1);
      }
      mbar_init(done, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   if (warp == 2) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                   "r"((uint32_t)W)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   const uint32_t tmem = tmem_base;
   if (warp == 0 && lane == 0) {
      int i = 0;
      for (; i < nk; i++) {
         const int slot = i % kWgradStages, round = i / kWgradStages;
         if (round > 0 && !mbar_wait(empty0 + 8 * slot, (round - 1) & 1, failed)) {
            *failed = 1;
            break;
         }
         const uint32_t sa = smem_u32(smem + slot * kWgradStage), sb = sa + 128 * BK * 2, bar = full0 + 8 * slot;
         mbar_expect_tx(bar, 128 * BK * 2 + N * BK * 2);
         tma_load_2d(sa, &maps.A[job], (kb0 + i) * BK, 128 * mt, bar);
         tma_load_2d(sb, &maps.B[job], (kb0 + i) * BK, 0, bar);
      }
      if (*failed)
         for (int k = max(0, i - kWgradStages); k < i; k++) mbar_wait(full0 + 8 * (k % kWgradStages), (k / kWgradStages) & 1);
   } else if (warp == 1 && lane == 0) {
      const uint32_t idesc = instr_desc(N);
      for (int i = 0; i < nk; i++) {
         const int slot = i % kWgradStages;
         if (!mbar_wait(full0 + 8 * slot, (i / kWgradStages) & 1, failed)) {
            *failed = 1;
            break;
         }
         asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
         const uint32_t sa = smem_u32(smem + slot * kWgradStage), sb = sa + 128 * BK * 2;
#pragma unroll
         for (int kk = 0; kk < BK / 16; kk++)
            mma_bf16(tmem, smem_desc(sa + 32 * kk), smem_desc(sb + 32 * kk), idesc, (i > 0 || kk > 0) ? 1u : 0u);
         mma_commit(empty0 + 8 * slot);
      }
      mma_commit(done);
   }
   __syncwarp();
   const bool ok = mbar_wait(done, 0);
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   if (!ok || *failed) {
      if (threadIdx.x == 0) *(volatile int*)a.err = 1;
   } else {
      const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
      float* out = a.out[job] + (size_t)split * N * W + 128 * mt + 32 * warp + lane;
#pragma unroll 1
      for (int c = 0; c < N; c += 16) {
         float v[16];
         tmem_ld16(taddr + c, v);
#pragma unroll
         for (int j = 0; j < 16; j++) out[(size_t)(c + j) * W] = v[j];
      }
   }
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   if (warp == 2)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)W) : "memory");
}

// ------------------------------------------------------------------
// gradients from the splits, in split order, and Adam (Kingma & Ba, 2015)
// ------------------------------------------------------------------
struct Tensor {
   float *p, *m, *v, *g;   // parameters, moments, gradient
};
struct UpdateArgs {
   Tensor W1, b1, W2, b2, W3, b3, W4, b4;   // W1 [256][64], W4 [16][256]; the rest as named
   bf16 *W1b, *W2b, *W2t, *W3b, *W3t, *W4b, *W4t;
   const float *part1, *part2, *part3, *part4;   // [split][16][256] (dW1^T), [256][256], [256][256], [16][256]
   int splits;
   const bf16* dZt[3];
   int ld, B;
   const double* lpart;
   const int* err;         // the pass's error word: nothing is updated after a wait that gave up
   int* host_err;
   double* loss;
   int adam;
   float lr, c1, c2;       // c1, c2: bias corrections
};

constexpr int kWeightThreads = 2 * W * W + NOUT * W + NIN * W;
constexpr int kWeightBlocks = kWeightThreads / 256;   // 521
constexpr int kBiasBlocks = 3 * W;                    // one to a bias
static_assert(kWeightThreads % 256 == 0, "whole blocks");

__device__ __forceinline__ float adam(const Tensor& t, int i, float g, const UpdateArgs& a)
{
   const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
   const float mi = b1 * t.m[i] + (1.f - b1) * g;
   const float vi = b2 * t.v[i] + (1.f - b2) * g * g;
   t.m[i] = mi;
   t.v[i] = vi;
   const float p = t.p[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + eps);
   t.p[i] = p;
   return p;
}

__device__ __forceinline__ float split_sum(const float* __restrict__ part, int splits, size_t stride, int i)
{
   float g = 0.f;
#pragma unroll 8
   for (int s = 0; s < splits; s++) g += part[s * stride + i];
   return g;
}

__global__ void __launch_bounds__(256) update_kernel(const __grid_constant__ UpdateArgs a)
{
   const int lane = threadIdx.x & 31;
   if (*a.err) {
      if (blockIdx.x == 0 && threadIdx.x == 0) *a.host_err = 1;
      return;
   }
   if (blockIdx.x < kWeightBlocks) {
      int i = blockIdx.x * 256 + threadIdx.x;
      if (i < 2 * W * W) {
         const bool second = i < W * W;
         const Tensor& t = second ? a.W2 : a.W3;
         i &= W * W - 1;
         const float g = split_sum(second ? a.part2 : a.part3, a.splits, (size_t)W * W, i);
         t.g[i] = g;
         if (a.adam) {
            const bf16 b = __float2bfloat16_rn(adam(t, i, g, a));
            (second ? a.W2b : a.W3b)[i] = b;
            (second ? a.W2t : a.W3t)[(i & (W - 1)) * W + i / W] = b;
         }
      } else if ((i -= 2 * W * W) < NOUT * W) {
         const float g = split_sum(a.part4, a.splits, (size_t)NOP * W, i);
         a.W4.g[i] = g;
         if (a.adam) {
            const bf16 b = __float2bfloat16_rn(adam(a.W4, i, g, a));
            a.W4b[i] = b;
            a.W4t[(i & (W - 1)) * KOP + i / W] = b;
         }
      } else {
         i -= NOUT * W;
         const float g = split_sum(a.part1, a.splits, (size_t)NOP * W, i);
         const int o = (i & (W - 1)) * KIN + i / W;
         a.W1.g[o] = g;
         if (a.adam) a.W1b[o] = __float2bfloat16_rn(adam(a.W1, o, g, a));
      }
   } else if (blockIdx.x < kWeightBlocks + kBiasBlocks) {
      // hidden biases: the row sums of the transposed dZ
      __shared__ float sum[256];
      const int r = blockIdx.x - kWeightBlocks, l = r / W, i = r & (W - 1);
      const bf16* z = a.dZt[l] + (size_t)i * a.ld;
      float g = 0.f;
#pragma unroll 8
      for (int b = threadIdx.x; b < a.B; b += 256) g += __bfloat162float(z[b]);
      sum[threadIdx.x] = g;
      __syncthreads();
      for (int k = 128; k > 0; k >>= 1) {
         if (threadIdx.x < k) sum[threadIdx.x] += sum[threadIdx.x + k];
         __syncthreads();
      }
      const Tensor& t = l == 0 ? a.b1 : l == 1 ? a.b2 : a.b3;
      if (threadIdx.x == 0) {
         t.g[i] = sum[0];
         if (a.adam) adam(t, i, sum[0], a);
      }
   } else if (threadIdx.x < 5 * 32) {
      // the loss and the output biases, a warp each over the partial sums
      const int q = threadIdx.x >> 5, i = q - 1;
      double t = 0.0;
#pragma unroll 4
      for (int k = lane; k < a.B / 32; k += 32) t += a.lpart[5 * (size_t)k + q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0 && q == 0) *a.loss = t;
      if (lane == 0 && q > 0) {
         a.b4.g[i] = (float)t;
         if (a.adam) adam(a.b4, i, (float)t, a);
      }
   }
}

// BF16 copies of an FP32 tensor [rows][cols] (no update)
__global__ void cast_kernel(const float* __restrict__ p, int rows, int cols, bf16* __restrict__ w, int ldw,
                            bf16* __restrict__ wt, int ldt)
{
   const int i = blockIdx.x * blockDim.x + threadIdx.x;
   if (i >= rows * cols) return;
   const int r = i / cols, c = i - r * cols;
   const bf16 b = __float2bfloat16_rn(p[i]);
   w[(size_t)r * ldw + c] = b;
   if (wt) wt[(size_t)c * ldt + r] = b;
}

int blocks(long long n, int t = 256) { return (int)((n + t - 1) / t); }

// splits actually used when nkb blocks are asked to go to `splits` (each at least one)
int used_splits(int nkb, int splits, int* per)
{
   splits = std::max(1, std::min(splits, nkb));
   *per = (nkb + splits - 1) / splits;
   return (nkb + *per - 1) / *per;
}

// a pass's result, in page-locked host memory that the kernels write: one
// synchronisation brings it, no copy
struct Result {
   double loss;
   int err, pad;
};

}  // namespace

struct hamstr_mlp {
   int Bmax = 0, nsm = 148;
   int max_splits = 1;   // of the weight gradients
   cudaStream_t st = nullptr;
   std::vector<void*> owned;
   // FP32 master parameters, Adam moments, gradients (W1 [256][64], W4 [16][256])
   Tensor W1, b1, W2, b2, W3, b3, W4, b4;
   // BF16 weights: W1 [256][64], W2/W3 [256][256] and transposes, W4 [16][256], W4t [256][64]
   bf16 *W1b, *W2b, *W2t, *W3b, *W3t, *W4b, *W4t;
   // for Bmax rows, transposed: inputs and outputs' gradients [16][Bmax], the rest [256][Bmax]
   bf16 *Xt, *Ht[3], *dZt[3], *dZ4t;
   float *G, *part1, *part2, *part3, *part4;
   double* lpart;
   Result* host = nullptr;   // and its device address
   Result* res = nullptr;
   int* err;                 // of the passes before an update, which leaves the parameters as they are then
   int give_up = -1;         // self-test (hamstr_check_mlp_wait)
   float* host_params = nullptr;   // [kNParams], page-locked: what get_params and get_grads bring (pack_kernel)
   float* dev_params = nullptr;    // its device address
   std::mutex params_mutex;        // of that buffer: threads may read parameters at the same time
   NetMaps net;
   WgradMaps wg;

   template <typename T>
   int alloc(T** p, size_t n)
   {
      if (cudaMalloc((void**)p, (n ? n : 1) * sizeof(T)) != cudaSuccess) return HAMSTR_GPU_ERR_NOMEM;
      owned.push_back(*p);
      return cudaMemsetAsync(*p, 0, (n ? n : 1) * sizeof(T), st) == cudaSuccess ? HAMSTR_GPU_OK : HAMSTR_GPU_ERR_CUDA;
   }
   int alloc(Tensor* t, size_t n)
   {
      int e = alloc(&t->p, n);
      if (!e) e = alloc(&t->m, n);
      if (!e) e = alloc(&t->v, n);
      if (!e) e = alloc(&t->g, n);
      return e;
   }
};

namespace {

int cuda_ok(cudaError_t e, const char* what)
{
   if (e == cudaSuccess) return HAMSTR_GPU_OK;
   set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
   return HAMSTR_GPU_ERR_CUDA;
}

constexpr int net_smem(int ew) { return kInBytes + net_stages(ew) * kStageBytes + 1024; }
constexpr int kWgradSmem = kWgradStages * kWgradStage + 1024;

int configure()
{
   auto allow = [](const void* k, int bytes) {
      return cuda_ok(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), "mlp shared memory");
   };
   int st = allow((const void*)net_kernel<false, 8>, net_smem(8));
   if (!st) st = allow((const void*)net_kernel<false, 16>, net_smem(16));
   if (!st) st = allow((const void*)net_kernel<true, 16>, net_smem(16));
   if (!st) st = allow((const void*)wgrad_kernel, kWgradSmem);
   return st;
}

int make_maps(hamstr_mlp* h)
{
   const int B = h->Bmax;
   bool ok = make_map(&h->net.w[0], h->W1b, W, KIN, 128) && make_map(&h->net.w[1], h->W2b, W, W, 128) &&
             make_map(&h->net.w[2], h->W3b, W, W, 128) && make_map(&h->net.w[3], h->W4b, NOP, W, NOP) &&
             make_map(&h->net.w[4], h->W4t, W, KOP, 128) && make_map(&h->net.w[5], h->W3t, W, W, 128) &&
             make_map(&h->net.w[6], h->W2t, W, W, 128);
   ok = ok && make_map(&h->wg.A[0], h->Ht[0], W, B, 128) && make_map(&h->wg.B[0], h->dZt[1], W, B, W) &&
        make_map(&h->wg.A[1], h->Ht[1], W, B, 128) && make_map(&h->wg.B[1], h->dZt[2], W, B, W) &&
        make_map(&h->wg.A[2], h->Ht[2], W, B, 128) && make_map(&h->wg.B[2], h->dZ4t, NOP, B, NOP) &&
        make_map(&h->wg.A[3], h->dZt[0], W, B, 128) && make_map(&h->wg.B[3], h->Xt, NOP, B, NOP);
   if (ok) return HAMSTR_GPU_OK;
   set_last_error("mlp: tensor map encoding failed");
   return HAMSTR_GPU_ERR_CUDA;
}

// BF16 copies of every weight from the FP32 masters
int refresh_bf16(hamstr_mlp* h)
{
   cast_kernel<<<blocks(W * KIN), 256, 0, h->st>>>(h->W1.p, W, KIN, h->W1b, KIN, nullptr, 0);
   cast_kernel<<<blocks(W * W), 256, 0, h->st>>>(h->W2.p, W, W, h->W2b, W, h->W2t, W);
   cast_kernel<<<blocks(W * W), 256, 0, h->st>>>(h->W3.p, W, W, h->W3b, W, h->W3t, W);
   cast_kernel<<<blocks(NOP * W), 256, 0, h->st>>>(h->W4.p, NOP, W, h->W4b, W, h->W4t, KOP);
   return cuda_ok(cudaGetLastError(), "mlp cast");
}

NetArgs net_args(hamstr_mlp* h)
{
   NetArgs a = {};
   a.b1 = h->b1.p;
   a.b2 = h->b2.p;
   a.b3 = h->b3.p;
   a.b4 = h->b4.p;
   a.err = &h->res->err;
   a.give_up = h->give_up;
   h->give_up = -1;
   return a;
}

int finish(hamstr_mlp* h, double* loss)
{
   const int st = cuda_ok(cudaStreamSynchronize(h->st), "mlp sync");
   if (st) return st;
   const volatile Result* r = h->host;
   if (r->err) {
      set_last_error("mlp: a tensor-core pipeline wait timed out");
      h->host->err = 0;
      cudaMemsetAsync(h->err, 0, sizeof(int), h->st);
      return HAMSTR_GPU_ERR_CUDA;
   }
   if (loss) *loss = r->loss;
   return HAMSTR_GPU_OK;
}

// forward, loss and backward of B rows (B_valid of them real), the gradients
// and, with adam, the update
int train(hamstr_mlp* h, const float* feat, const float* targ, long long n_all, int B, int B_valid,
          unsigned long long seed, unsigned long long step, bool adam, float lr, double* loss)
{
   NetArgs a = net_args(h);
   a.feat = feat;
   a.targ = targ;
   a.n_all = n_all;
   a.n = B;
   a.rows = B_valid;
   a.seed = seed;
   a.step = step;
   a.Xt = h->Xt;
   a.dZ4t = h->dZ4t;
   for (int l = 0; l < 3; l++) {
      a.Ht[l] = h->Ht[l];
      a.dZt[l] = h->dZt[l];
   }
   a.err = h->err;
   a.ld = h->Bmax;
   a.G = h->G;
   a.lpart = h->lpart;
   const int ntiles = B / 128;
   net_kernel<true, 16><<<std::min(ntiles, h->nsm), net_threads(16), net_smem(16), h->st>>>(h->net, a);
   int st = cuda_ok(cudaGetLastError(), "mlp pass");
   if (st) return st;
   WgradArgs w = {};
   w.nkb = B / BK;
   w.splits = used_splits(w.nkb, h->max_splits, &w.per);
   w.out[0] = h->part2;
   w.out[1] = h->part3;
   w.out[2] = h->part4;
   w.out[3] = h->part1;
   w.err = h->err;
   wgrad_kernel<<<8 * w.splits, 128, kWgradSmem, h->st>>>(h->wg, w);
   if ((st = cuda_ok(cudaGetLastError(), "mlp weight gradients"))) return st;
   UpdateArgs u = {};
   u.W1 = h->W1; u.b1 = h->b1; u.W2 = h->W2; u.b2 = h->b2;
   u.W3 = h->W3; u.b3 = h->b3; u.W4 = h->W4; u.b4 = h->b4;
   u.W1b = h->W1b; u.W2b = h->W2b; u.W2t = h->W2t; u.W3b = h->W3b; u.W3t = h->W3t; u.W4b = h->W4b; u.W4t = h->W4t;
   u.part1 = h->part1;
   u.part2 = h->part2;
   u.part3 = h->part3;
   u.part4 = h->part4;
   u.splits = w.splits;
   for (int l = 0; l < 3; l++) u.dZt[l] = h->dZt[l];
   u.ld = h->Bmax;
   u.B = B;
   u.lpart = h->lpart;
   u.err = h->err;
   u.host_err = &h->res->err;
   u.loss = &h->res->loss;
   u.adam = adam ? 1 : 0;
   u.lr = lr;
   u.c1 = 1.f - std::pow(0.9f, (float)(step + 1));   // t = step + 1
   u.c2 = 1.f - std::pow(0.999f, (float)(step + 1));
   update_kernel<<<kWeightBlocks + kBiasBlocks + 1, 256, 0, h->st>>>(u);
   if ((st = cuda_ok(cudaGetLastError(), "mlp update"))) return st;
   return finish(h, loss);
}

// (pointer, rows, cols, padded leading dimension) of each logical tensor
struct View {
   float* p;
   int rows, cols, ld;
};

constexpr int kViews = 8;

std::vector<View> views(hamstr_mlp* h, bool grads)
{
   auto at = [&](const Tensor& t) { return grads ? t.g : t.p; };
   return {{at(h->W1), W, NIN, KIN}, {at(h->b1), 1, W, W}, {at(h->W2), W, W, W},    {at(h->b2), 1, W, W},
           {at(h->W3), W, W, W},     {at(h->b3), 1, W, W}, {at(h->W4), NOUT, W, W}, {at(h->b4), 1, NOUT, NOP}};
}

// the logical tensors one after another, without their padding, into page-locked
// host memory.  A copy per tensor into the caller's pageable memory took 9.5 us
// each, eight of them and the synchronisation 92 us; this kernel, the
// synchronisation and one copy on the host 53 us.
struct PackArgs {
   View v[kViews];
   float* out;
};

__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ PackArgs a)
{
   int i = blockIdx.x * blockDim.x + threadIdx.x;
   const int o = i;
#pragma unroll
   for (int t = 0; t < kViews; t++) {
      const View& v = a.v[t];
      const int n = v.rows * v.cols;
      if (i >= 0 && i < n) a.out[o] = v.p[(size_t)(i / v.cols) * v.ld + i % v.cols];
      i -= n;
   }
}

}  // namespace

extern "C" {

int hamstr_mlp_nparams(void) { return kNParams; }

int hamstr_mlp_set_params(hamstr_mlp* h, const float* params);

int hamstr_mlp_destroy(hamstr_mlp* h)
{
   if (!h) return HAMSTR_GPU_OK;
   if (h->st) cudaStreamSynchronize(h->st);
   for (void* p : h->owned) cudaFree(p);
   if (h->host) cudaFreeHost(h->host);
   if (h->host_params) cudaFreeHost(h->host_params);
   if (h->st) cudaStreamDestroy(h->st);
   delete h;
   return HAMSTR_GPU_OK;
}

int hamstr_mlp_create(int Bmax, unsigned long long seed, hamstr_mlp** out)
{
   if (!out || Bmax < 128) return HAMSTR_GPU_ERR_ARG;
   *out = nullptr;
   hamstr_mlp* h = new hamstr_mlp;
   h->Bmax = (Bmax + 127) / 128 * 128;
   if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess) {
      delete h;
      return HAMSTR_GPU_ERR_CUDA;
   }
   int dev = 0;
   cudaGetDevice(&dev);
   cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, dev);
   h->max_splits = std::max(1, h->nsm / 2);   // two 128-row tiles to a split
   const size_t B = h->Bmax;
   int st = configure();
   // a smaller batch may use more splits than the largest one (used_splits evens them out)
   const size_t splits = std::min(h->Bmax / BK, h->max_splits);
#define A(x, n) \
   if (!st) st = h->alloc(&h->x, (n))
   A(W1, W * KIN); A(b1, W); A(W2, W * W); A(b2, W); A(W3, W * W); A(b3, W); A(W4, NOP * W); A(b4, NOP);
   A(W1b, W * KIN); A(W2b, W * W); A(W2t, W * W); A(W3b, W * W); A(W3t, W * W); A(W4b, NOP * W); A(W4t, W * KOP);
   A(Xt, NOP * B); A(dZ4t, NOP * B);
   A(Ht[0], W * B); A(Ht[1], W * B); A(Ht[2], W * B); A(dZt[0], W * B); A(dZt[1], W * B); A(dZt[2], W * B);
   A(G, 3 * W * B);
   A(part1, splits * NOP * W); A(part4, splits * NOP * W); A(part2, splits * W * W); A(part3, splits * W * W);
   A(lpart, 5 * (B / 32));
   A(err, 1);
#undef A
   if (!st) st = cuda_ok(cudaHostAlloc((void**)&h->host, sizeof(Result), cudaHostAllocMapped), "mlp result");
   if (!st) {
      *h->host = Result{};
      st = cuda_ok(cudaHostGetDevicePointer((void**)&h->res, h->host, 0), "mlp result");
   }
   if (!st) st = cuda_ok(cudaHostAlloc((void**)&h->host_params, kNParams * sizeof(float), cudaHostAllocMapped), "mlp parameters");
   if (!st) st = cuda_ok(cudaHostGetDevicePointer((void**)&h->dev_params, h->host_params, 0), "mlp parameters");
   if (!st) st = make_maps(h);
   if (st) {
      hamstr_mlp_destroy(h);
      return st;
   }
   // initial weights: uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)), seeded,
   // biases zero (the common default for GELU MLPs)
   std::vector<float> p(kNParams, 0.f);
   unsigned long long s = seed ? seed : 1;
   auto rnd = [&]() {
      s ^= s << 13;
      s ^= s >> 7;
      s ^= s << 17;   // xorshift64 (Marsaglia, 2003)
      return (double)(s >> 11) * (1.0 / 9007199254740992.0);
   };
   size_t o = 0;
   const int fan[4] = {NIN, W, W, W}, rows[4] = {W, W, W, NOUT};
   for (int l = 0; l < 4; l++) {
      const double a = 1.0 / std::sqrt((double)fan[l]);
      for (int i = 0; i < rows[l] * fan[l]; i++) p[o++] = (float)((2.0 * rnd() - 1.0) * a);
      o += rows[l];
   }
   *out = h;
   st = hamstr_mlp_set_params(h, p.data());
   if (st) {
      hamstr_mlp_destroy(h);
      *out = nullptr;
   }
   return st;
}

int hamstr_mlp_set_params(hamstr_mlp* h, const float* params)
{
   if (!h || !params) return HAMSTR_GPU_ERR_ARG;
   size_t o = 0;
   for (const View& v : views(h, false)) {
      std::vector<float> buf((size_t)v.rows * v.ld, 0.f);
      for (int r = 0; r < v.rows; r++)
         for (int c = 0; c < v.cols; c++) buf[(size_t)r * v.ld + c] = params[o++];
      int st = cuda_ok(cudaMemcpyAsync(v.p, buf.data(), buf.size() * sizeof(float), cudaMemcpyHostToDevice, h->st),
                       "mlp set params");
      if (st) return st;
   }
   int st = refresh_bf16(h);
   if (st) return st;
   return cuda_ok(cudaStreamSynchronize(h->st), "mlp set params sync");
}

static int get_tensors(hamstr_mlp* h, bool grads, float* out)
{
   PackArgs a = {};
   const std::vector<View> v = views(h, grads);
   std::copy(v.begin(), v.end(), a.v);
   a.out = h->dev_params;
   std::lock_guard<std::mutex> lock(h->params_mutex);
   pack_kernel<<<(kNParams + 255) / 256, 256, 0, h->st>>>(a);
   int st = cuda_ok(cudaGetLastError(), "mlp get");
   if (!st) st = cuda_ok(cudaStreamSynchronize(h->st), "mlp get sync");
   if (!st) std::memcpy(out, h->host_params, kNParams * sizeof(float));
   return st;
}

int hamstr_mlp_get_params(hamstr_mlp* h, float* out)
{
   if (!h || !out) return HAMSTR_GPU_ERR_ARG;
   return get_tensors(h, false, out);
}

int hamstr_mlp_get_grads(hamstr_mlp* h, float* out)
{
   if (!h || !out) return HAMSTR_GPU_ERR_ARG;
   return get_tensors(h, true, out);
}

int hamstr_check_mlp_wait(hamstr_mlp* h, int tile)
{
   if (!h || tile < 0) return HAMSTR_GPU_ERR_ARG;
   h->give_up = tile;
   return HAMSTR_GPU_OK;
}

int hamstr_mlp_forward(hamstr_mlp* h, const float* feat, int n, float* y)
{
   if (!h || !feat || !y || n < 1) return HAMSTR_GPU_ERR_ARG;
   NetArgs a = net_args(h);
   a.feat = feat;
   a.n_all = n;
   a.n = a.rows = n;
   a.y = y;
   const int ntiles = (n - 1) / 128 + 1;
   if (ntiles <= h->nsm) net_kernel<false, 16><<<ntiles, net_threads(16), net_smem(16), h->st>>>(h->net, a);
   else net_kernel<false, 8><<<std::min(ntiles, 2 * h->nsm), net_threads(8), net_smem(8), h->st>>>(h->net, a);
   const int st = cuda_ok(cudaGetLastError(), "mlp pass");
   return st ? st : finish(h, nullptr);
}

int hamstr_mlp_grad(hamstr_mlp* h, const float* feat, const float* targ, int n, double* loss_out)
{
   if (!h || !feat || !targ || n < 1 || n > h->Bmax) return HAMSTR_GPU_ERR_ARG;
   return train(h, feat, targ, n, (n + 127) / 128 * 128, n, 0, 0, false, 0.f, loss_out);
}

int hamstr_mlp_train_step(hamstr_mlp* h, const float* feat_all, const float* targ_all, long long n_all, int batch,
                          unsigned long long seed, unsigned long long step, float lr, double* loss_out)
{
   if (!h || !feat_all || !targ_all || n_all < 1 || batch < 128 || batch > h->Bmax || batch % 128 || !seed)
      return HAMSTR_GPU_ERR_ARG;
   return train(h, feat_all, targ_all, n_all, batch, batch, seed, step, true, lr, loss_out);
}

}  // extern "C"
