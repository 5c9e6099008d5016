// ##################################################################
//
// mixed.cu -- mixed-precision defect correction
//
// The residual that defines the steady state (reconstruction, Roe flux and
// the per-cell sums of computeRHS) stays in FP64 and is bit-identical to the
// reference.  The approximate operator of the implicit step -- the Roe
// Jacobians, the ADI block assembly and block-tridiagonal line solves, and
// the linearised residual of the sweeps (ADI.cpp, computeLinearRHS.cpp) --
// runs in FP32.  Near convergence the FP32 operator only changes how fast
// the FP64 residual falls, not where it goes to zero.
//
// GB300 issues FP32 about 70x faster than FP64 (64-cycle dependent FP64
// latency against 4 for FP32), so the line solves here are one thread per
// chain running the block Thomas elimination in registers, with chains of
// similar length sharing a warp.
// ##################################################################
#include <algorithm>
#include <type_traits>
#include "cell_sum.cuh"
#include "device_state.h"
#include "plan.h"
#include "recon.cuh"
#include "roe.cuh"

namespace hamstr {

namespace {

constexpr int kThreads = 256;
static_assert(kThreads == kNormBlock, "cell kernels run one norm block per thread block");

// ---------------- residual + FP32 Jacobian ----------------
constexpr int kFaceSmem = 9 * 16 + 16;
// PRE: the order-5 face states come from recon5_kernel
template <int ORDER, bool SD, bool PRE = false>
__global__ void __launch_bounds__(kThreads) mx_rhs_face_kernel(DeviceState d)
{
   // the FP32 Jacobians leave through shared memory, so their stores are
   // whole lines (8 float4 per slot, consecutive slots; row stride 9)
   extern __shared__ float4 sj[];   // kFaceSmem bytes a thread
   const int nb = blockDim.x, s0 = blockIdx.x * nb, s = s0 + threadIdx.x;
   unsigned char* live = reinterpret_cast<unsigned char*>(sj + 9 * nb);
   if (halted(d)) return;
   const bool act = s < d.nSlot && !frozen_slot(d, s);
   live[threadIdx.x] = act ? 1 : 0;
   if (act) {
      const int4 sl = d.slot[s];
      const double2 nv = d.normal[s];
      double L[4], R[4];
      if (ORDER == 5 && PRE) face_states_pre(d, s, (sl.w & 1) != 0, L, R);
      else face_states<ORDER, SD>(d, sl.x, (sl.w & 1) != 0, L, R);
      RoeOut o;
      if (!roe_face<false, SD>(nv.x, nv.y, L, R, d.fc.gamma, o, nullptr, nullptr))
         atomicOr(d.status, DEV_ERR_NAN_SPEC);
      st4(d.flux + 4 * (size_t)s, o.flux);
      d.spec[s] = o.spec;
      const float Lf[4] = {float(L[0]), float(L[1]), float(L[2]), float(L[3])};
      const float Rf[4] = {float(R[0]), float(R[1]), float(R[2]), float(R[3])};
      float lm[16], rm[16];
      roe_jacobian_only<float>(float(nv.x), float(nv.y), Lf, Rf, float(d.fc.gamma), lm, rm);
#pragma unroll
      for (int q = 0; q < 4; q++) {
         sj[threadIdx.x * 9 + q] = make_float4(lm[4 * q], lm[4 * q + 1], lm[4 * q + 2], lm[4 * q + 3]);
         sj[threadIdx.x * 9 + 4 + q] = make_float4(rm[4 * q], rm[4 * q + 1], rm[4 * q + 2], rm[4 * q + 3]);
      }
   }
   __syncthreads();
   const int nloc = min(nb, d.nSlot - s0);
   float4* __restrict__ dst = reinterpret_cast<float4*>(d.ff32 + 32 * (size_t)s0);
   for (int c = threadIdx.x; c < 8 * nloc; c += nb)
      if (live[c >> 3]) dst[c] = sj[(c >> 3) * 9 + (c & 7)];
}

// r (already scaled by CFL/sigma in FP64) -> FP32 r, r0; dq = 0
__global__ void __launch_bounds__(kThreads) mx_init_kernel(DeviceState d)
{
   const int c = blockIdx.x * blockDim.x + threadIdx.x;
   if (c >= d.nCell || halted(d) || frozen_cell(d, c)) return;
   double r[4];
   ld4(d.r + 4 * (size_t)c, r);
   const float rf[4] = {float(r[0]), float(r[1]), float(r[2]), float(r[3])};
   const float z[4] = {0.f, 0.f, 0.f, 0.f};
   st4(d.r32 + 4 * (size_t)c, rf);
   st4(d.r032 + 4 * (size_t)c, rf);
   st4(d.dq32 + 4 * (size_t)c, z);
}

// the tiled index of element e of tile row s in lane `lane` of a W-wide
// array (W a multiple of 4): each lane's elements 4k .. 4k+3 are one float4,
// and the 32 lanes' float4 of one group lie together, so a warp's access of
// one group is 512 contiguous bytes and takes one instruction per lane
__device__ __forceinline__ size_t tix(int s, int W, int e, int lane)
{
   return (((size_t)s * W + (e & ~3)) << 5) + 4 * lane + (e & 3);
}

// FP32 blocks in the reference's term order (ADI.cpp:62-217), one thread per
// row k of a mesh row's three blocks (a float4 of every term; the row's lists
// and scale once for the twelve entries); the alternative to mx_row below.
// Bound by the latency of the lookups, tile row to term list to face.  512 x 128,
// 30% split: 70 us with a thread per entry, 29 us with one per block row, 27 us
// so; 32 meshes of 983,040 cells 349 us with one per block row, 253 us so.
__global__ void __launch_bounds__(kThreads) mx_assemble_kernel(DeviceState d)
{
   // a warp: eight lanes of a tile row times the four rows k of its blocks, so
   // that a term's block is 64 contiguous bytes of four neighbouring lanes and
   // a store fills four whole lines of 128 bytes
   const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= 128 * (size_t)d.tile_rows || halted(d)) return;
   const int k = (int)(t & 3), lane = (int)((t >> 2) & 31), srow = (int)(t >> 7);
   const int row = d.tile_row[32 * (size_t)srow + lane];
   if (row < 0) return;
   const int sc = d.row_scell[row];
   if (frozen_cell(d, sc)) return;
   int4 list[3];
#pragma unroll
   for (int b = 0; b < 3; b++) list[b] = reinterpret_cast<const int4*>(d.row_ops + 3 * kOpsPerBlock * (size_t)row)[b];
   const float s = float(d.dtfac[sc]);
#pragma unroll
   for (int b = 0; b < 3; b++) {
      const int ops[kOpsPerBlock] = {list[b].x, list[b].y, list[b].z, list[b].w};
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int o = 0; o < kOpsPerBlock; o++) {
         const int op = ops[o];
         if (op < 0) break;
         const int slot = op >> 3, sel = (op >> 1) & 3;
         float v[4];
         ld4(d.ff32 + 32 * (size_t)slot + (sel == OP_SEL_L ? 0 : 16) + 4 * k, v);
         if (sel == OP_SEL_RREFL) {
            const double4 rf = d.refl[d.slot_face[slot]];
            const float r01 = v[1], r02 = v[2];
            v[1] = float(rf.x) * r01 + float(rf.y) * r02;
            v[2] = float(rf.z) * r01 + float(rf.w) * r02;
         }
#pragma unroll
         for (int m = 0; m < 4; m++) {
            if (op & 1) acc[m] -= v[m];
            else acc[m] += v[m];
         }
      }
#pragma unroll
      for (int m = 0; m < 4; m++) {
         acc[m] *= s;
         if (b == 1 && m == k) acc[m] += 1.f;
      }
      st4(d.blk32 + tix(srow, 48, 16 * b + 4 * k, lane), acc);
   }
}

// whether chain ich takes the segmented solve: sp_on 1 takes the long
// periodic chains, 2 the long open ones as well
__device__ __forceinline__ bool spike_active(const DeviceState& d, int ich)
{
   return d.sp_on && d.chain_spike[ich] >= 0 && (d.sp_on == 2 || d.chain_periodic[ich]);
}

// 16 consecutive elements of a tiled record (4 float4, 128 floats apart: each load of
// a warp is one 128-byte line)
__device__ __forceinline__ void ld16t(const float* __restrict__ p, float (&v)[16])
{
#pragma unroll
   for (int q = 0; q < 4; q++) {
      const float4 x = *reinterpret_cast<const float4*>(p + 128 * q);
      v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
   }
}

__device__ __forceinline__ void st16t(float* __restrict__ p, const float (&v)[16])
{
#pragma unroll
   for (int q = 0; q < 4; q++)
      *reinterpret_cast<float4*>(p + 128 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// ---------------- FP32 line solves, one thread per chain ----------------
// The same split as the FP64 path: the block factorisation runs once per
// step (mx_factor), each sweep replays the right-hand side (mx_solve).  One
// thread carries a whole chain in registers (FP32 latency is 4 cycles, so
// the recurrence is short), rows are loaded one ahead or several rows at a
// time, and products use FMA since this operator is approximate by design.  Record layout per row
// (80 floats): A, LU of B', C', fill-in a', c_{N-1} at elimination step i.
constexpr int kRec = 80;

struct LUf {
   float p0, u01, u02, u03, l10, p1, u12, u13, l20, l21, p2, u23, l30, l31, l32, p3;
};

__device__ __forceinline__ LUf luf_factor(const float (&b)[16])
{
   LUf u;
   u.p0 = 1.f / b[0];
   u.u01 = b[1] * u.p0; u.u02 = b[2] * u.p0; u.u03 = b[3] * u.p0;
   u.l10 = b[4];
   u.p1 = 1.f / __fmaf_rn(-u.l10, u.u01, b[5]);
   u.u12 = __fmaf_rn(-u.l10, u.u02, b[6]) * u.p1;
   u.u13 = __fmaf_rn(-u.l10, u.u03, b[7]) * u.p1;
   u.l20 = b[8];
   u.l21 = __fmaf_rn(-u.l20, u.u01, b[9]);
   u.p2 = 1.f / __fmaf_rn(-u.l21, u.u12, __fmaf_rn(-u.l20, u.u02, b[10]));
   u.u23 = __fmaf_rn(-u.l21, u.u13, __fmaf_rn(-u.l20, u.u03, b[11])) * u.p2;
   u.l30 = b[12];
   u.l31 = __fmaf_rn(-u.l30, u.u01, b[13]);
   u.l32 = __fmaf_rn(-u.l31, u.u12, __fmaf_rn(-u.l30, u.u02, b[14]));
   u.p3 = 1.f / __fmaf_rn(-u.l32, u.u23, __fmaf_rn(-u.l31, u.u13, __fmaf_rn(-u.l30, u.u03, b[15])));
   return u;
}

__device__ __forceinline__ void luf_solve(const LUf& u, float& x0, float& x1, float& x2, float& x3)
{
   const float d0 = x0 * u.p0;
   const float d1 = __fmaf_rn(-u.l10, d0, x1) * u.p1;
   const float d2 = __fmaf_rn(-u.l21, d1, __fmaf_rn(-u.l20, d0, x2)) * u.p2;
   const float d3 = __fmaf_rn(-u.l32, d2, __fmaf_rn(-u.l31, d1, __fmaf_rn(-u.l30, d0, x3))) * u.p3;
   x3 = d3;
   x2 = __fmaf_rn(-u.u23, x3, d2);
   x1 = __fmaf_rn(-u.u13, x3, __fmaf_rn(-u.u12, x2, d1));
   x0 = __fmaf_rn(-u.u03, x3, __fmaf_rn(-u.u02, x2, __fmaf_rn(-u.u01, x1, d0)));
}

__device__ __forceinline__ void luf_store(float* p, const LUf& u)
{
   const float v[16] = {u.p0, u.u01, u.u02, u.u03, u.l10, u.p1, u.u12, u.u13,
                        u.l20, u.l21, u.p2, u.u23, u.l30, u.l31, u.l32, u.p3};
#pragma unroll
   for (int m = 0; m < 16; m += 4) *reinterpret_cast<float4*>(p + m) = make_float4(v[m], v[m + 1], v[m + 2], v[m + 3]);
}

__device__ __forceinline__ LUf luf_of(const float (&v)[16])
{
   LUf u;
   u.p0 = v[0]; u.u01 = v[1]; u.u02 = v[2]; u.u03 = v[3]; u.l10 = v[4]; u.p1 = v[5]; u.u12 = v[6]; u.u13 = v[7];
   u.l20 = v[8]; u.l21 = v[9]; u.p2 = v[10]; u.u23 = v[11]; u.l30 = v[12]; u.l31 = v[13]; u.l32 = v[14]; u.p3 = v[15];
   return u;
}

__device__ __forceinline__ LUf luf_load(const float* p)
{
   float v[16];
#pragma unroll
   for (int m = 0; m < 16; m += 4) {
      const float4 a = *reinterpret_cast<const float4*>(p + m);
      v[m] = a.x; v[m + 1] = a.y; v[m + 2] = a.z; v[m + 3] = a.w;
   }
   return luf_of(v);
}

// the LU record of a tiled row
__device__ __forceinline__ void luf_store_t(float* p, const LUf& u)
{
   const float v[16] = {u.p0, u.u01, u.u02, u.u03, u.l10, u.p1, u.u12, u.u13,
                        u.l20, u.l21, u.p2, u.u23, u.l30, u.l31, u.l32, u.p3};
   st16t(p, v);
}

__device__ __forceinline__ void ld16f(const float* p, float (&v)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m += 4) {
      const float4 a = *reinterpret_cast<const float4*>(p + m);
      v[m] = a.x; v[m + 1] = a.y; v[m + 2] = a.z; v[m + 3] = a.w;
   }
}

// M <- LU^{-1} M, column by column
__device__ __forceinline__ void luf_cols(const LUf& u, float (&m)[16])
{
#pragma unroll
   for (int j = 0; j < 4; j++) luf_solve(u, m[j], m[4 + j], m[8 + j], m[12 + j]);
}

// out = acc - M * X (4x4), acc = nullptr for 0
__device__ __forceinline__ void mm_sub(const float (&M)[16], const float (&X)[16], float (&acc)[16])
{
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
         float a = acc[4 * k + j];
#pragma unroll
         for (int l = 0; l < 4; l++) a = __fmaf_rn(-M[4 * k + l], X[4 * l + j], a);
         acc[4 * k + j] = a;
      }
}

// One FP32 block from its term list, in the reference's term order
// (ADI.cpp:62-217): +/- L or R of a face slot, or R with its velocity
// columns reflected at a wall (ADI.cpp:151-163)
__device__ __forceinline__ void mx_block(const DeviceState& d, const int* __restrict__ ops, float (&M)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) M[m] = 0.f;
#pragma unroll
   for (int o = 0; o < kOpsPerBlock; o++) {
      const int op = ops[o];
      if (op < 0) break;
      const int slot = op >> 3, sel = (op >> 1) & 3;
      float v[16];
      ld16f(d.ff32 + 32 * (size_t)slot + (sel == OP_SEL_L ? 0 : 16), v);
      if (sel == OP_SEL_RREFL) {
         const double4 rf = d.refl[d.slot_face[slot]];
#pragma unroll
         for (int k = 0; k < 4; k++) {
            const float r01 = v[4 * k + 1], r02 = v[4 * k + 2];
            v[4 * k + 1] = float(rf.x) * r01 + float(rf.y) * r02;
            v[4 * k + 2] = float(rf.z) * r01 + float(rf.w) * r02;
         }
      }
      if (op & 1) {
#pragma unroll
         for (int m = 0; m < 16; m++) M[m] -= v[m];
      } else {
#pragma unroll
         for (int m = 0; m < 16; m++) M[m] += v[m];
      }
   }
}

// what the fused assembly of one row looks up first: its term lists and
// its scaled cell (the face Jacobians and the CFL/sigma factor follow from
// them), loaded a row earlier than the blocks so that each row waits on
// one memory round trip, not two
struct RowRef {
   int4 ops[3];
   int scell;
};

__device__ __forceinline__ RowRef mx_rowref(const DeviceState& d, int row)
{
   RowRef r;
   const int4* p = reinterpret_cast<const int4*>(d.row_ops + 3 * kOpsPerBlock * (size_t)row);
   r.ops[0] = p[0];
   r.ops[1] = p[1];
   r.ops[2] = p[2];
   r.scell = d.row_scell[row];
   return r;
}

// the three blocks of one ADI row from its looked-up references, scaled by
// CFL/sigma, B + I (ADI.cpp:197-217)
__device__ __forceinline__ void mx_row_ref(const DeviceState& d, const RowRef& r, float (&A)[16], float (&B)[16],
                                           float (&C)[16])
{
   const int oa[4] = {r.ops[0].x, r.ops[0].y, r.ops[0].z, r.ops[0].w};
   const int ob[4] = {r.ops[1].x, r.ops[1].y, r.ops[1].z, r.ops[1].w};
   const int oc[4] = {r.ops[2].x, r.ops[2].y, r.ops[2].z, r.ops[2].w};
   mx_block(d, oa, A);
   mx_block(d, ob, B);
   mx_block(d, oc, C);
   const float s = float(d.dtfac[r.scell]);
#pragma unroll
   for (int m = 0; m < 16; m++) {
      A[m] *= s;
      B[m] *= s;
      C[m] *= s;
   }
#pragma unroll
   for (int k = 0; k < 4; k++) B[5 * k] += 1.f;
}

// ---- fused assembly with the next row's terms staged in shared memory ----
// Each of a row's up to 3 x kOpsPerBlock face-Jacobian terms is a 64-byte
// block of ff32.  Summing them as they arrive makes the row wait on one
// round trip per term; instead the terms of row i+1 are copied into shared
// memory with asynchronous copies (cp.async, 16 bytes each) while row i is
// factored, and summed, in the same order as mx_block, after it.  Layout:
// float4 q of term t of thread `tid` at ((t * 4 + q) * blockDim + tid), so
// a warp's copies and reads of one float4 are one 512-byte span.
constexpr int kStageTerms = 3 * kOpsPerBlock;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
   const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
   asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// every copy of this thread has arrived, committed to a group or not
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// all but the newest N groups of this thread's copies have arrived
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// copies through L2 only: the rows are read once
__device__ __forceinline__ void cp_async16_cg(void* smem, const void* gmem)
{
   const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
   asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// A thread's rows on their way: a ring of DEPTH rows of V float4 in shared
// memory, each filled by the thread's own asynchronous copies, one group to a
// row, DEPTH - 1 rows ahead.  A row of a chain is a few dozen dependent FP32
// operations in the solve, some thousand cycles in the factorisation; a load is
// 600 to 1,000 cycles, and there are not registers for that many rows.  A
// row's slot is its number modulo DEPTH, known at compile time in loops unrolled
// by DEPTH; a warp's access of one float4 is 512 contiguous bytes.
template <int V, int DEPTH>
struct RowRing {
   float4* buf;
   __device__ __forceinline__ explicit RowRing(float4* stage)
       : buf(stage + (threadIdx.x >> 5) * (32 * V * DEPTH) + (threadIdx.x & 31))
   {
   }
   __device__ __forceinline__ float4* at(int slot, int v) const { return buf + 32 * (slot * V + v); }
   // N float4 of a tiled record (128 floats apart) into v, v + 1, ..
   template <int N>
   __device__ __forceinline__ void copy(int slot, int v, const float* src) const
   {
#pragma unroll
      for (int q = 0; q < N; q++) cp_async16_cg(at(slot, v + q), src + 128 * q);
   }
   template <int N>
   __device__ __forceinline__ void read(int slot, int v, float (&x)[N]) const
   {
#pragma unroll
      for (int q = 0; q < N / 4; q++) {
         const float4 y = *at(slot, v + q);
         x[4 * q] = y.x; x[4 * q + 1] = y.y; x[4 * q + 2] = y.z; x[4 * q + 3] = y.w;
      }
   }
};

__device__ __forceinline__ float4* stage_at(float4* stage, int term, int q)
{
   return stage + (size_t)(term * 4 + q) * blockDim.x + threadIdx.x;
}

// issue the copies of row r's terms (terms with op < 0 copy nothing)
__device__ __forceinline__ void mx_stage_row(const DeviceState& d, const RowRef& r, float4* stage)
{
   const int ops[kStageTerms] = {r.ops[0].x, r.ops[0].y, r.ops[0].z, r.ops[0].w, r.ops[1].x, r.ops[1].y,
                                 r.ops[1].z, r.ops[1].w, r.ops[2].x, r.ops[2].y, r.ops[2].z, r.ops[2].w};
#pragma unroll
   for (int t = 0; t < kStageTerms; t++) {
      const int op = ops[t];
      if (op < 0) continue;
      const float* src = d.ff32 + 32 * (size_t)(op >> 3) + (((op >> 1) & 3) == OP_SEL_L ? 0 : 16);
#pragma unroll
      for (int q = 0; q < 4; q++) cp_async16(stage_at(stage, t, q), src + 4 * q);
   }
   cp_async_commit();
}

// mx_block from the staged terms of block b (0, 1, 2 = A, B, C)
__device__ __forceinline__ void mx_block_staged(const DeviceState& d, const int (&ops)[kOpsPerBlock], int b,
                                                const float4* stage, float (&M)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) M[m] = 0.f;
#pragma unroll
   for (int o = 0; o < kOpsPerBlock; o++) {
      const int op = ops[o];
      if (op < 0) break;
      float v[16];
#pragma unroll
      for (int q = 0; q < 4; q++) {
         const float4 x = *stage_at(const_cast<float4*>(stage), b * kOpsPerBlock + o, q);
         v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
      }
      if (((op >> 1) & 3) == OP_SEL_RREFL) {
         const double4 rf = d.refl[d.slot_face[op >> 3]];
#pragma unroll
         for (int k = 0; k < 4; k++) {
            const float r01 = v[4 * k + 1], r02 = v[4 * k + 2];
            v[4 * k + 1] = float(rf.x) * r01 + float(rf.y) * r02;
            v[4 * k + 2] = float(rf.z) * r01 + float(rf.w) * r02;
         }
      }
      if (op & 1) {
#pragma unroll
         for (int m = 0; m < 16; m++) M[m] -= v[m];
      } else {
#pragma unroll
         for (int m = 0; m < 16; m++) M[m] += v[m];
      }
   }
}

// mx_row_ref from staged terms and the row's CFL/sigma factor s
__device__ __forceinline__ void mx_row_staged(const DeviceState& d, const RowRef& r, const float4* stage, float s,
                                              float (&A)[16], float (&B)[16], float (&C)[16])
{
   const int oa[4] = {r.ops[0].x, r.ops[0].y, r.ops[0].z, r.ops[0].w};
   const int ob[4] = {r.ops[1].x, r.ops[1].y, r.ops[1].z, r.ops[1].w};
   const int oc[4] = {r.ops[2].x, r.ops[2].y, r.ops[2].z, r.ops[2].w};
   mx_block_staged(d, oa, 0, stage, A);
   mx_block_staged(d, ob, 1, stage, B);
   mx_block_staged(d, oc, 2, stage, C);
#pragma unroll
   for (int m = 0; m < 16; m++) {
      A[m] *= s;
      B[m] *= s;
      C[m] *= s;
   }
#pragma unroll
   for (int k = 0; k < 4; k++) B[5 * k] += 1.f;
}

// rows of the periodic last-row elimination whose loads issue together
// where all chains are resident at once (1 otherwise: there the kernel is
// bound by throughput, not by one chain's round trips)
constexpr int kElimChunk = 2;

// all chains, thread p on the chain at position p of line_chains; ED rows of
// the last-row elimination per chunk.  FUSED: each thread builds its chain's
// blocks straight from the FP32 face Jacobians; otherwise it reads those that
// mx_assemble_kernel wrote, through its ring (512 x 128, 30% split: 124 us with
// the next row's blocks in registers, 50 us so; 32 meshes of 983,040 cells 75 us).
constexpr int kFactorDepth = 4, kFactorVec = 12;

template <bool FUSED, int ED>
__global__ void __launch_bounds__(256) mx_factor_kernel(DeviceState d, int count)
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= count || halted(d)) return;
   const int ich = d.line_chains[t];
   if (frozen_chain(d, ich) || spike_active(d, ich)) return;
   const int N = d.chain_nrows[ich], row0 = d.chain_row0[ich], lane = t & 31, s0 = d.grp_row0[t >> 5];
   const bool per = d.chain_periodic[ich] != 0;
   float A[16], B[16], C[16], cp[16], ap[16];
   bool bad = false;   // a reciprocal pivot is not finite (DEV_ERR_PIVOT)
   RowRef rnext{};   // fused: references of row i + 1, looked up a row ahead
   RowRef rstaged{};  // fused: references of the row whose terms are staged
   float snext = 0.f;  // fused: its CFL/sigma factor
   extern __shared__ float4 stage[];   // fused: kStageTerms x 4 float4 per thread; otherwise the ring
   const RowRing<kFactorVec, kFactorDepth> ring(stage);
   constexpr int AHEAD = kFactorDepth - 1;
   auto fetch = [&](int i, int slot) {   // unfused: row i's blocks, as mx_assemble_kernel left them
      if (i < N) ring.copy<12>(slot, 0, d.blk32 + tix(s0 + i, 48, 0, lane));
      cp_async_commit();
   };
   if (FUSED) {
      const RowRef r0 = mx_rowref(d, row0);
      if (N > 1) rnext = mx_rowref(d, row0 + 1);
      mx_row_ref(d, r0, A, B, C);
   } else {
#pragma unroll
      for (int i = 0; i < AHEAD; i++) fetch(i, i);
   }
   // the rows, with or without the fill-in column (periodic chains): the loop for
   // both was 380 instructions an open row, 85 us for 512 x 128; apart 67 us, and
   // 56 us with the ring's slots known at compile time
   auto rows = [&](auto fill_in) {
      constexpr bool PER = decltype(fill_in)::value;
      auto one = [&](int i, int slot) {
         if (FUSED) {
            if (i + 1 < N) {
               // row i+1's terms are copied while row i is factored
               mx_stage_row(d, rnext, stage);
               rstaged = rnext;
               snext = float(d.dtfac[rnext.scell]);
               if (i + 2 < N) rnext = mx_rowref(d, row0 + i + 2);
            }
         } else {
            cp_async_wait<AHEAD - 1>();
            ring.read(slot, 0, A);
            ring.read(slot, 4, B);
            ring.read(slot, 8, C);
            fetch(i + AHEAD, (slot + AHEAD) % kFactorDepth);
         }
         float* rec = d.fac32 + tix(s0 + i, kRec, 0, lane);
         st16t(rec, A);
         float fill[16];
         if (i > 0) {
            mm_sub(A, cp, B);
#pragma unroll
            for (int m = 0; m < 16; m++) fill[m] = 0.f;
            if (PER) mm_sub(A, ap, fill);
         } else {
#pragma unroll
            for (int m = 0; m < 16; m++) fill[m] = A[m];
         }
         const LUf u = luf_factor(B);
         luf_store_t(rec + 32 * 16, u);
         bad |= nonfinite(u.p0) || nonfinite(u.p1) || nonfinite(u.p2) || nonfinite(u.p3);
         if (PER && i == N - 2) {
#pragma unroll
            for (int m = 0; m < 16; m++) C[m] += fill[m];
            luf_cols(u, C);
#pragma unroll
            for (int m = 0; m < 16; m++) fill[m] = C[m];
         } else {
            luf_cols(u, C);
            if (PER) luf_cols(u, fill);
         }
         st16t(rec + 32 * 32, C);
         if (PER) st16t(rec + 32 * 48, fill);
#pragma unroll
         for (int m = 0; m < 16; m++) {
            cp[m] = C[m];
            if (PER) ap[m] = fill[m];
         }
         if (FUSED && i + 1 < N) {
            cp_async_wait_all();
            mx_row_staged(d, rstaged, stage, snext, A, B, C);
         }
      };
      constexpr int UNROLL = FUSED ? 1 : kFactorDepth;
      for (int i0 = 0; i0 < N; i0 += UNROLL) {
#pragma unroll
         for (int u = 0; u < UNROLL; u++) {
            if (i0 + u >= N) break;
            one(i0 + u, u);
         }
      }
   };
   if (per) rows(std::true_type{});
   else rows(std::false_type{});
   if (!FUSED) cp_async_wait_all();
   if (!per) {
      if (bad) atomicOr(d.status, DEV_ERR_PIVOT);
      return;
   }
   // last-row elimination (triSolvers.cpp:967-999).  A row's arithmetic is
   // short, so the loads of ED rows are issued before it; the main loop's
   // arrays are dead here, so a chunk of 2 adds no registers.
   constexpr int D = ED;
   float cN[16], bN[16];
#pragma unroll
   for (int m = 0; m < 16; m++) { cN[m] = cp[m]; bN[m] = ((m >> 2) == (m & 3)) ? 1.f : 0.f; }
   for (int i0 = 0; i0 < N - 1; i0 += D) {
      float ci[D][16], ai[D][16];
#pragma unroll
      for (int u = 0; u < D; u++)
         if (i0 + u < N - 1) {
            const float* rec = d.fac32 + tix(s0 + i0 + u, kRec, 0, lane);
            ld16t(rec + 32 * 32, ci[u]);
            ld16t(rec + 32 * 48, ai[u]);
         }
#pragma unroll
      for (int u = 0; u < D; u++)
         if (i0 + u < N - 1) {
            st16t(d.fac32 + tix(s0 + i0 + u, kRec, 64, lane), cN);
            float tt[16];
#pragma unroll
            for (int m = 0; m < 16; m++) tt[m] = 0.f;
            mm_sub(cN, ci[u], tt);
            mm_sub(cN, ai[u], bN);
#pragma unroll
            for (int m = 0; m < 16; m++) cN[m] = tt[m];
         }
   }
   const LUf uN = luf_factor(bN);
   luf_store(d.facN32 + 16 * d.chain_facN[ich], uN);
   bad |= nonfinite(uN.p0) || nonfinite(uN.p1) || nonfinite(uN.p2) || nonfinite(uN.p3);
   if (bad) atomicOr(d.status, DEV_ERR_PIVOT);
}

// y -= M x (4x4, 4-vector)
__device__ __forceinline__ void mv_sub(const float (&M)[16], const float (&x)[4], float (&y)[4])
{
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) y[k] = __fmaf_rn(-M[4 * k + j], x[j], y[k]);
}

__device__ __forceinline__ void mv_add(const float (&M)[16], const float (&x)[4], float (&y)[4])
{
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) y[k] = __fmaf_rn(M[4 * k + j], x[j], y[k]);
}

// The rings of the solves: a row's record by halves (A and LU, or two of C', V,
// W), and a 4-vector; cells are looked up a ring's rows before their copies.
constexpr int kSolveVec = 9;
constexpr size_t kFacRow = 32 * kRec, kFsRow = 128;   // floats from a tile row to the next

// f(i) = LU^{-1}(F(i) - A(i) f(i-1)) for a thread's n tiled rows, F(i) =
// r32[fcell[i]] (0 without a cell); f into fs, the last f in xp
template <int DEPTH>
__device__ __forceinline__ void forward_rows(const RowRing<kSolveVec, DEPTH>& ring, int n, const float* fac, float* fs, const int* fcell,
                                             const float* r32, float (&xp)[4])
{
   constexpr int AHEAD = DEPTH - 1;
   auto fetch = [&](int i, int slot, int cell) {
      if (i < n) {
         ring.template copy<8>(slot, 0, fac + kFacRow * i);
         if (cell >= 0) cp_async16_cg(ring.at(slot, 8), r32 + 4 * (size_t)cell);
         else *ring.at(slot, 8) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      cp_async_commit();
   };
   auto look = [&](int i) { return i < n ? fcell[i] : -1; };
#pragma unroll
   for (int i = 0; i < AHEAD; i++) fetch(i, i, look(i));
   int fc[DEPTH];
#pragma unroll
   for (int u = 0; u < DEPTH; u++) fc[u] = look(AHEAD + u);
   // a row leaves the ring while the one before it is solved
   float a[16], lu[16], x[4];
   cp_async_wait<AHEAD - 1>();
   ring.read(0, 0, a);
   ring.read(0, 4, lu);
   ring.read(0, 8, x);
   for (int i0 = 0; i0 < n; i0 += DEPTH) {
      int fcn[DEPTH];
#pragma unroll
      for (int u = 0; u < DEPTH; u++) fcn[u] = look(i0 + AHEAD + DEPTH + u);
#pragma unroll
      for (int u = 0; u < DEPTH; u++) {
         const int i = i0 + u;
         if (i >= n) break;
         float an[16], ln[16], y[4];
         cp_async_wait<AHEAD - 2>();
         ring.read((u + 1) % DEPTH, 0, an);   // (past the last row: what the slot holds, unused)
         ring.read((u + 1) % DEPTH, 4, ln);
         ring.read((u + 1) % DEPTH, 8, y);
         fetch(i + AHEAD, (u + AHEAD) % DEPTH, fc[u]);
         if (i > 0) mv_sub(a, xp, x);
         luf_solve(luf_of(lu), x[0], x[1], x[2], x[3]);
         *reinterpret_cast<float4*>(fs + kFsRow * i) = make_float4(x[0], x[1], x[2], x[3]);
#pragma unroll
         for (int k = 0; k < 4; k++) { xp[k] = x[k]; x[k] = y[k]; }
#pragma unroll
         for (int m = 0; m < 16; m++) { a[m] = an[m]; lu[m] = ln[m]; }
      }
#pragma unroll
      for (int u = 0; u < DEPTH; u++) fc[u] = fcn[u];
   }
   cp_async_wait_all();
   __threadfence_block();   // f, before copies of it into the ring
}

// One sweep's solve of one chain per thread (the chain at position first +
// t of line_chains).  The recurrence only carries the 4-vector x in
// registers; what a row needs comes through the thread's ring (its factor
// record, its right-hand side through the cell looked up a ring's rows before
// that, later the forward sweep's row).  Solutions go straight to r32 (each
// cell is written once per chain; chains of a wave share no cell).
// Bound by the chain: with the loads of four rows issued together a row of the
// longest chain took 650 cycles forward or back, through the ring 280 (512 x 128,
// 30% split: the four solves of a step 207 -> 103 us; unsplit 170 -> 79 us; 32
// meshes of 983,040 cells 270 -> 129 us).  With the slots
// computed each row and not unrolled it was 390.
constexpr int kSolveDepth = 8;

__global__ void __launch_bounds__(128) mx_solve_kernel(DeviceState d, int first, int count)
{
   const int t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= count || halted(d)) return;
   const int p = first + t;
   const int ich = d.line_chains[p];
   if (frozen_chain(d, ich) || spike_active(d, ich)) return;
   const int N = d.chain_nrows[ich], row0 = d.chain_row0[ich], lane = p & 31, s0 = d.grp_row0[p >> 5];
   const bool per = d.chain_periodic[ich] != 0;
   const int* fcell = d.row_fcell + row0;
   const int* scell = d.row_scell + row0;
   extern __shared__ float4 stage[];
   const RowRing<kSolveVec, kSolveDepth> ring(stage);
   constexpr int AHEAD = kSolveDepth - 1;
   const float* fac = d.fac32 + tix(s0, kRec, 0, lane);
   float* fsr = d.fsc32 + tix(s0, 4, 0, lane);
   float x[4], xp[4];
   forward_rows(ring, N, fac, fsr, fcell, d.r32, xp);
   float xn[4], fN[4] = {xp[0], xp[1], xp[2], xp[3]};
   if (per) {
      // last row: f(N-1) - sum over i < N-1 of cN(i) f(i), in row order
      auto fetch_last = [&](int i) {
         if (i < N - 1) {
            ring.copy<4>(i % kSolveDepth, 0, fac + kFacRow * i + 32 * 64);
            cp_async16_cg(ring.at(i % kSolveDepth, 8), fsr + kFsRow * i);
         }
         cp_async_commit();
      };
#pragma unroll
      for (int i = 0; i < AHEAD; i++) fetch_last(i);
      for (int i = 0; i < N - 1; i++) {
         cp_async_wait<AHEAD - 1>();
         float c[16], f[4];
         ring.read(i % kSolveDepth, 0, c);
         ring.read(i % kSolveDepth, 8, f);
         fetch_last(i + AHEAD);
         mv_sub(c, f, fN);
      }
      cp_async_wait_all();
      const LUf uN = luf_load(d.facN32 + 16 * d.chain_facN[ich]);
      luf_solve(uN, fN[0], fN[1], fN[2], fN[3]);
   }
#pragma unroll
   for (int k = 0; k < 4; k++) xn[k] = fN[k];
   st4(d.r32 + 4 * (size_t)scell[N - 1], xn);
   // back substitution, rows N-2 down to 0 (step s = N-2-i), periodic with the
   // fill-in column
   auto back = [&](auto fill_in) {
      constexpr bool PER = decltype(fill_in)::value;
      auto fetch_back = [&](int s, int slot) {
         const int i = N - 2 - s;
         if (i >= 0) {
            ring.copy<4>(slot, 0, fac + kFacRow * i + 32 * 32);
            if (PER) ring.copy<4>(slot, 4, fac + kFacRow * i + 32 * 48);
            cp_async16_cg(ring.at(slot, 8), fsr + kFsRow * i);
         }
         cp_async_commit();
      };
      auto look = [&](int i) { return i >= 0 ? scell[i] : -1; };
#pragma unroll
      for (int s = 0; s < AHEAD; s++) fetch_back(s, s);
      int sc[kSolveDepth];
#pragma unroll
      for (int u = 0; u < kSolveDepth; u++) sc[u] = look(N - 2 - u);
      float c[16], aa[16];
      cp_async_wait<AHEAD - 1>();
      ring.read(0, 0, c);
      if (PER) ring.read(0, 4, aa);
      ring.read(0, 8, x);
      for (int q0 = 0; q0 <= N - 2; q0 += kSolveDepth) {
         int scn[kSolveDepth];
#pragma unroll
         for (int u = 0; u < kSolveDepth; u++) scn[u] = look(N - 2 - q0 - kSolveDepth - u);
#pragma unroll
         for (int u = 0; u < kSolveDepth; u++) {
            const int s = q0 + u;
            if (s > N - 2) break;
            float cn[16], an[16], y[4];
            cp_async_wait<AHEAD - 2>();
            ring.read((u + 1) % kSolveDepth, 0, cn);
            if (PER) ring.read((u + 1) % kSolveDepth, 4, an);
            ring.read((u + 1) % kSolveDepth, 8, y);
            fetch_back(s + AHEAD, (u + AHEAD) % kSolveDepth);
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
               for (int j = 0; j < 4; j++) {
                  if (PER) {
                     const float v = c[4 * k + j] * xn[j];
                     x[k] -= (s == 0) ? v : __fmaf_rn(aa[4 * k + j], fN[j], v);
                  } else {
                     x[k] = __fmaf_rn(-c[4 * k + j], xn[j], x[k]);
                  }
               }
            st4(d.r32 + 4 * (size_t)sc[u], x);
#pragma unroll
            for (int k = 0; k < 4; k++) { xn[k] = x[k]; x[k] = y[k]; }
#pragma unroll
            for (int m = 0; m < 16; m++) {
               c[m] = cn[m];
               if (PER) aa[m] = an[m];
            }
         }
#pragma unroll
         for (int u = 0; u < kSolveDepth; u++) sc[u] = scn[u];
      }
   };
   if (per) back(std::true_type{});
   else back(std::false_type{});
   cp_async_wait_all();
}

// ---------------- long chains by segments -------------------------------
// A periodic chain of N rows (A_i x_{i-1} + B_i x_i + C_i x_{i+1} = f_i,
// indices mod N) is cut into P segments of about N/P rows, one lane of a
// warp each.  An open chain is the same system with A_0 and C_{N-1} (which
// its solve never reads) set to zero: its first segment's W and its last
// segment's V spikes vanish, and the cyclic boundary system below has zero
// coupling across the wrap.  With D_p the block-tridiagonal matrix of segment p alone
// (rows s..e), its solution is
//     x_i = y_i + V_i x_{e+1} + W_i x_{s-1},
// where D_p y = f, D_p V = -C_e (in the last row) and D_p W = -A_s (in the
// first row): V and W are the "spikes", the segment's responses to the
// couplings across its two ends.  With b_p = x_e and t_p = x_s of segment
// p, the rows at the segment ends give a cyclic system in the interface
// pairs Z_p = (b_p, t_{p+1}):
//     b_p     - V_e(p) t_{p+1} - W_e(p) b_{p-1}   = y_e(p)
//     t_{p+1} - V_s(p+1) t_{p+2} - W_s(p+1) b_p   = y_s(p+1)
// i.e. L_p Z_{p-1} + D_p Z_p + U_p Z_{p+1} = R_p with 8x8 blocks
//     D_p = [I, -V_e(p); -W_s(p+1), I],  L_p = [-W_e(p), 0; 0, 0],
//     U_p = [0, 0; 0, -V_s(p+1)],
// which lane 0 eliminates onto Z_{P-1} (a cyclic block Thomas of P rows).
// Their sparsity keeps every step in 4x4 blocks: the pivot blocks are
// M_p = [I, X_p; -W_s(p+1), I] and are solved through the 4x4 Schur
// complement S_p = I + W_s(p+1) X_p; the couplings G_p = M_p^{-1} U_p and
// H_p (to Z_{P-1}) have four non-zero columns each.  This is the same
// linear system the sequential cyclic block Thomas solves (in FP32 it
// differs in rounding only), with N/P + P rows of latency instead of N.
// The segment factors and spikes, and the boundary system's factors, are
// formed once per step; each sweep replays the right-hand side.
//
// Layout: the rows of a chain's segments are tiled like the other FP32 line
// data (element e of local row k of segment p at tix(R0 + k, W, e, p), R0
// the chain's first tile row), so every load and store of the warp is one
// 128-byte line.

// sp_fac record of one row: A, LU of the segment's B', C' (no C' on a
// segment's last row), V, W
constexpr int kSpRec = 80;

// sp_red layout of one chain: for p = 0 .. P-2, at kRedRow * p: X_p, LU(S_p),
// G_p (top 4 rows, bottom 4 rows; its non-zero columns 4-7), H_p (top,
// bottom; columns 0-3), W_e(p), W_s(p+1); then at kRedLast: LU(K) (8x8),
// W_e(P-1), V_s(0)
constexpr int kRedRow = 128;
constexpr int kRedLast = kRedRow * (kSpikeMaxSeg - 1);
static_assert(kRedLast + 64 + 32 <= kSpikeRedStride, "boundary-system factors fit their stride");
enum { RX = 0, RS = 16, RGT = 32, RGB = 48, RHT = 64, RHB = 80, RWE = 96, RWS = 112 };

// out = M X (4x4)
__device__ __forceinline__ void mm_mul(const float (&M)[16], const float (&X)[16], float (&out)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) out[m] = 0.f;
   mm_sub(M, X, out);
#pragma unroll
   for (int m = 0; m < 16; m++) out[m] = -out[m];
}

__device__ __forceinline__ void ld16s(const float* p, float (&v)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) v[m] = p[m];
}

__device__ __forceinline__ void st16s(float* p, const float (&v)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) p[m] = v[m];
}

// 8x8 row-major LU with reciprocal pivots (K, once per chain and step):
// M = L U, U unit upper; L below and on the diagonal (the diagonal holding
// 1/L_kk)
__device__ __forceinline__ void m8_lu(float (&M)[64])
{
#pragma unroll   // M stays in registers
   for (int k = 0; k < 8; k++) {
      const float piv = 1.f / M[9 * k];
      M[9 * k] = piv;
#pragma unroll
      for (int j = k + 1; j < 8; j++) M[8 * k + j] *= piv;
#pragma unroll
      for (int i = k + 1; i < 8; i++) {
         const float l = M[8 * i + k];
#pragma unroll
         for (int j = k + 1; j < 8; j++) M[8 * i + j] = __fmaf_rn(-l, M[8 * k + j], M[8 * i + j]);
      }
   }
}

// x <- M^{-1} x with the LU of m8_lu
__device__ void m8_solve(const float* LU, float (&x)[8])
{
   for (int i = 0; i < 8; i++) {
      float v = x[i];
      for (int k = 0; k < i; k++) v = __fmaf_rn(-LU[8 * i + k], x[k], v);
      x[i] = v * LU[9 * i];
   }
   for (int i = 6; i >= 0; i--) {
      float v = x[i];
      for (int j = i + 1; j < 8; j++) v = __fmaf_rn(-LU[8 * i + j], x[j], v);
      x[i] = v;
   }
}

// M [u; v] = [f; h] with M = [I, X; -Ws, I] and the LU of S = I + Ws X:
// v = S^{-1}(h + Ws f), u = f - X v, for the four columns of F and Hh
// (Hh = nullptr for h = 0)
__device__ __forceinline__ void schur_cols(const float (&X)[16], const LUf& s, const float (&Ws)[16],
                                           const float (&F)[16], const float* Hh, float (&U)[16], float (&Vv)[16])
{
#pragma unroll
   for (int m = 0; m < 16; m++) Vv[m] = Hh ? Hh[m] : 0.f;
   float WF[16];
   mm_mul(Ws, F, WF);
#pragma unroll
   for (int m = 0; m < 16; m++) Vv[m] += WF[m];
   luf_cols(s, Vv);
#pragma unroll
   for (int m = 0; m < 16; m++) U[m] = F[m];
   mm_sub(X, Vv, U);
}

// One warp per chain.  Bound by the chain of its rows, then of the boundary
// system's.  FUSED: as in mx_factor_kernel; otherwise the blocks that
// mx_assemble_kernel wrote, through the lane's ring (512 x 128: 82 us
// inside, 59 us so; 32 meshes of 983,040 cells 304 and 221 us).
template <bool FUSED>
__global__ void __launch_bounds__(32) mx_spike_factor_kernel(DeviceState d)
{
   extern __shared__ float4 stage[];
   __shared__ __align__(16) float tips[kSpikeMaxSeg * 64];   // per segment: V_s, W_s, V_e, W_e
   const int sp = blockIdx.x, lane = threadIdx.x;
   const int ich = d.sp_chain[sp];
   if (halted(d) || frozen_chain(d, ich) || !spike_active(d, ich)) return;
   const int P = d.sp_nseg[sp], row0 = d.chain_row0[ich], R0 = d.sp_rec0[sp];
   const bool per = d.chain_periodic[ich] != 0;
   const int* seg = d.sp_seg + (kSpikeMaxSeg + 1) * sp;
   bool bad = false;
   if (lane < P) {
      const int s = seg[lane], n = seg[lane + 1] - s;   // n >= 2
      // forward: B'_k = B_k - A_k C'_{k-1}; C'_k = B'^{-1} C_k; the left
      // spike's forward values g_0 = B'^{-1}(-A_0), g_k = B'^{-1}(-A_k g_{k-1});
      // at the last row the right spike B'^{-1}(-C_e).  The next row's blocks
      // are assembled from references looked up a row earlier.
      float A[16], B[16], C[16], cp[16], gw[16];
      RowRef rnext{};
      const RowRing<kFactorVec, kFactorDepth> ring(stage);
      constexpr int AHEAD = kFactorDepth - 1;
      const int pos = d.sp_pos[sp];
      const float* blk = FUSED ? nullptr : d.blk32 + tix(d.grp_row0[pos >> 5] + s, 48, 0, pos & 31);
      auto fetch = [&](int k) {
         if (k < n) ring.copy<12>(k % kFactorDepth, 0, blk + 32 * 48 * (size_t)k);
         cp_async_commit();
      };
      if (FUSED) {
         rnext = mx_rowref(d, row0 + s + 1);
         mx_row_ref(d, mx_rowref(d, row0 + s), A, B, C);
      } else {
#pragma unroll
         for (int k = 0; k < AHEAD; k++) fetch(k);
      }
      for (int k = 0; k < n; k++) {
         float An[16], Bn[16], Cn[16];
         if (FUSED) {
            if (k + 1 < n) {
               mx_row_ref(d, rnext, An, Bn, Cn);
               if (k + 2 < n) rnext = mx_rowref(d, row0 + s + k + 2);
            }
         } else {
            cp_async_wait<AHEAD - 1>();
            ring.read(k % kFactorDepth, 0, A);
            ring.read(k % kFactorDepth, 4, B);
            ring.read(k % kFactorDepth, 8, C);
            fetch(k + AHEAD);
         }
         // an open chain: no coupling from its first row back to its last
         if (k == 0 && !per && lane == 0) {
#pragma unroll
            for (int m = 0; m < 16; m++) A[m] = 0.f;
         }
         float* rec = d.sp_fac + tix(R0 + k, kSpRec, 0, lane);
         st16t(rec, A);
         float w[16];
         if (k == 0) {
#pragma unroll
            for (int m = 0; m < 16; m++) w[m] = -A[m];
         } else {
            mm_sub(A, cp, B);
#pragma unroll
            for (int m = 0; m < 16; m++) w[m] = 0.f;
            mm_sub(A, gw, w);
         }
         const LUf u = luf_factor(B);
         luf_store_t(rec + 32 * 16, u);
         bad |= nonfinite(u.p0) || nonfinite(u.p1) || nonfinite(u.p2) || nonfinite(u.p3);
         luf_cols(u, w);
         st16t(rec + 32 * 64, w);
#pragma unroll
         for (int m = 0; m < 16; m++) gw[m] = w[m];
         if (k + 1 < n) {
            luf_cols(u, C);
            st16t(rec + 32 * 32, C);
#pragma unroll
            for (int m = 0; m < 16; m++) cp[m] = C[m];
            if (FUSED) {
#pragma unroll
               for (int m = 0; m < 16; m++) { A[m] = An[m]; B[m] = Bn[m]; C[m] = Cn[m]; }
            }
         } else {
            // (an open chain's last row has no coupling forward to its first)
            const bool wrap = per || lane + 1 < P;
#pragma unroll
            for (int m = 0; m < 16; m++) C[m] = wrap ? -C[m] : 0.f;
            luf_cols(u, C);
            st16t(rec + 32 * 48, C);
         }
      }
      // back substitution of both spikes: V_k = -C'_k V_{k+1},
      // W_k = g_k - C'_k W_{k+1}, C' and g through the ring (step j: row n-2-j)
      cp_async_wait_all();
      __threadfence_block();   // the rows above, before copies of them
      float* rec = d.sp_fac + tix(R0, kSpRec, 0, lane);
      constexpr int BD = FUSED ? 2 : kFactorDepth, BA = BD - 1;
      const RowRing<8, BD> back(stage);
      auto fetch_back = [&](int j) {
         const int k = n - 2 - j;
         if (k >= 0) {
            back.template copy<4>(j % BD, 0, rec + kFacRow * k + 32 * 32);
            back.template copy<4>(j % BD, 4, rec + kFacRow * k + 32 * 64);
         }
         cp_async_commit();
      };
#pragma unroll
      for (int j = 0; j < BA; j++) fetch_back(j);
      float vn[16], wn[16];
#pragma unroll
      for (int m = 0; m < 16; m++) { vn[m] = C[m]; wn[m] = gw[m]; }
      float* tip = tips + 64 * lane;
      st16s(tip + 32, vn);   // V_e
      st16s(tip + 48, wn);   // W_e
      for (int k = n - 2; k >= 0; k--) {
         const int j = n - 2 - k;
         cp_async_wait<BA - 1>();
         float c[16], g[16], v[16];
         back.read(j % BD, 0, c);
         back.read(j % BD, 4, g);
         fetch_back(j + BA);
#pragma unroll
         for (int m = 0; m < 16; m++) v[m] = 0.f;
         mm_sub(c, vn, v);
         mm_sub(c, wn, g);
         st16t(rec + kFacRow * k + 32 * 48, v);
         st16t(rec + kFacRow * k + 32 * 64, g);
#pragma unroll
         for (int m = 0; m < 16; m++) { vn[m] = v[m]; wn[m] = g[m]; }
      }
      cp_async_wait_all();
      st16s(tip, vn);        // V_s
      st16s(tip + 16, wn);   // W_s
   }
   if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(d.status, DEV_ERR_PIVOT);
   __syncwarp();
   if (lane != 0) return;
   // boundary system, p = 0 .. P-2 (q = p + 1):
   //   X_p = -V_e(p) + W_e(p) Gtop_{p-1}  (X_0 = -V_e(0)),  S_p = I + W_s(q) X_p,
   //   G_p = M_p^{-1} [0; -V_s(q)],
   //   H_0 = M_0^{-1} [-W_e(0); 0],  H_p = M_p^{-1} [W_e(p) Htop_{p-1}; 0]
   float* red = d.sp_red + (size_t)kSpikeRedStride * sp;
   float Gt[16], Ht[16], Gb[16], Hb[16];
   bool kbad = false;
   for (int p = 0; p <= P - 2; p++) {
      const int q = p + 1;
      float X[16], We[16], Ws[16], T[16];
      ld16s(tips + 64 * p + 32, X);
      ld16s(tips + 64 * p + 48, We);
      ld16s(tips + 64 * q + 16, Ws);
#pragma unroll
      for (int m = 0; m < 16; m++) X[m] = -X[m];
      if (p > 0) {
         mm_mul(We, Gt, T);
#pragma unroll
         for (int m = 0; m < 16; m++) X[m] += T[m];
      }
      float S[16];
      mm_mul(Ws, X, S);
#pragma unroll
      for (int k = 0; k < 4; k++) S[5 * k] += 1.f;
      const LUf su = luf_factor(S);
      kbad |= nonfinite(su.p0) || nonfinite(su.p1) || nonfinite(su.p2) || nonfinite(su.p3);
      float F[16], Hh[16];
      // G_p: f = 0, h = -V_s(q): v = S^{-1}(-V_s(q)), u = -X v
      ld16s(tips + 64 * q, Hh);
#pragma unroll
      for (int m = 0; m < 16; m++) { Hh[m] = -Hh[m]; F[m] = 0.f; }
      schur_cols(X, su, Ws, F, Hh, Gt, Gb);
      // H_p
      if (p == 0) {
#pragma unroll
         for (int m = 0; m < 16; m++) F[m] = -We[m];
      } else {
         mm_mul(We, Ht, F);
      }
      schur_cols(X, su, Ws, F, nullptr, Ht, Hb);
      float* rr = red + kRedRow * p;
      st16s(rr + RX, X);
      luf_store(rr + RS, su);
      st16s(rr + RGT, Gt);
      st16s(rr + RGB, Gb);
      st16s(rr + RHT, Ht);
      st16s(rr + RHB, Hb);
      st16s(rr + RWE, We);
      st16s(rr + RWS, Ws);
   }
   // Z_p = a_p + B_p Z_{P-1}; only the rows of B_{P-2} (top) and B_0
   // (bottom) enter K: B_{P-2} = -[H_{P-2} | G_{P-2}],
   // B_p = -G_p Bbot_{p+1} - [H_p | 0], carried on its bottom rows
   float Bl[16], Br[16];   // bottom rows of B_p: columns 0-3, 4-7
#pragma unroll
   for (int m = 0; m < 16; m++) { Bl[m] = -Hb[m]; Br[m] = -Gb[m]; }
   float BtopL[16], BtopR[16];   // top rows of B_{P-2}
#pragma unroll
   for (int m = 0; m < 16; m++) { BtopL[m] = -Ht[m]; BtopR[m] = -Gt[m]; }
   for (int p = P - 3; p >= 0; p--) {
      float g[16], h[16], nl[16], nr[16];
      ld16s(red + kRedRow * p + RGB, g);
      ld16s(red + kRedRow * p + RHB, h);
      mm_mul(g, Bl, nl);
      mm_mul(g, Br, nr);
#pragma unroll
      for (int m = 0; m < 16; m++) { Bl[m] = -nl[m] - h[m]; Br[m] = -nr[m]; }
   }
   // K = D_{P-1} + L_{P-1} B_{P-2} + U_{P-1} B_0:
   //   top rows    [I, -V_e(P-1)] - W_e(P-1) Btop_{P-2}
   //   bottom rows [-W_s(0), I]   - V_s(0) Bbot_0
   float K[64], We[16], Vs0[16], M4[16], t[16];
   ld16s(tips + 64 * (P - 1) + 48, We);
   ld16s(tips, Vs0);
   ld16s(tips + 64 * (P - 1) + 32, t);   // V_e(P-1)
   mm_mul(We, BtopL, M4);
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
         K[8 * k + j] = ((k == j) ? 1.f : 0.f) - M4[4 * k + j];
      }
   mm_mul(We, BtopR, M4);
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) K[8 * k + 4 + j] = -t[4 * k + j] - M4[4 * k + j];
   ld16s(tips + 16, t);   // W_s(0)
   mm_mul(Vs0, Bl, M4);
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) K[8 * (4 + k) + j] = -t[4 * k + j] - M4[4 * k + j];
   mm_mul(Vs0, Br, M4);
#pragma unroll
   for (int k = 0; k < 4; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) K[8 * (4 + k) + 4 + j] = ((k == j) ? 1.f : 0.f) - M4[4 * k + j];
   m8_lu(K);
#pragma unroll
   for (int k = 0; k < 8; k++) kbad |= nonfinite(K[9 * k]);
   float* last = red + kRedLast;
#pragma unroll
   for (int m = 0; m < 64; m++) last[m] = K[m];
   st16s(last + 64, We);
   st16s(last + 80, Vs0);
   if (kbad) atomicOr(d.status, DEV_ERR_PIVOT);
}

// one sweep's solve of the spike chains sp = first .. first+count-1 of a
// wave: right-hand sides r32[fcell], solutions into r32[scell].  Every pass over
// a segment's rows goes through the lane's ring, the last one's first rows and
// the boundary system's factors while other work runs.  The two solves of a step
// (512 x 128): 90 us with each row's loads a row ahead, 58 us so; 32 meshes of
// 983,040 cells 330 and 259 us.
constexpr int kSpikeSolveDepth = 4;   // 36 KB a block with the boundary system's factors: six to an SM

__global__ void __launch_bounds__(32) mx_spike_solve_kernel(DeviceState d, int first)
{
   // (red_s is read with float4 loads: 16-byte aligned)
   __shared__ __align__(16) float red_s[kRedLast + 96];   // the chain's boundary-system factors
   __shared__ __align__(16) float ry[kSpikeMaxSeg * 8];   // per segment: y_s then y_e
   __shared__ __align__(16) float zs[kSpikeMaxSeg * 8];   // Z_p = (b_p, t_{p+1})
   const int sp = first + blockIdx.x, lane = threadIdx.x;
   const int ich = d.sp_chain[sp];
   if (halted(d) || frozen_chain(d, ich) || !spike_active(d, ich)) return;
   const int P = d.sp_nseg[sp], row0 = d.chain_row0[ich], R0 = d.sp_rec0[sp];
   const int* seg = d.sp_seg + (kSpikeMaxSeg + 1) * sp;
   {
      // the boundary-system factors into shared memory (lane 0 reads them
      // one step after another below)
      const float* red = d.sp_red + (size_t)kSpikeRedStride * sp;
      const int nrow = kRedRow * (P - 1);
      for (int m = 4 * lane; m < nrow; m += 128) cp_async16_cg(red_s + m, red + m);
      if (lane < 24) cp_async16_cg(red_s + kRedLast + 4 * lane, red + kRedLast + 4 * lane);
      cp_async_commit();   // a group of their own: each lane waits for its copies before the __syncwarp below
   }
   extern __shared__ float4 stage[];
   const RowRing<kSolveVec, kSpikeSolveDepth> ring(stage);
   constexpr int AHEAD = kSpikeSolveDepth - 1;
   const float* fac = d.sp_fac + tix(R0, kSpRec, 0, lane);
   float* ys = d.sp_y + tix(R0, 4, 0, lane);
   auto fetch_rows = [&](int k, int n) {   // V, W and y of row k
      if (k < n) {
         ring.copy<8>(k % kSpikeSolveDepth, 0, fac + kFacRow * k + 32 * 48);
         cp_async16_cg(ring.at(k % kSpikeSolveDepth, 8), ys + kFsRow * k);
      }
      cp_async_commit();
   };
   int s = 0, n = 0;
   if (lane < P) {
      s = seg[lane];
      n = seg[lane + 1] - s;
      // forward: y'_k = B'^{-1}(f_k - A_k y'_{k-1})
      float yp[4];
      forward_rows(ring, n, fac, ys, d.row_fcell + row0 + s, d.r32, yp);
      // back: y_k = y'_k - C'_k y_{k+1} (step j: row n-2-j)
#pragma unroll
      for (int c = 0; c < 4; c++) ry[8 * lane + 4 + c] = yp[c];
      auto fetch_back = [&](int j) {
         const int k = n - 2 - j;
         if (k >= 0) {
            ring.copy<4>(j % kSpikeSolveDepth, 0, fac + kFacRow * k + 32 * 32);
            cp_async16_cg(ring.at(j % kSpikeSolveDepth, 8), ys + kFsRow * k);
         }
         cp_async_commit();
      };
#pragma unroll
      for (int j = 0; j < AHEAD; j++) fetch_back(j);
      for (int k = n - 2; k >= 0; k--) {
         const int j = n - 2 - k;
         cp_async_wait<AHEAD - 1>();
         float cm[16], yk[4];
         ring.read(j % kSpikeSolveDepth, 0, cm);
         ring.read(j % kSpikeSolveDepth, 8, yk);
         fetch_back(j + AHEAD);
         mv_sub(cm, yp, yk);
         *reinterpret_cast<float4*>(ys + kFsRow * k) = make_float4(yk[0], yk[1], yk[2], yk[3]);
#pragma unroll
         for (int c = 0; c < 4; c++) yp[c] = yk[c];
      }
      cp_async_wait_all();
      __threadfence_block();   // y, before copies of it
#pragma unroll
      for (int c = 0; c < 4; c++) ry[8 * lane + c] = yp[c];
      // on their way while lane 0 solves the boundary system
#pragma unroll
      for (int k = 0; k < AHEAD; k++) fetch_rows(k, n);
   } else {
      cp_async_wait_all();
   }
   __syncwarp();
   if (lane == 0) {
      // R_p = (y_e(p), y_s(p+1));
      //   g_p: f = y_e(p) + W_e(p) gtop_{p-1}, h = y_s(p+1):
      //        v = S_p^{-1}(h + W_s(p+1) f), u = f - X_p v;
      //   a_{P-2} = g_{P-2}, a_p = g_p - G_p abot_{p+1};
      //   Z_{P-1} = K^{-1}(R_{P-1} + [W_e(P-1) atop_{P-2}; V_s(0) abot_0]);
      //   Z_{P-2} = g_{P-2} - G_{P-2} zbot - H_{P-2} ztop,
      //   Z_p = g_p - G_p Zbot_{p+1} - H_p ztop
      float gt[4] = {0.f, 0.f, 0.f, 0.f};
      for (int p = 0; p <= P - 2; p++) {
         const float* rr = red_s + kRedRow * p;
         float f[4], v[4], M[16];
#pragma unroll
         for (int c = 0; c < 4; c++) { f[c] = ry[8 * p + 4 + c]; v[c] = ry[8 * (p + 1) + c]; }
         if (p > 0) {
            ld16s(rr + RWE, M);
            mv_add(M, gt, f);
         }
         ld16s(rr + RWS, M);
         mv_add(M, f, v);
         const LUf su = luf_load(rr + RS);
         luf_solve(su, v[0], v[1], v[2], v[3]);
         ld16s(rr + RX, M);
         mv_sub(M, v, f);
#pragma unroll
         for (int c = 0; c < 4; c++) { zs[8 * p + c] = f[c]; zs[8 * p + 4 + c] = v[c]; gt[c] = f[c]; }
      }
      // a_p: only atop_{P-2} and abot_0 enter Z_{P-1}, so the recurrence
      // carries the bottom rows
      float at[4], ab[4], an[4];
#pragma unroll
      for (int c = 0; c < 4; c++) { at[c] = zs[8 * (P - 2) + c]; ab[c] = zs[8 * (P - 2) + 4 + c]; }
      const float yeL[4] = {ry[8 * (P - 1) + 4], ry[8 * (P - 1) + 5], ry[8 * (P - 1) + 6], ry[8 * (P - 1) + 7]};
      const float ys0[4] = {ry[0], ry[1], ry[2], ry[3]};
      const float atL[4] = {at[0], at[1], at[2], at[3]};
      for (int p = P - 3; p >= 0; p--) {
         const float* rr = red_s + kRedRow * p;
         float M[16], ub[4];
#pragma unroll
         for (int c = 0; c < 4; c++) { ub[c] = zs[8 * p + 4 + c]; an[c] = ab[c]; }
         ld16s(rr + RGB, M);
         mv_sub(M, an, ub);
#pragma unroll
         for (int c = 0; c < 4; c++) ab[c] = ub[c];
      }
      // ab = abot_0
      float z[8], M[16];
      const float* last = red_s + kRedLast;
#pragma unroll
      for (int c = 0; c < 4; c++) { z[c] = yeL[c]; z[4 + c] = ys0[c]; }
      {
         float zt[4] = {z[0], z[1], z[2], z[3]}, zb[4] = {z[4], z[5], z[6], z[7]};
         ld16s(last + 64, M);
         mv_add(M, atL, zt);
         ld16s(last + 80, M);
         mv_add(M, ab, zb);
#pragma unroll
         for (int c = 0; c < 4; c++) { z[c] = zt[c]; z[4 + c] = zb[c]; }
      }
      m8_solve(last, z);
      const float ztop[4] = {z[0], z[1], z[2], z[3]};
      float zb[4] = {z[4], z[5], z[6], z[7]};   // bottom of Z_{p+1} (Z_{P-1} = z first)
#pragma unroll
      for (int c = 0; c < 8; c++) zs[8 * (P - 1) + c] = z[c];
      for (int p = P - 2; p >= 0; p--) {
         const float* rr = red_s + kRedRow * p;
         float ut[4], ub[4];
#pragma unroll
         for (int c = 0; c < 4; c++) { ut[c] = zs[8 * p + c]; ub[c] = zs[8 * p + 4 + c]; }
         ld16s(rr + RGT, M);
         mv_sub(M, zb, ut);
         ld16s(rr + RGB, M);
         mv_sub(M, zb, ub);
         ld16s(rr + RHT, M);
         mv_sub(M, ztop, ut);
         ld16s(rr + RHB, M);
         mv_sub(M, ztop, ub);
#pragma unroll
         for (int c = 0; c < 4; c++) { zs[8 * p + c] = ut[c]; zs[8 * p + 4 + c] = ub[c]; zb[c] = ub[c]; }
      }
   }
   __syncwarp();
   if (lane < P) {
      // x_k = y_k + V_k t_{p+1} + W_k b_{p-1}
      float tn[4], bp[4];
      const int pm = (lane == 0) ? P - 1 : lane - 1;
#pragma unroll
      for (int c = 0; c < 4; c++) {
         tn[c] = zs[8 * lane + 4 + c];
         bp[c] = zs[8 * pm + c];
      }
      const int* scell = d.row_scell + row0 + s;
      int sc[kSpikeSolveDepth];
#pragma unroll
      for (int u = 0; u < kSpikeSolveDepth; u++) sc[u] = u < n ? scell[u] : 0;
      for (int k0 = 0; k0 < n; k0 += kSpikeSolveDepth) {
         int scn[kSpikeSolveDepth];
#pragma unroll
         for (int u = 0; u < kSpikeSolveDepth; u++) scn[u] = k0 + kSpikeSolveDepth + u < n ? scell[k0 + kSpikeSolveDepth + u] : 0;
#pragma unroll
         for (int u = 0; u < kSpikeSolveDepth; u++) {
            const int k = k0 + u;
            if (k >= n) break;
            cp_async_wait<AHEAD - 1>();
            float v[16], w[16], x[4];
            ring.read(u, 0, v);
            ring.read(u, 4, w);
            ring.read(u, 8, x);
            fetch_rows(k + AHEAD, n);
            mv_add(w, bp, x);
            mv_add(v, tn, x);
            st4(d.r32 + 4 * (size_t)sc[u], x);
         }
#pragma unroll
         for (int u = 0; u < kSpikeSolveDepth; u++) sc[u] = scn[u];
      }
      cp_async_wait_all();
   }
}

__global__ void __launch_bounds__(kThreads) mx_dq_update_kernel(DeviceState d)
{
   const int c = blockIdx.x * blockDim.x + threadIdx.x;
   if (c >= d.nCell || halted(d) || frozen_cell(d, c)) return;
   float r[4], dq[4];
   ld4(d.r32 + 4 * (size_t)c, r);
   ld4(d.dq32 + 4 * (size_t)c, dq);
#pragma unroll
   for (int k = 0; k < 4; k++) dq[k] += r[k];
   st4(d.dq32 + 4 * (size_t)c, dq);
   if (nonfinite(dq[0]) || nonfinite(dq[1]) || nonfinite(dq[2]) || nonfinite(dq[3])) atomicOr(d.status, DEV_ERR_DQ);
}

template <int ORDER>
__global__ void __launch_bounds__(kThreads) mx_lin_face_kernel(DeviceState d)
{
   // the block's face Jacobians staged through shared memory: read with
   // whole-line loads (8 float4 per slot, consecutive slots), then each
   // thread takes its own (row stride 9 float4: no bank conflicts)
   __shared__ float4 sj[kThreads * 9];
   const int nb = blockDim.x, s0 = blockIdx.x * nb, s = s0 + threadIdx.x;
   const int nloc = min(nb, d.nSlot - s0);
   const float4* __restrict__ src = reinterpret_cast<const float4*>(d.ff32 + 32 * (size_t)s0);
   for (int c = threadIdx.x; c < 8 * nloc; c += nb) sj[(c >> 3) * 9 + (c & 7)] = src[c];
   __syncthreads();
   if (s >= d.nSlot || halted(d) || frozen_slot(d, s)) return;
   const int4 sl = d.slot[s];
   float dL[4], dR[4];
   face_dstates<ORDER, float>(d, d.dq32, sl.x, (sl.w & 1) != 0, dL, dR);
   // the Jacobian kept for this face is its owner slot's (a periodic
   // chain's repeated face); almost always the slot itself
   const int own = sl.w >> 1;
   float m[32];
#pragma unroll
   for (int q = 0; q < 8; q++) {
      const float4 v = (own == s) ? sj[threadIdx.x * 9 + q]
                                  : reinterpret_cast<const float4*>(d.ff32 + 32 * (size_t)own)[q];
      m[4 * q] = v.x;
      m[4 * q + 1] = v.y;
      m[4 * q + 2] = v.z;
      m[4 * q + 3] = v.w;
   }
   float g[4];
#pragma unroll
   for (int j = 0; j < 4; j++) {
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; k++) acc += ((m[4 * j + k] * dL[k]) + (m[16 + 4 * j + k] * dR[k]));
      g[j] = acc;
   }
   st4(d.g32 + 4 * (size_t)s, g);
}

template <bool UPDATE_Q>
__global__ void __launch_bounds__(kThreads) mx_lin_cell_kernel(DeviceState d)
{
   if (halted(d)) return;
   const int c = norm_cell(d);
   double sq = 0.0, am = 0.0;
   if (c >= 0) {
      float r[4], r0[4], dq[4];
      ld4(d.r032 + 4 * (size_t)c, r0);
      ld4(d.dq32 + 4 * (size_t)c, dq);
#pragma unroll
      for (int k = 0; k < 4; k++) r[k] = r0[k] - dq[k];
      const float dt = float(d.dtfac[c]);
      const int e1 = d.cell_ptr[c + 1];
      for (int e = d.cell_ptr[c]; e < e1; e += kGather) {
         int ent[kGather];
         float g[kGather][4];
         cell_entries(d, e, e1, ent);
#pragma unroll
         for (int u = 0; u < kGather; u++) {
            if (e + u >= e1) break;
            ld4(d.g32 + 4 * (size_t)(ent[u] >> 1), g[u]);
         }
#pragma unroll
         for (int u = 0; u < kGather; u++) {
            if (e + u >= e1) break;
            if (ent[u] & 1) {
#pragma unroll
               for (int k = 0; k < 4; k++) r[k] += g[u][k] * dt;
            } else {
#pragma unroll
               for (int k = 0; k < 4; k++) r[k] -= g[u][k] * dt;
            }
         }
      }
      st4(d.r32 + 4 * (size_t)c, r);
      sq = double(r[0]) * double(r[0]);
      am = fabs(double(r[0]));
      if (UPDATE_Q) {
         double q[4];
         ld4(d.q + 4 * (size_t)c, q);
#pragma unroll
         for (int k = 0; k < 4; k++) q[k] += double(dq[k]);
         st4(d.q + 4 * (size_t)c, q);
      }
   }
   block_norm(d, sq, am);
}

inline int blocks_for(int n) { return (n + kThreads - 1) / kThreads; }

}  // namespace

namespace {
template <bool SD>
void mx_rhs_face_go(const DeviceState& d, int b, int t, cudaStream_t st)
{
   switch (d.recon) {
      case 1: mx_rhs_face_kernel<1, SD><<<b, t, kFaceSmem * t, st>>>(d); break;
      case 3: mx_rhs_face_kernel<3, SD><<<b, t, kFaceSmem * t, st>>>(d); break;
      case 5:
         if (d.qface) mx_rhs_face_kernel<5, SD, true><<<b, t, kFaceSmem * t, st>>>(d);
         else mx_rhs_face_kernel<5, SD><<<b, t, kFaceSmem * t, st>>>(d);
         break;
      case 31: mx_rhs_face_kernel<31, SD><<<b, t, kFaceSmem * t, st>>>(d); break;
      default: mx_rhs_face_kernel<32, SD><<<b, t, kFaceSmem * t, st>>>(d); break;
   }
}
}  // namespace

void launch_mx_rhs_face(const DeviceState& d, cudaStream_t st)
{
   const int t = face_threads(d);
   const int b = (d.nSlot + t - 1) / t;
   if (d.face_soft) mx_rhs_face_go<true>(d, b, t, st);
   else mx_rhs_face_go<false>(d, b, t, st);
}

void launch_mx_assemble(const DeviceState& d, cudaStream_t st)
{
   const size_t n = 128 * (size_t)d.tile_rows;
   if (!d.mx_fused && n > 0) mx_assemble_kernel<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st>>>(d);
}

void launch_mx_init(const DeviceState& d, cudaStream_t st) { mx_init_kernel<<<blocks_for(d.nCell), kThreads, 0, st>>>(d); }

// dynamic shared memory of the factorisation (staged terms or ring) and of the solve (ring)
size_t mx_factor_stage_bytes(int block) { return (size_t)std::max(kStageTerms * 4, kFactorDepth * kFactorVec) * sizeof(float4) * block; }
size_t mx_solve_ring_bytes(int block) { return (size_t)kSolveDepth * kSolveVec * sizeof(float4) * block; }
constexpr size_t kSpikeRingBytes = (size_t)kSpikeSolveDepth * kSolveVec * sizeof(float4) * 32;

int mx_configure()
{
   const int want = (int)mx_factor_stage_bytes(128), ring = (int)mx_solve_ring_bytes(128);
   const void* factor[] = {(const void*)mx_factor_kernel<true, kElimChunk>, (const void*)mx_factor_kernel<true, 1>,
                           (const void*)mx_factor_kernel<false, kElimChunk>, (const void*)mx_factor_kernel<false, 1>};
   for (const void* f : factor)
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, want) != cudaSuccess) return 1;
   if (cudaFuncSetAttribute(mx_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ring) != cudaSuccess) return 1;
   // these run beside each other: an SM takes blocks of two kernels at a time
   // only where both ask for the same split of its L1 (eight steps of 512 x 128
   // with the assembly inside 6.6 -> 5.1 ms)
   const void* beside[] = {factor[0], factor[1], factor[2], factor[3], (const void*)mx_solve_kernel,
                           (const void*)mx_spike_factor_kernel<true>, (const void*)mx_spike_factor_kernel<false>,
                           (const void*)mx_spike_solve_kernel};
   for (const void* f : beside)
      if (cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
          cudaSuccess)
         return 1;
   return 0;
}

void launch_mx_factor(const DeviceState& d, cudaStream_t st)
{
   const int tb = d.mx_block;
   const unsigned nb = (d.nChain + tb - 1) / tb;
   const bool chunk = d.nChain <= d.mx_chunk_chains;
   const size_t sm = mx_factor_stage_bytes(tb);
   if (d.mx_fused) {
      if (chunk) mx_factor_kernel<true, kElimChunk><<<nb, tb, sm, st>>>(d, d.nChain);
      else mx_factor_kernel<true, 1><<<nb, tb, sm, st>>>(d, d.nChain);
   } else {
      if (chunk) mx_factor_kernel<false, kElimChunk><<<nb, tb, sm, st>>>(d, d.nChain);
      else mx_factor_kernel<false, 1><<<nb, tb, sm, st>>>(d, d.nChain);
   }
}

void launch_mx_solve(const DeviceState& d, int first, int count, cudaStream_t st)
{
   const int tb = d.mx_block;
   if (count <= 0) return;
   mx_solve_kernel<<<(count + tb - 1) / tb, tb, mx_solve_ring_bytes(tb), st>>>(d, first, count);
}

int mx_factor_chunk_capacity(int block, bool fused)
{
   int dev = 0, sms = 0, per_sm = 0;
   if (mx_configure() || cudaGetDevice(&dev) != cudaSuccess) return 0;   // (the query refuses shared memory not allowed yet)
   if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
   const cudaError_t e = fused ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mx_factor_kernel<true, kElimChunk>,
                                                                               block, mx_factor_stage_bytes(block))
                               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mx_factor_kernel<false, kElimChunk>,
                                                                               block, mx_factor_stage_bytes(block));
   return e == cudaSuccess ? sms * per_sm * block : 0;
}

void launch_mx_spike_factor(const DeviceState& d, cudaStream_t st)
{
   if (!d.sp_on || d.nSpike <= 0) return;
   if (d.mx_fused) mx_spike_factor_kernel<true><<<d.nSpike, 32, 2 * 8 * 32 * sizeof(float4), st>>>(d);
   else mx_spike_factor_kernel<false><<<d.nSpike, 32, mx_factor_stage_bytes(32), st>>>(d);
}

void launch_mx_spike_solve(const DeviceState& d, int first, int count, cudaStream_t st)
{
   if (d.sp_on && count > 0) mx_spike_solve_kernel<<<count, 32, kSpikeRingBytes, st>>>(d, first);
}

void launch_mx_dq_update(const DeviceState& d, cudaStream_t st)
{
   mx_dq_update_kernel<<<blocks_for(d.nCell), kThreads, 0, st>>>(d);
}

void launch_mx_lin_face(const DeviceState& d, cudaStream_t st)
{
   const int kThreads = d.face_block;
   const int b = (d.nSlot + kThreads - 1) / kThreads;
   if (d.lin_order == 1) {
      mx_lin_face_kernel<1><<<b, kThreads, 0, st>>>(d);
      return;
   }
   switch (d.recon) {
      case 1: mx_lin_face_kernel<1><<<b, kThreads, 0, st>>>(d); break;
      case 3: mx_lin_face_kernel<3><<<b, kThreads, 0, st>>>(d); break;
      case 5: mx_lin_face_kernel<5><<<b, kThreads, 0, st>>>(d); break;
      case 31: mx_lin_face_kernel<31><<<b, kThreads, 0, st>>>(d); break;
      default: mx_lin_face_kernel<32><<<b, kThreads, 0, st>>>(d); break;
   }
}

void launch_mx_lin_cell(const DeviceState& d, bool update_q, cudaStream_t st)
{
   if (update_q) mx_lin_cell_kernel<true><<<d.norm_blocks, kThreads, 0, st>>>(d);
   else mx_lin_cell_kernel<false><<<d.norm_blocks, kThreads, 0, st>>>(d);
}

}  // namespace hamstr
