// ##################################################################
//
// pointwise.cu -- function-level entry points of the reference's numerics
//
// The solver handle fuses the reference's per-face and per-chain functions
// into whole-mesh kernels.  A caller that uses those functions directly --
// SOLVER::fluxRoe2D / jacobianRoe2D (interfaceFlux.cpp:24-169,
// jacobianRoe.cpp:9-70) and RECONSTRUCTION::MUSCL / WENO / MUSCL_DERIV /
// WENO_DERIV (reconstruction.cpp:16-386) -- gets them here, batched over
// faces or over lines, on device arrays, one thread per face or per value
// of a line (WENO: per value and side).  Every expression keeps the
// reference's operands and association (the unit is compiled with
// -fmad=false), so each output equals one reference call's bit for bit.
// (WENO entries above 2^1021 in magnitude are outside of that: there a doubled
// entry alone overflows in the reference, and here only its sum with others.)
//
// These are bound by FP64 issue (15.8 G warp instructions/s), and a hardware
// division takes 7 of its slots: the divisions, the small constants and, in
// WENO, the multiplies run on the integer pipes as in the solver's kernels
// (softdiv.cuh, recon.cuh, identical results).  Blocks are small so that the
// last ones fill the SMs.  Measured, before -> now: flux and Jacobian of 164,399
// faces 369 -> 184 us; WENO and its linearisation on 128 lines of 518 x 4 values
// 287 -> 150 us.
//
// Line arrays are [nlines][imax][nq] doubles: entry i, component n of
// line l at (l*imax + i)*nq + n, the reference's f[i][n] per chain.  Threads
// follow that order, so a warp's accesses are contiguous.
// ##################################################################
#include <cuda_runtime.h>

#include <string>

#include "../../include/hamstr_gpu.h"
#include "recon.cuh"
#include "roe.cuh"

namespace hamstr {
void set_last_error(const std::string& m);
}

namespace {

using namespace hamstr;

constexpr int kThreads = 64;

int launched(const char* what)
{
   const cudaError_t e = cudaGetLastError();
   if (e == cudaSuccess) return HAMSTR_GPU_OK;
   set_last_error(std::string(what) + " launch: " + cudaGetErrorString(e));
   return HAMSTR_GPU_ERR_CUDA;
}

unsigned blocks(size_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// ---------------- Roe flux and Jacobian, one thread per face -------------
// (Blocks to an SM: with no bound given the compiler stays at 128 registers and
// keeps two values of the Jacobian in local memory, 189 us for 164,399 faces' flux
// and Jacobian; six blocks leave it 146 and none, 180 us.)
template <bool JAC>
__global__ void __launch_bounds__(kThreads, JAC ? 6 : 9) roe_faces_kernel(int n, const double* __restrict__ nxy,
                                                             const double* __restrict__ ql,
                                                             const double* __restrict__ qr, double gamma,
                                                             double* __restrict__ flux, double* __restrict__ spec,
                                                             double* __restrict__ lmat, double* __restrict__ rmat)
{
   const int f = blockIdx.x * blockDim.x + threadIdx.x;
   if (f >= n) return;
   double L[4], R[4];
#pragma unroll
   for (int k = 0; k < 4; k++) {
      L[k] = ql[4 * (size_t)f + k];
      R[k] = qr[4 * (size_t)f + k];
   }
   RoeOut o;
   double lm[16], rm[16];
   roe_face<JAC, true>(nxy[2 * (size_t)f], nxy[2 * (size_t)f + 1], L, R, gamma, o, lm, rm);
   if (JAC) {
#pragma unroll
      for (int e = 0; e < 16; e++) {
         lmat[16 * (size_t)f + e] = lm[e];
         rmat[16 * (size_t)f + e] = rm[e];
      }
   } else {
#pragma unroll
      for (int k = 0; k < 4; k++) flux[4 * (size_t)f + k] = o.flux[k];
      spec[f] = o.spec;
   }
}

// ---------------- reconstructions along lines ----------------------------
struct Lines {
   int nlines, imax, nq;
};

// thread t -> value t of entries [i0, i0 + ni) of all lines, in memory order:
// its index in the line arrays and its entry (32-bit division where the count
// allows it)
__device__ __forceinline__ bool line_index(const Lines& g, int i0, int ni, size_t& at, int& i)
{
   const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
   const size_t per_line = (size_t)g.nq * ni, all = per_line * g.nlines;
   if (t >= all) return false;
   size_t l, r;
   if (all <= 0xFFFFFFFFull) {
      l = (unsigned)t / (unsigned)per_line;
      r = (unsigned)t - (unsigned)l * (unsigned)per_line;
   } else {
      l = t / per_line;
      r = t - l * per_line;
   }
   at = (l * g.imax + i0) * g.nq + r;
   i = i0 + (int)(per_line <= 0xFFFFFFFFull ? (unsigned)r / (unsigned)g.nq : r / g.nq);
   return true;
}

// MUSCL (reconstruction.cpp:16-70): first order copies f; otherwise the
// kappa scheme with the reference's limiter, which also leaves the differences
// f2[i] = f[i+1] - f[i], i < imax-1, in the caller's f2 (reconstruction.cpp:54-55).
// Every entry of the line has a thread; entries is .. ie get ql and qr.
__global__ void __launch_bounds__(kThreads) muscl_kernel(Lines g, const double* __restrict__ f,
                                                         double* __restrict__ ql, double* __restrict__ qr,
                                                         double* __restrict__ f2, int is, int ie, double th, double qt,
                                                         double eps)
{
   size_t at;
   int i;
   if (!line_index(g, 0, g.imax, at, i)) return;
   const double fi = f[at];
   const bool in = i >= is && i <= ie;
   if (qt == 0.0) {
      if (in) {
         ql[at] = fi;
         qr[at] = fi;
      }
      return;
   }
   if (i + 1 >= g.imax) return;
   const double f2i = f[at + g.nq] - fi;
   f2[at] = f2i;
   if (!in) return;
   const double thm = 1.0 - th;
   const double thp = 1.0 + th;
   const double f2i1 = fi - f[at - g.nq];
   const double a1 = pc<3, true>(f2i * f2i1 + eps);
   const double a2 = 2.0 * (f2i - f2i1) * (f2i - f2i1) + a1;
   const double f3i = Dv<double, true>(a2).div(a1);
   const double f3qt = qt * f3i;
   ql[at] = fi + f3qt * (thm * f2i1 + thp * f2i);
   qr[at] = fi - f3qt * (thp * f2i1 + thm * f2i);
}

// MUSCL_DERIV (reconstruction.cpp:168-236): the linearisation of MUSCL
// about f applied to dq
__global__ void __launch_bounds__(kThreads) muscl_deriv_kernel(Lines g, const double* __restrict__ f,
                                                               const double* __restrict__ dq, double* __restrict__ ql,
                                                               double* __restrict__ qr, double* __restrict__ f2, int is,
                                                               int ie, double th, double qt, double eps)
{
   size_t at;
   int i;
   if (!line_index(g, 0, g.imax, at, i)) return;
   const bool in = i >= is && i <= ie;
   if (qt == 0.0) {
      if (in) {
         ql[at] = dq[at];
         qr[at] = dq[at];
      }
      return;
   }
   if (i + 1 >= g.imax) return;
   const double fi = f[at];
   const double f2i = f[at + g.nq] - fi;
   f2[at] = f2i;
   if (!in) return;
   const double dqi = dq[at];
   const double thm = 1.0 - th;
   const double thp = 1.0 + th;
   const double f2i1 = fi - f[at - g.nq];
   const double df2i = dq[at + g.nq] - dqi;
   const double df2i1 = dqi - dq[at - g.nq];
   const double a1 = pc<3, true>(f2i * f2i1 + eps);
   const double da1 = pc<3, true>(df2i * f2i1 + f2i * df2i1);
   const double a2 = 2.0 * (f2i - f2i1) * (f2i - f2i1) + a1;
   const double da2 = 2.0 * 2.0 * (f2i - f2i1) * (df2i - df2i1) + da1;
   const Dv<double, true> r2(a2);
   const double f3i = r2.div(a1);
   const double df3i = r2.div(da1) - Dv<double, true>(a2 * a2).div(a1 * da2);
   const double f3qt = qt * f3i;
   const double df3qt = qt * df3i;
   ql[at] = dqi + df3qt * (thm * f2i1 + thp * f2i) + f3qt * (thm * df2i1 + thp * df2i);
   qr[at] = dqi - df3qt * (thp * f2i1 + thm * f2i) - f3qt * (thp * df2i1 + thm * df2i);
}

// WENO (reconstruction.cpp:133-160) and, with DERIV, WENO_DERIV
// (reconstruction.cpp:353-386): entries is .. imax-3; blockIdx.y 0 the left
// values, 1 the right ones (the same formulas on the entries reversed)
template <bool DERIV>
__global__ void __launch_bounds__(kThreads) weno_kernel(Lines g, const double* __restrict__ f,
                                                        const double* __restrict__ dq, double* __restrict__ ql,
                                                        double* __restrict__ qr, int is, double eps)
{
   size_t at;
   int i;
   if (!line_index(g, is, g.imax - 2 - is, at, i)) return;
   const ptrdiff_t step = blockIdx.y ? -(ptrdiff_t)g.nq : (ptrdiff_t)g.nq;
   double* out = blockIdx.y ? qr : ql;
   double v[5], dv[5];
#pragma unroll
   for (int k = 0; k < 5; k++) {
      v[k] = f[at + (k - 2) * step];
      if (DERIV) dv[k] = dq[at + (k - 2) * step];
   }
   out[at] = DERIV ? weno5_lin_apply<double, true>(weno5_lin_pre<double, true>(v[0], v[1], v[2], v[3], v[4], eps), dv[0],
                                                   dv[1], dv[2], dv[3], dv[4])
                   : weno5<true>(v[0], v[1], v[2], v[3], v[4]);
}

// shared argument checks of the line entry points: the reference reads
// f2[i-1], f2[i] (MUSCL: entries i-1 .. i+1) for i in [is, ie] and, WENO,
// f[i-2 .. i+2] for i in [is, imax-3]
int check_lines(const char* what, int nlines, int imax, int nq, int is, int ie, int lo, int hi_off)
{
   if (nlines < 0 || imax < 1 || nq < 1 || is < lo || ie < is - 1 || ie > imax - 1 - hi_off) {
      set_last_error(std::string(what) + ": need nlines >= 0, imax >= 1, nq >= 1 and " + std::to_string(lo) +
                     " <= is <= ie + 1, ie <= imax - " + std::to_string(1 + hi_off) + " (is = " +
                     std::to_string(is) + ", ie = " + std::to_string(ie) + ", imax = " + std::to_string(imax) + ")");
      return HAMSTR_GPU_ERR_ARG;
   }
   return HAMSTR_GPU_OK;
}

}  // namespace

extern "C" {

int hamstr_gpu_flux_roe2d(int n, const double* nxy, const double* ql, const double* qr, double* flux, double* spec,
                          double gamma, void* stream)
{
   if (n < 0 || (n > 0 && (!nxy || !ql || !qr || !flux || !spec))) {
      set_last_error("flux_roe2d: n >= 0 and non-null arrays");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (n == 0) return HAMSTR_GPU_OK;
   roe_faces_kernel<false><<<blocks(n), kThreads, 0, (cudaStream_t)stream>>>(n, nxy, ql, qr, gamma, flux, spec,
                                                                             nullptr, nullptr);
   return launched("flux_roe2d");
}

int hamstr_gpu_jacobian_roe2d(int n, const double* nxy, const double* ql, const double* qr, double* lmat,
                              double* rmat, double gamma, void* stream)
{
   if (n < 0 || (n > 0 && (!nxy || !ql || !qr || !lmat || !rmat))) {
      set_last_error("jacobian_roe2d: n >= 0 and non-null arrays");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (n == 0) return HAMSTR_GPU_OK;
   roe_faces_kernel<true><<<blocks(n), kThreads, 0, (cudaStream_t)stream>>>(n, nxy, ql, qr, gamma, nullptr,
                                                                            nullptr, lmat, rmat);
   return launched("jacobian_roe2d");
}

int hamstr_gpu_muscl(int nlines, int imax, int nq, const double* f, double* ql, double* qr, double* f2, int is,
                     int ie, double th, double qt, double eps, void* stream)
{
   const bool third = qt != 0.0;
   int st = check_lines("muscl", nlines, imax, nq, is, ie, third ? 1 : 0, third ? 1 : 0);
   if (st) return st;
   if (nlines > 0 && (!f || !ql || !qr || (third && !f2))) {
      set_last_error("muscl: null array");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (nlines == 0) return HAMSTR_GPU_OK;
   const Lines g{nlines, imax, nq};
   const cudaStream_t s = (cudaStream_t)stream;
   muscl_kernel<<<blocks((size_t)nlines * nq * imax), kThreads, 0, s>>>(g, f, ql, qr, f2, is, ie, th, qt, eps);
   return launched("muscl");
}

int hamstr_gpu_muscl_deriv(int nlines, int imax, int nq, const double* f, const double* dq, double* ql, double* qr,
                           double* f2, int is, int ie, double th, double qt, double eps, void* stream)
{
   const bool third = qt != 0.0;
   int st = check_lines("muscl_deriv", nlines, imax, nq, is, ie, third ? 1 : 0, third ? 1 : 0);
   if (st) return st;
   if (nlines > 0 && (!dq || !ql || !qr || (third && (!f || !f2)))) {
      set_last_error("muscl_deriv: null array");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (nlines == 0) return HAMSTR_GPU_OK;
   const Lines g{nlines, imax, nq};
   const cudaStream_t s = (cudaStream_t)stream;
   muscl_deriv_kernel<<<blocks((size_t)nlines * nq * imax), kThreads, 0, s>>>(g, f, dq, ql, qr, f2, is, ie, th, qt,
                                                                              eps);
   return launched("muscl_deriv");
}

int hamstr_gpu_weno(int nlines, int imax, int nq, const double* f, double* ql, double* qr, int is, int ie,
                    double epsw, void* stream)
{
   (void)epsw;   // the reference overwrites its epsw argument with 1e-15 (reconstruction.cpp:145)
   int st = check_lines("weno", nlines, imax, nq, is, ie, 2, 0);
   if (st) return st;
   if (nlines > 0 && (!f || !ql || !qr)) {
      set_last_error("weno: null array");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (nlines == 0 || imax - 2 <= is) return HAMSTR_GPU_OK;
   const Lines g{nlines, imax, nq};
   const dim3 nb(blocks((size_t)nlines * nq * (imax - 2 - is)), 2);
   weno_kernel<false><<<nb, kThreads, 0, (cudaStream_t)stream>>>(g, f, nullptr, ql, qr, is, 1e-15);
   return launched("weno");
}

int hamstr_gpu_weno_deriv(int nlines, int imax, int nq, const double* f, const double* dq, double* ql, double* qr,
                          int is, int ie, double eps, void* stream)
{
   int st = check_lines("weno_deriv", nlines, imax, nq, is, ie, 2, 0);
   if (st) return st;
   if (nlines > 0 && (!f || !dq || !ql || !qr)) {
      set_last_error("weno_deriv: null array");
      return HAMSTR_GPU_ERR_ARG;
   }
   if (nlines == 0 || imax - 2 <= is) return HAMSTR_GPU_OK;
   const Lines g{nlines, imax, nq};
   const dim3 nb(blocks((size_t)nlines * nq * (imax - 2 - is)), 2);
   weno_kernel<true><<<nb, kThreads, 0, (cudaStream_t)stream>>>(g, f, dq, ql, qr, is, eps);
   return launched("weno_deriv");
}

}  // extern "C"
