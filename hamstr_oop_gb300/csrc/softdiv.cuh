// ##################################################################
//
// softdiv.cuh -- correctly rounded FP64 division on the integer pipes
//
// GB300 issues one FP64 warp instruction per ~70-80 cycles per SM
// sub-partition, and an IEEE division takes several of them; the
// integer units sit idle in the FP64-bound kernels.  These functions
// divide binary64 numbers with integer arithmetic only (plus one FP32
// division for a seed), giving the round-to-nearest-even quotient, i.e.
// exactly what the `/` operator gives, for normal operands.  Anything
// else (zero, subnormal, infinite or NaN divisor; infinite or NaN
// dividend; subnormal quotient) falls back to `/`.
//
// Method: the divisor's 53-bit significand mb (value m = mb/2^52 in [1,2))
// gets r ~ 2^64/m in one 64-bit word, a few units below the true value: an
// FP32 reciprocal estimate y of m's leading 24 bits, kept below 1/m, the
// exact integer residual e = 1 - m y (it fits one word) and the first
// terms of 1/m = y (1 + e + e^2 + ...), the Newton-Raphson series of the
// reciprocal.  A quotient is then the high word of ma * r, with 10 or 11 bits
// beyond the 53 kept.  The rounding follows from those bits except where they
// lie within the error of r of the midpoint (about 1 in 150 quotients); there
// the sign of the exact remainder at the midpoint decides, one 64-bit
// product.  A quotient of two 53-bit numbers is never a midpoint itself
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990).
//
// What it replaced: a division by the exact word floor((2^128-1)/d) - 2^64 and
// an exact quotient and remainder (Moller & Granlund, IEEE Trans. Computers
// 60(2), 2011), about twice the integer instructions.  Measured on 512 x 128
// half split, WENO, per launch: lin_recon5 189 -> 169 us, recon5 205 -> 183,
// rhs_face 224 -> 196.  A dependent reciprocal takes 177 cycles (the hardware
// sequence 354), so the line factorisations use it on every mesh: 128-row
// loops 420 -> 377 us.
// ##################################################################
#ifndef HAMSTR_GPU_SOFTDIV_CUH
#define HAMSTR_GPU_SOFTDIV_CUH

#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace hamstr {
namespace sd {

__host__ __device__ __forceinline__ uint64_t mulhi(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
   return __umul64hi(a, b);
#else
   return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

__host__ __device__ __forceinline__ uint64_t bits(double x)
{
#ifdef __CUDA_ARCH__
   return (uint64_t)__double_as_longlong(x);
#else
   uint64_t u;
   std::memcpy(&u, &x, 8);
   return u;
#endif
}

__host__ __device__ __forceinline__ double from_bits(uint64_t u)
{
#ifdef __CUDA_ARCH__
   return __longlong_as_double((long long)u);
#else
   double x;
   std::memcpy(&x, &u, 8);
   return x;
#endif
}

// The exact reciprocal word, kept as the check of 64-bit arithmetic that the
// tests run on the host: v = floor((2^128 - 1) / d) - 2^64 for 2^63 <= d < 2^64 (Algorithm 2 of
// Moller & Granlund; v0 = floor((2^19 - 3*2^8) / d9) from a correctly
// rounded FP32 division: the true quotient is never within 1/d9 > 2^-13
// below an integer, so the floor of the rounded quotient is exact)
__host__ __device__ __forceinline__ uint64_t reciprocal_word(uint64_t d)
{
   const uint64_t d0 = d & 1;
   const uint64_t d9 = d >> 55;
   const uint64_t d40 = (d >> 24) + 1;
   const uint64_t d63 = (d >> 1) + d0;
#ifdef __CUDA_ARCH__
   const uint64_t v0 = (uint64_t)__float2uint_rz(__fdiv_rn(523520.0f, (float)(uint32_t)d9));
#else
   const uint64_t v0 = (uint64_t)(523520u / (uint32_t)d9);
#endif
   const uint64_t v1 = (v0 << 11) - ((v0 * v0 * d40) >> 40) - 1;
   const uint64_t v2 = (v1 << 13) + ((v1 * ((1ull << 60) - v1 * d40)) >> 47);
   const uint64_t e = ((v2 >> 1) & (0 - d0)) - v2 * d63;
   const uint64_t v3 = (mulhi(v2, e) >> 1) + (v2 << 31);
   // v4 = v3 - floor((v3 + 2^64 + 1) d / 2^64)
   const uint64_t lo = v3 * d, hi = mulhi(v3, d);
   const uint64_t lo2 = lo + d;
   const uint64_t hi2 = hi + d + (lo2 < lo ? 1 : 0);
   return v3 - hi2;
}

// an FP32 estimate of 1/m, m = mb / 2^52 in [1, 2): of the reciprocal of m
// rounded to 24 bits, within 1.5 * 2^-23 of 1/m relative
__host__ __device__ __forceinline__ float recip_seed(uint64_t mb)
{
   const uint32_t u = 0x3F800000u + (uint32_t)((mb - 0x10000000000000ull + (1u << 28)) >> 29);
   float y;
#ifdef __CUDA_ARCH__
   asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(u)));
#else
   float f;
   std::memcpy(&f, &u, 4);
   y = 1.0f / f;
#endif
   return y;
}

// 2^64 / m as a 64-bit word from such an estimate: less than 8 below the true
// value and never above it.  The estimate is lowered by 3 * 2^-24 so that
// Y = y 2^32 stays below 2^32/m: then e = 1 - m y is in [0, 2^-20.8) and
// E = e 2^84 is exact in one word, (e + e^2) 2^64 is formed with both terms
// floored, and e^3 and what follows (less than 3 units) is left out.
__host__ __device__ __forceinline__ uint64_t recip64(uint64_t mb, float y)
{
#ifdef __CUDA_ARCH__
   uint32_t u = __float_as_uint(y);
#else
   uint32_t u;
   std::memcpy(&u, &y, 4);
#endif
   u = u < 0x3F000000u ? 0x3F000000u : u > 0x3F7FFFFFu ? 0x3F7FFFFFu : u;   // [1/2, 1)
   const uint32_t Y = ((u << 8) | 0x80000000u) - 0x300u;
   const uint64_t E = 0 - mb * (uint64_t)Y;
   const uint32_t Eh = (uint32_t)(E >> 32);
   const uint64_t S = (E >> 20) + (((uint64_t)Eh * Eh) >> 40);
   return ((uint64_t)Y << 32) + (uint64_t)(uint32_t)(S >> 32) * Y + (((uint64_t)(uint32_t)S * Y) >> 32);
}

// a divisor prepared once for several divisions
struct Divisor {
   double b;
   uint64_t mb, r;   // significand, recip64 of it
   int eb;           // biased exponent
   uint64_t sign;
   bool ok;          // normal and finite: the integer path applies
};

__host__ __device__ __forceinline__ Divisor divisor(double b)
{
   Divisor D;
   const uint64_t B = bits(b);
   D.b = b;
   D.eb = (int)((B >> 52) & 0x7FF);
   D.sign = B & 0x8000000000000000ull;
   D.ok = D.eb != 0 && D.eb != 0x7FF;
   D.mb = (B & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
   D.r = recip64(D.mb, recip_seed(D.mb));
   return D;
}

// the operands the integer path leaves to the `/` operator; kept out of
// line so that the many inlined divisions of a kernel share one copy of the
// hardware division sequence
#ifdef __CUDA_ARCH__
__device__ __noinline__ double div_other(double a, double b) { return a / b; }
#else
inline double div_other(double a, double b) { return a / b; }
#endif

// (2^K a) / D.b rounded to nearest even, equal to the multiply and the `/` operator
template <int K = 0>
__host__ __device__ __forceinline__ double div(double a, const Divisor& D)
{
   const uint64_t A = bits(a);
   const int ea = (int)((A >> 52) & 0x7FF);
   const uint64_t ma = (A & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
   // quotient significand in [1, 2): s = 1 where ma < mb
   const int s = ma < D.mb ? 1 : 0;
   const int e = ea - D.eb + 1023 + K - s;
   if (!D.ok || ea == 0 || ea >= 0x7FF - K || e <= 0 || e >= 0x7FE) {
      // zero dividends are exact; subnormal, infinite and NaN operands and
      // quotients near or past the normal range go to the operator
      if (D.ok && (A << 1) == 0) return from_bits((A ^ D.sign) & 0x8000000000000000ull);
      return div_other(K == 0 ? a : a * (double)(1 << K), D.b);
   }
   // floor of (ma/mb) 2^63 less an error in [0, 9); 10 + (1 - s) bits are
   // beyond the significand
   const uint64_t H = mulhi(ma << 11, D.r);
   const int sh = 11 - s;
   uint64_t q = H >> sh;
   const uint32_t half = 0x400u >> s, f = (uint32_t)H & (2 * half - 1);
   bool up = f >= half;
   if (f - (half - 9) <= 8u) up = (int64_t)((ma << (53 + s)) - D.mb * (2 * q + 1)) > 0;
   q += up ? 1 : 0;
   // q in [2^52, 2^53]; 2^53 carries into the exponent
   return from_bits(((A ^ D.sign) & 0x8000000000000000ull) | (((uint64_t)e << 52) + q - 0x10000000000000ull));
}

// 1 / b rounded to nearest even, equal to the `/` operator unless `rare` is
// raised: for the operands the integer path does not take (zero, subnormal,
// inf, NaN, a subnormal result) and the words too close to a midpoint (1 in
// 228), which the caller leaves to the operator
__host__ __device__ __forceinline__ double rcp_try(double b, bool& rare)
{
   const uint64_t B = bits(b);
   const uint32_t eb = (uint32_t)(B >> 52) & 0x7FFu;
   const uint64_t mb = (B & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
   const uint64_t r = recip64(mb, recip_seed(mb));
   const uint64_t q = (r >> 11) + ((r >> 10) & 1);
   rare |= eb - 1u >= 2044u || ((uint32_t)r & 0x7FFu) - 0x3F7u <= 8u;
   return from_bits((B & 0x8000000000000000ull) | (((uint64_t)(2044u - eb) << 52) + q));
}

// 1 / b rounded to nearest even, equal to the `/` operator
__host__ __device__ __forceinline__ double rcp(double b)
{
   bool rare = false;
   double y = rcp_try(b, rare);
   if (rare) y = div_other(1., b);
   return y;
}

__host__ __device__ __forceinline__ double div(double a, double b) { return div(a, divisor(b)); }

// x * 2^K on the integer pipes: for a normal x whose product stays normal
// the exponent field moves by K and the significand is unchanged, which is
// exactly the rounded product; zeros stay; anything else (subnormal,
// infinite, NaN, a product that overflows or turns subnormal) goes to the
// multiply.  Equal to x * 2^K for every x.
#ifdef __CUDA_ARCH__
__device__ __noinline__ double mul_other(double x, double s) { return x * s; }
#else
inline double mul_other(double x, double s) { return x * s; }
#endif

template <int K>
__host__ __device__ __forceinline__ double scale2(double x)
{
   constexpr double kScale = K >= 0 ? double(1ull << (K >= 0 ? K : 0)) : 1.0 / double(1ull << (K < 0 ? -K : 0));
   const uint64_t u = bits(x);
   const int e = (int)((u >> 52) & 0x7FF);
   if (e >= 1 && e <= 0x7FE && e + K >= 1 && e + K <= 0x7FE) return from_bits(u + (uint64_t)((int64_t)K << 52));
   if ((u << 1) == 0) return x;   // +-0
   return mul_other(x, kScale);
}

// (2^K a) * b rounded to nearest even on the integer pipes, equal to the FP64
// multiplies (K >= 0: a doubling is exact, and moves the exponent here at no
// cost): for normal operands with a normal product the 53-bit
// significands multiply exactly in 128 bits (each shifted to the top of a
// 64-bit word), the top 53 bits round on the next bit and the OR of the
// rest; a zero times a zero or a normal number is a signed zero; anything
// else (subnormal, infinite or NaN operands, a product that overflows or
// turns subnormal) goes to the multiply.
template <int K = 0>
__host__ __device__ __forceinline__ double mul(double a, double b)
{
   constexpr uint64_t kMant = 0xFFFFFFFFFFFFFull, kHidden = 0x10000000000000ull;
   const uint64_t ua = bits(a), ub = bits(b);
   const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
   const int ea = (int)((ua >> 52) & 0x7FF), eb = (int)((ub >> 52) & 0x7FF);
   const bool na = (unsigned)(ea - 1) < 0x7FEu - K, nb = (unsigned)(eb - 1) < 0x7FEu;
   if (!na || !nb) {
      const bool za = (ua << 1) == 0, zb = (ub << 1) == 0;
      if ((za && (zb || nb)) || (zb && na)) return from_bits(sign);
      return mul_other(K == 0 ? a : a * (double)(1 << K), b);
   }
   int e = ea + eb - 1023 + K;   // biased exponent of a product in [1, 2)
   const uint64_t A = ((ua & kMant) | kHidden) << 11, B = ((ub & kMant) | kHidden) << 11;
   uint64_t hi = mulhi(A, B), lo = A * B;
   if (hi >> 63) {
      e += 1;
   } else {
      hi = (hi << 1) | (lo >> 63);
      lo <<= 1;
   }
   if (e < 1) return mul_other(K == 0 ? a : a * (double)(1 << K), b);   // subnormal or zero product
   uint64_t m = hi >> 11;
   const uint64_t g = (hi >> 10) & 1;
   const bool st = ((hi & 0x3FF) | lo) != 0;
   if (g && (st || (m & 1))) m = m + 1;
   if (m >> 53) {
      m >>= 1;
      e += 1;
   }
   if (e > 0x7FE) return mul_other(K == 0 ? a : a * (double)(1 << K), b);   // overflow
   return from_bits(sign | ((uint64_t)e << 52) | (m & kMant));
}

// x * C for a small odd C (3, 5, 7, 11) on the integer pipes, equal to the FP64
// multiply: the product of the significand fits one word, so it costs about
// half of mul
#ifdef __CUDA_ARCH__
__device__ __noinline__ double mulc_other(double x, double c) { return x * c; }
#else
inline double mulc_other(double x, double c) { return x * c; }
#endif

template <int C>
__host__ __device__ __forceinline__ double mulc(double x)
{
   static_assert(C == 3 || C == 5 || C == 7 || C == 11, "small odd constants");
   constexpr int kShift = C == 3 ? 1 : C == 11 ? 3 : 2;   // floor(log2 C)
   const uint64_t u = bits(x);
   const uint32_t e = (uint32_t)(u >> 52) & 0x7FFu;
   if (e - 1u >= 0x7FAu) {   // zero, subnormal, inf, NaN, or a product that may overflow
      if ((u << 1) == 0) return x;
      return mulc_other(x, (double)C);
   }
   uint64_t p = ((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) * (uint64_t)C;
   const int s = kShift + (int)(p >> (53 + kShift));
   p += (1ull << (s - 1)) - 1 + ((p >> s) & 1);   // to nearest even
   const uint64_t m = p >> s;                      // 2^53 carries into the exponent
   return from_bits((u & 0x8000000000000000ull) | (((uint64_t)(e + s - 1) << 52) + m));
}

// 0.0 + v (sub false) or 0.0 - v (sub true) on the integer pipes, equal to
// the FP64 add: +-v with the sign flipped for sub, except that a zero v
// gives +0.0 either way
__host__ __device__ __forceinline__ double zero_plus(double v, bool sub)
{
   const uint64_t u = bits(v);
   return from_bits(((u << 1) == 0) ? 0ull : (sub ? u ^ 0x8000000000000000ull : u));
}

}  // namespace sd

// a * b in the reconstructions and fluxes: with SOFT (FP64) on the integer
// pipes (sd::mul, identical results), otherwise the multiply
template <bool SOFT>
__host__ __device__ __forceinline__ double pm(double a, double b)
{
   return SOFT ? sd::mul(a, b) : a * b;
}
template <bool SOFT>
__host__ __device__ __forceinline__ float pm(float a, float b)
{
   return a * b;
}

// (2^K a) * b, as pm
template <int K, bool SOFT>
__host__ __device__ __forceinline__ double pm2(double a, double b)
{
   return SOFT ? sd::mul<K>(a, b) : ((double)(1 << K) * a) * b;
}
template <int K, bool SOFT>
__host__ __device__ __forceinline__ float pm2(float a, float b)
{
   return ((float)(1 << K) * a) * b;
}

// C * x for a small odd C, as pm
template <int C, bool SOFT>
__host__ __device__ __forceinline__ double pc(double x)
{
   return SOFT ? sd::mulc<C>(x) : (double)C * x;
}
template <int C, bool SOFT>
__host__ __device__ __forceinline__ float pc(float x)
{
   return (float)C * x;
}

// 2^K x + y with one rounding of the sum: the product is exact wherever it
// neither overflows nor turns subnormal, so this is the reference's multiply
// and add, in one FP64 instruction instead of one and a scaling on the integer
// pipes.  For K > 0 it is that for every x up to 2^(1023-K) in magnitude; beyond,
// the product alone would be infinite and the sum here may not be.  For K < 0 it
// is that unless 2^K x is subnormal and y not far larger.  S = -1: y - 2^K x.
template <int K, int S = 1>
__host__ __device__ __forceinline__ double add2(double x, double y)
{
   constexpr double kScale = S * (K >= 0 ? double(1ull << (K >= 0 ? K : 0)) : 1.0 / double(1ull << (K < 0 ? -K : 0)));
#ifdef __CUDA_ARCH__
   return __fma_rn(kScale, x, y);
#else
   return kScale * x + y;
#endif
}
template <int K, int S = 1>
__host__ __device__ __forceinline__ float add2(float x, float y)
{
   constexpr float kScale = S * (K >= 0 ? float(1u << (K >= 0 ? K : 0)) : 1.0f / float(1u << (K < 0 ? -K : 0)));
   return kScale * x + y;
}

// x * 2^K in the reconstructions: with SOFT (FP64 only) on the integer
// pipes (sd::scale2, identical results), otherwise the multiply
template <int K, bool SOFT>
__host__ __device__ __forceinline__ double p2(double x)
{
   constexpr double kScale = K >= 0 ? double(1ull << (K >= 0 ? K : 0)) : 1.0 / double(1ull << (K < 0 ? -K : 0));
   return SOFT ? sd::scale2<K>(x) : kScale * x;
}
template <int K, bool SOFT>
__host__ __device__ __forceinline__ float p2(float x)
{
   constexpr float kScale = K >= 0 ? float(1u << (K >= 0 ? K : 0)) : 1.0f / float(1u << (K < 0 ? -K : 0));
   return kScale * x;
}

// Division by one divisor, possibly several times: in FP64 with SOFT the
// correctly rounded integer-pipe division above (identical results to `/`,
// off the FP64 pipe the FP64 kernels are bound by); otherwise the
// operator.  Which is faster depends on the kernel and the mesh (the
// autotuner picks).
template <typename T, bool SOFT = true>
struct Dv {
   T b;
   __device__ __forceinline__ explicit Dv(T b_) : b(b_) {}
   __device__ __forceinline__ T div(T a) const { return a / b; }
   template <int K>
   __device__ __forceinline__ T div2(T a) const { return (T(1 << K) * a) / b; }   // (2^K a) / b
};
template <>
struct Dv<double, true> {
   sd::Divisor D;
   __device__ __forceinline__ explicit Dv(double b) : D(sd::divisor(b)) {}
   __device__ __forceinline__ double div(double a) const { return sd::div(a, D); }
   template <int K>
   __device__ __forceinline__ double div2(double a) const { return sd::div<K>(a, D); }
};

}  // namespace hamstr
#endif
