// The sine-product + Gaussian solution (ADV_IC_SINE_GAUSS) in fixed point.
//
// Three sines and an exponential in binary64 cost about 130 FP64
// instructions per point, 65 clocks of an SM's FP64 pipe each; on the integer
// pipes they take about 600 instructions, 10 clocks.  The fraction of a turn
// is carried to 2^-62, the polynomials (Taylor series on |angle| <= pi/4 and on
// |x| <= ln 2 / 2, their last terms in binary32) to a few 2^-57 of 1, and the sum
// of the sine product and the Gaussian is rounded to binary64 once.  Largest
// errors in units of 2^-57, over 20,000 points each in 200-bit arithmetic: sine 4.2, sine
// product 3.6, exponential of a given argument 2.9; the Gaussian 14.7, since its
// argument 50 r^2 is formed in binary64, and the rounded sum 18.2 (one binary64
// rounding of a result in [1/2, 1) is 8).  These are absolute: far out the Gaussian
// keeps few bits of its own.
#pragma once

#include "fixed.cuh"

namespace adv
{
constexpr int kSinTerms = 7, kSinTail = 4;  // fixed-point and binary32 terms
constexpr int kExpTerms = 10, kExpTail = 5;

struct FxMathTables
{
  int2  sc[2][kSinTerms];                // sine (of w = 4 angle / pi, over w) and cosine, in w^2: c 2^57
  float sct[2][kSinTail];                // the following terms, c 2^57
  int2  ex[kExpTerms];                   // 2^(-1/2) exp(-ln 2 / 2 w) in w: c 2^57
  float ext[kExpTail];
  int2  log2e;                           // mantissa of log2 e: c 2^57 as limbs (58 bits)
};
static __constant__ FxMathTables c_tab_fxm;

static inline int2 fx_host_limbs2(long double c, int bits)
{
  const long long X = llrintl(ldexpl(c, bits));
  const long long l = ((X + (1ll << 28)) & ((1ll << 29) - 1)) - (1ll << 28);
  return make_int2((int)((X - l) >> 29), (int)l);
}

static inline cudaError_t upload_fx_math_local()
{
  FxMathTables      t;
  const long double q = 0.785398163397448309615660845819875721L, h = 0.346573590279972654708616060729088284L;
  for (int p = 0; p < 2; ++p)
    {
      long double c = p == 0 ? q : 1.0L; // p = 0: q^(2k+1) / (2k+1)!, 1: q^(2k) / (2k)!
      for (int k = 0; k < kSinTerms + kSinTail; ++k)
        {
          if (k < kSinTerms)
            t.sc[p][k] = fx_host_limbs2(c, 57);
          else
            t.sct[p][k - kSinTerms] = (float)ldexpl(c, 57);
          const long double a = p == 0 ? 2 * k + 2 : 2 * k + 1;
          c *= -q * q / (a * (a + 1));
        }
    }
  long double c = 0.707106781186547524400844362104849039L;
  for (int k = 0; k < kExpTerms + kExpTail; ++k)
    {
      if (k < kExpTerms)
        t.ex[k] = fx_host_limbs2(c, 57);
      else
        t.ext[k - kExpTerms] = (float)ldexpl(c, 57);
      c *= -h / (k + 1);
    }
  const long double l2e = 1.44269504088896340735992468100189214L;
  const long long   X   = llrintl(ldexpl(l2e, 57)); // unsigned limbs, as fx_product's
  t.log2e = make_int2((int)(X >> 29), (int)(X & ((1ll << 29) - 1)));
  return cudaMemcpyToSymbol(c_tab_fxm, &t, sizeof(t));
}

// fraction of y in units of 2^-62, |y| < 2^20 (bits below are cut off)
__device__ __forceinline__ unsigned long long fx_turn(double y)
{
  const long long          b  = __double_as_longlong(y);
  const int                sh = (int)((b >> 52) & 0x7FF) - 1013;
  const unsigned long long m  = ((unsigned long long)b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  unsigned long long       v  = sh >= 0 ? m << min(sh, 63) : m >> min(-sh, 63);
  v                           = b < 0 ? 0ull - v : v;
  return v & ((1ull << 62) - 1);
}

// limbs of a 58-bit value, the second factor of fx_times
__device__ __forceinline__ int2 fx_limbs58(long long v)
{
  const long long Y = v + (1ll << 28);
  return make_int2((int)(Y >> 29), (int)((unsigned)Y & 0x1FFFFFFFu) - (1 << 28));
}

__device__ __forceinline__ long long fx_join(const Limbs &x)
{
  return (long long)x.h * (1 << 29) + x.l;
}

// sin(2 pi u 2^-62) 2^57
__device__ __forceinline__ Limbs fx_sin_turn(unsigned long long u)
{
  const long long k = (long long)((u + (1ull << 59)) >> 60);
  const long long r = (long long)u - (k << 60); // w 2^59, angle = pi / 4 w
  const bool      p = k & 1;
  const Limbs     X = fx_split(r >> 1);
  // w^2 2^58 = X^2 2^-56
  const long long zz = (mul_wide(X.h, X.h) << 2) + (mul_wide(X.h, 2 * X.l) >> 27);
  const int2      z  = fx_limbs58(zz);
  const float     zf = (float)z.x * 0x1p-29f;
  float           t  = p ? c_tab_fxm.sct[1][kSinTail - 1] : c_tab_fxm.sct[0][kSinTail - 1];
#pragma unroll
  for (int i = kSinTail - 2; i >= 0; --i)
    t = fmaf(t, zf, p ? c_tab_fxm.sct[1][i] : c_tab_fxm.sct[0][i]);
  Limbs a{0, (int)t};
#pragma unroll
  for (int i = kSinTerms - 1; i >= 0; --i)
    {
      a = fx_times(a, z);
      a.h += p ? c_tab_fxm.sc[1][i].x : c_tab_fxm.sc[0][i].x;
      a.l += p ? c_tab_fxm.sc[1][i].y : c_tab_fxm.sc[0][i].y;
    }
  // the odd polynomial's factor w (2^58 units), or 1
  a            = fx_times(a, p ? make_int2(1 << 29, 0) : fx_limbs58(r >> 1));
  const int sg = (k & 2) ? -1 : 1;
  return Limbs{a.h * sg, a.l * sg};
}

// exp(-x) 2^57 for 0 <= x < 64
__device__ __forceinline__ long long fx_exp_neg(double x)
{
  const unsigned hv = (unsigned)__double2hiint(x), lv = (unsigned)__double2loint(x);
  const int      ev = (int)((hv << 1) >> 21);
  const int2     c  = c_tab_fxm.log2e;
  // T = 2 (log2 e x) 2^(57 - E) as fx_product, then t 2^56
  const int       yh = (int)__funnelshift_l(lv, (hv & 0xFFFFFu) | 0x100000u, 7), yl = (int)((lv & 0x1FFFFFFu) << 4);
  const long long mid = mad_wide(c.y, yh, mad_wide(c.x, yl, (long long)__umulhi((unsigned)c.y << 3, (unsigned)yl)));
  const long long T   = (mul_wide(c.x, yh) << 1) + (mid >> 28);
  const int       s   = ev - 1023;
  const long long t   = ev == 0 ? 0 : s >= 0 ? T << s : T >> min(-s, 63);
  const int       n   = (int)(t >> 56);
  // 2^-f = 2^(-1/2) exp(-ln 2 / 2 w), w = 2 f - 1
  const long long w = ((t & ((1ll << 56) - 1)) - (1ll << 55)) << 3; // w 2^58
  const int2      W = fx_limbs58(w);
  const float     wf = (float)W.x * 0x1p-29f;
  float           e  = c_tab_fxm.ext[kExpTail - 1];
#pragma unroll
  for (int i = kExpTail - 2; i >= 0; --i)
    e = fmaf(e, wf, c_tab_fxm.ext[i]);
  Limbs a{0, (int)e};
#pragma unroll
  for (int i = kExpTerms - 1; i >= 0; --i)
    {
      a = fx_times(a, W);
      a.h += c_tab_fxm.ex[i].x;
      a.l += c_tab_fxm.ex[i].y;
    }
  return n < 60 ? fx_join(a) >> n : 0;
}

// exact_value of ADV_IC_SINE_GAUSS from the three phases y_d = (x_d - v_d t -
// lo_d) / L_d - p_d, |y_d| < 2^20
__device__ __forceinline__ double fx_sine_gauss(double y0, double y1, double y2)
{
  const unsigned long long u[3] = {fx_turn(y0), fx_turn(y1), fx_turn(y2)};
  double                   r2   = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    {
      const double c = fx_to_double((long long)u[d] - (1ll << 61), -62);
      r2             = d ? fma(c, c, r2) : c * c;
    }
  Limbs p = fx_sin_turn(u[0]);
#pragma unroll 1
  for (int d = 1; d < 3; ++d)
    {
      const Limbs q = fx_sin_turn(u[d]);
      p             = fx_times(p, make_int2(2 * q.h, 2 * q.l));
    }
  return fx_to_double(fx_join(p) + fx_exp_neg(50.0 * r2), -57);
}
} // namespace adv
