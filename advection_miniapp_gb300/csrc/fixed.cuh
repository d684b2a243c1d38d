// Block fixed-point arithmetic for the contractions of the FP64 operator.
//
// On this GPU the FP64 pipe retires 2 instructions per clock and SM, the
// integer multiply-add pipe about 55-64 32 x 32 -> 64 bit products (measured:
// 1.6 DFMA, 53 mad.wide.s32, 61 shifts, 65 logic operations per clock and
// SM), so a contraction carried as integers of 57 bits costs a fraction of
// its binary64 form and is at least as exact: a block of values (a cell) is
// scaled by one power of two above its largest entry and each value becomes
//     X = x 2^(57 - E),  |X| <= 2^57,   X = h 2^29 + l,  |l| <= 2^28,
// two signed 32-bit limbs (round to nearest).  A product with a constant of
// the same form keeps h h', h l' + l h' in two 64-bit accumulators; the
// dropped l l' is at most 2^-1 of the unit.  Rounding errors are thus a few
// times 2^-57 of the block's largest entry per contraction, where binary64
// commits 2^-53 of each intermediate result.
//
// Blocks whose scale leaves a safe window (infinities, NaN, values near the
// ends of the binary64 range) are computed in binary64 by the caller.
#pragma once

#include "device_common.cuh"

namespace adv
{
// resident threads per SM the register allocation allows for (80 registers a
// thread).  One three-stage step with 768 / 640 / 512, in us: upwind field
// geometry 40^3 degree 4 627 / 656 / 718, 24^3 degree 6 514 / 514 / 510; affine
// 48^3 degree 2 276 / 289 / 308, 24^3 degree 6 403 / 450 / 451; SIPG 40^3 degree 4
// 1331 / 1339 / 1434, 32^3 degree 5 1162 / 1275 / 1275; apply 40^3 degree 4 322 / 328 / 360.
// The variants that read every trace of field geometry spill (180-410 bytes of loads)
// and still prefer 768 at 3 and 5 points (rotating 48^3 degree 2 370 / 371 / 399,
// Lax-Friedrichs 40^3 degree 4 915 / 919 / 964), but not at 7 (24^3: 618 / 589 /
// 589 and 690 / 652 / 653); without traces (BDF2) 512 gives 832 instead of 862.
constexpr int kFxThreadsPerSM = 768;

struct Limbs
{
  int h, l; // h 2^29 + l, |l| <= 2^28
};

__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
  // inline PTX: the compiler splits the C expression into a product and a
  // 64-bit addition, half the rate
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(c) : "r"(a), "r"(b));
  return c;
}
__device__ __forceinline__ long long mul_wide(int a, int b)
{
  return (long long)a * b;
}

// a constant's limbs h, l, and h shifted up by the bits between the high
// accumulator and the result's unit
struct FxConst
{
  int h, l, hs;
};

// Sum of products of limb pairs X with constants c 2^b, SHIFT the shift of
// the constants' hs: hi + (mid >> (29 - SHIFT)) is X c 2^(b + SHIFT - 58),
// rounded to nearest (mid starts at half a unit: a truncation's bias would be
// the same in every stage and add up over the steps)
template <int SHIFT>
struct FxAcc
{
  long long hi, mid;
  __device__ __forceinline__ void set(int h, int l, const FxConst &c)
  {
    hi  = mul_wide(h, c.hs);
    mid = mad_wide(l, c.h, mad_wide(h, c.l, 1ll << (28 - SHIFT)));
  }
  __device__ __forceinline__ void add(int h, int l, const FxConst &c)
  {
    hi  = mad_wide(h, c.hs, hi);
    mid = mad_wide(h, c.l, mid);
    mid = mad_wide(l, c.h, mid);
  }
  __device__ __forceinline__ long long value() const { return hi + (mid >> (29 - SHIFT)); }
};

// Limbs of T / 2 rounded to nearest, |T| < 2^60
__device__ __forceinline__ Limbs fx_split(long long T)
{
  const long long Y = T + ((1ll << 29) + 1);
  Limbs           r;
  r.h = (int)(Y >> 30);
  r.l = (int)(((unsigned)Y >> 1) & 0x1FFFFFFFu) - (1 << 28);
  return r;
}

// biased binary64 exponent and magnitude bits of the high word
__device__ __forceinline__ unsigned abs_hi(double x)
{
  return (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
}

// The largest of them: 0 for zeros and for values below 2^-1042 (fx_subnormal)
template <int N>
__device__ __forceinline__ unsigned fx_magnitude(const double (&x)[N])
{
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < N; ++k)
    m = max(m, abs_hi(x[k]));
  return m;
}

// Whether values of magnitude 0 are not all zero (some low word is not)
template <int N>
__device__ __forceinline__ bool fx_subnormal(const double (&x)[N])
{
  unsigned lo = 0;
#pragma unroll
  for (int k = 0; k < N; ++k)
    lo |= (unsigned)__double2loint(x[k]);
  return lo != 0u;
}

// x 2^(57 - E) as limbs for |x| < 2^E: top = E + 1022, the largest biased
// exponent in the block
__device__ __forceinline__ Limbs fx_from_double(double x, int top)
{
  const int      hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int      s  = min(top - (int)(((unsigned)hi << 1) >> 21), 63);
  const unsigned long long m = ((unsigned long long)(((unsigned)hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
  const int      sg = (hi >> 31) | 1;
  Limbs          r  = fx_split((long long)((m << 5) >> s));
  r.h *= sg;
  r.l *= sg;
  return r;
}

// top exponent of the product c v (|c v| < 2^(top - 1022)), at least 1; 0 for a product
// with zero (v may then be a trace that nobody wrote), 2047 if v is not finite
__device__ __forceinline__ unsigned fx_product_top(double c, double v)
{
  const unsigned ec = abs_hi(c) >> 20, ev = abs_hi(v) >> 20;
  const bool     zero = ec == 0u || (abs_hi(v) | (unsigned)__double2loint(v)) == 0u;
  return zero ? 0u : ev == 0x7FFu ? 0x7FFu : (unsigned)max((int)(ec + ev) - 1022, 1);
}

// (-)c v 2^(57 - E) as limbs for top = E + 1022 >= fx_product_top(c, v)
__device__ __forceinline__ Limbs fx_product(double c, double v, int top, bool negative)
{
  const unsigned hc = (unsigned)__double2hiint(c), hv = (unsigned)__double2hiint(v);
  const unsigned lc = (unsigned)__double2loint(c), lv = (unsigned)__double2loint(v);
  const int      ec = (int)((hc << 1) >> 21), ev = (int)((hv << 1) >> 21);
  // a factor of zero (or subnormal): shift everything out
  const int      s = ec == 0 || ev == 0 ? 63 : min(top - (ec + ev - 1022), 63);
  // mantissas of 58 and 57 bits as limbs of 29 and 28 + 29
  const int      xh = (int)__funnelshift_l(lc, (hc & 0xFFFFFu) | 0x100000u, 8), xl = (int)((lc & 0xFFFFFFu) << 5);
  const int      yh = (int)__funnelshift_l(lv, (hv & 0xFFFFFu) | 0x100000u, 7), yl = (int)((lv & 0x1FFFFFFu) << 4);
  const long long mid = mad_wide(xl, yh, mad_wide(xh, yl, (long long)__umulhi((unsigned)xl << 3, (unsigned)yl)));
  const int       sg  = ((int)(hc ^ hv) >> 31) | 1;
  Limbs           r   = fx_split(((mul_wide(xh, yh) << 1) + (mid >> 28)) >> s);
  r.h *= negative ? -sg : sg;
  r.l *= negative ? -sg : sg;
  return r;
}

// X W 2^-58 as limbs, |X| <= 2^57, |W| <= 2^58 (W: a metric value of the
// cell geometry or a uniform constant, y 2^(58 - Ey) as limbs)
__device__ __forceinline__ Limbs fx_times(Limbs X, int2 W)
{
  // the shift of mid rounds to nearest, and 2^28 is added to balance l
  const long long hi  = mul_wide(X.h, W.x);
  const long long mid = mad_wide(X.l, W.x, mad_wide(X.h, W.y, (1ll << 57) + (1ll << 28)));
  const long long Y   = hi + (mid >> 29);
  Limbs           r;
  r.h = (int)(Y >> 29);
  r.l = (int)((unsigned)Y & 0x1FFFFFFFu) - (1 << 28);
  return r;
}

__device__ __forceinline__ unsigned long long fx_abs(long long x)
{
  const unsigned long long s = (unsigned long long)(x >> 63);
  return ((unsigned long long)x ^ s) - s;
}

// Z 2^e rounded to binary64, |Z| < 2^62, for normal results (on the integer
// pipes: the conversion instruction issues on the FP64 pipe)
__device__ __forceinline__ double fx_to_double(long long Z, int e)
{
  const unsigned long long s  = (unsigned long long)(Z >> 63);
  const unsigned long long m  = fx_abs(Z);
  const int                lz = __clzll((long long)m);
  // leading bit to 62, round half up at bit 10; a carry moves the exponent on
  const unsigned long long n = ((m << (lz - 1)) + 0x200u) >> 10;
  const unsigned long long b = n + ((unsigned long long)(unsigned)(1023 + 62 - lz + e) << 52);
  return __longlong_as_double((long long)(m ? (b | (s & 0x8000000000000000ull)) : 0ull));
}

// Constant tables.  The entries of the antisymmetric even-odd form of Dw
// and of the face lifts are c 2^(57 - kd): 2^kd bounds the largest of them.
// A product with a value X is kept at 2^(kFxGuard - kd) of X's unit, so
// that the sum over three directions and six lifts of a cell stays below
// 2^62: 3 (||Dw||_inf + max_q (|lw0| + |lw1|)) 2^(57 + kFxGuard - kd) is at
// most 2^61.55 for n = 2..7 (20.8, 39.7, 64.0, 93.9, 129.4, 170.6 for the
// bracket).
constexpr int kFxGuard = 2, kFxShift = 1 + kFxGuard;
template <int N>
constexpr int fx_kd()
{
  return N == 2 ? 2 : N == 3 ? 3 : N <= 5 ? 4 : 5;
}

struct FxEvenOdd
{
  FxConst e[3][3], o[3][3], ce[3], mid[3], cc;
};

struct FxTables
{
  FxEvenOdd Dw;
  FxConst   lwe[4], lwo[4];
};

static __constant__ FxTables c_tab_fx[kMaxNDev + 1];

// c 2^bits as balanced limbs
inline FxConst fx_host_limbs(double c, int bits, int shift)
{
  const long long X = llrint(ldexp(c, bits));
  const long long l = ((X + (1ll << 28)) & ((1ll << 29) - 1)) - (1ll << 28);
  const long long h = (X - l) >> 29;
  return FxConst{(int)h, (int)l, (int)(h << shift)};
}

// (static: every translation unit fills its own copy of the symbol.)
// shift: that of the accumulators the translation unit's kernels use
static inline cudaError_t upload_fx_local(const DevTables<double> *d, int shift = kFxShift)
{
  static FxTables t[kMaxNDev + 1];
  memset(t, 0, sizeof(t));
  const int kd[kMaxNDev + 1] = {0, 0, fx_kd<2>(), fx_kd<3>(), fx_kd<4>(), fx_kd<5>(), fx_kd<6>(), fx_kd<7>()};
  for (int n = 2; n <= kMaxNDev; ++n)
    {
      const EvenOdd<double> &M    = d[n].Dw_eo;
      const int              bits = 57 - kd[n], h = n / 2;
      for (int q = 0; q < h; ++q)
        {
          for (int i = 0; i < h; ++i)
            {
              t[n].Dw.e[q][i] = fx_host_limbs(M.e[q][i], bits, shift);
              t[n].Dw.o[q][i] = fx_host_limbs(M.o[q][i], bits, shift);
            }
          t[n].Dw.ce[q]  = fx_host_limbs(M.ce[q], bits, shift);
          t[n].Dw.mid[q] = fx_host_limbs(M.mid[q], bits, shift);
          t[n].lwo[q]    = fx_host_limbs(d[n].lwo[q], bits, shift);
        }
      for (int q = 0; q < (n + 1) / 2; ++q)
        t[n].lwe[q] = fx_host_limbs(d[n].lwe[q], bits, shift);
    }
  return cudaMemcpyToSymbol(c_tab_fx, t, sizeof(t));
}

// Volume and lift terms of one pencil: out = Dw V + lw0 F_lo + lw1 F_hi from
// the even-odd halves, in units of 2^(kFxGuard - kd) of V's and F's
template <int N>
__device__ __forceinline__ void fx_sweep_lift(const FxTables &tb, const Limbs (&V)[N], Limbs Flo, Limbs Fhi,
                                              long long (&out)[N])
{
  constexpr int H   = N / 2;
  const int     psh = Flo.h + Fhi.h, psl = Flo.l + Fhi.l;
  const int     pdh = Flo.h - Fhi.h, pdl = Flo.l - Fhi.l;
  int           eh[H], el[H], oh[H], ol[H];
#pragma unroll
  for (int i = 0; i < H; ++i)
    {
      eh[i] = V[i].h + V[N - 1 - i].h, el[i] = V[i].l + V[N - 1 - i].l;
      oh[i] = V[i].h - V[N - 1 - i].h, ol[i] = V[i].l - V[N - 1 - i].l;
    }
#pragma unroll
  for (int q = 0; q < H; ++q)
    {
      FxAcc<kFxShift> E, O;
      O.set(psh, psl, tb.lwe[q]);
      E.set(pdh, pdl, tb.lwo[q]);
#pragma unroll
      for (int i = 0; i < H; ++i)
        {
          E.add(eh[i], el[i], tb.Dw.e[q][i]);
          O.add(oh[i], ol[i], tb.Dw.o[q][i]);
        }
      if (N % 2)
        E.add(V[H].h, V[H].l, tb.Dw.ce[q]);
      const long long a = O.value(), b = E.value();
      out[q]         = a + b;
      out[N - 1 - q] = a - b;
    }
  if (N % 2)
    {
      FxAcc<kFxShift> m;
      m.set(psh, psl, tb.lwe[H]);
#pragma unroll
      for (int i = 0; i < H; ++i)
        m.add(oh[i], ol[i], tb.Dw.mid[i]);
      out[H] = m.value();
    }
}

// Biased top exponents of a block inside the window: 2^-722 .. 2^600.  Lower end,
// with metric factors within 2^+-200: a subnormal value, which the conversions shift
// out, adds at most 2^-822 to a block, 2^-100 of it; zeros, converted as 2^-1022, lie
// 2^64 below the unit; 2^-57 of the block times 1 / det J is a normal number.  (It was 2^-400; blocks below run twice, in fixed point
// as far as their scale and in binary64.  A blob of width 0.05 on the unit cube
// has cells of 2^-571: on 40^3 affine cells of degree 2 a step took 214 us, now
// 166, apply 117, now 74.)
constexpr int kFxLow = 300, kFxHigh = 1623;

// Scale of a block of magnitude m (fx_magnitude): whether it lies in the
// window, and the biased top exponent (1023 for a zero block)
__device__ __forceinline__ bool fx_window(unsigned m, int &top)
{
  const int e = (int)(m >> 20);
  top         = m ? e : 1023;
  return m == 0 || (e > kFxLow && e < kFxHigh);
}
} // namespace adv
