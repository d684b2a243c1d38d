// Changes of basis in block fixed-point arithmetic: tables and sweeps of S,
// S^-1 and S^T (a header of its own: constant memory holds the tables only in
// the translation units that sweep).
#pragma once

#include "fixed.cuh"

namespace adv
{
// changes of basis (entries at most 1: c 2^57) and face values (c 2^56)
struct FxBasisTables
{
  FxEvenOdd S, Si, St;
  FxConst   l0[7], l1[7];
};

static __constant__ FxBasisTables c_tab_fxb[kMaxNDev + 1];

static inline cudaError_t upload_fx_basis_local(const DevTables<double> *d)
{
  static FxBasisTables t[kMaxNDev + 1];
  memset(t, 0, sizeof(t));
  for (int n = 2; n <= kMaxNDev; ++n)
    {
      const int              h       = n / 2;
      const EvenOdd<double> *from[3] = {&d[n].S_eo, &d[n].Si_eo, &d[n].St_eo};
      FxEvenOdd             *to[3]   = {&t[n].S, &t[n].Si, &t[n].St};
      for (int m = 0; m < 3; ++m)
        {
          for (int q = 0; q < h; ++q)
            {
              for (int i = 0; i < h; ++i)
                {
                  to[m]->e[q][i] = fx_host_limbs(from[m]->e[q][i], 57, 2);
                  to[m]->o[q][i] = fx_host_limbs(from[m]->o[q][i], 57, 2);
                }
              to[m]->ce[q]  = fx_host_limbs(from[m]->ce[q], 57, 2);
              to[m]->mid[q] = fx_host_limbs(from[m]->mid[q], 57, 2);
            }
          to[m]->cc = fx_host_limbs(from[m]->cc, 57, 2);
        }
      for (int q = 0; q < n; ++q)
        {
          t[n].l0[q] = fx_host_limbs(d[n].l0[q], 56, 2);
          t[n].l1[q] = fx_host_limbs(d[n].l1[q], 56, 2);
        }
    }
  return cudaMemcpyToSymbol(c_tab_fxb, t, sizeof(t));
}

// One sweep of a change of basis, M symmetric under reflection (even-odd
// form, entries at most 1): out = 2 M X (one extra bit, for fx_split), rounded
// to nearest.  |X| < 2^59; sums of limbs stay within 32 bits, |out| < 2^62.
template <int N>
__device__ __forceinline__ void fx_sweep_sym(const FxEvenOdd &M, const Limbs (&X)[N], long long (&out)[N])
{
  constexpr int H = N / 2;
  int           eh[H], el[H], oh[H], ol[H];
#pragma unroll
  for (int i = 0; i < H; ++i)
    {
      eh[i] = X[i].h + X[N - 1 - i].h, el[i] = X[i].l + X[N - 1 - i].l;
      oh[i] = X[i].h - X[N - 1 - i].h, ol[i] = X[i].l - X[N - 1 - i].l;
    }
#pragma unroll
  for (int q = 0; q < H; ++q)
    {
      FxAcc<2> E, O;
      E.set(eh[0], el[0], M.e[q][0]);
      O.set(oh[0], ol[0], M.o[q][0]);
#pragma unroll
      for (int i = 1; i < H; ++i)
        {
          E.add(eh[i], el[i], M.e[q][i]);
          O.add(oh[i], ol[i], M.o[q][i]);
        }
      if (N % 2)
        E.add(X[H].h, X[H].l, M.ce[q]);
      const long long a = E.value(), b = O.value();
      out[q]         = a + b;
      out[N - 1 - q] = a - b;
    }
  if (N % 2)
    {
      FxAcc<2> m;
      m.set(X[H].h, X[H].l, M.cc);
#pragma unroll
      for (int i = 0; i < H; ++i)
        m.add(eh[i], el[i], M.mid[i]);
      out[H] = m.value();
    }
}

// Rounded right shift of a sweep's output
template <int BITS>
__device__ __forceinline__ long long fx_shift(long long T)
{
  return BITS ? (T + (1ll << (BITS > 0 ? BITS - 1 : 0))) >> BITS : T;
}

// Bits the values of a cell grow by in sweeps of S, S^T and S^-1, as the
// shifts that keep the limbs in range.  ||S||_inf is 1, 1.17, 1.30, 1.39,
// 1.51, 1.62 and ||S^T||_inf 1, 1.80, 1.73, 1.79, 1.76, 1.78 for n = 2..7: two
// sweeps of 2^57 stay below 2^59.  ||S^-1||_inf is 1.73, 2.33, 2.86, 3.32,
// 3.75, 4.14: its second and third input are shifted down by fx_si1 and
// fx_si2 bits (about 17 2^57 >> 3 for n = 7).
template <int N>
constexpr int fx_si1()
{
  return N == 7 ? 1 : 0;
}
template <int N>
constexpr int fx_si2()
{
  return N == 2 ? 0 : N == 3 ? 1 : 2;
}
} // namespace adv
