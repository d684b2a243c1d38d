// Collocation-form stage of the FP64 advection-diffusion operator (SIPG on
// affine meshes) in block fixed-point arithmetic (fixed.cuh): the counterpart
// of stage_gauss_cta<..., VISC> (stage_gauss.cuh) without a skew term.
//
// Per direction the pencil's volume term is D U, then Dw of s vt U - nu V / h^2 D U
// (s the velocity's time factor) with the lifts of the fluxes and of the SIPG
// jumps in the same accumulators; the binary64 kernel spent 100 FP64
// instructions per point at degree 5.  (One symmetric contraction with Dw D
// instead of two in a row costs the same but loses up to 5 bits: its entries
// are 2^4 times Dw's and its operand has to share the unit of s vt U.)
// Fluxes, jumps, 1 / det J and the update stay binary64; the traces (value and
// normal derivative at six faces) are integer contractions at their pencil's own
// scale.  Cells outside the window of exponents take the binary64 path (see
// stage_fx.cuh).
// Bound: integer and FP64 issue (46 % and 42 % of their pipes) at three CTAs
// per SM.  Measured on GB300 on 32^3 cells of degree 5, one LSRK(5,4) step: 1.82
// instead of 6.23 ms; with binary64 traces 2.29, with the geometry staged in
// shared memory (two CTAs) 1.93.
#pragma once

#include "fixed.cuh"
#include "stage_fx.cuh"

namespace adv
{
// Tables of the diffusive terms: D as c 2^(57 - kdd) and the split derivative
// lifts lde, ldo as c 2^(57 - kld).  Their operands are carried 2^kdd and
// 2^(kld - kd) times larger, so that all terms share the unit of the Dw terms.
// ||D||_inf / 2^kdd is 1.7, 1.3, 2.7, 2.4, 3.9, 2.9 for n = 2..7: with one bit of
// headroom in the block's scale s vt U - nu V / h^2 D U stays below 2^58.3 (its limbs
// and sums of two of them within 32 bits: h below 2^30.3, l below 2^30), and with one
// guard bit less than the advection stage the sum over three directions, lifts
// included, below 2^61.25 (n = 7).
template <int N>
constexpr int fx_kdd()
{
  return N == 2 ? 1 : N <= 4 ? 3 : N <= 6 ? 4 : 5;
}
template <int N>
constexpr int fx_kld()
{
  return N == 2 ? 2 : N == 3 ? 4 : N == 4 ? 6 : N <= 6 ? 7 : 8;
}
constexpr int kFxViscBits = 1, kFxViscGuard = 1, kFxViscShift = 1 + kFxViscGuard;

// face derivatives of the traces: c 2^(57 - kle)
template <int N>
constexpr int fx_kle()
{
  return N == 2 ? 1 : N <= 5 ? N : 6;
}

struct FxViscTables
{
  FxEvenOdd D;
  FxConst   lde[4], ldo[4];
  FxConst   l[2][kMaxNDev], ld[2][kMaxNDev]; // at the low and high face
};
static __constant__ FxViscTables c_tab_fxv[kMaxNDev - 1];

static inline cudaError_t upload_fx_visc_local(const DevTables<double> *d)
{
  static FxViscTables t[kMaxNDev - 1];
  memset(t, 0, sizeof(t));
  const int kdd[kMaxNDev - 1] = {fx_kdd<2>(), fx_kdd<3>(), fx_kdd<4>(), fx_kdd<5>(), fx_kdd<6>(), fx_kdd<7>()};
  const int kld[kMaxNDev - 1] = {fx_kld<2>(), fx_kld<3>(), fx_kld<4>(), fx_kld<5>(), fx_kld<6>(), fx_kld<7>()};
  const int kle[kMaxNDev - 1] = {fx_kle<2>(), fx_kle<3>(), fx_kle<4>(), fx_kle<5>(), fx_kle<6>(), fx_kle<7>()};
  for (int n = 2; n <= kMaxNDev; ++n)
    {
      FxViscTables          &T = t[n - 2];
      const EvenOdd<double> &M = d[n].D_eo;
      const int              h = n / 2, bd = 57 - kdd[n - 2], bl = 57 - kld[n - 2];
      for (int q = 0; q < h; ++q)
        {
          for (int i = 0; i < h; ++i)
            {
              T.D.e[q][i] = fx_host_limbs(M.e[q][i], bd, 2);
              T.D.o[q][i] = fx_host_limbs(M.o[q][i], bd, 2);
            }
          T.D.ce[q]  = fx_host_limbs(M.ce[q], bd, 2);
          T.D.mid[q] = fx_host_limbs(M.mid[q], bd, 2);
          T.ldo[q]   = fx_host_limbs(d[n].ldo[q], bl, kFxViscShift);
        }
      for (int q = 0; q < (n + 1) / 2; ++q)
        T.lde[q] = fx_host_limbs(d[n].lde[q], bl, kFxViscShift);
      for (int q = 0; q < n; ++q)
        {
          T.l[0][q]  = fx_host_limbs(d[n].l0[q], 56, 2);
          T.l[1][q]  = fx_host_limbs(d[n].l1[q], 56, 2);
          T.ld[0][q] = fx_host_limbs(d[n].ld0[q], 57 - kle[n - 2], 2);
          T.ld[1][q] = fx_host_limbs(d[n].ld1[q], 57 - kle[n - 2], 2);
        }
    }
  return cudaMemcpyToSymbol(c_tab_fxv, t, sizeof(t));
}

__device__ __forceinline__ Limbs fx_add(const Limbs &a, const Limbs &b)
{
  return Limbs{a.h + b.h, a.l + b.l};
}
__device__ __forceinline__ Limbs fx_sub(const Limbs &a, const Limbs &b)
{
  return Limbs{a.h - b.h, a.l - b.l};
}

// out = 2^-kdd D X as limbs
template <int N>
__device__ __forceinline__ void fx_sweep_d(const FxViscTables &tv, const Limbs (&X)[N], Limbs (&out)[N])
{
  constexpr int H = N / 2;
  Limbs         e[H], o[H];
#pragma unroll
  for (int i = 0; i < H; ++i)
    e[i] = fx_add(X[i], X[N - 1 - i]), o[i] = fx_sub(X[i], X[N - 1 - i]);
#pragma unroll
  for (int q = 0; q < H; ++q)
    {
      FxAcc<2> E, O;
      E.set(e[0].h, e[0].l, tv.D.e[q][0]);
      O.set(o[0].h, o[0].l, tv.D.o[q][0]);
#pragma unroll
      for (int i = 1; i < H; ++i)
        {
          E.add(e[i].h, e[i].l, tv.D.e[q][i]);
          O.add(o[i].h, o[i].l, tv.D.o[q][i]);
        }
      if (N % 2)
        E.add(X[H].h, X[H].l, tv.D.ce[q]);
      const long long a = E.value(), b = O.value();
      out[q]         = fx_split(b + a);
      out[N - 1 - q] = fx_split(b - a);
    }
  if (N % 2)
    {
      FxAcc<2> m;
      m.set(o[0].h, o[0].l, tv.D.mid[0]);
#pragma unroll
      for (int i = 1; i < H; ++i)
        m.add(o[i].h, o[i].l, tv.D.mid[i]);
      out[H] = fx_split(m.value());
    }
}

// out = Dw V + value lifts of Flo, Fhi + derivative lifts of dlo, dhi
template <int N>
__device__ __forceinline__ void fx_sweep_visc(const FxTables &tb, const FxViscTables &tv, const Limbs (&V)[N],
                                              Limbs Flo, Limbs Fhi, Limbs dlo, Limbs dhi, long long (&out)[N])
{
  constexpr int H  = N / 2;
  const Limbs   ps = fx_add(Flo, Fhi), pd = fx_sub(Flo, Fhi), ds = fx_sub(dlo, dhi), dd = fx_add(dlo, dhi);
  Limbs         e[H], o[H];
#pragma unroll
  for (int i = 0; i < H; ++i)
    e[i] = fx_add(V[i], V[N - 1 - i]), o[i] = fx_sub(V[i], V[N - 1 - i]);
#pragma unroll
  for (int q = 0; q < H; ++q)
    {
      FxAcc<kFxViscShift> a, b; // out = a + b at q, a - b at n - 1 - q
      a.set(ps.h, ps.l, tb.lwe[q]);
      a.add(ds.h, ds.l, tv.lde[q]);
      b.set(pd.h, pd.l, tb.lwo[q]);
      b.add(dd.h, dd.l, tv.ldo[q]);
#pragma unroll
      for (int i = 0; i < H; ++i)
        {
          a.add(o[i].h, o[i].l, tb.Dw.o[q][i]);
          b.add(e[i].h, e[i].l, tb.Dw.e[q][i]);
        }
      if (N % 2)
        b.add(V[H].h, V[H].l, tb.Dw.ce[q]);
      const long long x = a.value(), y = b.value();
      out[q]         = x + y;
      out[N - 1 - q] = x - y;
    }
  if (N % 2)
    {
      FxAcc<kFxViscShift> m;
      m.set(ps.h, ps.l, tb.lwe[H]);
      m.add(ds.h, ds.l, tv.lde[H]);
#pragma unroll
      for (int i = 0; i < H; ++i)
        m.add(o[i].h, o[i].l, tb.Dw.mid[i]);
      out[H] = m.value();
    }
}

template <int N, bool TR>
struct FxViscShape
{
  using SH                     = StageShape<N, double, false, true>;
  static constexpr int C       = SH::C;
  static constexpr int THREADS = SH::THREADS;
  static_assert(C * N * N <= THREADS && C <= 32, "one pencil per thread and a bit per cell");
  // U, s U, Z [C][NQ], block maxima and the mask
  static constexpr int OWN  = 3 * C * N * N * N * 8 + (3 * C + 1) * 4;
  static constexpr int BIN  = GaussShape<N, double, false, true, TR>::SMEM;
  static constexpr int SMEM = OWN > BIN ? OWN : BIN;
};

// the binary64 path for the cells of `mask`
template <int N, bool TR>
__device__ __noinline__ void stage_visc_masked(const StageArgs &A, long long cell0, unsigned char *smem, unsigned mask)
{
  stage_gauss_cta<N, double, false, true, TR>(A, cell0, smem, mask);
}

// Value and reference normal derivative of a pencil x at its low (s = 0) or
// high face, in fixed point at the pencil's own scale (a pencil outside the
// window of exponents in binary64).  The caller converts the pencil once.
template <int N>
struct ViscPencil
{
  Limbs X[N];
  int   top;
  bool  ok;
  __device__ __forceinline__ void set(const double (&x)[N])
  {
    const unsigned m = fx_magnitude(x);
    ok               = fx_window(m, top) && !(m == 0u && fx_subnormal(x));
#pragma unroll
    for (int q = 0; q < N; ++q)
      X[q] = fx_from_double(x[q], top);
  }
  __device__ __forceinline__ double2 at(const DevTables<double> &tb, const FxViscTables &tv, const double (&x)[N],
                                        int s) const
  {
    if (!ok)
      {
        const double *l = s ? tb.l1 : tb.l0, *ld = s ? tb.ld1 : tb.ld0;
        double2       t = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int i = 0; i < 1; ++i)
#pragma unroll
          for (int q = 0; q < N; ++q)
            {
              t.x = fma(l[q], x[q], t.x);
              t.y = fma(ld[q], x[q], t.y);
            }
        return t;
      }
    FxAcc<2> v, d;
    v.set(X[0].h, X[0].l, tv.l[s][0]);
    d.set(X[0].h, X[0].l, tv.ld[s][0]);
#pragma unroll
    for (int q = 1; q < N; ++q)
      {
        v.add(X[q].h, X[q].l, tv.l[s][q]);
        d.add(X[q].h, X[q].l, tv.ld[s][q]);
      }
    return make_double2(fx_to_double(v.value(), top - 1022 - 57), fx_to_double(d.value(), top - 1022 - 58 + fx_kle<N>()));
  }
};

template <int N, bool TR>
__device__ __forceinline__ void stage_fx_visc_cta(const StageArgs &A, const long long cell0, unsigned char *smem_raw)
{
  using FS         = FxViscShape<N, TR>;
  constexpr int C  = FS::C;
  constexpr int NQ = N * N * N;
  constexpr int NF = N * N;
  constexpr int NT = FS::THREADS;
  int2      *Ub    = reinterpret_cast<int2 *>(smem_raw);         // [C][NQ] U as limbs
  int2      *Sb    = Ub + C * NQ;                                // [C][NQ] s 2^-es U / 2 (es = adv_exp)
  long long *Qb    = reinterpret_cast<long long *>(Sb + C * NQ); // [C][NQ] Z, then the next input
  unsigned  *s_eu = reinterpret_cast<unsigned *>(Qb + C * NQ), *s_ef = s_eu + C, *s_bad = s_ef + C;

  const DevTables<double> &tb    = tab<double>(N);
  const FxTables          &fx    = c_tab_fx[N];
  const FxViscTables      &fv    = c_tab_fxv[N - 2];
  const int                tid   = threadIdx.x;
  const int                ncell = (int)min((long long)C, A.n_cells - cell0);
  const bool               mine  = tid < ncell * NF;
  const int                cl = tid / NF, r = tid % NF;
  const int                ox = cl * NQ + N * r, oy = cl * NQ + (r % N) + NF * (r / N), oz = cl * NQ + r;
  const long long          gb    = (cell0 + cl) * NQ + r;
  const double            *tr_in = static_cast<const double *>(A.tr_in);

  double U[N]; // the z pencil
  if (mine)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        U[k] = __ldg(A.r_in + gb + k * NF);
    }
  if (tid < C)
    s_eu[tid] = s_ef[tid] = 0u;
  if (tid == 0)
    *s_bad = 0u;
  __syncthreads();

  // ---- fluxes and jumps at the pencil's six face points: F[j] the value
  //      lifted with l(s) / w (low face: s (M u_own + P u_nbr) + K1 J - K2 (d u_own + d u_nbr),
  //      high face: -s (P u_own + M u_nbr) + K1 J + K2 (...)), J = u_nbr - u_own
  double   F[6], J[6];
  const double kj = (double)(1 << (fx_kld<N>() > fx_kd<N>() ? fx_kld<N>() - fx_kd<N>() : 0));
  if (mine)
    {
      const unsigned c = (unsigned)(cell0 + cl), nx = A.nc[0], ny = A.nc[1];
      const unsigned row = c / nx;
      const int      ix = (int)(c - row * nx), iz = (int)(row / ny), iy = (int)(row - (unsigned)iz * ny);
#pragma unroll
      for (int j = 0; j < 6; ++j)
        {
          const int d = j >> 1;
          int       nb;
          unsigned  face;
          cell_face(A, ix, iy, iz, j, nb, face);
          const double *fg = static_cast<const double *>(A.face_geo[d]);
          double2       pm = __ldg(reinterpret_cast<const double2 *>(fg + ((size_t)face * NF + r) * 2));
          if (A.swap_pm)
            pm = make_double2(pm.y, pm.x);
          const double co = (j & 1) ? pm.x : pm.y, cn = (j & 1) ? pm.y : pm.x;
          // value and reference normal derivative on both sides
          double2 o, n;
          if (TR)
            {
              const double *to = tr_in + ((cell0 + cl) * 6 + j) * 2 * NF + r;
              const double *tn = tr_in + ((long long)(nb < 0 ? cell0 + cl : nb) * 6 + (nb < 0 ? j : j ^ 1)) * 2 * NF + r;
              o = make_double2(__ldg(to), __ldg(to + NF));
              n = make_double2(__ldg(tn), __ldg(tn + NF));
            }
          else
            {
              const int     st = j < 2 ? 1 : j < 4 ? N : NF, at = j < 2 ? N * r : j < 4 ? oy - cl * NQ : r;
              const double *go = A.r_in + (cell0 + cl) * NQ + at;
              const double *gn = A.r_in + (nb < 0 ? cell0 + cl : (long long)nb) * NQ + at;
              double        x[N], y[N];
#pragma unroll
              for (int q = 0; q < N; ++q)
                x[q] = __ldg(go + q * st), y[q] = __ldg(gn + q * st);
              ViscPencil<N> p;
              p.set(x);
              o = p.at(tb, fv, x, j & 1);
              p.set(y);
              n = p.at(tb, fv, y, (j & 1) ^ 1);
            }
          double un = n.x; // the neighbour's value of the advective flux
          if (nb < 0)
            {
              un  = boundary_value(A, d, face, r, NF);
              n.x = 2.0 * un - o.x; // mirror data
              n.y = o.y;
            }
          const double adv  = A.adv_scale * fma(co, o.x, cn * un);
          const double jump = n.x - o.x, flux = fma(A.K1[d], jump, (j & 1) ? -adv : adv);
          const double k2   = (j & 1) ? A.K2[d] : -A.K2[d];
          F[j]              = fma(k2, n.y + o.y, flux);
          J[j]              = (A.K2[d] * kj) * jump;
        }
      atomicMax(s_eu + cl, fx_magnitude(U));
      atomicMax(s_ef + cl, max(fx_magnitude(F), fx_magnitude(J)));
    }
  __syncthreads();

  // ---- the block's scale, kFxViscBits above the largest term
  Limbs f[6], jl[6];
  int2  cd[3];
  bool  live = mine;
  int   topz = 0, topw = 0;
  if (mine)
    {
      const unsigned mu = s_eu[cl], mf = s_ef[cl];
      const int      eu = (int)(mu >> 20), ef = (int)(mf >> 20);
      // the velocity term at its own size, s vt, |s| <= 2^es (a velocity near its
      // reversal in time would set a unit far above the terms of the cell)
      topw = A.cell_exp[cell0 + cl] + A.adv_exp;
      double c2[3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        {
          c2[d] = -A.cdiff[d] * (double)(1 << fx_kdd<N>());
          topw  = max(topw, (int)(abs_hi(c2[d]) >> 20));
        }
      const bool zero = (mu | mf) == 0;
      topz            = (zero ? 1023 : max(eu + topw - 1022, ef)) + kFxViscBits;
      live            = eu < kFxHigh && ef < kFxHigh && topz > kFxLow + kFxViscBits;
      // (values of magnitude 0 that are not zero: the binary64 path)
      if ((!live && r == 0) || (mu == 0 && fx_subnormal(U)) || (mf == 0 && (fx_subnormal(F) || fx_subnormal(J))))
        atomicOr(s_bad, 1u << cl);
      const int topu = topz - topw + 1022;
      if (live)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            {
              const Limbs x   = fx_from_double(U[k], topu);
              Ub[oz + k * NF] = make_int2(x.h, x.l);
              const Limbs s   = fx_times(x, A.adv_limbs); // s 2^-es U / 2: vt takes the factor 2^(es + 1) below
              Sb[oz + k * NF] = make_int2(s.h, s.l);
            }
#pragma unroll
          for (int j = 0; j < 6; ++j)
            {
              f[j]  = fx_from_double(F[j], topz);
              jl[j] = fx_from_double((j & 1) ? -J[j] : J[j], topz);
            }
#pragma unroll
          for (int d = 0; d < 3; ++d)
            cd[d] = fx_const58(c2[d], topw);
        }
    }
  __syncthreads();
  live = live && !((*s_bad >> cl) & 1u);

  auto pass = [&](int off, int st, const double *v, int d, long long(&out)[N]) {
    Limbs X[N], V[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      X[k] = Limbs{Ub[off + k * st].x, Ub[off + k * st].y};
    fx_sweep_d<N>(fv, X, V);
#pragma unroll
    for (int k = 0; k < N; ++k)
      {
        const int2 s = Sb[off + k * st];
        V[k]         = fx_add(fx_times(V[k], cd[d]), fx_times(Limbs{s.x, s.y}, fx_const58(__ldg(v + k * st), topw - 1 - A.adv_exp)));
      }
    fx_sweep_visc<N>(fx, fv, V, f[2 * d], f[2 * d + 1], jl[2 * d], jl[2 * d + 1], out);
  };
  // the geometry is read from global memory (staged it would take half of the
  // shared memory and two of the three resident CTAs)
  const double *G = static_cast<const double *>(A.cell_geo) + (cell0 + cl) * 4 * NQ;
  long long     out[N];
  if (live)
    {
      pass(ox, 1, G + N * r, 0, out);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[ox + k] = out[k];
    }
  __syncthreads();
  if (live)
    {
      pass(oy, N, G + NQ + (oy - cl * NQ), 1, out);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[oy + k * N] += out[k];
    }
  const bool upd = A.mode == kModeStage || A.mode == kModeLastStage;
  double     ui[N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    ui[k] = live && upd && A.u_in ? __ldcs(A.u_in + gb + k * NF) : 0.0;
  __syncthreads();
  if (live)
    {
      pass(oz, NF, G + 2 * NQ + r, 2, out);
      const int ez = topz - 1022 - 57 + fx_kd<N>() - kFxViscGuard;
      double    kd[N], next[N];
#pragma unroll
      for (int k = 0; k < N; ++k)
        kd[k] = fx_to_double(Qb[oz + k * NF] + out[k], ez) * __ldg(G + 3 * NQ + r + k * NF);
      if (!upd)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            A.r_out[gb + k * NF] = A.out_scale * kd[k];
        }
      else
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            next[k] = fma(A.b, kd[k], ui[k]);
#pragma unroll
          for (int k = 0; k < N; ++k)
            A.u_out[gb + k * NF] = next[k];
          if (A.mode == kModeStage)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                next[k] = fma(A.a, kd[k], ui[k]);
#pragma unroll
              for (int k = 0; k < N; ++k)
                A.r_out[gb + k * NF] = next[k];
            }
#pragma unroll
          for (int k = 0; k < N; ++k)
            Qb[oz + k * NF] = __double_as_longlong(next[k]);
        }
    }
  if (TR && A.tr_out)
    {
      // value and derivative traces of the next input along the three directions
      __syncthreads();
      if (live)
        {
#pragma unroll 1
          for (int d = 0; d < 3; ++d)
            {
              const long long *p  = Qb + (d == 0 ? ox : d == 1 ? oy : oz);
              const int        st = d == 0 ? 1 : d == 1 ? N : NF;
              double           x[N];
#pragma unroll
              for (int k = 0; k < N; ++k)
                x[k] = __longlong_as_double(p[k * st]);
              double       *to = static_cast<double *>(A.tr_out) + ((cell0 + cl) * 6 + 2 * d) * 2 * NF + r;
              ViscPencil<N> t;
              t.set(x);
              const double2 lo = t.at(tb, fv, x, 0), hi = t.at(tb, fv, x, 1);
              to[0]      = lo.x;
              to[NF]     = lo.y;
              to[2 * NF] = hi.x;
              to[3 * NF] = hi.y;
            }
        }
    }
  // ---- cells outside the window
  const unsigned bad = *s_bad;
  if (bad)
    {
      __syncthreads();
      stage_visc_masked<N, TR>(A, cell0, smem_raw, bad);
    }
}

template <int N, bool TR>
__global__ void __launch_bounds__(FxViscShape<N, TR>::THREADS, kFxThreadsPerSM / FxViscShape<N, TR>::THREADS)
  stage_fx_visc_kernel(const __grid_constant__ StageArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_fx_visc_cta<N, TR>(A, A.cell_begin + (long long)blockIdx.x * FxViscShape<N, TR>::C, smem_raw);
}

template <int N, bool TR>
cudaError_t launch_stage_fx_visc_t(const StageArgs &args, cudaStream_t stream)
{
  using FS              = FxViscShape<N, TR>;
  constexpr auto kernel = stage_fx_visc_kernel<N, TR>;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t                            e = opt_in_smem(kernel, FS::SMEM, configured);
  if (e != cudaSuccess)
    return e;
  const long long blocks = (args.n_cells - args.cell_begin + FS::C - 1) / FS::C;
  kernel<<<(unsigned)blocks, FS::THREADS, FS::SMEM, stream>>>(args);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_stage_fx_visc_n(const StageArgs &args, cudaStream_t stream)
{
  return args.tr_in ? launch_stage_fx_visc_t<N, true>(args, stream) : launch_stage_fx_visc_t<N, false>(args, stream);
}
} // namespace adv
