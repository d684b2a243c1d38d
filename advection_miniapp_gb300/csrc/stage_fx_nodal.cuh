// Nodal (Gauss-Lobatto) stage of the FP64 advection operator in block
// fixed-point arithmetic (fixed.cuh): the counterpart of stage_cta
// (stage_kernel.cuh) with a binary64 operator and no diffusion or skew term,
// for apply, perform_stage, the weak-form vmult and the nodal step loop.
//
// Every contraction of the binary64 kernel (three sweeps of S, two sweeps of S
// over six neighbour face layers, the face values, three volume passes with
// lifts, three sweeps of S^-1 or S^T; 8.3 k FP64 instructions per cell at degree 4)
// runs on the integer pipes.  Blocks and their scales: the cell's nodal
// values; each neighbour face layer by itself; the cell's fluxes with vt U (as
// stage_fx_cta); the cell's result before S^-1.  Face values become binary64
// for the flux, Z for 1 / det J, and the result for the update.
// Bound: integer issue (48 % of the slots) and the latencies between its
// eleven barriers at six resident CTAs (degree 4).  Measured on GB300 against
// the binary64 kernel: five perform_stage calls on 32^3 curved cells of degree 4
// 0.91 instead of 2.92 ms, apply on 17 x 13 x 11 curved cells of degree 6 146 instead
// of 268 us; with the binary64 path's staged face coefficients in the same shared
// memory (four CTAs, one at degree 6) 1.01 ms and 172 us.
// A cell with a block outside the window of exponents is left to the binary64
// kernel afterwards, cell by cell.
#pragma once

#include "fixed_basis.cuh"
#include "stage_kernel.cuh"

namespace adv
{
template <int N, bool UNI>
struct FxNodalShape
{
  using SH                     = StageShape<N, double, UNI, false>;
  static constexpr int C       = SH::C;
  static constexpr int THREADS = SH::THREADS;
  static constexpr int ROWS    = (6 * C * N + THREADS - 1) / THREADS; // neighbour rows per thread
  // U, Z [C][NQ], neighbour layers [C][6][NF], geometry [C][4][NQ], the block
  // maxima (cell, layers, flux, result), neighbours and faces, the mask
  static constexpr int OWN = ((UNI ? 2 : 6) * C * N * N * N + 6 * C * N * N) * 8 + (4 * C + 6 * C + 12 * C + 1) * 4;
  // the binary64 path without staged face coefficients
  static constexpr int BIN  = SH::SMEM - (UNI ? 0 : 12 * C * N * N * 8);
  static constexpr int SMEM = OWN > BIN ? OWN : BIN;
  static_assert((2 * C * N * N * N + 6 * C * N * N) % 2 == 0, "cp.async destinations need 16-byte alignment");
};

// the binary64 path for the cells of `mask`
template <int N, bool UNI>
__device__ __noinline__ void stage_nodal_masked(const StageArgs &A, long long cell0, unsigned char *smem, unsigned mask)
{
  stage_cta<N, double, UNI, false, !UNI>(A, cell0, smem, mask);
}

template <int N, bool UNI>
__device__ __forceinline__ void stage_fx_nodal_cta(const StageArgs &A, const long long cell0, unsigned char *smem_raw)
{
  using FS         = FxNodalShape<N, UNI>;
  constexpr int C  = FS::C;
  constexpr int NQ = N * N * N;
  constexpr int NF = N * N;
  constexpr int NT = FS::THREADS;
  int2      *Ub    = reinterpret_cast<int2 *>(smem_raw);         // [C][NQ] U: binary64, then limbs; result limbs
  long long *Qb    = reinterpret_cast<long long *>(Ub + C * NQ); // [C][NQ] Z
  double    *Nb    = reinterpret_cast<double *>(Qb + C * NQ);    // [C][6][NF] neighbour layers: limbs, binary64
  double    *Gb    = Nb + 6 * C * NF;                            // field: [C][4][NQ] geometry
  unsigned  *s_eu = reinterpret_cast<unsigned *>(Gb + (UNI ? 0 : 4 * C * NQ)), *s_ef = s_eu + C, *s_ez = s_ef + C;
  unsigned  *s_e3 = s_ez + C, *s_en = s_e3 + C; // [C], [C][6]
  int       *s_nbr = reinterpret_cast<int *>(s_en + 6 * C), *s_face = s_nbr + 6 * C;
  unsigned  *s_bad = reinterpret_cast<unsigned *>(s_face + 6 * C);

  const DevTables<double> &tb    = tab<double>(N);
  const FxTables          &fx    = c_tab_fx[N];
  const FxBasisTables     &fxb   = c_tab_fxb[N];
  const int                tid   = threadIdx.x;
  const int                ncell = (int)min((long long)C, A.n_cells - cell0);
  const bool               mine  = tid < ncell * NF;
  const int                cl = tid / NF, r = tid % NF;
  const int                ox = cl * NQ + N * r, oy = cl * NQ + (r % N) + NF * (r / N), oz = cl * NQ + r;
  const long long          gb = (cell0 + cl) * NQ + r;

  // ---- loads: geometry by cp.async, the own z pencil, later the rows of the
  //      neighbours' face layers
  if (!UNI)
    {
      const char *geo = reinterpret_cast<const char *>(static_cast<const double *>(A.cell_geo) + cell0 * 4 * NQ);
      for (int i = tid; i < ncell * 2 * NQ; i += NT)
        __pipeline_memcpy_async(reinterpret_cast<char *>(Gb) + 16 * i, geo + 16 * i, 16);
      __pipeline_commit();
    }
  double x[N];
  if (mine)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        x[k] = __ldg(A.r_in + gb + k * NF);
    }
  for (int i = tid; i < 10 * C; i += NT)
    s_eu[i] = 0u;
  if (tid == 0)
    *s_bad = 0u;
  cell_neighbours(A, cell0, ncell, s_nbr, s_face, tid, NT);
  __syncthreads();

  // row i of the neighbour layers: face cf = i / N, position b = i % N along
  // the second tangential direction; the layer next to the shared face
  double rows[FS::ROWS][N];
#pragma unroll
  for (int q = 0; q < FS::ROWS; ++q)
    {
      const int i = tid + q * NT, cf = i / N, b = i % N;
      if (i < ncell * 6 * N && s_nbr[cf] >= 0)
        {
          const int     j = cf % 6, d = j >> 1, layer = (j & 1) ? 0 : N - 1;
          const int     base   = d == 0 ? layer + NF * b : d == 1 ? N * layer + NF * b : N * b + NF * layer;
          const double *g      = A.r_in + (long long)s_nbr[cf] * NQ + base;
#pragma unroll
          for (int a = 0; a < N; ++a)
            rows[q][a] = __ldg(g + a * (d == 0 ? N : 1));
          atomicMax(s_en + cf, fx_magnitude(rows[q]));
        }
    }
  if (mine)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        reinterpret_cast<double *>(Ub)[oz + k * NF] = x[k];
      atomicMax(s_eu + cl, fx_magnitude(x));
    }
  __syncthreads();

  Limbs     X[N];
  long long T[N];
  auto      load = [&](const int2 *p, int st) {
#pragma unroll
    for (int k = 0; k < N; ++k)
      X[k].h = p[k * st].x, X[k].l = p[k * st].y;
  };
  auto store = [&](int2 *p, int st) {
#pragma unroll
    for (int k = 0; k < N; ++k)
      {
        const Limbs l = fx_split(T[k]);
        p[k * st]     = make_int2(l.h, l.l);
      }
  };

  // ---- S along x (own cell) and along the layers' first tangential direction
  int  top  = 1023;
  bool live = mine && fx_window(s_eu[cl], top);
  // (values of magnitude 0 that are not zero: the binary64 path)
  if (live && s_eu[cl] == 0u && fx_subnormal(x))
    atomicOr(s_bad, 1u << cl);
  if (live)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        X[k] = fx_from_double(reinterpret_cast<const double *>(Ub)[ox + k], top);
      fx_sweep_sym<N>(fxb.S, X, T);
      store(Ub + ox, 1);
    }
  else if (mine && r == 0)
    atomicOr(s_bad, 1u << cl);
  int2 *Nl = reinterpret_cast<int2 *>(Nb);
#pragma unroll
  for (int q = 0; q < FS::ROWS; ++q)
    {
      const int i = tid + q * NT, cf = i / N, b = i % N;
      if (i < ncell * 6 * N && s_nbr[cf] >= 0)
        {
          int topn;
          const bool in = fx_window(s_en[cf], topn);
          if (s_en[cf] == 0u ? fx_subnormal(rows[q]) : !in && b == 0)
            atomicOr(s_bad, 1u << (cf / 6));
          if (!in)
            continue;
#pragma unroll
          for (int a = 0; a < N; ++a)
            X[a] = fx_from_double(rows[q][a], topn);
          fx_sweep_sym<N>(fxb.S, X, T);
          store(Nl + cf * NF + N * b, 1);
        }
    }
  __syncthreads();

  // ---- S along y; the layers' second tangential direction, or Dirichlet data
  if (live)
    {
      load(Ub + oy, N);
      fx_sweep_sym<N>(fxb.S, X, T);
      store(Ub + oy, N);
    }
#pragma unroll 1
  for (int i = tid; i < ncell * 6 * N; i += NT)
    {
      const int cf = i / N, b = i % N;
      double   *p  = Nb + cf * NF + b;
      if (s_nbr[cf] >= 0)
        {
          int topn;
          fx_window(s_en[cf], topn);
          load(Nl + cf * NF + b, N);
          fx_sweep_sym<N>(fxb.S, X, T);
#pragma unroll
          for (int k = 0; k < N; ++k)
            p[k * N] = fx_to_double(T[k], topn - 1022 - 58);
        }
      else
        {
          const int d = (cf % 6) >> 1;
          for (int k = 0; k < N; ++k)
            {
              double g = 0.0;
              if (A.bc_exact)
                {
                  const double *fxp = d == 0 ? A.face_x[0] : d == 1 ? A.face_x[1] : A.face_x[2];
                  const double *xp  = fxp + ((size_t)s_face[cf] * NF + b + N * k) * 3;
                  g                 = exact_value(A.ex, xp[0], xp[1], xp[2], A.t);
                }
              p[k * N] = g;
            }
        }
    }
  __syncthreads();

  // a cell with a layer outside the window is left to the binary64 path
  live = live && !((*s_bad >> cl) & 1u);

  // ---- S along z: U at the Gauss points, limbs in units of 2^(top3 - 1079)
  //      with top3 from the largest |U| (the bound of the three sweeps would
  //      cost up to 3 bits)
  if (live)
    {
      load(Ub + oz, NF);
      fx_sweep_sym<N>(fxb.S, X, T);
      unsigned m = 0;
#pragma unroll
      for (int k = 0; k < N; ++k)
        m = max(m, (unsigned)(fx_abs(T[k]) >> 32));
      atomicMax(s_e3 + cl, m);
    }
  __syncthreads();
  int top3 = top;
  if (live)
    {
      const int sh = 6 - __clz((int)s_e3[cl]); // |T| = 2 |X| < 2^(64 - clz) -> 2^58
      top3 += sh;
#pragma unroll
      for (int k = 0; k < N; ++k)
        T[k] = sh > 0 ? (T[k] + (1ll << (sh - 1))) >> sh : T[k] << -sh;
      store(Ub + oz, NF);
    }
  __syncthreads();

  // ---- fluxes at the pencil's six face points
  double F[6];
  if (live)
    {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        {
          load(Ub + (d == 0 ? ox : d == 1 ? oy : oz), d == 0 ? 1 : d == 1 ? N : NF);
          FxAcc<2> lo, hi;
          lo.set(X[0].h, X[0].l, fxb.l0[0]);
          hi.set(X[0].h, X[0].l, fxb.l1[0]);
#pragma unroll
          for (int q = 1; q < N; ++q)
            {
              lo.add(X[q].h, X[q].l, fxb.l0[q]);
              hi.add(X[q].h, X[q].l, fxb.l1[q]);
            }
          // l is tabulated as c 2^56: the sums are in units of X
          const double uo[2] = {fx_to_double(lo.value(), top3 - 1022 - 57), fx_to_double(hi.value(), top3 - 1022 - 57)};
#pragma unroll
          for (int s = 0; s < 2; ++s)
            {
              const int cf = cl * 6 + 2 * d + s;
              double    P, M;
              if (UNI)
                P = A.P[d], M = A.M[d];
              else
                {
                  const double *fg = static_cast<const double *>(A.face_geo[d]);
                  const double2 pm = __ldg(reinterpret_cast<const double2 *>(fg + ((size_t)s_face[cf] * NF + r) * 2));
                  P = pm.x, M = pm.y;
                }
              if (A.swap_pm)
                {
                  const double tmp = P;
                  P = M, M = tmp;
                }
              const double un = Nb[cf * NF + r];
              F[2 * d + s]    = s ? -fma(P, uo[1], M * un) : fma(M, uo[0], P * un);
            }
        }
      atomicMax(s_ef + cl, fx_magnitude(F));
    }
  if (!UNI)
    __pipeline_wait_prior(0);
  __syncthreads();

  // ---- scale of vt U and the fluxes (as stage_fx_cta), direction passes
  int   topv = 0, topz = 0;
  Limbs f[6];
  int2  cv[3];
  int   dz = 0;
  bool  tiny = false;
  if (live)
    {
      topv = UNI ? (int)(max(max(abs_hi(A.cv[0]), abs_hi(A.cv[1])), abs_hi(A.cv[2])) >> 20) : A.cell_exp[cell0 + cl];
      const unsigned mf = s_ef[cl];
      const int      ef = (int)(mf >> 20);
      // (a cell of zeros takes its fluxes' scale)
      topz = s_eu[cl] ? max(top3 + topv - 1022, ef) : mf ? ef : 1023;
      if (ef >= kFxHigh || topz <= kFxLow)
        {
          live = false;
          if (r == 0)
            atomicOr(s_bad, 1u << cl);
        }
      tiny = mf == 0;
      if (tiny && fx_subnormal(F))
        atomicOr(s_bad, 1u << cl);
      dz = min(max(topz - (top3 + topv - 1022), 0), 63);
#pragma unroll
      for (int j = 0; j < 6; ++j)
        f[j] = fx_from_double(F[j], topz);
      if (UNI)
        {
#pragma unroll
          for (int d = 0; d < 3; ++d)
            cv[d] = fx_const58(A.cv[d], topv);
        }
    }
  const double *G    = Gb + cl * 4 * NQ;
  auto          pass = [&](const int2 *p, int st, const double *v, const int2 &c, const Limbs &flo, const Limbs &fhi) {
    load(p, st);
    Limbs V[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      V[k] = fx_times(X[k], UNI ? c : reinterpret_cast<const int2 *>(v)[k * st]);
    if (dz) // the fluxes set the scale: cells of zeros or beside much larger ones
      {
#pragma unroll
        for (int k = 0; k < N; ++k)
          V[k] = fx_split((2 * ((long long)V[k].h * (1 << 29) + V[k].l)) >> dz);
      }
    fx_sweep_lift<N>(fx, V, flo, fhi, T);
  };
  if (live)
    {
      pass(Ub + ox, 1, G + N * r, cv[0], f[0], f[1]);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[ox + k] = T[k];
    }
  __syncthreads();
  if (tiny)
    live = live && !((*s_bad >> cl) & 1u);
  if (live)
    {
      pass(Ub + oy, N, G + (oy - cl * NQ) + NQ, cv[1], f[2], f[3]);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[oy + k * N] += T[k];
    }
  __syncthreads();
  const bool weak = A.mode == kModeVmult;
  if (live)
    {
      pass(Ub + oz, NF, G + 2 * NQ + r, cv[2], f[4], f[5]);
      const int ez = topz - 1022 - 57 + fx_kd<N>() - kFxGuard;
#pragma unroll
      for (int k = 0; k < N; ++k)
        {
          const double z = fx_to_double(Qb[oz + k * NF] + T[k], ez);
          if (weak)
            {
              // implicit operator in weak form, JxW (c U - bracket), then S^T
              const double wq = tb.gw[r % N] * tb.gw[r / N] * tb.gw[k];
              const double br = A.out_scale * z;
              const double U  = fx_to_double((long long)X[k].h * (1 << 29) + X[k].l, top3 - 1022 - 57);
              x[k] = UNI ? wq * A.vol * (A.mass_factor * U - br) : wq * (A.mass_factor * U / G[3 * NQ + r + k * NF] - br);
            }
          else
            x[k] = UNI ? z : z * G[3 * NQ + r + k * NF];
        }
      atomicMax(s_ez + cl, fx_magnitude(x));
    }
  __syncthreads();

  // ---- S^-1 (or S^T) along x, y, z, from the result's own scale
  int topr = 1023;
  if (live && !fx_window(s_ez[cl], topr))
    {
      live = false;
      if (r == 0)
        atomicOr(s_bad, 1u << cl);
    }
  const FxEvenOdd &B = weak ? fxb.St : fxb.Si;
  if (live)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        {
          const Limbs l    = fx_from_double(x[k], topr);
          Ub[oz + k * NF] = make_int2(l.h, l.l);
        }
    }
  // the update's reads ahead of the last sweeps
  const bool upd = A.mode == kModeStage || A.mode == kModeLastStage;
  double     ui[N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    ui[k] = live && upd && A.u_in ? __ldcs(A.u_in + gb + k * NF) : 0.0;
  __syncthreads();
  if (live)
    {
      load(Ub + ox, 1);
      fx_sweep_sym<N>(B, X, T);
#pragma unroll
      for (int k = 0; k < N; ++k)
        T[k] = fx_shift<fx_si1<N>()>(T[k]);
      store(Ub + ox, 1);
    }
  __syncthreads();
  if (live)
    {
      load(Ub + oy, N);
      fx_sweep_sym<N>(B, X, T);
#pragma unroll
      for (int k = 0; k < N; ++k)
        T[k] = fx_shift<fx_si2<N>()>(T[k]);
      store(Ub + oy, N);
    }
  __syncthreads();
  if (live)
    {
      load(Ub + oz, NF);
      fx_sweep_sym<N>(B, X, T);
      const int er = topr - 1022 - 58 + fx_si1<N>() + fx_si2<N>();
#pragma unroll
      for (int k = 0; k < N; ++k)
        x[k] = fx_to_double(T[k], er);
      // (branches around whole loops, not predicated FP64 instructions)
      if (!upd)
        {
          if (!weak)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                x[k] *= A.out_scale;
            }
#pragma unroll
          for (int k = 0; k < N; ++k)
            A.r_out[gb + k * NF] = x[k];
        }
      else
        {
          if (A.k_add)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                x[k] += __ldcs(A.k_add + gb + k * NF);
            }
          double un[N];
#pragma unroll
          for (int k = 0; k < N; ++k)
            un[k] = fma(A.b, x[k], ui[k]);
          if (A.mode == kModeLastStage && A.u_base)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                un[k] += A.u_base[gb + k * NF];
            }
#pragma unroll
          for (int k = 0; k < N; ++k)
            A.u_out[gb + k * NF] = un[k];
          if (A.mode == kModeStage)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                A.r_out[gb + k * NF] = fma(A.a, x[k], ui[k]);
              if (A.k_out)
                {
#pragma unroll
                  for (int k = 0; k < N; ++k)
                    A.k_out[gb + k * NF] = x[k];
                }
            }
        }
    }
  // ---- cells outside the window
  __syncthreads();
  const unsigned bad = *s_bad;
  if (bad)
    {
      __syncthreads();
      stage_nodal_masked<N, UNI>(A, cell0, smem_raw, bad);
    }
}

template <int N, bool UNI>
__global__ void __launch_bounds__(FxNodalShape<N, UNI>::THREADS, kFxThreadsPerSM / FxNodalShape<N, UNI>::THREADS)
  stage_fx_nodal_kernel(const __grid_constant__ StageArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_fx_nodal_cta<N, UNI>(A, A.cell_begin + (long long)blockIdx.x * FxNodalShape<N, UNI>::C, smem_raw);
}

template <int N, bool UNI>
cudaError_t launch_stage_fx_nodal_t(const StageArgs &args, cudaStream_t stream)
{
  using FS              = FxNodalShape<N, UNI>;
  constexpr auto kernel = stage_fx_nodal_kernel<N, UNI>;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t                            e = opt_in_smem(kernel, FS::SMEM, configured);
  if (e != cudaSuccess)
    return e;
  const long long blocks = (args.n_cells - args.cell_begin + FS::C - 1) / FS::C;
  kernel<<<(unsigned)blocks, FS::THREADS, FS::SMEM, stream>>>(args);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_stage_fx_nodal_n(const StageArgs &args, cudaStream_t stream)
{
  return args.uniform ? launch_stage_fx_nodal_t<N, true>(args, stream)
                      : launch_stage_fx_nodal_t<N, false>(args, stream);
}
} // namespace adv
