// Collocation-form stage of the FP64 advection operator in block fixed-point
// arithmetic (fixed.cuh).
//
// The mathematics, data layout and outputs are those of stage_gauss_cta
// (stage_gauss.cuh) with a binary64 operator; the volume and lift
// contractions of the three direction passes, which were 75 % of its FP64
// instructions, run on the integer pipes.  Per cell: the largest |U| and the
// largest face flux give the power of two of the block, U is converted once
// to limb pairs in shared memory, each pass multiplies its pencil with vt
// (mantissa products), contracts it with Dw and the lifts, and adds 64-bit
// integers into Z, which becomes binary64 again once, in the Runge-Kutta
// update.  Face values, fluxes, 1 / det J, the update and the next face
// traces stay binary64.
//
// Bound: the latency of the two dependent reads of a CTA (coefficients, then
// the upwind traces), then the FP64 pipe (9 instead of 27 instructions per
// point: fluxes, 1 / det J, update, traces) and HBM; the geometry comes by
// cp.async behind the fluxes and the solution ahead of the last pass.
// Measured on GB300 against the binary64 kernel: 64^3 curved cells of degree
// 4, LSRK(5,4): 16.6 instead of 36.1 ms per 4 steps (with both changes of
// basis); 29 x 23 x 37 affine cells of degree 2, 4 steps of the 7-stage scheme:
// 0.69 instead of 1.94 ms; 512 affine cells of degree 3, one step: 56 instead
// of 76 us.
//
// Cells whose block leaves the safe window of exponents (infinities, NaN,
// magnitudes outside about 2^-400 .. 2^600) are left out here and computed
// by the binary64 path afterwards, cell by cell, so that a cell's result
// does not depend on its neighbours in the CTA.
#pragma once

#include "fixed.cuh"
#include "stage_gauss.cuh"

namespace adv
{
template <int N, bool UNI, bool TR>
struct FxShape
{
  using SH                     = StageShape<N, double, UNI, false>;
  static constexpr int C       = SH::C;
  static constexpr int THREADS = SH::THREADS;
  static_assert(C * N * N <= THREADS && C <= 32, "one pencil per thread and a bit per cell");
  // U and Z [C][NQ], field geometry [C][4][NQ], the block maxima and the mask
  static constexpr int OWN  = (UNI ? 2 : 6) * C * N * N * N * 8 + (2 * C + 1) * 4;
  static constexpr int BIN  = GaussShape<N, double, UNI, false, TR>::SMEM;
  static constexpr int SMEM = OWN > BIN ? OWN : BIN;
  static_assert(2 * C * N * N * N * 8 % 16 == 0, "cp.async destinations need 16-byte alignment");
};

// the binary64 path for the cells of `mask`
template <int N, bool UNI, bool TR, bool INC, bool UPW>
__device__ __noinline__ void stage_gauss_masked(const StageArgs &A, long long cell0, unsigned char *smem,
                                                unsigned mask)
{
  stage_gauss_cta<N, double, UNI, false, TR, INC, UPW>(A, cell0, smem, mask);
}

template <int N, bool UNI, bool TR, bool INC, bool UPW>
__device__ __forceinline__ void stage_fx_cta(const StageArgs &A, const long long cell0, unsigned char *smem_raw)
{
  using FS         = FxShape<N, UNI, TR>;
  constexpr int C  = FS::C;
  constexpr int NQ = N * N * N;
  constexpr int NF = N * N;
  constexpr int NT = FS::THREADS;
  static_assert(!UPW || (TR && !UNI), "upwind traces are written on field geometry");
  int2      *Ub    = reinterpret_cast<int2 *>(smem_raw);         // [C][NQ] U: binary64, then limbs
  long long *Qb    = reinterpret_cast<long long *>(Ub + C * NQ); // [C][NQ] Z, then the next input
  double    *Gb    = reinterpret_cast<double *>(Qb + C * NQ);    // field: [C][4][NQ] geometry
  unsigned  *s_eu = reinterpret_cast<unsigned *>(Gb + (UNI ? 0 : 4 * C * NQ)), *s_ef = s_eu + C, *s_bad = s_ef + C;

  const DevTables<double> &tb    = tab<double>(N);
  const FxTables          &fx    = c_tab_fx[N];
  const int                tid   = threadIdx.x;
  const int                ncell = (int)min((long long)C, A.n_cells - cell0);
  const bool               mine  = tid < ncell * NF;
  const int                cl    = tid / NF, r = tid % NF;
  const int                offy  = (r % N) + NF * (r / N);
  const double            *tr_in = static_cast<const double *>(A.tr_in);

  // the cells' geometry, one contiguous range, while the fluxes are formed
  if (!UNI)
    {
      const char *geo = reinterpret_cast<const char *>(static_cast<const double *>(A.cell_geo) + cell0 * 4 * NQ);
      for (int i = tid; i < ncell * 2 * NQ; i += NT)
        __pipeline_memcpy_async(reinterpret_cast<char *>(Gb) + 16 * i, geo + 16 * i, 16);
      __pipeline_commit();
    }
  double U[N]; // the z pencil
  if (mine)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        U[k] = __ldg(A.r_in + (cell0 + cl) * NQ + r + k * NF);
    }
  if (tid < C)
    s_eu[tid] = s_ef[tid] = 0u;
  if (tid == 0)
    *s_bad = 0u;
  // face coefficients and where the pencil's six face values are
  int      nb[6];
  unsigned face[6];
  double   P[6], M[6];
  if (mine)
    {
      const unsigned c = (unsigned)(cell0 + cl), nx = A.nc[0], ny = A.nc[1];
      const unsigned row = c / nx;
      const int      ix = (int)(c - row * nx), iz = (int)(row / ny), iy = (int)(row - (unsigned)iz * ny);
#pragma unroll
      for (int j = 0; j < 6; ++j)
        {
          cell_face(A, ix, iy, iz, j, nb[j], face[j]);
          if (UNI)
            P[j] = A.P[j >> 1], M[j] = A.M[j >> 1];
          else
            {
              const double *fg = static_cast<const double *>(A.face_geo[j >> 1]);
              const double2 pm = __ldg(reinterpret_cast<const double2 *>(fg + ((size_t)face[j] * NF + r) * 2));
              P[j] = pm.x, M[j] = pm.y;
            }
          if (A.swap_pm)
            {
              const double tmp = P[j];
              P[j] = M[j], M[j] = tmp;
            }
        }
    }
  if (!TR)
    {
      if (mine)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            reinterpret_cast<double *>(Ub)[cl * NQ + r + k * NF] = U[k];
        }
    }
  __syncthreads();

  // ---- face fluxes at the pencil's six face points, binary64
  double   F[6];
  unsigned own = 0; // upwind traces: bit j: the own trace of face j is read
  if (mine)
    {
      unsigned mf = 0, mu = 0;
      // Dirichlet data of face j
      auto boundary = [&](int j) -> double {
        if (!A.bc_exact)
          return 0.0;
        const double *x = A.face_x[j >> 1] + ((size_t)face[j] * NF + r) * 3;
        return exact_value(A.ex, x[0], x[1], x[2], A.t);
      };
      if (UPW)
        {
          // one read per face point: the trace on the side whose coefficient
          // is not zero (the own side: M of a low face, P of a high one)
#pragma unroll
          for (int j = 0; j < 6; ++j)
            {
              const bool      mine_j = nonzero((j & 1) ? P[j] : M[j]);
              const long long c      = mine_j || nb[j] < 0 ? cell0 + cl : (long long)nb[j];
              own |= mine_j ? 1u << j : 0u;
              F[j] = __ldg(tr_in + (c * 6 + (mine_j || nb[j] < 0 ? j : j ^ 1)) * NF + r);
            }
#pragma unroll
          for (int j = 0; j < 6; ++j)
            {
              if (nb[j] < 0 && !((own >> j) & 1))
                F[j] = boundary(j);
              F[j] = or_bits(P[j], M[j]) * F[j];
            }
        }
      else
        {
          double uo[6], un[6];
#pragma unroll
          for (int j = 0; j < 6; ++j)
            {
              const int     d  = j >> 1;
              const int     st = d == 0 ? 1 : d == 1 ? N : NF;
              const int     at = d == 0 ? N * r : d == 1 ? offy : r;
              if (TR)
                {
                  uo[j] = __ldg(tr_in + ((cell0 + cl) * 6 + j) * NF + r);
                  un[j] = nb[j] < 0 ? boundary(j) : __ldg(tr_in + ((long long)nb[j] * 6 + (j ^ 1)) * NF + r);
                }
              else
                {
                  // contractions of the own pencil and of the neighbour's, in
                  // the order the traces are formed in
                  const double *p  = reinterpret_cast<const double *>(Ub) + cl * NQ + at;
                  const double *lo = (j & 1) ? tb.l1 : tb.l0, *ln = (j & 1) ? tb.l0 : tb.l1;
                  double        v[N];
                  if (nb[j] >= 0)
                    {
#pragma unroll
                      for (int q = 0; q < N; ++q)
                        v[q] = __ldg(A.r_in + (long long)nb[j] * NQ + at + q * st);
                    }
                  uo[j] = lo[0] * p[0];
#pragma unroll
                  for (int q = 1; q < N; ++q)
                    uo[j] = fma(lo[q], p[q * st], uo[j]);
                  if (nb[j] < 0)
                    un[j] = boundary(j);
                  else
                    {
                      un[j] = ln[0] * v[0];
#pragma unroll
                      for (int q = 1; q < N; ++q)
                        un[j] = fma(ln[q], v[q], un[j]);
                    }
                }
            }
          // as direction_pass_pm: low face M u_own + P u_nbr, high face
          // -(P u_own + M u_nbr)
#pragma unroll
          for (int j = 0; j < 6; ++j)
            F[j] = (j & 1) ? fma(P[j], uo[j], M[j] * un[j]) : fma(M[j], uo[j], P[j] * un[j]);
        }
#pragma unroll
      for (int j = 0; j < 6; ++j)
        {
          if (j & 1)
            F[j] = -F[j];
          mf = max(mf, abs_hi(F[j]));
        }
#pragma unroll
      for (int k = 0; k < N; ++k)
        mu = max(mu, abs_hi(U[k]));
      atomicMax(s_eu + cl, mu);
      atomicMax(s_ef + cl, mf);
    }
  __syncthreads();

  // ---- the block's scale: biased exponents of the tops of U, vt U and Z
  Limbs f[6], cv[3];
  bool  live = mine;
  int   topv = 0, topz = 0, dz = 0;
  if (mine)
    {
      const unsigned mu = s_eu[cl], mf = s_ef[cl];
      const int      eu = (int)(mu >> 20), ef = (int)(mf >> 20);
      if (UNI)
        topv = (int)(max(max(abs_hi(A.cv[0]), abs_hi(A.cv[1])), abs_hi(A.cv[2])) >> 20);
      else
        topv = A.cell_exp[cell0 + cl];
      const bool zero = (mu | mf) == 0;
      topz            = zero ? 1023 : max(eu + topv - 1022, ef);
      live            = eu < 1623 && ef < 1623 && topz > 623;
      if (!live && r == 0)
        atomicOr(s_bad, 1u << cl);
      const int topu = max(eu, topz - topv + 1022 - 64);
      dz             = topz - (topu + topv - 1022);
      if (live)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            {
              const Limbs x                = fx_from_double(U[k], topu);
              Ub[cl * NQ + r + k * NF]     = make_int2(x.h, x.l);
            }
#pragma unroll
          for (int j = 0; j < 6; ++j)
            f[j] = fx_from_double(F[j], topz);
          if (UNI)
            {
#pragma unroll
              for (int d = 0; d < 3; ++d)
                cv[d] = fx_from_double(A.cv[d], topv);
            }
        }
    }
  if (!UNI)
    __pipeline_wait_prior(0);
  __syncthreads();

  // one direction pass: the pencil at p (stride st) with vt at v (stride st)
  auto pass = [&](const int2 *p, int st, const double *v, const Limbs &c, const Limbs &flo, const Limbs &fhi,
                  long long(&out)[N]) {
    Limbs V[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      {
        const int2 u = p[k * st];
        Limbs      X;
        X.h = u.x, X.l = u.y;
        V[k] = UNI ? fx_times(X, c, min(dz, 63)) : fx_times_double(X, v[k * st], topv + dz);
      }
    fx_sweep_lift<N>(fx, V, flo, fhi, out);
  };
  const double *G = Gb + cl * 4 * NQ;

  // ---- x, y and z terms
  long long out[N];
  if (live)
    {
      const int off = cl * NQ + N * r;
      pass(Ub + off, 1, G + N * r, cv[0], f[0], f[1], out);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[off + k] = out[k];
    }
  __syncthreads();
  if (live)
    {
      const int off = cl * NQ + offy;
      pass(Ub + off, N, G + NQ + offy, cv[1], f[2], f[3], out);
#pragma unroll
      for (int k = 0; k < N; ++k)
        Qb[off + k * N] += out[k];
    }
  // the update's read of the solution ahead of the last pass
  const long long gb        = (cell0 + cl) * NQ + r;
  const bool      reads_u   = !INC && (A.mode == kModeStage || A.mode == kModeLastStage) && (TR || A.u_in);
  double          ui[N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    ui[k] = live && reads_u ? __ldcs(A.u_in + gb + k * NF) : 0.0;
  __syncthreads();
  if (live)
    {
      const int off = cl * NQ + r;
      pass(Ub + off, NF, G + 2 * NQ + r, cv[2], f[4], f[5], out);
      // Z = integer x 2^(topz - 1022 - 57 + kd - guard), times 1 / det J
      const int ez = topz - 1022 - 57 + fx_kd<N>() - kFxGuard;
      double          next[N];
#pragma unroll
      for (int k = 0; k < N; ++k)
        {
          const double    zi = fx_to_double(Qb[off + k * NF] + out[k], ez);
          const long long gi = gb + k * NF;
          if (!TR && !INC && A.mode == kModeVmult)
            {
              // implicit operator in weak form: JxW (c U - bracket), as stage_gauss_cta
              const double wq = tb.gw[r % N] * tb.gw[r / N] * tb.gw[k];
              const double br = A.out_scale * zi, u = __ldg(A.r_in + gi);
              A.r_out[gi]     = UNI ? wq * A.vol * (A.mass_factor * u - br)
                                    : wq * (A.mass_factor * u / G[3 * NQ + r + k * NF] - br);
              next[k]         = 0.0;
              continue;
            }
          const double kd = UNI ? zi : zi * G[3 * NQ + r + k * NF];
          if (INC)
            {
              // the FP32 increments' FP64 anchor: K0 and the first G
              A.k_out[gi]   = kd;
              A.k_out32[gi] = d2f_int(kd);
              A.r_out32[gi] = d2f_int(A.a * kd);
              next[k]       = 0.0;
            }
          else if (A.mode == kModeStage)
            {
              const double kk = !TR && A.k_add ? kd + __ldcs(A.k_add + gi) : kd;
              next[k]         = fma(A.a, kk, ui[k]);
              A.u_out[gi]     = fma(A.b, kk, ui[k]);
              A.r_out[gi]     = next[k];
              if (!TR && A.k_out)
                A.k_out[gi] = kk;
            }
          else if (A.mode == kModeLastStage)
            {
              const double kk = !TR && A.k_add ? kd + __ldcs(A.k_add + gi) : kd;
              next[k]         = fma(A.b, kk, ui[k]);
              if (!TR && A.u_base)
                next[k] += A.u_base[gi];
              A.u_out[gi] = next[k];
            }
          else
            {
              A.r_out[gi] = A.out_scale * kd;
              next[k]     = 0.0;
            }
        }
      if (TR && !INC && A.tr_out)
        {
          double *to = static_cast<double *>(A.tr_out) + ((cell0 + cl) * 6 + 4) * NF + r, lo, hi;
          if (UPW)
            {
              if (upwind_pencil_traces<N, double>(tb, next, (own >> 4) & 1, (own >> 5) & 1, to, to + NF))
                {
                  pencil_traces<N, double>(tb, next, lo, hi);
                  to[NF] = hi;
                }
            }
          else
            {
              pencil_traces<N, double>(tb, next, lo, hi);
              to[0]  = lo;
              to[NF] = hi;
            }
#pragma unroll
          for (int k = 0; k < N; ++k)
            Qb[off + k * NF] = __double_as_longlong(next[k]);
        }
    }
  if (TR && !INC && A.tr_out)
    {
      __syncthreads();
      if (live)
        {
#pragma unroll 1
          for (int d = 0; d < 2; ++d)
            {
              const long long *p  = Qb + cl * NQ + (d == 0 ? N * r : offy);
              const int        st = d == 0 ? 1 : N;
              double           x[N], lo, hi;
#pragma unroll
              for (int k = 0; k < N; ++k)
                x[k] = __longlong_as_double(p[k * st]);
              double *to = static_cast<double *>(A.tr_out) + ((cell0 + cl) * 6 + 2 * d) * NF + r;
              if (UPW)
                {
                  if (upwind_pencil_traces<N, double>(tb, x, (own >> (2 * d)) & 1, (own >> (2 * d + 1)) & 1, to, to + NF))
                    {
                      pencil_traces<N, double>(tb, x, lo, hi);
                      to[NF] = hi;
                    }
                }
              else
                {
                  pencil_traces<N, double>(tb, x, lo, hi);
                  to[0]  = lo;
                  to[NF] = hi;
                }
            }
        }
    }
  // ---- cells outside the window
  const unsigned bad = *s_bad;
  if (bad)
    {
      __syncthreads();
      stage_gauss_masked<N, UNI, TR, INC, UPW>(A, cell0, smem_raw, bad);
    }
}

template <int N, bool UNI, bool TR, bool INC, bool UPW>
__global__ void __launch_bounds__(FxShape<N, UNI, TR>::THREADS, kFxThreadsPerSM / FxShape<N, UNI, TR>::THREADS)
  stage_fx_kernel(const __grid_constant__ StageArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_fx_cta<N, UNI, TR, INC, UPW>(A, A.cell_begin + (long long)blockIdx.x * FxShape<N, UNI, TR>::C, smem_raw);
}

template <int N, bool UNI, bool TR, bool INC = false, bool UPW = false>
cudaError_t launch_stage_fx_t(const StageArgs &args, cudaStream_t stream)
{
  using FS              = FxShape<N, UNI, TR>;
  constexpr auto kernel = stage_fx_kernel<N, UNI, TR, INC, UPW>;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t                            e = opt_in_smem(kernel, FS::SMEM, configured);
  if (e != cudaSuccess)
    return e;
  const long long blocks = (args.n_cells - args.cell_begin + FS::C - 1) / FS::C;
  kernel<<<(unsigned)blocks, FS::THREADS, FS::SMEM, stream>>>(args);
  return cudaGetLastError();
}

// Advection stages without a skew term; fx_ok: vt and 1 / det J within
// 2^+-200 (checked when the geometry is built)
template <int N>
cudaError_t launch_stage_fx_n(const StageArgs &args, cudaStream_t stream)
{
  if (args.tr_in)
    {
      if (args.uniform)
        return launch_stage_fx_t<N, true, true>(args, stream);
      if (args.inc32)
        return args.upwind_tr ? launch_stage_fx_t<N, false, true, true, true>(args, stream)
                              : launch_stage_fx_t<N, false, true, true>(args, stream);
      return args.upwind_tr ? launch_stage_fx_t<N, false, true, false, true>(args, stream)
                            : launch_stage_fx_t<N, false, true>(args, stream);
    }
  if (args.inc32)
    return args.uniform ? launch_stage_fx_t<N, true, false, true>(args, stream)
                        : launch_stage_fx_t<N, false, false, true>(args, stream);
  return args.uniform ? launch_stage_fx_t<N, true, false>(args, stream)
                      : launch_stage_fx_t<N, false, false>(args, stream);
}
} // namespace adv
