// Collocation-form stage of the FP64 advection operator in block fixed-point
// arithmetic (fixed.cuh).
//
// The mathematics, data layout and outputs are those of stage_gauss_cta
// (stage_gauss.cuh) with a binary64 operator; the volume and lift
// contractions of the three direction passes, which were 75 % of its FP64
// instructions, run on the integer pipes, and so do the fluxes.  Per cell: the
// largest |U| and the largest face flux give the power of two of the block, U is
// converted once to limb pairs in shared memory, each pass multiplies its pencil
// with vt (stored as limbs), contracts it with Dw and the lifts, and adds 64-bit
// integers into Z, which becomes binary64 again once, in the Runge-Kutta
// update.  1 / det J, the update and the next face traces stay binary64.
//
// Bound: FP64 issue (6.5 instead of 27 instructions per point: 1 / det J,
// update, traces) and integer issue, both near 60 %, at 63 % of the HBM
// bandwidth on curved cells; the geometry comes by cp.async behind the fluxes and
// the solution ahead of the last pass.  Measured on GB300 against the binary64
// kernel: 64^3 curved cells of degree 4, LSRK(5,4): 12.6 instead of 36.1 ms per 4 steps
// (with both changes of basis); 37 x 23 x 29 affine cells of degree 2, 4 steps of the
// 7-stage scheme: 0.54 instead of 1.94 ms; 512 affine cells of degree 3, one step: 44
// instead of 76 us.  On the way (4 steps at 64^3): geometry read in the passes 25.6 ms,
// staged by cp.async with one trace read per face point 16.6, fluxes as integer
// products 13.8, no predicated FP64 code 12.6.
//
// Cells whose block leaves the safe window of exponents (infinities, NaN,
// magnitudes outside about 2^-722 .. 2^600) are left out here and computed
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
  static constexpr int BIN  = GaussShape<N, double, UNI, false, TR, !UNI>::SMEM;
  static constexpr int SMEM = OWN > BIN ? OWN : BIN;
  static_assert(2 * C * N * N * N * 8 % 16 == 0, "cp.async destinations need 16-byte alignment");
};

// the binary64 path for the cells of `mask`
template <int N, bool UNI, bool TR, bool UPW>
__device__ __noinline__ void stage_gauss_masked(const StageArgs &A, long long cell0, unsigned char *smem,
                                                unsigned mask)
{
  stage_gauss_cta<N, double, UNI, false, TR, false, UPW, !UNI>(A, cell0, smem, mask);
}

// The traces of a pencil x that the next stage reads: at the low face if bit 0
// of `own` is set, at the high face if bit 1 is.  A loop, so that one chain
// serves lanes with either face and a second one runs only in warps that
// have a pencil with both (as predicated code both would issue on the FP64 pipe).
template <int N>
__device__ __forceinline__ void write_traces(const DevTables<double> &tb, const double (&x)[N], unsigned own, double *to)
{
#pragma unroll 1
  for (int s = own & 1u ? 0 : 1; s < (own & 2u ? 2 : 1); ++s)
    {
      const double *l = s ? tb.l1 : tb.l0;
      double        h = l[0] * x[0];
#pragma unroll
      for (int q = 1; q < N; ++q)
        h = fma(l[q], x[q], h);
      to[s * N * N] = h;
    }
}

// Dirichlet data at face point r of a face normal to d (out of line: rare, and
// long with the exact solution)
static __device__ __noinline__ double boundary_value(const StageArgs &A, int d, unsigned face, int r, int nf)
{
  if (!A.bc_exact)
    return 0.0;
  const double *x = (d == 0 ? A.face_x[0] : d == 1 ? A.face_x[1] : A.face_x[2]) + ((size_t)face * nf + r) * 3;
  return exact_value(A.ex, x[0], x[1], x[2], A.t);
}

// LATE: low words are looked at only in blocks of magnitude 0, after the scale, and
// the mask of cells left out is read again; else they join the maximum of every
// block.  The first for the uniform launches of one mesh (a stage on 512 cells of
// degree 3 6.4 us, 6.8 with the second form, 6.4 without the check), the second for
// field geometry (64^3 curved cells of degree 4, 4 steps 12.62 ms, 12.65 with
// the first, 12.61 without) and the batched launches (a burst of 16 requests
// 48.3 ms, 49.3-50.3 with the first, which spills at 7 points, 48.4 without).
template <int N, bool UNI, bool TR, bool UPW, bool LATE = false>
__device__ __forceinline__ void stage_fx_cta(const StageArgs &A, const long long cell0, unsigned char *smem_raw)
{
  using FS         = FxShape<N, UNI, TR>;
  constexpr int C  = FS::C;
  constexpr int NQ = N * N * N;
  constexpr int NF = N * N;
  constexpr int NT = FS::THREADS;
  static_assert(!UPW || (TR && !UNI), "upwind traces are written on field geometry");
  int2      *Ub    = reinterpret_cast<int2 *>(smem_raw);         // [C][NQ] U as limbs
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
  __syncthreads();

  // ---- face fluxes at the pencil's six face points as pairs of factors
  //      c v: where one of P, M is zero (upwind flux) the other times the value
  //      on its side, formed in fixed point below; else 1 times the binary64 flux.
  //      Low face M u_own + P u_nbr, high face -(P u_own + M u_nbr).
  double   fc[6], fv[6];
  unsigned own = 0; // bit j: the own trace of face j is read
  if (mine)
    {
      unsigned mf = 0;
      // coefficients of the own and the neighbour's value at face j
      auto co = [&](int j) { return (j & 1) ? P[j] : M[j]; };
      auto cn = [&](int j) { return (j & 1) ? M[j] : P[j]; };
      // value of cell c on its side of face j: its trace, or the contraction
      // of its pencil in the order the traces are formed in
      auto face_value = [&](long long c, bool self, int j) -> double {
        if (TR)
          return __ldg(tr_in + (c * 6 + (self ? j : j ^ 1)) * NF + r);
        const int     st = j < 2 ? 1 : j < 4 ? N : NF;
        const double *g  = A.r_in + c * NQ + (j < 2 ? N * r : j < 4 ? offy : r);
        const double *l  = self == (bool)(j & 1) ? tb.l1 : tb.l0;
        double        v[N], u;
#pragma unroll
        for (int q = 0; q < N; ++q)
          v[q] = __ldg(g + q * st);
        u = l[0] * v[0];
#pragma unroll
        for (int q = 1; q < N; ++q)
          u = fma(l[q], v[q], u);
        return u;
      };
      // one value per face point: the side whose coefficient is not zero
      unsigned two = 0, edge = 0; // faces that need both, that take Dirichlet data
#pragma unroll
      for (int j = 0; j < 6; ++j)
        {
          const bool ro = nonzero(co(j)), self = ro || nb[j] < 0;
          own |= ro ? 1u << j : 0u;
          edge |= !ro && nb[j] < 0 ? 1u << j : 0u;
          if (!UPW)
            two |= ro && nonzero(cn(j)) ? 1u << j : 0u;
          fv[j] = face_value(self ? cell0 + cl : (long long)nb[j], self, j);
          fc[j] = or_bits(P[j], M[j]);
        }
      // a velocity that changes sign in time exchanges P and M between the
      // stages: all traces are written for the next one
      if (!UPW && !UNI)
        own = 63u;
      if (edge)
        {
#pragma unroll
          for (int j = 0; j < 6; ++j)
            if ((edge >> j) & 1u)
              fv[j] = boundary_value(A, j >> 1, face[j], r, NF);
        }
      if (!UPW && two)
        {
#pragma unroll
          for (int j = 0; j < 6; ++j)
            if ((two >> j) & 1u)
              {
                const double un = nb[j] < 0 ? boundary_value(A, j >> 1, face[j], r, NF) : face_value(nb[j], false, j);
                fv[j]           = fma(co(j), fv[j], cn(j) * un);
                fc[j]           = 1.0;
              }
        }
#pragma unroll
      for (int j = 0; j < 6; ++j)
        mf = max(mf, fx_product_top(fc[j], fv[j]));
      atomicMax(s_eu + cl, LATE ? fx_magnitude(U) : fx_magnitude(U) | (unsigned)fx_subnormal(U));
      atomicMax(s_ef + cl, mf);
    }
  __syncthreads();

  // ---- the block's scale: biased exponents of the tops of U, vt U and Z
  Limbs f[6];
  int2  cv[3];
  bool  live = mine, tiny = false;
  int   topz = 0;
  if (mine)
    {
      const unsigned mu = s_eu[cl], mf = s_ef[cl];
      const int      eu = (int)(mu >> 20), ef = (int)mf;
      const int topv = UNI ? (int)(max(max(abs_hi(A.cv[0]), abs_hi(A.cv[1])), abs_hi(A.cv[2])) >> 20)
                           : A.cell_exp[cell0 + cl];
      const bool zero = (mu | mf) == 0;
      topz            = zero ? 1023 : max(eu + topv - 1022, ef);
      live            = eu < kFxHigh && ef < kFxHigh && topz > kFxLow;
      // (values of magnitude 0 that are not zero: the binary64 path)
      tiny = LATE && mu == 0;
      if ((!live && r == 0) || (tiny && fx_subnormal(U)))
        atomicOr(s_bad, 1u << cl);
      // U so that vt U is in Z's scale (topu >= eu)
      const int topu = topz - topv + 1022;
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
            f[j] = fx_product(fc[j], fv[j], topz, j & 1);
          if (UNI)
            {
#pragma unroll
              for (int d = 0; d < 3; ++d)
                cv[d] = fx_const58(A.cv[d], topv);
            }
        }
    }
  if (!UNI)
    __pipeline_wait_prior(0);
  __syncthreads();
  if (tiny)
    live = live && !((*s_bad >> cl) & 1u);

  // one direction pass: the pencil at p (stride st) with vt at v (stride st)
  auto pass = [&](const int2 *p, int st, const double *v, const int2 &c, const Limbs &flo, const Limbs &fhi,
                  long long(&out)[N]) {
    Limbs V[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      {
        const int2 u = p[k * st];
        Limbs      X;
        X.h = u.x, X.l = u.y;
        V[k] = fx_times(X, UNI ? c : reinterpret_cast<const int2 *>(v)[k * st]);
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
  const bool      reads_u   = (A.mode == kModeStage || A.mode == kModeLastStage) && (TR || A.u_in);
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
      double    kd[N], next[N];
      // (the mode's branches around whole loops: as predicated code the
      // instructions of every mode would issue on the FP64 pipe)
#pragma unroll
      for (int k = 0; k < N; ++k)
        kd[k] = fx_to_double(Qb[off + k * NF] + out[k], ez);
      if (!TR && A.mode == kModeVmult)
        {
          // implicit operator in weak form: JxW (c U - bracket), as
          // stage_gauss_cta; with JxW given, without the division by 1 / det J (half
          // of this mode's FP64 instructions: 135 instead of 187 us on 32^3 curved
          // cells of degree 4)
          if (!UNI && A.jxw)
            {
              const double wxy = tb.gw[r % N] * tb.gw[r / N];
#pragma unroll
              for (int k = 0; k < N; ++k)
                U[k] = (A.mass_factor * __ldg(A.r_in + gb + k * NF)) * __ldg(A.jxw + gb + k * NF);
#pragma unroll
              for (int k = 0; k < N; ++k)
                A.r_out[gb + k * NF] = fma(-(wxy * tb.gw[k]), A.out_scale * kd[k], U[k]);
            }
          else
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                {
                  const double wq = tb.gw[r % N] * tb.gw[r / N] * tb.gw[k];
                  const double br = A.out_scale * kd[k], u = __ldg(A.r_in + gb + k * NF);
                  A.r_out[gb + k * NF] = UNI ? wq * A.vol * (A.mass_factor * u - br)
                                             : wq * (A.mass_factor * u / G[3 * NQ + r + k * NF] - br);
                }
            }
        }
      else
        {
          if (!UNI)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                kd[k] *= G[3 * NQ + r + k * NF];
            }
          if (A.mode == kModeApply)
            {
#pragma unroll
              for (int k = 0; k < N; ++k)
                A.r_out[gb + k * NF] = A.out_scale * kd[k];
            }
          else
            {
              if (!TR && A.k_add)
                {
#pragma unroll
                  for (int k = 0; k < N; ++k)
                    kd[k] += __ldcs(A.k_add + gb + k * NF);
                }
#pragma unroll
              for (int k = 0; k < N; ++k)
                next[k] = fma(A.b, kd[k], ui[k]);
              if (!TR && A.mode == kModeLastStage && A.u_base)
                {
#pragma unroll
                  for (int k = 0; k < N; ++k)
                    next[k] += A.u_base[gb + k * NF];
                }
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
                  if (!TR && A.k_out)
                    {
#pragma unroll
                      for (int k = 0; k < N; ++k)
                        A.k_out[gb + k * NF] = kd[k];
                    }
                }
            }
        }
      if (TR && A.tr_out)
        {
          write_traces<N>(tb, next, own >> 4, static_cast<double *>(A.tr_out) + ((cell0 + cl) * 6 + 4) * NF + r);
#pragma unroll
          for (int k = 0; k < N; ++k)
            Qb[off + k * NF] = __double_as_longlong(next[k]);
        }
    }
  if (TR && A.tr_out)
    {
      __syncthreads();
      if (live)
        {
#pragma unroll 1
          for (int d = 0; d < 2; ++d)
            {
              const long long *p  = Qb + cl * NQ + (d == 0 ? N * r : offy);
              const int        st = d == 0 ? 1 : N;
              double           x[N];
#pragma unroll
              for (int k = 0; k < N; ++k)
                x[k] = __longlong_as_double(p[k * st]);
              write_traces<N>(tb, x, own >> (2 * d),
                              static_cast<double *>(A.tr_out) + ((cell0 + cl) * 6 + 2 * d) * NF + r);
            }
        }
    }
  // ---- cells outside the window
  const unsigned bad = *s_bad;
  if (bad)
    {
      __syncthreads();
      stage_gauss_masked<N, UNI, TR, UPW>(A, cell0, smem_raw, bad);
    }
}

template <int N, bool UNI, bool TR, bool UPW>
__global__ void __launch_bounds__(FxShape<N, UNI, TR>::THREADS, kFxThreadsPerSM / FxShape<N, UNI, TR>::THREADS)
  stage_fx_kernel(const __grid_constant__ StageArgs A)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  stage_fx_cta<N, UNI, TR, UPW, UNI>(A, A.cell_begin + (long long)blockIdx.x * FxShape<N, UNI, TR>::C, smem_raw);
}

template <int N, bool UNI, bool TR, bool UPW = false>
cudaError_t launch_stage_fx_t(const StageArgs &args, cudaStream_t stream)
{
  using FS              = FxShape<N, UNI, TR>;
  constexpr auto kernel = stage_fx_kernel<N, UNI, TR, UPW>;
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
    return args.uniform     ? launch_stage_fx_t<N, true, true>(args, stream)
           : args.upwind_tr ? launch_stage_fx_t<N, false, true, true>(args, stream)
                            : launch_stage_fx_t<N, false, true>(args, stream);
  return args.uniform ? launch_stage_fx_t<N, true, false>(args, stream)
                      : launch_stage_fx_t<N, false, false>(args, stream);
}
} // namespace adv
