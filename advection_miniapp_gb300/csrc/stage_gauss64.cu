// Instantiations of the collocation-form stage kernel with a binary64
// operator, and the change of basis of the fused LSRK loop.
#include "fixed_basis.cuh"
#include "stage_fx.cuh"
#include "stage_fx_visc.cuh"

namespace adv
{
namespace
{
// u <- (M x M x M) u per cell, M = S (to the Gauss points) or S^-1, through
// shared memory: one thread per pencil, C cells per CTA.  MODE 1: to the
// Gauss points (optionally with the face traces of the result), 0: back to
// the Gauss-Lobatto nodes, 2: only the face traces of u (no change of basis),
// 3: M = S^T (dual coefficients from the Gauss-point to the nodal basis).
// UPW: upwind traces (StageArgs::upwind_tr; F carries the mesh and the FP64
// face coefficients): only the traces the first stage reads, as the stage
// kernel writes them.
// The sweeps run in block fixed point, one power of two per cell (fixed.cuh);
// a cell outside the window of exponents (infinities, NaN, magnitudes outside
// 2^-722 .. 2^600) in binary64.  The shared buffer holds binary64 values or
// limbs, 8 bytes each.  Measured on GB300 at 32^3 cells of degree 4: 30
// instead of 106 us per change of basis with binary64 sweeps (79 % of the FP64
// peak); a step through host memory at 48^3 2.53 instead of 2.84 ms.
template <int N, int MODE, bool UPW>
__global__ void __launch_bounds__(StageShape<N, double, true, false>::THREADS)
  basis_kernel(double *u, long long cell_begin, long long cell_end, double *traces, int width,
               const __grid_constant__ StageArgs F)
{
  using SH         = StageShape<N, double, true, false>;
  constexpr int C  = SH::C;
  constexpr int NQ = SH::NQ;
  constexpr int NF = SH::NF;
  __shared__ double        buf[C * NQ];
  __shared__ unsigned      s_max[C];
  const DevTables<double> &tb    = tab<double>(N);
  const FxBasisTables     &fx    = c_tab_fxb[N];
  const FxEvenOdd         &M     = MODE == 1 ? fx.S : MODE == 3 ? fx.St : fx.Si;
  const long long          cell0 = cell_begin + (long long)blockIdx.x * C;
  const int                ncell = (int)min((long long)C, cell_end - cell0);
  const int                tid   = threadIdx.x;
  const int                cl = tid / NF, r = tid % NF;
  const bool               mine = tid < ncell * NF;
  const int                ox = cl * NQ + N * r, oy = cl * NQ + (r % N) + NF * (r / N), oz = cl * NQ + r;
  double                  *g  = u + cell0 * NQ + oz;
  double                   x[N];
  if (mine)
    {
#pragma unroll
      for (int k = 0; k < N; ++k)
        x[k] = g[k * NF];
    }
  // face coefficients decide which traces the first stage reads
  unsigned own = 0;
  if (UPW && mine)
    {
      const unsigned c = (unsigned)(cell0 + cl), nx = F.nc[0], ny = F.nc[1];
      const unsigned row = c / nx;
      const int      ix = (int)(c - row * nx), iz = (int)(row / ny), iy = (int)(row - (unsigned)iz * ny);
#pragma unroll
      for (int j = 0; j < 6; ++j)
        {
          int      nb;
          unsigned face;
          cell_face(F, ix, iy, iz, j, nb, face);
          // own trace read on the low face where M != 0, on the high face where P != 0
          const double *fg = static_cast<const double *>(F.face_geo[j >> 1]) + (size_t)face * 2 * NF + 2 * r;
          own |= nonzero(__ldg(fg + ((j & 1) ? 0 : 1))) ? 1u << j : 0u;
        }
    }
  if (MODE != 2)
    {
      if (tid < C)
        s_max[tid] = 0u;
      __syncthreads();
      if (mine)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            buf[oz + k * NF] = x[k];
          const unsigned m = fx_magnitude(x);
          // (1: not zero although of magnitude 0, outside the window)
          atomicMax(s_max + cl, m == 0u && fx_subnormal(x) ? 1u : m);
        }
      __syncthreads();
      int        top  = 1023;
      const bool live = mine && fx_window(s_max[cl], top);
      int2      *lb   = reinterpret_cast<int2 *>(buf);
      // a sweep in binary64, of a cell outside the window
      auto sweep64 = [&](double *p, int st, double(&out)[N]) {
        double in[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
          in[k] = p[k * st];
        if (MODE == 1)
          sweep2<N, double, false>(tb.S, tb.S_eo, in, out);
        else if (MODE == 3)
          sweep2<N, double, false>(tb.St, tb.St_eo, in, out);
        else
          sweep2<N, double, false>(tb.Si, tb.Si_eo, in, out);
      };
      constexpr int SH1 = MODE == 0 ? fx_si1<N>() : 0, SH2 = MODE == 0 ? fx_si2<N>() : 0;
      Limbs         X[N];
      long long     T[N];
      if (live)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            X[k] = fx_from_double(buf[ox + k], top);
          fx_sweep_sym<N>(M, X, T);
#pragma unroll
          for (int k = 0; k < N; ++k)
            {
              const Limbs l = fx_split(fx_shift<SH1>(T[k]));
              lb[ox + k]    = make_int2(l.h, l.l);
            }
        }
      else if (mine)
        {
          double out[N];
          sweep64(buf + ox, 1, out);
#pragma unroll
          for (int k = 0; k < N; ++k)
            buf[ox + k] = out[k];
        }
      __syncthreads();
      if (live)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            X[k].h = lb[oy + k * N].x, X[k].l = lb[oy + k * N].y;
          fx_sweep_sym<N>(M, X, T);
#pragma unroll
          for (int k = 0; k < N; ++k)
            {
              const Limbs l  = fx_split(fx_shift<SH2>(T[k]));
              lb[oy + k * N] = make_int2(l.h, l.l);
            }
        }
      else if (mine)
        {
          double out[N];
          sweep64(buf + oy, N, out);
#pragma unroll
          for (int k = 0; k < N; ++k)
            buf[oy + k * N] = out[k];
        }
      __syncthreads();
      if (live)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            X[k].h = lb[oz + k * NF].x, X[k].l = lb[oz + k * NF].y;
          fx_sweep_sym<N>(M, X, T);
#pragma unroll
          for (int k = 0; k < N; ++k)
            x[k] = fx_to_double(T[k], top - 1022 - 58 + SH1 + SH2);
        }
      else if (mine)
        sweep64(buf + oz, NF, x);
      if (mine)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            g[k * NF] = x[k];
        }
    }
  if (MODE != 0 && MODE != 3 && traces)
    {
      // face traces of the result, [6][width][NF] per cell (StageArgs::tr_in):
      // values, and with width 2 also reference normal derivatives
      if (mine)
        {
#pragma unroll
          for (int k = 0; k < N; ++k)
            buf[oz + k * NF] = x[k]; // this thread's own column
        }
      __syncthreads();
#pragma unroll 1
      for (int d = 0; mine && d < 3; ++d)
        {
          const double *p  = buf + (d == 0 ? ox : d == 1 ? oy : oz);
          const int     st = d == 0 ? 1 : d == 1 ? N : NF;
          double        v[N], lo, hi;
#pragma unroll
          for (int k = 0; k < N; ++k)
            v[k] = p[k * st];
          double *to = traces + ((cell0 + cl) * 6 + 2 * d) * width * NF + r;
          if (UPW)
            {
              write_traces<N>(tb, v, own >> (2 * d), to);
              continue;
            }
          if (width == 2 && F.fx_visc)
            {
              // as the block fixed-point stages form them
              ViscPencil<N> p2;
              p2.set(v);
              const double2 a = p2.at(tb, c_tab_fxv[N - 2], v, 0), b = p2.at(tb, c_tab_fxv[N - 2], v, 1);
              to[0]      = a.x;
              to[NF]     = a.y;
              to[2 * NF] = b.x;
              to[3 * NF] = b.y;
              continue;
            }
          pencil_traces<N, double>(tb, v, lo, hi);
          to[0]          = lo;
          to[width * NF] = hi;
          if (width == 2)
            {
              pencil_dtraces<N, double>(tb, v, lo, hi);
              to[NF]     = lo;
              to[3 * NF] = hi;
            }
        }
    }
}

// The same in binary64 (modes 0 and 1), for the FP32 operator and increments:
// a change in the last bit of their input turns single binary32 roundings,
// which the stages spread, so their solutions would move by their own round-off.
template <int N, int MODE, bool UPW>
__global__ void __launch_bounds__(StageShape<N, double, true, false>::THREADS)
  basis64_kernel(double *u, long long cell_begin, long long cell_end, double *traces, int width, const StageArgs F)
{
  using SH         = StageShape<N, double, true, false>;
  constexpr int C  = SH::C;
  constexpr int NQ = SH::NQ;
  constexpr int NF = SH::NF;
  constexpr int NT = SH::THREADS;
  __shared__ double    buf[C * NQ];
  // upwind traces: face ids, and the pencils whose high trace is deferred
  __shared__ int           s_face[UPW ? 6 * C : 1], s_nbr[UPW ? 6 * C : 1], s_nboth, s_both[UPW ? 3 * C * NF : 1];
  const DevTables<double> &tb    = tab<double>(N);
  const long long          cell0 = cell_begin + (long long)blockIdx.x * C;
  const int                ncell = (int)min((long long)C, cell_end - cell0);
  const int                tid   = threadIdx.x;
  double                  *g     = u + cell0 * NQ;
  constexpr bool TO_GAUSS = MODE == 1;
  if (UPW)
    {
      cell_neighbours(F, cell0, ncell, s_nbr, s_face, tid, NT);
      if (tid == 0)
        s_nboth = 0;
    }
  for (int i = tid; i < ncell * NQ; i += NT)
    buf[i] = g[i];
  __syncthreads();
#pragma unroll
  for (int d = 0; d < 3; ++d)
    {
      for (int w = tid; w < ncell * NF; w += NT)
        {
          const int cl = w / NF, r = w % NF;
          const int off = d == 0 ? N * r : d == 1 ? (r % N) + NF * (r / N) : r;
          const int st  = d == 0 ? 1 : d == 1 ? N : NF;
          double   *p   = buf + cl * NQ + off;
          double    in[N], out[N];
#pragma unroll
          for (int k = 0; k < N; ++k)
            in[k] = p[k * st];
          if (TO_GAUSS)
            sweep2<N, double, false>(tb.S, tb.S_eo, in, out);
          else
            sweep2<N, double, false>(tb.Si, tb.Si_eo, in, out);
#pragma unroll
          for (int k = 0; k < N; ++k)
            p[k * st] = out[k];
        }
      __syncthreads();
    }
  for (int i = tid; i < ncell * NQ; i += NT)
    g[i] = buf[i];
  if (MODE != 0 && traces)
    {
      // face traces of the result, [6][width][NF] per cell (StageArgs::tr_in):
      // values, and with width 2 also reference normal derivatives
      for (int w = tid; w < 3 * ncell * NF; w += NT)
        {
          const int d = w / (ncell * NF), v = w % (ncell * NF);
          const int cl = v / NF, r = v % NF;
          const int off = d == 0 ? N * r : d == 1 ? (r % N) + NF * (r / N) : r;
          const int st  = d == 0 ? 1 : d == 1 ? N : NF;
          double    x[N], lo, hi;
#pragma unroll
          for (int k = 0; k < N; ++k)
            x[k] = buf[cl * NQ + off + k * st];
          double *to = traces + ((cell0 + cl) * 6 + 2 * d) * width * NF + r;
          if (UPW)
            {
              // own trace read on the low face where M != 0, on the high face where P != 0
              const double *fg = d == 0 ? static_cast<const double *>(F.face_geo[0])
                               : d == 1 ? static_cast<const double *>(F.face_geo[1])
                                        : static_cast<const double *>(F.face_geo[2]);
              const double2 pl = *reinterpret_cast<const double2 *>(fg + (size_t)s_face[cl * 6 + 2 * d] * 2 * NF + 2 * r);
              const double2 ph =
                *reinterpret_cast<const double2 *>(fg + (size_t)s_face[cl * 6 + 2 * d + 1] * 2 * NF + 2 * r);
              if (upwind_pencil_traces<N, double>(tb, x, nonzero(pl.y), nonzero(ph.x), to, to + NF))
                s_both[atomicAdd(&s_nboth, 1)] = (d * C + cl) * NF + r;
              continue;
            }
          pencil_traces<N, double>(tb, x, lo, hi);
          to[0]          = lo;
          to[width * NF] = hi;
          if (width == 2)
            {
              pencil_dtraces<N, double>(tb, x, lo, hi);
              to[NF]     = lo;
              to[3 * NF] = hi;
            }
        }
      if (UPW)
        {
          // the deferred high traces (usually none)
          __syncthreads();
          for (int i = tid; i < s_nboth; i += NT)
            {
              const int code = s_both[i];
              const int d = code / (C * NF), cl = (code / NF) % C, r = code % NF;
              const int off = d == 0 ? N * r : d == 1 ? (r % N) + NF * (r / N) : r;
              const int st  = d == 0 ? 1 : d == 1 ? N : NF;
              double    h   = tb.l1[0] * buf[cl * NQ + off];
#pragma unroll
              for (int q = 1; q < N; ++q)
                h = fma(tb.l1[q], buf[cl * NQ + off + q * st], h);
              traces[((cell0 + cl) * 6 + 2 * d + 1) * NF + r] = h;
            }
        }
    }
}

template <int N>
cudaError_t launch_basis_n(double *u, long long cell_begin, long long cell_end, int mode, cudaStream_t s,
                           double *traces, int width, const StageArgs *upwind, bool fixed)
{
  using SH               = StageShape<N, double, true, false>;
  const long long blocks = (cell_end - cell_begin + SH::C - 1) / SH::C;
  if (blocks <= 0)
    return cudaSuccess;
  StageArgs F;
  if (upwind)
    F = *upwind;
  else
    memset(&F, 0, sizeof(F));
  const bool upw  = upwind && traces && width == 1;
  auto       call = [&](auto kernel, double *tr, int w) {
    kernel<<<(unsigned)blocks, SH::THREADS, 0, s>>>(u, cell_begin, cell_end, tr, w, F);
  };
  if (mode == 1 && upw)
    call(fixed ? basis_kernel<N, 1, true> : basis64_kernel<N, 1, true>, traces, width);
  else if (mode == 1)
    call(fixed ? basis_kernel<N, 1, false> : basis64_kernel<N, 1, false>, traces, width);
  else if (mode == 2 && upw)
    call(basis_kernel<N, 2, true>, traces, width);
  else if (mode == 2)
    call(basis_kernel<N, 2, false>, traces, width);
  else if (mode == 3)
    call(basis_kernel<N, 3, false>, nullptr, 1);
  else
    call(fixed ? basis_kernel<N, 0, false> : basis64_kernel<N, 0, false>, nullptr, 1);
  return cudaGetLastError();
}
} // namespace

cudaError_t upload_tables_gauss64(const DevTables<double> *d, const DevTables<float> *f)
{
  cudaError_t e = upload_tables_local(d, f);
  if (e == cudaSuccess)
    e = upload_fx_basis_local(d);
  return e != cudaSuccess ? e : upload_fx_visc_local(d);
}

cudaError_t launch_stage_gauss_fp64(int n, const StageArgs &args, cudaStream_t stream)
{
  // block fixed-point contractions wherever they apply: advection without a
  // skew term, metric within the window of exponents
  if (args.fx_ok && !args.visc && !args.has_skew)
    return n <= 3 ? launch_stage_fx_a(n, args, stream)
         : n <= 5 ? launch_stage_fx_b(n, args, stream)
                  : launch_stage_fx_c(n, args, stream);
  if (args.fx_visc && !args.inc32 && args.mode != kModeVmult && !args.k_add && !args.k_out && !args.u_base)
    return launch_stage_fx_visc(n, args, stream);
  return launch_stage_gauss_any<double>(n, args, stream);
}

namespace
{
cudaError_t launch_basis_mode(int n, double *u, long long cell_begin, long long cell_end, int mode,
                              cudaStream_t stream, double *traces, int width, const StageArgs *upwind = nullptr,
                              bool fixed = true)
{
  switch (n)
    {
      case 2: return launch_basis_n<2>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      case 3: return launch_basis_n<3>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      case 4: return launch_basis_n<4>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      case 5: return launch_basis_n<5>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      case 6: return launch_basis_n<6>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      case 7: return launch_basis_n<7>(u, cell_begin, cell_end, mode, stream, traces, width, upwind, fixed);
      default: return cudaErrorInvalidValue;
    }
}
} // namespace

cudaError_t launch_basis_change(int n, double *u, long long cell_begin, long long cell_end, bool to_gauss,
                                cudaStream_t stream, double *traces, int width, const StageArgs *upwind, bool fixed)
{
  return launch_basis_mode(n, u, cell_begin, cell_end, to_gauss ? 1 : 0, stream, traces, width, upwind, fixed);
}

cudaError_t launch_basis_dual_to_nodal(int n, double *u, long long cell_begin, long long cell_end,
                                       cudaStream_t stream)
{
  return launch_basis_mode(n, u, cell_begin, cell_end, 3, stream, nullptr, 1);
}

cudaError_t launch_face_traces(int n, const double *u, long long cell_begin, long long cell_end,
                               cudaStream_t stream, double *traces, int width, const StageArgs *upwind)
{
  return launch_basis_mode(n, const_cast<double *>(u), cell_begin, cell_end, 2, stream, traces, width, upwind);
}
} // namespace adv
