// Set-up and diagnostics kernels: L2 projection of the initial data
// (project_initial, advection_solver.cc:760-784), mass/energy/H1 seminorm
// (compute_mass_and_energy, advection_solver.cc:787-818), the L2 error
// against the analytic solution (output_results, advection_solver.cc:1183-1208)
// and an FMA throughput probe for roofline denominators.
//
// FP64, one CTA per cell at a time (grid-stride), every evaluation by sum
// factorization: 1D matrices applied direction by direction in shared memory,
// one thread per output entry.  No geometry is stored for the diagnostics: the
// deformation is a sum of products of 1D functions, so its tensor-product
// interpolant on the Gauss-Lobatto support points (the degree-k mapping) is
// the same sum of products of 1D interpolants, x_c = linear + A L_c S_{c+1} S_{c+2}
// with S_d the interpolated sin(2 pi s_d): 6 m values per cell and rule instead
// of 27 sweeps over the cell (the projection excepted, see there).  The
// sine-product + Gaussian solution is evaluated on the integer pipes
// (fixed_math.cuh).  Reductions are
// deterministic: per-CTA partials, summed by the caller.
// Bound: the FP64 pipe (sweeps, phases, quadrature sums).  Measured on GB300 on
// 32^3 curved cells of degree 4: projection 1.60 instead of 3.09 ms, L2 error 1.27
// instead of 7.82, mass and energy 0.86 instead of 2.84 (with 27 mapping
// sweeps per rule, binary64 sines and exponentials).
#include "fixed_math.cuh"
#include "kernels.h"

namespace adv
{
namespace
{
constexpr int kDiagThreads = 128;

__device__ __forceinline__ void cell_origin(const DiagArgs &g, long long c, double lo[3])
{
  const int ix = (int)(c % g.nc[0]), iy = (int)((c / g.nc[0]) % g.nc[1]),
            iz = (int)(c / ((long long)g.nc[0] * g.nc[1])) + g.zoff;
  lo[0] = g.lo[0] + ix * g.h[0];
  lo[1] = g.lo[1] + iy * g.h[1];
  lo[2] = g.lo[2] + iz * g.h[2];
}

// out = A applied along direction D of `in` (D0 x D1 x D2 entries, first
// fastest), A MO x NI row-major; the output has MO entries along D.  Ends with
// a barrier.
template <int MO, int NI, int D, int D0, int D1, int D2>
__device__ __forceinline__ void tsweep(const double *A, const double *in, double *out)
{
  constexpr int o0 = D == 0 ? MO : D0, o1 = D == 1 ? MO : D1, o2 = D == 2 ? MO : D2;
  constexpr int st = D == 0 ? 1 : D == 1 ? D0 : D0 * D1;
  for (int idx = threadIdx.x; idx < o0 * o1 * o2; idx += kDiagThreads)
    {
      const int i0 = idx % o0, i1 = (idx / o0) % o1, i2 = idx / (o0 * o1);
      const int q  = D == 0 ? i0 : D == 1 ? i1 : i2;
      const int b  = (D == 0 ? 0 : i0) + D0 * ((D == 1 ? 0 : i1) + D1 * (D == 2 ? 0 : i2));
      double    s  = A[q * NI] * in[b];
#pragma unroll
      for (int k = 1; k < NI; ++k)
        s = fma(A[q * NI + k], in[b + k * st], s);
      out[idx] = s;
    }
  __syncthreads();
}

// 1D sines of the deformation at the support points, sn[d n + a] = sin(2 pi s_d)
// (0 on affine meshes).  Ends with a barrier.
template <int N>
__device__ __forceinline__ void support_sines(const DiagArgs &g, const double lo[3], double *sn)
{
  for (int i = threadIdx.x; i < 3 * N; i += kDiagThreads)
    {
      const int    d = i / N, a = i % N;
      const double x = lo[d] + g.h[d] * g.gl[a];
      sn[i]          = g.curved ? fx_to_double(fx_join(fx_sin_turn(fx_turn((x - g.lo[d]) / g.L[d]))), -57) : 0.0;
    }
  __syncthreads();
}

// What a rule with M points per direction needs of the mapping, per direction
// and point: S, the interpolated sine (nodal-basis values V), dS its derivative
// (weights W; from differences to the first node: the weights sum to zero),
// x the linear part of the position and y its phase (x - v t - lo) / L - p in
// the exact solution, with the products below folded in.
template <int M>
struct RuleSines
{
  double S[3][M], dS[3][M], AS[3][M], y[3][M];
};

// fills it (no barrier)
template <int N, int M>
__device__ __forceinline__ void rule_sines(const DiagArgs &g, const double lo[3], const double *V, const double *W,
                                           const double *pts, double t, const double *sn, RuleSines<M> &R)
{
  for (int i = threadIdx.x; i < 9 * M; i += kDiagThreads)
    {
      const int e = i / (3 * M), d = i / M % 3, q = i % M;
      if (e == 2)
        {
          const double tt = g.ex.constant_velocity ? t : 0.0;
          R.y[d][q]       = (lo[d] + g.h[d] * pts[q] - g.ex.velocity[d] * tt - g.lo[d]) / g.L[d] - g.ex.p[d];
          continue;
        }
      const double *T = (e ? W : V) + q * N, *f = sn + d * N;
      double        s = e ? 0.0 : T[0] * f[0];
#pragma unroll
      for (int a = 1; a < N; ++a)
        s = fma(T[a], e ? f[a] - f[0] : f[a], s);
      (e ? R.dS : R.S)[d][q] = s;
      if (e == 0)
        R.AS[d][q] = g.deformation * s;
    }
}

// det J of a curved cell's point.  With J[c][c] = h_c, J[c][c+1] = A L_c dS_{c+1}
// S_{c+2}, J[c][c+2] = A L_c S_{c+1} dS_{c+2} both cyclic products are the
// same: det J = h0 h1 h2 + 2 A^3 L0 L1 L2 S0 S1 S2 dS0 dS1 dS2 - sum_c h_c
// A^2 L_{c+1} L_{c+2} S_c^2 dS_{c+1} dS_{c+2}.
struct DetConstants
{
  double hhh, k3, k2[3];
  __device__ __forceinline__ DetConstants(const DiagArgs &g)
  {
    const double A = g.deformation;
    hhh            = g.h[0] * g.h[1] * g.h[2];
    k3             = 2.0 * A * A * A * g.L[0] * g.L[1] * g.L[2];
    for (int c = 0; c < 3; ++c)
      k2[c] = -A * A * g.L[(c + 1) % 3] * g.L[(c + 2) % 3] * g.h[c];
  }
};
template <int M>
__device__ __forceinline__ double point_det(const DetConstants &k, const RuleSines<M> &R, const int (&q)[3])
{
  const double s0 = R.S[0][q[0]], s1 = R.S[1][q[1]], s2 = R.S[2][q[2]];
  const double d0 = R.dS[0][q[0]], d1 = R.dS[1][q[1]], d2 = R.dS[2][q[2]];
  const double d01 = d0 * d1;
  double       det = fma(k.k3 * (s0 * s1), s2 * (d01 * d2), k.hhh);
  det              = fma(k.k2[0] * (s0 * s0), d1 * d2, det);
  det              = fma(k.k2[1] * (s1 * s1), d2 * d0, det);
  return fma(k.k2[2] * (s2 * s2), d01, det);
}

// Jacobian J[c][d] = dx_c / dxi_d there
template <int M>
__device__ __forceinline__ void point_jacobian(const DiagArgs &g, const RuleSines<M> &R, const int (&q)[3],
                                               double (&J)[3][3])
{
#pragma unroll
  for (int c = 0; c < 3; ++c)
    {
      const int    c1 = (c + 1) % 3, c2 = (c + 2) % 3;
      const double l = g.L[c] * g.deformation;
      J[c][c]        = g.h[c];
      J[c][c1]       = l * R.dS[c1][q[c1]] * R.S[c2][q[c2]];
      J[c][c2]       = l * R.S[c1][q[c1]] * R.dS[c2][q[c2]];
    }
}

// cofactors C[d][i] = det J (J^{-1})_{di}; returns det J
__device__ __forceinline__ double cofactors(const double (&J)[3][3], double (&C)[3][3])
{
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      {
        const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, d1 = (d + 1) % 3, d2 = (d + 2) % 3;
        C[d][i] = fma(J[i1][d1], J[i2][d2], -(J[i1][d2] * J[i2][d1]));
      }
  return fma(J[0][0], C[0][0], fma(J[0][1], C[1][0], J[0][2] * C[2][0]));
}

// binary64 solution at the point (other initial data, phases out of the
// fixed-point range)
template <int M>
__device__ __noinline__ double exact_binary64(const DiagArgs &g, const double *pts, const double lo0, const double lo1,
                                              const double lo2, const RuleSines<M> &R, int q0, int q1, int q2, double t)
{
  const double lo[3] = {lo0, lo1, lo2};
  const int    q[3]  = {q0, q1, q2};
  double       x[3];
  for (int c = 0; c < 3; ++c)
    x[c] = lo[c] + g.h[c] * pts[q[c]] +
           g.deformation * g.L[c] * R.S[(c + 1) % 3][q[(c + 1) % 3]] * R.S[(c + 2) % 3][q[(c + 2) % 3]];
  return exact_value(g.ex, x[0], x[1], x[2], t);
}

template <int M>
__device__ __forceinline__ double exact_at(const DiagArgs &g, const double *pts, const double lo[3],
                                           const RuleSines<M> &R, const int (&q)[3], double t)
{
  if (g.ex.type == ADV_IC_SINE_GAUSS)
    {
      double y[3];
      bool   in = true;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        {
          const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          y[c]         = fma(R.AS[c1][q[c1]], R.S[c2][q[c2]], R.y[c][q[c]]);
          in           = in && abs_hi(y[c]) < 0x41300000u; // 2^20
        }
      if (in)
        return fx_sine_gauss(y[0], y[1], y[2]);
    }
  return exact_binary64<M>(g, pts, lo[0], lo[1], lo[2], R, q[0], q[1], q[2], t);
}

__device__ void block_reduce3(double v0, double v1, double v2, double *out)
{
  __shared__ double red[3][kDiagThreads / 32];
  for (int o = 16; o > 0; o >>= 1)
    {
      v0 += __shfl_down_sync(0xffffffffu, v0, o);
      v1 += __shfl_down_sync(0xffffffffu, v1, o);
      v2 += __shfl_down_sync(0xffffffffu, v2, o);
    }
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (lane == 0)
    red[0][warp] = v0, red[1][warp] = v1, red[2][warp] = v2;
  __syncthreads();
  if (threadIdx.x == 0)
    {
      double s0 = 0, s1 = 0, s2 = 0;
      for (int w = 0; w < kDiagThreads / 32; ++w)
        s0 += red[0][w], s1 += red[1][w], s2 += red[2][w];
      out[0] = s0, out[1] = s1, out[2] = s2;
    }
}

// The projection keeps binary64 arithmetic in a fixed order (mapping by
// interpolation of the support points, sines and exponential of the binary64
// library): initial data that differ in their last bit grow to differences of
// the size of its round-off in the FP32 operator's solutions, so a rounding
// here would change them all.  Only the position is interpolated (three sweeps
// per component).
template <int N>
__global__ void __launch_bounds__(kDiagThreads) project_kernel(const __grid_constant__ DiagArgs g, double t, double *dst)
{
  constexpr int     NQ = N * N * N;
  __shared__ double X[3][NQ], T1[NQ], T2[NQ], sn[3 * N];
  // the translation v t rounded by itself (a product with 1 below), whether or
  // not the compiler fuses it into the subtraction
  ExactParams  ex = g.ex;
  const double tt = ex.constant_velocity ? 1.0 : t;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (ex.constant_velocity)
      ex.velocity[d] = __dmul_rn(g.ex.velocity[d], t);
  for (long long c = g.cell_begin + blockIdx.x; c < g.n_cells; c += gridDim.x)
    {
      double lo[3];
      cell_origin(g, c, lo);
      if (g.curved)
        {
          for (int i = threadIdx.x; i < 3 * N; i += kDiagThreads)
            {
              const int    d = i / N, a = i % N;
              const double x = lo[d] + g.h[d] * g.gl[a];
              sn[i]          = sinpi(2.0 * ((x - g.lo[d]) / g.L[d]));
            }
          __syncthreads();
#pragma unroll
          for (int k = 0; k < 3; ++k)
            {
              for (int i = threadIdx.x; i < NQ; i += kDiagThreads)
                {
                  const int    a[3] = {i % N, (i / N) % N, i / (N * N)};
                  const int    c1 = (k + 1) % 3, c2 = (k + 2) % 3;
                  const double p  = lo[k] + g.h[k] * g.gl[a[k]];
                  T1[i]           = p + g.deformation * g.L[k] * sn[c1 * N + a[c1]] * sn[c2 * N + a[c2]];
                }
              __syncthreads();
              tsweep<N, N, 2, N, N, N>(g.S, T1, T2);
              tsweep<N, N, 1, N, N, N>(g.S, T2, T1);
              tsweep<N, N, 0, N, N, N>(g.S, T1, X[k]);
            }
        }
      for (int p = threadIdx.x; p < NQ; p += kDiagThreads)
        {
          const int q[3] = {p % N, p / N % N, p / (N * N)};
          double    x[3];
#pragma unroll
          for (int k = 0; k < 3; ++k)
            x[k] = g.curved ? X[k][p] : lo[k] + g.h[k] * g.gp[q[k]];
          T1[p] = exact_value(ex, x[0], x[1], x[2], tt);
        }
      __syncthreads();
      // transform_from_q_points_to_basis: S^{-1} in every direction
      tsweep<N, N, 0, N, N, N>(g.Si, T1, T2);
      tsweep<N, N, 1, N, N, N>(g.Si, T2, T1);
      tsweep<N, N, 2, N, N, N>(g.Si, T1, T2);
      for (int i = threadIdx.x; i < NQ; i += kDiagThreads)
        dst[c * NQ + i] = T2[i];
    }
}

template <int N>
__global__ void __launch_bounds__(kDiagThreads)
  mass_energy_kernel(const __grid_constant__ DiagArgs g, const double *u, double *partials)
{
  constexpr int     NQ = N * N * N;
  __shared__ double T1[NQ], T2[NQ], G0[NQ], G1[NQ], G2[NQ], sn[3 * N];
  __shared__ RuleSines<N> R;
  double            m = 0.0, e = 0.0, hs = 0.0;
  for (long long c = g.cell_begin + blockIdx.x; c < g.n_cells; c += gridDim.x)
    {
      double lo[3];
      cell_origin(g, c, lo);
      for (int i = threadIdx.x; i < NQ; i += kDiagThreads)
        T1[i] = u[c * NQ + i];
      if (g.curved)
        {
          support_sines<N>(g, lo, sn);
          rule_sines<N, N>(g, lo, g.S, g.Sd, g.gp, 0.0, sn, R);
        }
      __syncthreads();
      tsweep<N, N, 0, N, N, N>(g.S, T1, T2);
      tsweep<N, N, 1, N, N, N>(g.S, T2, T1);
      tsweep<N, N, 2, N, N, N>(g.S, T1, T2); // values at the Gauss points
      tsweep<N, N, 0, N, N, N>(g.Dc, T2, G0);
      tsweep<N, N, 1, N, N, N>(g.Dc, T2, G1);
      tsweep<N, N, 2, N, N, N>(g.Dc, T2, G2);
      for (int p = threadIdx.x; p < NQ; p += kDiagThreads)
        {
          const int    q[3] = {p % N, p / N % N, p / (N * N)};
          const double w    = g.gw[q[0]] * g.gw[q[1]] * g.gw[q[2]], v = T2[p];
          const double d[3] = {G0[p], G1[p], G2[p]};
          double       det, gg = 0.0; // |det J grad u|^2
          if (g.curved)
            {
              double J[3][3], C[3][3];
              point_jacobian<N>(g, R, q, J);
              det = cofactors(J, C);
#pragma unroll
              for (int i = 0; i < 3; ++i)
                {
                  const double gi = fma(C[0][i], d[0], fma(C[1][i], d[1], C[2][i] * d[2]));
                  gg              = fma(gi, gi, gg);
                }
            }
          else
            {
              det = g.h[0] * g.h[1] * g.h[2];
#pragma unroll
              for (int i = 0; i < 3; ++i)
                {
                  const double gi = g.h[(i + 1) % 3] * g.h[(i + 2) % 3] * d[i];
                  gg              = fma(gi, gi, gg);
                }
            }
          const double jxw = det * w, vj = v * jxw;
          m += vj;
          e  = fma(v, vj, e);
          hs = fma(gg, w / det, hs);
        }
      __syncthreads();
    }
  block_reduce3(m, e, hs, partials + 3 * blockIdx.x);
}

template <int N>
__global__ void __launch_bounds__(kDiagThreads)
  l2_error_kernel(const __grid_constant__ DiagArgs g, const double *u, double t, double *partials)
{
  constexpr int     NQ = N * N * N, M = N + 1, M3 = M * M * M;
  __shared__ double T0[M3], T1[M3], sn[3 * N];
  __shared__ RuleSines<M> R;
  __shared__ RuleSines<N> Rn;
  const DetConstants      K(g);
  double                  err = 0.0, nrm = 0.0;
  for (long long c = g.cell_begin + blockIdx.x; c < g.n_cells; c += gridDim.x)
    {
      double lo[3];
      cell_origin(g, c, lo);
      for (int i = threadIdx.x; i < NQ; i += kDiagThreads)
        T0[i] = u[c * NQ + i];
      support_sines<N>(g, lo, sn);
      rule_sines<N, M>(g, lo, g.SE, g.SEd, g.ep, t, sn, R);
      rule_sines<N, N>(g, lo, g.S, g.Sd, g.gp, t, sn, Rn);
      __syncthreads();
      // u_h at the QGauss(k+2) points
      tsweep<M, N, 0, N, N, N>(g.SE, T0, T1);
      tsweep<M, N, 1, M, N, N>(g.SE, T1, T0);
      tsweep<M, N, 2, M, M, N>(g.SE, T0, T1);
      for (int p = threadIdx.x; p < M3; p += kDiagThreads)
        {
          const int    q[3] = {p % M, p / M % M, p / (M * M)};
          const double w    = g.ew[q[0]] * g.ew[q[1]] * g.ew[q[2]];
          const double det  = g.curved ? point_det<M>(K, R, q) : K.hhh;
          const double d    = T1[p] - exact_at<M>(g, g.ep, lo, R, q, t);
          err               = fma(d * d, det * w, err);
        }
      // norm of the exact solution with QGauss(k+1)
      for (int p = threadIdx.x; p < NQ; p += kDiagThreads)
        {
          const int    q[3] = {p % N, p / N % N, p / (N * N)};
          const double w    = g.gw[q[0]] * g.gw[q[1]] * g.gw[q[2]];
          const double det  = g.curved ? point_det<N>(K, Rn, q) : K.hhh;
          const double ue   = exact_at<N>(g, g.gp, lo, Rn, q, t);
          nrm               = fma(ue * ue, det * w, nrm);
        }
      __syncthreads();
    }
  block_reduce3(err, nrm, 0.0, partials + 3 * blockIdx.x);
}

template <typename T>
__global__ void fma_peak_kernel(T *out, int iters, T a, T b)
{
  T x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
    x7 = x0 + 7;
  for (int i = 0; i < iters; ++i)
    {
      x0 = fma(x0, a, b), x1 = fma(x1, a, b), x2 = fma(x2, a, b), x3 = fma(x3, a, b);
      x4 = fma(x4, a, b), x5 = fma(x5, a, b), x6 = fma(x6, a, b), x7 = fma(x7, a, b);
    }
  out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

// FP64 with the stage kernel's mix of FP64 instructions: per iteration 14
// independent chains, 7 FMA, 4 MUL and 3 ADD (the collocation stage with
// upwind traces issues about 51 % FMA, 28 % MUL and 21 % ADD)
constexpr int kMixF = 7, kMixM = 4, kMixA = 3;
__global__ void fp64_mix_kernel(double *out, int iters, double a, double b)
{
  double f[kMixF], m[kMixM], d[kMixA];
#pragma unroll
  for (int i = 0; i < kMixF; ++i)
    f[i] = threadIdx.x + i;
#pragma unroll
  for (int i = 0; i < kMixM; ++i)
    m[i] = threadIdx.x + kMixF + i;
#pragma unroll
  for (int i = 0; i < kMixA; ++i)
    d[i] = threadIdx.x + kMixF + kMixM + i;
  for (int it = 0; it < iters; ++it)
    {
#pragma unroll
      for (int i = 0; i < kMixF; ++i)
        f[i] = fma(f[i], a, b);
#pragma unroll
      for (int i = 0; i < kMixM; ++i)
        m[i] = m[i] * a;
#pragma unroll
      for (int i = 0; i < kMixA; ++i)
        d[i] = d[i] + b;
    }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kMixF; ++i)
    s += f[i];
#pragma unroll
  for (int i = 0; i < kMixM; ++i)
    s += m[i];
#pragma unroll
  for (int i = 0; i < kMixA; ++i)
    s += d[i];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

} // namespace

cudaError_t upload_tables_diag(const DevTables<double> *d, const DevTables<float> *f)
{
  cudaError_t e = upload_tables_local(d, f);
  return e != cudaSuccess ? e : upload_fx_math_local();
}

int diag_max_blocks(long long n_cells)
{
  return (int)(n_cells < 4096 ? n_cells : 4096);
}

#define ADV_DIAG_CASES(kernel, ...)                                              \
  switch (g.n)                                                                   \
    {                                                                            \
      case 2: kernel<2><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      case 3: kernel<3><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      case 4: kernel<4><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      case 5: kernel<5><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      case 6: kernel<6><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      case 7: kernel<7><<<blocks, kDiagThreads, 0, s>>>(g, __VA_ARGS__); break; \
      default: return cudaErrorInvalidValue;                                     \
    }                                                                            \
  return cudaGetLastError()

cudaError_t launch_project(const DiagArgs &g, double t, double *dst, cudaStream_t s)
{
  const int blocks = diag_max_blocks(g.n_cells - g.cell_begin);
  ADV_DIAG_CASES(project_kernel, t, dst);
}

cudaError_t launch_mass_energy(const DiagArgs &g, const double *u, double *partials, int *n_blocks,
                               cudaStream_t s)
{
  const int blocks = *n_blocks = diag_max_blocks(g.n_cells - g.cell_begin);
  ADV_DIAG_CASES(mass_energy_kernel, u, partials);
}

cudaError_t launch_l2_error(const DiagArgs &g, const double *u, double t, double *partials,
                            int *n_blocks, cudaStream_t s)
{
  const int blocks = *n_blocks = diag_max_blocks(g.n_cells - g.cell_begin);
  ADV_DIAG_CASES(l2_error_kernel, u, t, partials);
}
#undef ADV_DIAG_CASES

// out must hold blocks * 256 values of the precision's type
int fma_peak_chains(int precision)
{
  return precision == 2 ? kMixF + kMixM + kMixA : 8;
}

cudaError_t launch_fma_peak(int precision, double *out, int iters, int blocks, cudaStream_t s)
{
  if (precision == 2)
    fp64_mix_kernel<<<blocks, 256, 0, s>>>(out, iters, 1.0000001, 1e-9);
  else if (precision == 0)
    fma_peak_kernel<double><<<blocks, 256, 0, s>>>(out, iters, 1.0000001, 1e-9);
  else
    fma_peak_kernel<float><<<blocks, 256, 0, s>>>(reinterpret_cast<float *>(out), iters, 1.0000001f,
                                                   1e-9f);
  return cudaGetLastError();
}
} // namespace adv
