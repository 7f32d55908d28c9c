// Mixture-averaged diffusion coefficients on the device: the per-cell
// transport-property kernel of the Fickian diffusion solver
// (fickean_diffusion_solver.f90:358-395, calculate_diffusivity_coeff, over
// thermophysical_properties_class.f90:560-577 calculate_omega, :737-762
// binary_diffusion_coefficient, :768-814
// mixture_averaged_diffusion_coefficients).
//
// One thread per cell.  The collision integral is evaluated once per distinct
// sqrt(eps_i * eps_j) of the mechanism (36 pairs but 17 values for KEROMNES).
// Its power of the reduced temperature splits into a constant of the pair and
// one power of T per cell, and an exponential below half an ulp of the sum is
// not formed (the third above a reduced temperature of 10.8, the second above
// 27.4).  A species' sum over its partners is (1 - Y_i) W_i sum_j Y_j / (W_j
// D_ij) + Y_i sum_j Y_j / D_ij with 1 / D_ij = Omega_ij / bdc_ij p / T^1.5: the
// cell's factor comes out of the sums, and a pair costs one product and four
// fused multiply-adds on registers (all terms are positive).  The power of T
// and the cell's factor are in every term of a cell, so their rounding does
// not average out as the pairs' does; the sums therefore carry their rounding
// errors along, and the factor and the constant of the power their low parts.
// The form that divided five times per pair and took a power, three
// exponentials and five divisions per collision integral was bound by the
// FP64 pipe: 2.06 ms for 4.19 M cells of 9 species, now 0.80 ms.
#include <cuda_runtime.h>

#include <cstdint>

#include "diffusion.hpp"

namespace nrg {

namespace {

// calculate_omega(T_red, 1, 1): Neufeld, Janzen and Aziz (1972) fit of the
// (1,1) collision integral with the coefficients set in set_properties;
// first = 1.06036 / T_red^0.15610.
__device__ __forceinline__ double omega11(double T_red, double first) {
  if (!(T_red < 70.0)) return first;
  double om = first + 0.19300 * exp(-0.47635 * T_red);
  if (T_red < 27.4) {
    om = om + 1.03587 * exp(-1.52996 * T_red);
    if (T_red < 10.8) om = om + 1.76474 * exp(-3.89411 * T_red);
  }
  return om;
}

}  // namespace

template <int N>
__global__ void __launch_bounds__(128) k_mixture_diffusivity(const __grid_constant__ DiffusivityArgs a) {
  extern __shared__ double sm[];
  const int BS = blockDim.x;
  const long c = (long)blockIdx.x * BS + threadIdx.x;
  if (c >= a.n) return;
  double* om = sm + threadIdx.x;  // [value][thread]
  const double T = a.T[c], p = a.p[c], mm = a.m_mix[c];
  const bool valid = (!a.bc || a.bc[c] == 0) && T > 0.0 && p > 0.0 && mm > 0.0;
  if (!valid) {
#pragma unroll
    for (int k = 0; k < N; ++k) a.D[(long)k * a.ld + c] = 0.0;
    return;
  }
  double Y[N];
#pragma unroll
  for (int k = 0; k < N; ++k) Y[k] = a.Y[(long)k * a.ld + c];
  const double Tp = pow(T * (1.0 / 1024.0), -0.15610);
  if (a.n_uniq == 0) om[0] = 0.0;  // no pair diffuses: every ibdc is zero
#pragma unroll 2
  for (int u = 0; u < a.n_uniq; ++u)
    om[u * BS] = omega11(T * a.uniq_isq[u], fma(a.uniq_pow[u], Tp, a.uniq_pow_lo[u] * Tp));
  double Z[N], sy[N], sz[N], ey[N], ez[N];  // sums and their accumulated rounding errors
#pragma unroll
  for (int k = 0; k < N; ++k) {
    Z[k] = Y[k] / a.W[k];
    sy[k] = sz[k] = ey[k] = ez[k] = 0.0;
  }
  const auto add = [](double& s, double& e, double x, double y) {
    const double t = fma(x, y, s);
    e = e + fma(x, y, s - t);
    s = t;
  };
#pragma unroll
  for (int i = 0; i < N - 1; ++i)
#pragma unroll
    for (int j = i + 1; j < N; ++j) {
      const int q = i * (2 * N - i - 1) / 2 + j - i - 1;
      const double x = om[a.pair_u[q] * BS] * a.ibdc[q];
      add(sy[i], ey[i], x, Y[j]);
      add(sz[i], ez[i], x, Z[j]);
      add(sy[j], ey[j], x, Y[i]);
      add(sz[j], ez[j], x, Z[i]);
    }
  // f + f_lo = p / T^1.5
  const double t15 = pow(T, 1.5);
  const double f = p / t15;
  const double f_lo = fma(-f, t15, p) / t15;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double u = (1.0 - Y[k]) * a.W[k];
    const double s = fma(u, sz[k], Y[k] * sy[k]);
    const double s_lo = fma(u, sz[k], -(s - Y[k] * sy[k])) + fma(Y[k], sy[k], -(Y[k] * sy[k])) +
                        fma(u, ez[k], Y[k] * ey[k]);
    const double acc = fma(s, f, fma(s, f_lo, s_lo * f));
    double d = 0.0;
    if (a.W[k] > 0.0 && acc > 1.0e-10) d = u / (acc * mm);
    a.D[(long)k * a.ld + c] = d;
  }
}

template <int N>
static cudaError_t launch_n(const DiffusivityArgs& a, cudaStream_t s) {
  const size_t per_thread = (size_t)(a.n_uniq > 0 ? a.n_uniq : 1) * sizeof(double);
  const int BS = per_thread * 128 <= 48 * 1024 ? 128 : 64;
  const size_t smem = per_thread * BS;
  cudaError_t e = cudaFuncSetAttribute(k_mixture_diffusivity<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const long grid = (a.n + BS - 1) / BS;
  if (grid > 0x7fffffffL) return cudaErrorInvalidValue;
  k_mixture_diffusivity<N><<<(unsigned)grid, BS, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mixture_diffusivity(const DiffusivityArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  switch (a.N) {  // the compiled mechanism sizes of up to kDiffMaxSpecies species
    case 9: return launch_n<9>(a, s);
    case 10: return launch_n<10>(a, s);
    case 13: return launch_n<13>(a, s);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace nrg
