// Mixture-averaged diffusion coefficients (diffusion.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace nrg {

constexpr int kDiffMaxSpecies = 16;
constexpr int kDiffMaxPairs = kDiffMaxSpecies * (kDiffMaxSpecies - 1) / 2;

// Flat cells, species-major fields at [k * ld + c].  Pair tables in the order
// (0,1), (0,2), ..., (1,2), ...: ibdc = 1 / binary diffusivity constant (0: the
// pair has none, or a well depth that is not positive), pair_u = index of the
// pair's sqrt(eps_i * eps_j) among the n_uniq distinct values (first-seen
// order): pairs with equal values share one collision-integral evaluation.
// uniq_isq: the values' reciprocals; uniq_pow + uniq_pow_lo: 1.06036
// (value / 1024)^0.15610, the factor of (T / 1024)^-0.15610 in the fit's first
// term.
struct DiffusivityArgs {
  long n = 0, ld = 0;
  int N = 0;
  const double* T = nullptr;
  const double* p = nullptr;
  const double* Y = nullptr;
  const double* m_mix = nullptr;
  const int8_t* bc = nullptr;
  double* D = nullptr;
  double W[kDiffMaxSpecies] = {};
  double ibdc[kDiffMaxPairs] = {};
  double uniq_isq[kDiffMaxPairs] = {};
  double uniq_pow[kDiffMaxPairs] = {}, uniq_pow_lo[kDiffMaxPairs] = {};
  int n_uniq = 0;
  unsigned char pair_u[kDiffMaxPairs] = {};
};

cudaError_t launch_mixture_diffusivity(const DiffusivityArgs& a, cudaStream_t s);

}  // namespace nrg
