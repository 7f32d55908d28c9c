// Chemistry-step kernels, variant "ref": finite-difference Jacobian as the reference (DDPST MITER=2), FP64 LU.
#include "chem_kernels.cuh"

namespace nrg {

void upload_mechanism_ref(const DevMech& m, cudaStream_t s) {
  cudaMemcpyToSymbolAsync(c_mech, &m, sizeof(DevMech), 0, cudaMemcpyHostToDevice, s);
}

cudaError_t launch_chem_ref(const StepArgs& a, const LaunchCfg& cfg, int* queue,
                              unsigned long long* counters, cudaStream_t s, int spec, int n_species, int n_reactions) {
  // The reference's mechanisms, KEROMNES in all launch shapes, the others on the
  // thread-per-cell grid, each with its generated right-hand side (the table
  // walk's bits; a Jacobian column is one right-hand side: 20,453 wide-range
  // cells, KEROMNES, 53.6 -> 23.4 ms) when the lists match.
  constexpr int kF = kJacFD;
  if (n_species == 9 && n_reactions == 24)
    return spec == kSpecKeromnes ? launch_variant<9, 9, 24, kF, double, kSpecKeromnes>(a, cfg, queue, counters, s)
                                 : launch_variant<9, 9, 24, kF, double, 0>(a, cfg, queue, counters, s);
  if (n_species == 9 && n_reactions == 28)
    return spec == kSpecZhang ? launch_grid<9, 9, 28, kF, double, kSpecZhang>(a, cfg, queue, counters, s)
                              : launch_grid<9, 9, 28, kF, double>(a, cfg, queue, counters, s);
  if (n_species == 10 && n_reactions == 24)
    return spec == kSpecTereza ? launch_grid<10, 10, 24, kF, double, kSpecTereza>(a, cfg, queue, counters, s)
                               : launch_grid<10, 10, 24, kF, double>(a, cfg, queue, counters, s);
  if (n_species == 13 && n_reactions == 71)
    return spec == kSpecKonnov ? launch_grid<13, 13, 71, kF, double, kSpecKonnov>(a, cfg, queue, counters, s)
                               : launch_grid<13, 13, 71, kF, double>(a, cfg, queue, counters, s);
  if (n_species == 17 && n_reactions == 25)
    return spec == kSpecAcetylene ? launch_grid<17, 17, 25, kF, double, kSpecAcetylene>(a, cfg, queue, counters, s)
                                  : launch_grid<17, 17, 25, kF, double>(a, cfg, queue, counters, s);
  return cudaErrorNotSupported;
}

}  // namespace nrg
