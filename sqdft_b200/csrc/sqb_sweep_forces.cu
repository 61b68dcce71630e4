// ForcesNonLocal on the sweep kernel (node_forces in sqb_sweep.cuh), in its
// own translation unit so its register allocation is its own.
#include "sqb_sweep.cuh"

namespace sqb {

namespace {

template <int PM, typename T>
struct ForceKernels {
  template <int MAXT, int MINB>
  static const void *get() {
    return reinterpret_cast<const void *>(&sweep::sweep_force_kernel<PM, T, MAXT, sweep::TILE_RY, MINB>);
  }
};

const void *force_kernel(const SweepArgs &a, int single) {
  if (a.pmax == 1)
    return single ? sweep::pick_tile<ForceKernels<1, float>>(a.n)
                  : sweep::pick_tile<ForceKernels<1, double>>(a.n);
  if (a.pmax == 3)
    return single ? sweep::pick_tile<ForceKernels<3, float>>(a.n)
                  : sweep::pick_tile<ForceKernels<3, double>>(a.n);
  return nullptr;
}

}  // namespace

cudaError_t sweep_forces_per_sm(const SweepArgs &a, int single, int *per_sm) {
  return sweep::tile_setup(force_kernel(a, single), a, per_sm);
}

cudaError_t launch_sweep_forces(const SweepArgs &a, int single, int grid, cudaStream_t s) {
  const void *kernel = force_kernel(a, single);
  cudaError_t e = sweep::tile_setup(kernel, a, nullptr);
  if (e != cudaSuccess) return e;
  SweepArgs args = a;
  void *argv[] = {&args};
  return cudaLaunchKernel(kernel, dim3(grid), dim3(a.nsweep), argv, sweep_smem(a.n, a.pmax, a.n_gproj), s);
}

}  // namespace sqb
