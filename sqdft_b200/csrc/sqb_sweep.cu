// Sweep kernel group (sqb_sweep.cuh): instantiations, launch set-up, and the
// kernel that builds the layered projector fields from the projector tables.
#include "sqb_sweep.cuh"

namespace sqb {

namespace {

// Per replica and ball point: its projector values into the replica's layer
// of the fields, and its first projector id into the point's id word.  The
// balls of one layer do not overlap, so every field value has one writer.
__global__ void fill_layers_kernel(int n_rep, const int4 *rep_box, const int *rep_gpb, const int *typ_nlocc,
                                   const long long *rep_off, const double *tab64, int ex, int ey, int ez, int pitch, int pmax,
                                   unsigned short *lay_id16, double *lay_chi) {
  const long long evol = (long long)pitch * ey * ez;
  for (int r = blockIdx.x; r < n_rep; r += gridDim.x) {
    const int4 b = rep_box[r];
    const int x0 = (short)(b.x & 0xffff), y0 = (short)(b.y & 0xffff), z0 = (short)(b.z & 0xffff);
    const int k = b.w & 0xff, np = (b.w >> 8) & 0xff, t = (b.w >> 16) & 0xff;
    const int Sd = 2 * typ_nlocc[t] + 1, sp2 = plane_stride(Sd);
    const int nb = Sd * Sd * Sd;
    const double *U = tab64 + rep_off[r];
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
      const int bx = i % Sd, by = (i / Sd) % Sd, bz = i / (Sd * Sd);
      const int X = x0 + bx, Yc = y0 + by, Z = z0 + bz;
      if (X < 0 || X >= ex || Yc < 0 || Yc >= ey || Z < 0 || Z >= ez) continue;
      const long long g = ((long long)Z * ey + Yc) * pitch + X;
      lay_id16[g * 4 + k] = (unsigned short)rep_gpb[r];
      for (int q = 0; q < np && q < pmax; q++)
        lay_chi[(long long)(k * pmax + q) * evol + g] = U[(long long)(q * Sd + bz) * sp2 + by * Sd + bx];
    }
  }
}

__global__ void fill_empty_kernel(unsigned long long *lay_id, long long evol, unsigned long long empty) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < evol; i += (long long)gridDim.x * blockDim.x)
    lay_id[i] = empty;
}

template <int PM, int FORM>
struct SqKernels {
  template <int MAXT, int MINB>
  static const void *get() {
    return reinterpret_cast<const void *>(&sweep::sweep_kernel<PM, FORM, MAXT, sweep::TILE_RY, MINB>);
  }
};

const void *sq_kernel(const SweepArgs &a) {
  if (a.pmax == 1)
    return a.form == 0   ? sweep::pick_tile<SqKernels<1, 0>>(a.n)
           : a.form == 1 ? sweep::pick_tile<SqKernels<1, 1>>(a.n)
                         : sweep::pick_tile<SqKernels<1, 2>>(a.n);
  if (a.pmax == 3)
    return a.form == 0   ? sweep::pick_tile<SqKernels<3, 0>>(a.n)
           : a.form == 1 ? sweep::pick_tile<SqKernels<3, 1>>(a.n)
                         : sweep::pick_tile<SqKernels<3, 2>>(a.n);
  return nullptr;
}

}  // namespace

int sweep_threads(int n) { return sweep::sweep_threads_of(n, sweep::TILE_RY); }

bool sweep_window_supported(int n) { return n <= sweep::TILE_N_MAX; }

size_t sweep_smem(int n, int pmax, int n_gproj) {
  return sweep::shared_fixed() + sweep::planes_bytes(n, sweep::TILE_RY) +
         sweep::ring_bytes(sweep::tile_bound(n), sweep::TILE_RY) +
         (((size_t)(n_gproj + pmax) * sizeof(double) + 127) & ~size_t(127));
}

size_t sweep_scratch_bytes(int n, int pmax) {
  return ((3 * sweep::vec_points(n) + sweep::flush_doubles(n, pmax)) * sizeof(double) + 255) & ~size_t(255);
}

namespace sweep {

cudaError_t kernel_setup(const void *kernel, int threads, size_t smem, int *per_sm) {
  if (kernel == nullptr) return cudaErrorInvalidConfiguration;
  // the device's limit, not this launch's size: contexts of other windows on
  // other threads share the kernel's attribute
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  if (e == cudaSuccess && per_sm) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, threads, smem);
    if (e == cudaSuccess && *per_sm < 1) e = cudaErrorInvalidConfiguration;
  }
  return e;
}

cudaError_t tile_setup(const void *kernel, const SweepArgs &a, int *per_sm) {
  if (a.n > MAXN || sweep_threads_of(a.n, TILE_RY) != a.nsweep) return cudaErrorInvalidConfiguration;
  return kernel_setup(kernel, a.nsweep, sweep_smem(a.n, a.pmax, a.n_gproj), per_sm);
}

}  // namespace sweep

cudaError_t sweep_per_sm(const SweepArgs &a, int *per_sm) { return sweep::tile_setup(sq_kernel(a), a, per_sm); }

cudaError_t launch_sweep(const SweepArgs &a, int grid, cudaStream_t s) {
  const void *kernel = sq_kernel(a);
  cudaError_t e = sweep::tile_setup(kernel, a, nullptr);
  if (e != cudaSuccess) return e;
  SweepArgs args = a;
  void *argv[] = {&args};
  return cudaLaunchKernel(kernel, dim3(grid), dim3(a.nsweep), argv, sweep_smem(a.n, a.pmax, a.n_gproj), s);
}

cudaError_t launch_fill_layers(int n_rep, const int4 *rep_box, const int *rep_gpb, const int *typ_nlocc,
                               const long long *rep_off, const double *tab64, int ex, int ey, int ez, int pitch, int pmax,
                               int n_gproj, unsigned long long *lay_id, double *lay_chi, cudaStream_t s) {
  const long long evol = (long long)pitch * ey * ez;
  cudaError_t e = cudaMemsetAsync(lay_chi, 0, (size_t)LAYERS * pmax * evol * sizeof(double), s);
  if (e != cudaSuccess) return e;
  const unsigned long long empty = 0x0001000100010001ull * (unsigned long long)n_gproj;
  fill_empty_kernel<<<1024, 256, 0, s>>>(lay_id, evol, empty);
  e = cudaGetLastError();
  if (e != cudaSuccess || n_rep == 0) return e;
  fill_layers_kernel<<<n_rep < 4096 ? n_rep : 4096, 256, 0, s>>>(n_rep, rep_box, rep_gpb, typ_nlocc, rep_off, tab64,
                                                                  ex, ey, ez, pitch, pmax,
                                                                  reinterpret_cast<unsigned short *>(lay_id), lay_chi);
  return cudaGetLastError();
}

}  // namespace sqb
