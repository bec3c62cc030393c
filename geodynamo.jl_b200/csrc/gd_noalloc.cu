// gd_noalloc.cu -- scalar synthesis that allocates no device memory.
//
// gd_spectral_to_physical() stages host arrays through buffers the handle
// allocates on first use.  Some callers cannot allow any allocation at call
// time: a Julia session whose GPU memory belongs to CUDA.jl's pool (a direct
// cudaMalloc from a ccall'd library bypasses that pool and can fail once the
// pool holds the free memory), or a solver loop in a framework that forbids
// allocation between its own set-up and tear-down.  This entry point serves
// them: inputs and outputs are the caller's device buffers, and the Fourier
// intermediate is the one the handle allocated when it was created, so calls on
// handles of their own, each on its own stream, have nothing in common.
#include <cuda_runtime.h>

#include <string>

#include "gd_handle.cuh"
#include "gd_internal.cuh"

// Most Fourier coefficients a call takes: min(nfield, 4) x nr x (mmax+1) x nlat
// complex doubles (the documented limit of the call).
static const size_t kScratchBytes = size_t(64) << 20;

// Makes the handle's device current for the call and restores the caller's
// current device afterwards.
namespace {
struct DeviceScope {
  int prev = -1;
  cudaError_t enter(int device) {
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess) return e;
    return cudaSetDevice(device);
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};
}  // namespace

extern "C" int gd_spectral_to_physical_noalloc(gd_handle* h, int nfield, const double* d_coef, double* d_grid) {
  if (!h) return GD_ERR_ARG;
  if (!d_coef || !d_grid || nfield < 1) return gd::set_error(h, GD_ERR_ARG, "null device pointer or nfield < 1");
  const gd::Dims& d = h->d;
  const size_t per_field = (size_t)d.nr * (d.M + 1) * d.nlat * sizeof(double2);
  const int group = nfield < 4 ? nfield : 4;
  if (per_field * group > kScratchBytes)
    return gd::set_error(h, GD_ERR_CONFIG,
                         "gd_spectral_to_physical_noalloc needs " + std::to_string(per_field * group) +
                             " bytes of Fourier scratch (min(nfield,4) x nr x (mmax+1) x nlat x 16); the fixed "
                             "maximum is " + std::to_string(kScratchBytes) + " bytes");
  DeviceScope scope;
  cudaError_t e = scope.enter(h->device);
  if (e != cudaSuccess) return gd::set_error(h, GD_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
  double2* const F = h->d_F;  // four components
  const size_t plane = (size_t)2 * d.nr * d.nlm;  // one field: Re and Im planes
  const size_t G = (size_t)d.nlat * d.nlon * d.nr;
  for (int f0 = 0; f0 < nfield; f0 += 4) {
    const int nf = nfield - f0 < 4 ? nfield - f0 : 4;
    gd::SynthArgs a{};
    a.table0 = h->d_P;
    for (int i = 0; i < nf; ++i) a.coef[i] = d_coef + plane * (f0 + i);
    a.nf = nf;
    a.out = F;
    gd::launch_synth_fp64(h->stream, d, h->d_moff, a, false);
    gd::launch_fft_synth<double>(h->stream, d, h->plan, h->d_tw, F, d_grid + G * f0, nf, G);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return gd::set_error(h, GD_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
  return GD_OK;
}
