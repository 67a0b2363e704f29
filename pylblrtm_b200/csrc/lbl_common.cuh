// Shared constants, record layouts and launch helpers of the line-by-line engine.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/lblgpu.h"

namespace lbl {

// Physical constants of the reference forward model (pylblrtm/forward.py:32-36).
constexpr double T_REF = 296.0;
constexpr double C2 = 1.4387752;            // second radiation constant [cm K]
constexpr double DOPPLER = 3.5810e-7;       // Doppler HWHM factor
constexpr double SQRT_LN2 = 0.83255461115769775635;   // sqrt(ln 2)
constexpr double VOIGT_K = 0.46971863934982566689;    // sqrt(ln 2 / pi)
// Hydrostatic constants (pylblrtm/atmosphere.py:15-18).
constexpr double P_STD_HPA = 1013.25;

// Grid point nu_i = nu_min + i * step, rounded exactly like the reference's
// nu_min + np.arange(n) * step (pylblrtm/forward.py:141-142).
__device__ __forceinline__ double grid_nu(double nu_min, double step, long long i) {
  return __dadd_rn(nu_min, __dmul_rn((double)i, step));
}

// Record the first failing (layer, group) position in reference loop order.
__device__ __forceinline__ void flag_error(int* err, int key) {
  if (err) atomicMin(err, key);
}

// Programmatic dependent launch: a kernel started with launch_dependent may begin while its
// predecessor in the stream still runs. It calls dependency_wait before it touches global
// memory (returns when the predecessor has finished and its writes are visible), and
// dependency_trigger to let its own successor begin.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependency_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename K, typename... A>
inline cudaError_t launch_dependent(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace lbl

// Status plumbing of the C ABI (capi.cu).
int lbl_set_error(int code, const char* fmt, ...);
int lbl_check_launch(const char* what);
// How far (cm^-1) from a tile's grid values the centres of its inner lines (forward) and of
// its 16-node level-1 lines (Jacobian) can lie, shifts apart.
double lbl_ml_inner_reach(int tile_samples, double step);    // voigt_ml.cu
double lbl_jac_near_reach(int tile_samples, double step);    // voigt_ml_jac.cu
