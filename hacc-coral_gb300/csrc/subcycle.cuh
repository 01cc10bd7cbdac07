// subcycle.cuh -- device kernels of the sub-cycle around the kick
// (Particles::map1 and Particles::resortParticles, src/cpu/Particles.cxx).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "rcb_device.cuh"

namespace hsr {

// x += pt * v (the half-stream; pt = prefactor * tau rounded in float).
cudaError_t launch_stream(float *x, float *y, float *z, const float *vx, const float *vy,
                          const float *vz, int64_t n, float pt, cudaStream_t s);

// The half-stream (pt may be null: none), a stable sort of the particles by
// unit grid cell of an ng[0] x ng[1] x ng[2] box, particles outside it last
// (Particles::resortParticles), and all masses set to one.  *n_inbox receives
// the in-box count.  scratch needs resort_scratch_bytes(n, ng) bytes.
// Synchronizes s.
size_t resort_scratch_bytes(int64_t n, const int32_t ng[3]);
cudaError_t drift_and_resort(int64_t n, const int32_t ng[3], const KickArrays &arrays,
                             const float *pt, void *scratch, int64_t *n_inbox, cudaStream_t s);

}  // namespace hsr
