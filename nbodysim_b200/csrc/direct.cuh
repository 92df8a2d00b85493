// FP64 direct-sum accelerations (direct.cu).
#pragma once

#include "common.cuh"

namespace nbody {

// Bytes of `part` below: the sources' chunk sums of one slab of targets.
size_t direct_scratch_bytes(uint32_t n, uint32_t m);
// out[3w..3w+2] = the all-pairs FP64 acceleration of particle targets[w]
// (or w when targets is null), w < m. Asynchronous.
cudaError_t launch_direct(const double *pos, const double *mass, uint32_t n, int damping, const uint32_t *targets,
                          uint32_t m, double *out, double *part, cudaStream_t st, unsigned *launches);

}  // namespace nbody
