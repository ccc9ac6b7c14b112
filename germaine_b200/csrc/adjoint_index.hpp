// Index arithmetic of the adjoint-source kernel (epilogue.cu), shared with its
// host check.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace gm {

struct AdjointItem {
    int receiver, shot;
    bool in;   // false beyond the last (receiver, shot) pair
};

// (receiver, shot) of flat item t = receiver * ns + shot.  In 64 bits: the
// pairs of a call may exceed 2^31 (many receivers on shared grid points).
__host__ __device__ inline AdjointItem adjoint_item(size_t t, int ns, int ntr) {
    const size_t q = t / (size_t)ns;
    return {(int)q, (int)(t - q * (size_t)ns), q < (size_t)ntr};
}

}  // namespace gm
