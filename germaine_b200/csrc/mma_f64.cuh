// FP64 matrix instructions (mma.sync m8n8k4)
// and the complex128 product made of four of them.
#pragma once
#include <cuda_runtime.h>

namespace gm {

// d = a b + d on one 8 x 8 x 4 FP64 block (warp-wide; a: this lane's entry
// of the 8 x 4 row-major left block, b: of the 4 x 8 column-major right
// block, d: this lane's two entries of the 8 x 8 result)
__device__ __forceinline__ void dmma_884(double a, double b, double &d0, double &d1) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// one complex 8 x 8 x 4 block
__device__ __forceinline__ void cmma_884(const double2 &a, const double2 &b, double2 &d0, double2 &d1) {
    dmma_884(a.x, b.x, d0.x, d1.x);    // Re += Ar Br
    dmma_884(-a.y, b.y, d0.x, d1.x);   //     - Ai Bi
    dmma_884(a.x, b.y, d0.y, d1.y);    // Im += Ar Bi
    dmma_884(a.y, b.x, d0.y, d1.y);    //     + Ai Br
}

}  // namespace gm
