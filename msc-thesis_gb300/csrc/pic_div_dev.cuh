// pic_div_dev.cuh -- FP64 division by a divisor known in advance
// (pic_compat.cu).
#pragma once
#include <cuda_runtime.h>

namespace pic {

// a / b for a divisor known in advance, y = 1/b rounded to nearest: one
// product, its residual and one correction (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990; N. Brisebarre, J.-M. Muller and S. K. Raina, IEEE Trans.
// Computers 53(8), 2004).  Three operations on the FP64 pipe, which issues
// one warp instruction per 16 cycles and SM and bounds the particle pass; the
// general division takes several times as many.  The same result for operands
// and quotients of 2^-900 .. 2^900 in size (the residual is then exact); a zero
// may lose its sign, and an infinite operand gives NaN (in the solve a transform
// has then made NaN of it already; positions are checked in cell_of).
__device__ __forceinline__ double div_known(double a, double b, double y)
{
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

}  // namespace pic
