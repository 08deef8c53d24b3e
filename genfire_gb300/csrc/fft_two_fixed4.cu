// fft_two_fixed4.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(7, 12) X(9, 12) X(10, 14) X(12, 14) X(10, 20) X(9, 27) X(14, 21) X(14, 25) X(20, 20) X(18, 25) \
    X(20, 27) X(25, 25) X(25, 28) X(28, 28) X(30, 30)

namespace gf {

const TwoFixed *two_fixed_part4(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
