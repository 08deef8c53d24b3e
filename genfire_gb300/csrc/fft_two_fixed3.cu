// fft_two_fixed3.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(9, 9) X(7, 15) X(9, 15) X(9, 18) X(14, 14) X(15, 16) X(16, 18) X(16, 21) X(14, 28) X(16, 28) \
    X(21, 25) X(24, 25) X(25, 27) X(24, 32) X(28, 32)

namespace gf {

const TwoFixed *two_fixed_part3(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
