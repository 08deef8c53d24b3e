// fft_two_fixed2.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(8, 10) X(10, 10) X(9, 14) X(10, 16) X(12, 16) X(15, 15) X(14, 20) X(18, 18) X(16, 24) X(21, 21) \
    X(21, 24) X(21, 28) X(24, 28) X(27, 28) X(27, 32)

namespace gf {

const TwoFixed *two_fixed_part2(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
