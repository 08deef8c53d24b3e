// fft_two_fixed1.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(5, 15) X(7, 14) X(5, 25) X(10, 15) X(9, 21) X(14, 16) X(15, 18) X(16, 20) X(18, 21) X(18, 24) \
    X(20, 25) X(24, 24) X(24, 27) X(25, 30) X(28, 30)

namespace gf {

const TwoFixed *two_fixed_part1(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
