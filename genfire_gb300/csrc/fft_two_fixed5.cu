// fft_two_fixed5.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(9, 10) X(8, 14) X(12, 12) X(7, 25) X(14, 15) X(10, 25) X(15, 20) X(18, 20) X(15, 27) X(20, 24) \
    X(20, 28) X(21, 30) X(24, 30) X(25, 32) X(30, 32)

namespace gf {

const TwoFixed *two_fixed_part5(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
