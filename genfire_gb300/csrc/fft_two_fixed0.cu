// fft_two_fixed0.cu -- complex64 lengths R1 R2 of the two-stage engine with
// kernels of their own (every sixth of the lengths from 72 to 1024 that are no
// power of two; split over files so that they compile in parallel).
#include "fft_two.cuh"
#include "internal.h"

#define GF_LENGTHS(X) \
    X(8, 9) X(8, 12) X(10, 12) X(7, 21) X(12, 15) X(12, 18) X(14, 18) X(15, 21) X(15, 25) X(20, 21) \
    X(18, 27) X(21, 27) X(20, 32) X(27, 27) X(27, 30)

namespace gf {

const TwoFixed *two_fixed_part0(int n)
{
#define X(r1, r2) make_two_fixed<r1, r2>(),
    static const TwoFixed part[] = {GF_LENGTHS(X)};
#undef X
    for (const TwoFixed &f : part)
        if (f.n == n) return &f;
    return nullptr;
}

}  // namespace gf
