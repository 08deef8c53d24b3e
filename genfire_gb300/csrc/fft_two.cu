// fft_two.cu -- instantiations of the two-stage passes (fft_two.cuh) for float.
#include "fft_two.cuh"
#include "internal.h"

namespace gf {

const TwoFixed *two_fixed_part0(int n);
const TwoFixed *two_fixed_part1(int n);
const TwoFixed *two_fixed_part2(int n);
const TwoFixed *two_fixed_part3(int n);
const TwoFixed *two_fixed_part4(int n);
const TwoFixed *two_fixed_part5(int n);

const TwoFixed *two_fixed(int n)
{
    for (auto part : {two_fixed_part0, two_fixed_part1, two_fixed_part2, two_fixed_part3, two_fixed_part4, two_fixed_part5})
        if (const TwoFixed *f = part(n)) return f;
    return nullptr;
}

// squared length of the rounded root WR^j, less 1
double root_gain(int j, int R)
{
    const double c = (float)root_cos(j, R), s = (float)root_sin(j, R);
    return c * c + s * s - 1.0;
}
// an R-point butterfly's: its factors' and the twiddles' between them; of a
// base radix the mean over its matrix
double radix_gain(int R)
{
    const int A = rdft_split(R), B = R / A;
    double g = 0;
    if (A == 1) {
        if (R == 2 || R == 4) return 0.0;
        for (int i = 0; i < R; ++i)
            for (int k = 0; k < R; ++k) g += root_gain(i * k % R, R);
        return g / (R * R);
    }
    for (int b = 0; b < B; ++b)
        for (int k = 0; k < A; ++k) g += root_gain(b * k, R);
    return g / R + radix_gain(A) + radix_gain(B);
}
double two_gain(int n)
{
    TwoPlan p;
    if (!make_two_plan(n, p)) return 0.0;
    double g = 0;
    for (int k = 0; k < p.R1; ++k)
        for (int t = 0; t < p.R2; ++t) g += root_gain(k * t, n);
    return g / n + radix_gain(p.R1) + radix_gain(p.R2);
}

template <> bool launch_col_two<float>(const ColPassArgs<float> &a, int other, cudaStream_t st)
{
    return launch_col_two_impl<float>(a, other, st);
}
template <> bool launch_rows_two<float>(const RowPassArgs<float> &a, bool forward, cudaStream_t st)
{
    return launch_rows_two_impl<float>(a, forward, st);
}

}  // namespace gf
