// fft_two_fp64.cu -- instantiations of the two-stage passes (fft_two.cuh) for double.
#include "fft_two.cuh"
#include "internal.h"

namespace gf {

template <> bool launch_col_two<double>(const ColPassArgs<double> &a, int other, cudaStream_t st)
{
    return launch_col_two_impl<double>(a, other, st);
}
template <> bool launch_rows_two<double>(const RowPassArgs<double> &a, bool forward, cudaStream_t st)
{
    return launch_rows_two_impl<double>(a, forward, st);
}

}  // namespace gf
