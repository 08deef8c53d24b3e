// fft_two.cuh -- FFT passes of two register stages for lengths N = R1 * R2 with
// both factors up to 32 (any product of 2, 3, 5 and 7 that splits so, up to
// 1024): the lengths that are no power of two, among them the grids of the
// class's default oversampling of 3.
//
// Thread t of a column (t < R2) takes the elements t + R2 m (m < R1), forms
// their R1-point DFT in registers, multiplies by WN^(t k1) and exchanges
// through shared memory; then thread k1 (k1 < R1) takes row k1 and forms the
// R2-point DFT, which gives the elements k1 + R1 k2.  One exchange per
// transform, the first stage loads from global memory and the last one stores
// there.  An inverse transform is the forward one with its output index
// reversed, X_inv[k] = X[(N - k) mod N], so both directions of a pass run the
// same code.
//
// Bound: instruction issue and the exchange's barriers.  The generic engine
// (k_colpass) these passes replace makes one shared-memory round trip per
// small radix (300 points: 4, 3, 5, 5), with an index division per butterfly.
// One iteration, complex64, generic engine -> here (F3 the fused pass in
// brackets):
//   300 x 225 x 300 grid of a 100 x 75 x 100 box  0.661 (0.446) -> 0.097 (0.056) ms
//   450 x 315 x 450 grid of a 150 x 105 x 150 box 2.21 (1.42) -> 0.342 (0.227) ms
//   450^3 grid of a 225^3 box                     3.68 (2.21) -> 0.601 (0.329) ms
// complex128 is bound by the FP64 pipe: 300 x 225 x 300 grid 3.68 -> 2.46 ms.
//
// Complex64 lengths from 72 points have kernels of their own (FixedPlan:
// every offset of the exchange an immediate; with the run-time split the 450^3
// iteration took 1.37 ms).  The shorter ones, where the launches bound an
// iteration, and complex128 take the radices from a uniform switch inside one
// kernel; RMAX 16 or 32 is the largest radix compiled in, so that the short
// lengths keep the registers (and the occupancy) of theirs.
#pragma once

#include "fft_reg.cuh"

#include <type_traits>

namespace gf {

// ---------------------------------------------------------------------------
// R-point DFTs in registers, R a product of 2, 3, 5 and 7 up to 32
// ---------------------------------------------------------------------------
// cos(2 pi j / R) at compile time: reduced to [0, pi/4] and summed as the
// Taylor series of cos or sin (terms beyond x^23 are below 1e-25)
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double taylor_cos(double x)
{
    double t = 1, s = 1;
    for (int k = 1; k <= 11; ++k) { t *= -x * x / ((2 * k - 1) * (2 * k)); s += t; }
    return s;
}
constexpr double taylor_sin(double x)
{
    double t = x, s = x;
    for (int k = 1; k <= 11; ++k) { t *= -x * x / ((2 * k) * (2 * k + 1)); s += t; }
    return s;
}
constexpr double root_cos(int j, int R)
{
    j %= R;
    if (j < 0) j += R;
    if (2 * j > R) j = R - j;                             // [0, 1/2] turn
    const bool neg = 4 * j > R;
    const double sg = neg ? -1.0 : 1.0;
    const int num = neg ? R - 2 * j : 2 * j;              // angle = pi num / R, in [0, pi/2]
    if (4 * num <= R) return sg * taylor_cos(kTwoPi / 2 * num / R);
    return sg * taylor_sin(kTwoPi / 4 * (R - 2 * num) / R);
}
constexpr double root_sin(int j, int R) { return root_cos(4 * j - R, 4 * R); }  // sin x = cos(x - pi/2)

// sums, differences and real multiples of complex values: packed FP32 pairs for
// complex64 (one instruction for both halves)
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return upk2(add2(pk2(a), pk2(b))); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return upk2(sub2(pk2(a), pk2(b))); }
__device__ __forceinline__ float2 vfma(float c, float2 a, float2 b) { return upk2(fma2(pk2(mk(c, c)), pk2(a), pk2(b))); }
__device__ __forceinline__ float2 vmul(float c, float2 a) { return upk2(mul2(pk2(mk(c, c)), pk2(a))); }
// a - i b and a + i b
__device__ __forceinline__ float2 vadd_mi(float2 a, float2 b) { return upk2(fma2(swap2(pk2(b)), pk2(mk(1.f, -1.f)), pk2(a))); }
__device__ __forceinline__ float2 vadd_pi(float2 a, float2 b) { return upk2(fma2(swap2(pk2(b)), pk2(mk(-1.f, 1.f)), pk2(a))); }
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return csub(a, b); }
__device__ __forceinline__ double2 vfma(double c, double2 a, double2 b) { return mk(fma(c, a.x, b.x), fma(c, a.y, b.y)); }
__device__ __forceinline__ double2 vmul(double c, double2 a) { return mk(c * a.x, c * a.y); }
__device__ __forceinline__ double2 vadd_mi(double2 a, double2 b) { return mk(a.x + b.y, a.y - b.x); }
__device__ __forceinline__ double2 vadd_pi(double2 a, double2 b) { return mk(a.x - b.y, a.y + b.x); }

// v * WR^j, j and R known at compile time
template <typename T, int J, int R> __device__ __forceinline__ cplx<T> mul_root(cplx<T> v)
{
    constexpr int j = J % R;
    if constexpr (j == 0) return v;
    else if constexpr (4 * j == R) return mul_mi(v);
    else if constexpr (2 * j == R) return mk(-v.x, -v.y);
    else if constexpr (4 * j == 3 * R) return mul_pi(v);
    else {
        constexpr T c = (T)root_cos(j, R), s = (T)-root_sin(j, R);
        return mk(v.x * c - v.y * s, v.x * s + v.y * c);
    }
}

constexpr int rdft_split(int R)  // the first of the two factors of a composite radix (1: a base radix)
{
    return R == 6 ? 2 : R == 9 ? 3 : R == 10 ? 2 : R == 12 ? 4 : R == 14 ? 2 : R == 15 ? 3 : R == 16 ? 4
         : R == 18 ? 2 : R == 20 ? 4 : R == 21 ? 3 : R == 24 ? 8 : R == 25 ? 5 : R == 27 ? 3 : R == 28 ? 4
         : R == 30 ? 5 : R == 32 ? 4 : 1;
}
constexpr bool rdft_radix(int R) { return R == 2 || R == 3 || R == 4 || R == 5 || R == 7 || R == 8 || rdft_split(R) > 1; }

// x[m] -> X[k] = sum_m x[m] WR^(m k), in natural order
template <typename T, int R> struct RDft {
    static constexpr int A = rdft_split(R), B = R / (A > 1 ? A : 1);
    template <int I> static __device__ __forceinline__ void twiddle(cplx<T> (&z)[R])
    {
        if constexpr (I < R) {  // z[A b + ka] *= WR^(b ka)
            z[I] = mul_root<T, (I / A) * (I % A), R>(z[I]);
            twiddle<I + 1>(z);
        }
    }
    static __device__ __forceinline__ void run(cplx<T> (&x)[R])
    {
        if constexpr (A == 1) {
            if constexpr (R % 2 == 1) run_odd(x);
            else if constexpr (R == 2) {
                const cplx<T> u = x[0];
                x[0] = vadd(u, x[1]);
                x[1] = vsub(u, x[1]);
            } else Dft<R, T>::run(x, false, nullptr, R);
        } else {
            // m = B a + b, k = ka + A kb
            cplx<T> z[R];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                cplx<T> u[A];
#pragma unroll
                for (int q = 0; q < A; ++q) u[q] = x[B * q + b];
                RDft<T, A>::run(u);
#pragma unroll
                for (int q = 0; q < A; ++q) z[A * b + q] = u[q];
            }
            twiddle<0>(z);
#pragma unroll
            for (int q = 0; q < A; ++q) {
                cplx<T> u[B];
#pragma unroll
                for (int b = 0; b < B; ++b) u[b] = z[A * b + q];
                RDft<T, B>::run(u);
#pragma unroll
                for (int k = 0; k < B; ++k) x[q + A * k] = u[k];
            }
        }
    }
    // an odd prime radix through the sums and differences of x[m] and x[R - m]
    static __device__ __forceinline__ void run_odd(cplx<T> (&x)[R])
    {
        constexpr int H = (R - 1) / 2;
        cplx<T> p[H], d[H], o[R];
        o[0] = x[0];
#pragma unroll
        for (int m = 0; m < H; ++m) {
            p[m] = vadd(x[m + 1], x[R - 1 - m]);
            d[m] = vsub(x[m + 1], x[R - 1 - m]);
            o[0] = vadd(o[0], p[m]);
        }
        odd_outputs<1>(x[0], p, d, o);
#pragma unroll
        for (int k = 0; k < R; ++k) x[k] = o[k];
    }
    template <int K, int M, int H>
    static __device__ __forceinline__ void odd_terms(const cplx<T> (&p)[H], const cplx<T> (&d)[H], cplx<T> &e, cplx<T> &f)
    {
        if constexpr (M <= H) {
            constexpr T c = (T)root_cos(K * M, R), q = (T)root_sin(K * M, R);
            e = vfma(c, p[M - 1], e);
            if constexpr (M == 1) f = vmul(q, d[0]);
            else f = vfma(q, d[M - 1], f);
            odd_terms<K, M + 1>(p, d, e, f);
        }
    }
    template <int K, int H>
    static __device__ __forceinline__ void odd_outputs(cplx<T> x0, const cplx<T> (&p)[H], const cplx<T> (&d)[H], cplx<T> (&o)[R])
    {
        if constexpr (K <= H) {
            cplx<T> e = x0, f;
            odd_terms<K, 1>(p, d, e, f);
            o[K] = vadd_mi(e, f);
            o[R - K] = vadd_pi(e, f);
            odd_outputs<K + 1>(x0, p, d, o);
        }
    }
};

// ---------------------------------------------------------------------------
// the split of a length
// ---------------------------------------------------------------------------
// The split of a length at run time, or (FixedPlan) at compile time: then every
// offset of the exchange is an immediate.
struct TwoPlan {
    static constexpr bool fixed = false;
    int R1, R2;
    int row;  // exchange row stride: R2 made odd, so that the rows read by a half-warp start in different banks
    int N;
};
template <int A, int B> struct FixedPlan {
    static constexpr bool fixed = true;
    static constexpr int R1 = A, R2 = B, row = B | 1, N = A * B;
};

// The most balanced split with both factors radices of the engine (threads per
// column = the larger factor); false when there is none.
inline bool make_two_plan(int n, TwoPlan &p)
{
    for (int r = 2; r <= 32; ++r)
        if (n % r == 0 && n / r <= r && n / r >= 2 && rdft_radix(r) && rdft_radix(n / r)) {
            p = TwoPlan{n / r, r, r | 1, n};
            return true;
        }
    return false;
}
template <class Plan> constexpr int two_threads(const Plan &p, int W) { return (W * p.R2 + 31) / 32 * 32; }
template <class Plan> constexpr int two_tile(const Plan &p) { return p.R1 * p.row; }  // elements per column (>= R1 R2)

// Calls fn with the radix R (the plan's R1 or R2) as a compile-time constant
template <int RMAX, class Fn> __device__ __forceinline__ void with_radix(int R, Fn &&fn)
{
#define GF_RADIX(r) \
    case r:         \
        if constexpr (r <= RMAX) fn(std::integral_constant<int, r>{}); \
        break;
    switch (R) {
        GF_RADIX(2) GF_RADIX(3) GF_RADIX(4) GF_RADIX(5) GF_RADIX(6) GF_RADIX(7) GF_RADIX(8) GF_RADIX(9) GF_RADIX(10)
        GF_RADIX(12) GF_RADIX(14) GF_RADIX(15) GF_RADIX(16) GF_RADIX(18) GF_RADIX(20) GF_RADIX(21) GF_RADIX(24)
        GF_RADIX(25) GF_RADIX(27) GF_RADIX(28) GF_RADIX(30) GF_RADIX(32)
    default: break;
    }
#undef GF_RADIX
}
template <int RMAX, class Plan, class Fn> __device__ __forceinline__ void with_r1(const Plan &p, Fn &&fn)
{
    if constexpr (Plan::fixed) fn(std::integral_constant<int, Plan::R1>{});
    else with_radix<RMAX>(p.R1, fn);
}
template <int RMAX, class Plan, class Fn> __device__ __forceinline__ void with_r2(const Plan &p, Fn &&fn)
{
    if constexpr (Plan::fixed) fn(std::integral_constant<int, Plan::R2>{});
    else with_radix<RMAX>(p.R2, fn);
}

// threads a CTA may have (8 columns of 32 threads), and the CTAs per SM its
// registers are held to: 16 values of complex64 fit 64 registers, 32 need 128
constexpr int kTwoMaxThreads = 256;
template <typename T, int RMAX> constexpr int two_min_blocks() { return (RMAX <= 16 ? 4 : 2) / (sizeof(T) == 8 ? 2 : 1); }
// a fixed plan's: its own thread count, and registers for its larger radix
constexpr int two_fixed_threads(int R2, int W) { return (W * R2 + 31) / 32 * 32; }
constexpr int two_fixed_blocks(int R2, int W)
{
    const int regs = R2 <= 16 ? 64 : R2 <= 21 ? 80 : R2 <= 25 ? 96 : 128;
    return 65536 / (regs * two_fixed_threads(R2, W));
}
template <typename T> constexpr int two_width(int n)  // tile_width<T>(n) as a constant
{
    int W = sizeof(T) == 4 ? 8 : 4;
    while (W > 1 && n * W > 8 * (sizeof(T) == 4 ? 512 : 256)) W /= 2;
    return W;
}

// One transform of a column pass (dir 0 forward, 1 inverse): from global memory
// or the natural-order tile, to the tile or, for the pass's last, to global
// memory.  Not inlined: with the two directions as one inlined loop the
// compiler hoists every radix's twiddle loads, offsets and constants out of
// it, and spills them.
template <typename T, int RMAX, class Plan>
__device__ __noinline__ void two_transform(const ColPassArgs<T> &a, const Plan &tp, int lw_, int dir, bool from_tile,
                                           bool last)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T> *s = reinterpret_cast<cplx<T> *>(smem_raw);
    const int N = tp.N;
    const int lw = Plan::fixed ? ilog2c(two_width<T>(tp.N)) : lw_, W = 1 << lw;
    const int c = threadIdx.x & (W - 1), t = threadIdx.x >> lw;
    const int other = blockIdx.y, col = blockIdx.x * W + c;
    const bool cv = col < a.ncols;
    // a thread beyond a stage's count repeats the last one's work without
    // storing it: a branch around the stage makes the compiler keep (and
    // spill) every radix's values at its join
    const bool onA = t < tp.R2, onB = t < tp.R1;
    const int tA = min(t, tp.R2 - 1), tB = min(t, tp.R1 - 1);
    with_r1<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
        if (from_tile) {
#pragma unroll
            for (int m = 0; m < R; ++m) x[m] = s[((tA + tp.R2 * m) << lw) + c];
            __syncthreads();  // the natural-order tile is read before the exchange overwrites it
        } else {
            const cplx<T> *in = a.in + (long long)other * a.in_other + tile_at(a, (int)blockIdx.x, a.in_blk) +
                (long long)c * a.col_stride;
            const unsigned idim = (unsigned)a.in_dim;
            int e = tA + a.in_c;
            if (e >= N) e -= N;
#pragma unroll
            for (int m = 0; m < R; ++m) {
                x[m] = (cv && e < a.in_cnt) ? in[(unsigned)e * idim] : mk((T)0, (T)0);
                e += tp.R2;
                if (e >= N) e -= N;
            }
        }
        RDft<T, R>::run(x);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (k) x[k] = cmul(x[k], __ldg(a.tw + tA * k));
            if (onA) s[((k * tp.row + t) << lw) + c] = x[k];
        }
    });
    __syncthreads();
    with_r2<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
#pragma unroll
        for (int m = 0; m < R; ++m) x[m] = s[((tB * tp.row + m) << lw) + c];
        RDft<T, R>::run(x);
        // element k = t + R1 k2, an inverse's at (N - k) mod N
        const int step = dir ? -tp.R1 : tp.R1;
        if (last) {
            cplx<T> *out = a.out + (long long)other * a.out_other + tile_at(a, (int)blockIdx.x, a.out_blk) +
                (long long)c * a.col_stride;
            const unsigned odim = (unsigned)a.out_dim;
            int e = (dir && tB ? N - tB : tB) + a.out_c;
            if (e >= N) e -= N;
            const int cnt = (onB && cv) ? a.out_cnt : 0;
#pragma unroll
            for (int m = 0; m < R; ++m) {
                if (e < cnt) out[(unsigned)e * odim] = mk(x[m].x * a.scale, x[m].y * a.scale);
                e += step;
                if (e >= N) e -= N;
                if (e < 0) e += N;
            }
        } else {
            __syncthreads();  // every exchange row is read before the tile overwrites it
#pragma unroll
            for (int m = 0; m < R; ++m)
                if (onB) s[((t + tp.R1 * m) << lw) + c] = x[m];
            __syncthreads();
        }
    });
}

// Column pass (contract of k_colpass); lw = log2 of the tile width.
template <typename T, int RMAX, class Plan>
__device__ __forceinline__ void col_two(const ColPassArgs<T> &a, const Plan &tp, int lw)
{
    pass_begin();
    if (a.ctl && blockIdx.x == 0 && blockIdx.y == 0) ctl_mid_update(a.ctl, a.partial, a.nparts, a.denom, a.hist);
    const bool both = (a.mode & 3) == 3;
    if (a.mode & 1) two_transform<T, RMAX>(a, tp, lw, 0, false, !both);
    if (a.mode & 4) {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        cplx<T> *s = reinterpret_cast<cplx<T> *>(smem_raw);
        const int W = 1 << lw;
        const auto idx = [lw](int q3, int cl) { return (q3 << lw) + cl; };
        if (a.rtab) {
            capture_rfree<T>(s, a, blockIdx.x, W, blockIdx.y, idx);
            __syncthreads();
        }
        const ErrPair<T> err = apply_table_at<T, ErrPair<T>>(s, a, blockIdx.x, W, blockIdx.y, idx);
        block_partial(err, a.partial + (long long)blockIdx.y * gridDim.x + blockIdx.x);
        __syncthreads();
    }
    if (a.mode & 2) two_transform<T, RMAX>(a, tp, lw, 1, both, true);
}
template <typename T, int RMAX>
__global__ void __launch_bounds__(kTwoMaxThreads, two_min_blocks<T, RMAX>())
    k_col_two(const __grid_constant__ ColPassArgs<T> a, const __grid_constant__ TwoPlan tp, int lw)
{
    col_two<T, RMAX>(a, tp, lw);
}
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(two_fixed_threads(R2, two_width<T>(R1 * R2)), two_fixed_blocks(R2, two_width<T>(R1 * R2)))
    k_col_fixed(const __grid_constant__ ColPassArgs<T> a)
{
    col_two<T, 32>(a, FixedPlan<R1, R2>{}, ilog2c(two_width<T>(R1 * R2)));
}

// Row passes (contracts of k_rows_r2c / k_rows_c2r): pair c of the CTA, the
// index along the row fastest within a warp; cp = elements per pair of the
// shared-memory tile.
template <typename T, int RMAX, class Plan>
__device__ __forceinline__ void row_r2c_two(const RowPassArgs<T> &a, const Plan &tp, int cp)
{
    pass_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (a.ctl && blockIdx.x == 0 && threadIdx.x == 0) ctl_begin_update(a.ctl, a.changes);
    if (row_pairs_empty(a, a.W)) {
        zero_half_rows(a, a.W);
        return;
    }
    const int N = tp.N;
    const int c = threadIdx.x / tp.R2, t = threadIdx.x - c * tp.R2;
    const bool cv = c < a.W;  // (the tile has room for the last warp's threads beyond it)
    const bool onB = t < tp.R1;
    const int tB = min(t, tp.R1 - 1);
    cplx<T> *s = reinterpret_cast<cplx<T> *>(smem_raw) + c * cp;
    const T *xs = (a.xsel && *a.xsel) ? a.xs[1] : a.xs[0];
    const int r0 = (blockIdx.x * a.W + c) * 2;
    const bool ok0 = cv && r0 < a.nrows, ok1 = cv && r0 + 1 < a.nrows;
    const long long o0 = (long long)r0 * a.B1, o1 = o0 + a.B1;
    with_r1<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
        int e = t + a.c1;
        if (e >= N) e -= N;
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const bool in = e < a.B1;
            T va = (in && ok0) ? xs[o0 + e] : (T)0, vb = (in && ok1) ? xs[o1 + e] : (T)0;
            if (a.support) {
                const uint8_t sa = (in && ok0) ? a.support[o0 + e] : (uint8_t)0, sb = (in && ok1) ? a.support[o1 + e] : (uint8_t)0;
                va *= (T)sa;
                vb *= (T)sb;
            }
            if (a.positivity) {
                if (va < (T)0) va = 0;
                if (vb < (T)0) vb = 0;
            }
            x[m] = mk(va, vb);
            e += tp.R2;
            if (e >= N) e -= N;
        }
        RDft<T, R>::run(x);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (k) x[k] = cmul(x[k], __ldg(a.tw + t * k));
            s[k * tp.row + t] = x[k];
        }
    });
    __syncthreads();
    with_r2<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
#pragma unroll
        for (int m = 0; m < R; ++m) x[m] = s[tB * tp.row + m];
        RDft<T, R>::run(x);
        __syncthreads();
#pragma unroll
        for (int m = 0; m < R; ++m)
            if (onB) s[t + tp.R1 * m] = x[m];
    });
    __syncthreads();
    // Xa(q) = (Z(q) + conj Z(-q)) / 2, Xb(q) = (Z(q) - conj Z(-q)) / 2i
    if (!cv) return;
    cplx<T> *ya = a.Y + (long long)r0 * a.ld1, *yb = ya + a.ld1;
    for (int q = t; q < a.h1; q += tp.R2) {
        const cplx<T> Z = s[q], Zm = s[q == 0 ? 0 : N - q];
        if (ok0) ya[q] = mk((T)0.5 * (Z.x + Zm.x), (T)0.5 * (Z.y - Zm.y));
        if (ok1) yb[q] = mk((T)0.5 * (Z.y + Zm.y), (T)0.5 * (Zm.x - Z.x));
    }
}

template <typename T, int RMAX, class Plan>
__device__ __forceinline__ void row_c2r_two(const RowPassArgs<T> &a, const Plan &tp, int cp)
{
    pass_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (row_pairs_empty(a, a.W)) return;
    const int N = tp.N;
    const int c = threadIdx.x / tp.R2, t = threadIdx.x - c * tp.R2;
    const bool cv = c < a.W;  // (the tile has room for the last warp's threads beyond it)
    const bool onB = t < tp.R1;
    const int tB = min(t, tp.R1 - 1);
    cplx<T> *s = reinterpret_cast<cplx<T> *>(smem_raw) + c * cp;
    T *xs = (a.xsel && *a.xsel) ? a.xs[1] : a.xs[0];
    const int r0 = (blockIdx.x * a.W + c) * 2;
    const bool ok0 = cv && r0 < a.nrows, ok1 = cv && r0 + 1 < a.nrows;
    with_r1<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
        // Z = Ha + i Hb; entry i >= h1 is the conjugate pair of N - i
        const cplx<T> *ya = a.Y + (long long)r0 * a.ld1, *yb = ya + a.ld1;
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int i = t + tp.R2 * m;
            const bool up = i >= a.h1;
            const int q = up ? N - i : i;
            cplx<T> ha = ok0 ? ya[q] : mk((T)0, (T)0), hb = ok1 ? yb[q] : mk((T)0, (T)0);
            if (q == 0 || 2 * q == N) { ha.y = 0; hb.y = 0; }
            if (up) { ha.y = -ha.y; hb.y = -hb.y; }
            x[m] = mk(ha.x - hb.y, ha.y + hb.x);
        }
        RDft<T, R>::run(x);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (k) x[k] = cmul(x[k], __ldg(a.tw + t * k));
            s[k * tp.row + t] = x[k];
        }
    });
    __syncthreads();
    with_r2<RMAX>(tp, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        cplx<T> x[R];
#pragma unroll
        for (int m = 0; m < R; ++m) x[m] = s[tB * tp.row + m];
        RDft<T, R>::run(x);
        int e = (tB ? N - tB : 0) + a.c1;
        if (e >= N) e -= N;
        const int cnt = onB ? a.B1 : 0;  // (ok0 and ok1 are false beyond the CTA's pairs)
#pragma unroll
        for (int m = 0; m < R; ++m) {
            if (e < cnt) {
                if (ok0) xs[(long long)r0 * a.B1 + e] = scaled(x[m].x, a);
                if (ok1) xs[(long long)(r0 + 1) * a.B1 + e] = scaled(x[m].y, a);
            }
            e -= tp.R1;
            if (e < 0) e += N;
        }
    });
}

template <typename T, int RMAX>
__global__ void __launch_bounds__(kTwoMaxThreads, two_min_blocks<T, RMAX>()) k_row_r2c_two(RowPassArgs<T> a, TwoPlan tp, int cp)
{
    row_r2c_two<T, RMAX>(a, tp, cp);
}
template <typename T, int RMAX>
__global__ void __launch_bounds__(kTwoMaxThreads, two_min_blocks<T, RMAX>()) k_row_c2r_two(RowPassArgs<T> a, TwoPlan tp, int cp)
{
    row_c2r_two<T, RMAX>(a, tp, cp);
}
template <int R1, int R2> constexpr int two_fixed_cp() { return two_tile(FixedPlan<R1, R2>{}) | 1; }
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(two_fixed_threads(R2, two_width<T>(R1 * R2)), two_fixed_blocks(R2, two_width<T>(R1 * R2)))
    k_row_r2c_fixed(RowPassArgs<T> a)
{
    row_r2c_two<T, 32>(a, FixedPlan<R1, R2>{}, two_fixed_cp<R1, R2>());
}
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(two_fixed_threads(R2, two_width<T>(R1 * R2)), two_fixed_blocks(R2, two_width<T>(R1 * R2)))
    k_row_c2r_fixed(RowPassArgs<T> a)
{
    row_c2r_two<T, 32>(a, FixedPlan<R1, R2>{}, two_fixed_cp<R1, R2>());
}

// ---------------------------------------------------------------------------
// host side (fft_two.cu and fft_two_fp64.cu hold the run-time kernels, the
// fft_two_fixed*.cu the complex64 lengths with a kernel of their own)
// ---------------------------------------------------------------------------
// Both launchers return false when the length has no two-factor split.  The
// run-time kernels with radices above 16 are built for complex128 only: the
// complex64 lengths that need them have kernels of their own (two_fixed).
template <typename T> bool launch_col_two(const ColPassArgs<T> &a, int other, cudaStream_t st);
template <typename T> bool launch_rows_two(const RowPassArgs<T> &a, bool forward, cudaStream_t st);

// one length's launchers
struct TwoFixed {
    int n;
    void (*col)(const ColPassArgs<float> &a, int other, cudaStream_t st);
    void (*rows)(const RowPassArgs<float> &a, bool forward, cudaStream_t st);
};
const TwoFixed *two_fixed(int n);  // nullptr: no kernel of its own

// complex128 lengths up to 256 with a second factor above 16 and at least 1.5
// times the first (125, 162, 200, 216, 243 and 250) stay with the generic engine:
// the run-time kernels' 32 values a thread leave two CTAs per SM, and a third or
// more of their threads are idle in the second stage.  An iteration of a cube, us,
// two-stage / generic: 200 points 1751 / 1510, 216 points 1890 / 1740, 250 points 4389 /
// 3239, and of the whole cube 125 points 1618 / 707, 243 points 6897 / 5164.  With a
// factor of 7 the generic engine's butterfly is the slower one (252 points 3049 / 5669),
// and above 256 points its passes are (270 points 3781 / 5987).
inline bool two_unbalanced(const TwoPlan &p) { return p.N <= 256 && p.N % 7 && p.R2 > 16 && 2 * p.R2 >= 3 * p.R1; }

template <typename T> bool two_capable(int n)
{
    TwoPlan p;
    if (n > 1024 || !make_two_plan(n, p)) return false;
    return sizeof(T) == 8 ? !two_unbalanced(p) : p.R2 <= 16 || two_fixed(n);
}

// Mean gains (squared length, less 1) of complex64 arithmetic, from the rounding
// of its constants: of the root WR^j, of an R-point butterfly of this engine, of a
// whole transform of n points on it.
double root_gain(int j, int R);
double radix_gain(int R);
double two_gain(int n);

inline size_t two_row_smem(int nt, int R2, int cp, size_t es) { return (size_t)cp * ((nt + R2 - 1) / R2) * es; }

template <int R1, int R2> TwoFixed make_two_fixed()
{
    using P = FixedPlan<R1, R2>;
    constexpr int W = two_width<float>(P::N), NT = two_fixed_threads(R2, W);
    TwoFixed f;
    f.n = P::N;
    f.col = [](const ColPassArgs<float> &a, int other, cudaStream_t st) {
        launch_pass(k_col_fixed<float, R1, R2>, dim3(cdiv(a.ncols, W), other), NT, (size_t)two_tile(P{}) * W * sizeof(float2), st, a);
    };
    f.rows = [](const RowPassArgs<float> &a, bool forward, cudaStream_t st) {
        const dim3 grid(cdiv((a.nrows + 1) / 2, W));
        const size_t sm = two_row_smem(NT, R2, two_fixed_cp<R1, R2>(), sizeof(float2));
        if (forward) launch_pass(k_row_r2c_fixed<float, R1, R2>, grid, NT, sm, st, a);
        else launch_pass(k_row_c2r_fixed<float, R1, R2>, grid, NT, sm, st, a);
    };
    return f;
}

template <typename T> bool launch_col_two_impl(const ColPassArgs<T> &a, int other, cudaStream_t st)
{
    TwoPlan p;
    if (!two_capable<T>(a.pl.n) || !make_two_plan(a.pl.n, p)) return false;
    int lw = 0;
    while ((1 << lw) < a.W) ++lw;
    if ((1 << lw) != a.W || two_threads(p, a.W) > kTwoMaxThreads) return false;
    if constexpr (sizeof(T) == 4) {
        if (const TwoFixed *f = two_fixed(a.pl.n)) {
            f->col(a, other, st);
            return true;
        }
    }
    const dim3 grid(cdiv(a.ncols, a.W), other);
    const size_t sm = (size_t)two_tile(p) * a.W * sizeof(cplx<T>);
    if (p.R2 <= 16) launch_pass(k_col_two<T, 16>, grid, two_threads(p, a.W), sm, st, a, p, lw);
    else if constexpr (sizeof(T) == 8) launch_pass(k_col_two<T, 32>, grid, two_threads(p, a.W), sm, st, a, p, lw);
    return true;
}
template <typename T> bool launch_rows_two_impl(const RowPassArgs<T> &a, bool forward, cudaStream_t st)
{
    TwoPlan p;
    if (!two_capable<T>(a.pl.n) || !make_two_plan(a.pl.n, p) || two_threads(p, a.W) > kTwoMaxThreads) return false;
    if constexpr (sizeof(T) == 4) {
        if (const TwoFixed *f = two_fixed(a.pl.n)) {
            f->rows(a, forward, st);
            return true;
        }
    }
    const dim3 grid(cdiv((a.nrows + 1) / 2, a.W));
    const int cp = two_tile(p) | 1, nt = two_threads(p, a.W);
    const size_t sm = two_row_smem(nt, p.R2, cp, sizeof(cplx<T>));
    if (p.R2 <= 16) {
        if (forward) launch_pass(k_row_r2c_two<T, 16>, grid, nt, sm, st, a, p, cp);
        else launch_pass(k_row_c2r_two<T, 16>, grid, nt, sm, st, a, p, cp);
    } else if constexpr (sizeof(T) == 8) {
        if (forward) launch_pass(k_row_r2c_two<T, 32>, grid, nt, sm, st, a, p, cp);
        else launch_pass(k_row_c2r_two<T, 32>, grid, nt, sm, st, a, p, cp);
    }
    return true;
}

}  // namespace gf
