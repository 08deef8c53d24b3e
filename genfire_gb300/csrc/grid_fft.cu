// grid_fft.cu -- FFT gridding, @GENFIRE_Reconstructor/fillInFourierGrid.m
// (griddingMethod = 1, the class default), on the GPU.
//
//   1. k_pad_ishift    each projection zero-padded to m x m with its centre kept
//                      (My_paddzero) and ifftshifted, in the pass precision
//   2. 2-D FFT         the column passes of fft.cuh along dims 1 and 2, batched
//                      over the projections (my_fft, fillInFourierGrid.m:59-61)
//   3. k_fft_gather    one CTA per pair of rows (k2, k3), (-k2, -k3) of the cube:
//                    the samples R'(kx, ky, 0) (FP32, :80-89) within the cutoff of
//                    the rows' voxels and their shift range (:108-139), weights
//                    1/(d + 1e-5) (:155-157), FP64 sums of w*F and w (:159-160) in
//                    shared memory, then FS = sum(w F) / sum(w) (:161) and
//                    hermitianSymmetrize (:163, src/hermitianSymmetrize.m:22-65),
//                    cast to the output precision: every voxel written once
//                      (or k_fft_scatter and k_fft_finalize, the same by atomics
//                    on the cube, where those are faster: scatter_faster)
//   4. recIFFT         rec_ifft (dr.cu): My_stripzero(real(my_ifft(K))) (:165)
//
// Differences from the reference, by design: the sums are FP64 (the reference
// accumulates single-precision products with accumarray), and they are atomic,
// so their order -- and the last bits of a sum with several terms -- does not
// follow the reference's list order.  The FP64 path also transforms the
// projections in FP64 (the reference pads to single precision); the MIXED
// path transforms in FP32 as the reference does.
#include "internal.h"

namespace gf {

int fft_grid_size(int Dim2, double ratio)
{
    const double m = (Dim2 % 2 == 0) ? (double)Dim2 * ratio : 1.0 + (double)(Dim2 - 1) * ratio;
    const double r = mround(m);
    if (std::fabs(m - r) > 1e-9 || r < 1 || r > 65535) return -1;
    return (int)r;
}

void grid_dims(const genfire_params &p, int &n1, int &n2)
{
    if (p.griddingMethod == 1) {
        const int m = fft_grid_size(p.Dim2, p.oversamplingRatio);
        if (m < 0)
            fail(GENFIRE_ERR_ARG, "FFT gridding: Dim2 * oversamplingRatio (1 + (Dim2-1) * oversamplingRatio for odd "
                                  "Dim2) must be an integer.");
        n1 = n2 = m;
    } else {
        n1 = oversampled(p.Dim1, p.oversamplingRatio);
        n2 = oversampled(p.Dim2, p.oversamplingRatio);
    }
}

__device__ __forceinline__ int wrap(int a, int n)
{
    a %= n;
    return a < 0 ? a + n : a;
}

// grid: x over dim 1 of the projection, y = dim-2 index, z = projection
template <typename T>
__global__ void k_pad_ishift(const double *__restrict__ proj, int D1, int D2, int m, cplx<T> *__restrict__ X)
{
    const int y = blockIdx.y, p = blockIdx.z;
    const int ty = wrap(y - D2 / 2, m);
    const double *src = proj + (size_t)p * D1 * D2 + (size_t)D1 * y;
    cplx<T> *dst = X + (size_t)p * m * m + (size_t)m * ty;
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < D1; x += gridDim.x * blockDim.x)
        dst[wrap(x - D1 / 2, m)] = mk((T)src[x], (T)0);
}

struct FftGridGeom {
    int m, s, P;        // cube size, shift range, projections
    float cut_le;       // for a float d: d <= cutoff (in double) iff d <= cut_le, the largest float not above it
    float reach;        // cutoff + 0.01: covers the FP32 rounding of the coordinates (below 1e-3 for grids up to 2^11)
};

// One projection's slice: sample (kx, ky) lies at (r0 kx + r1 ky, r2 kx + r3 ky,
// r4 kx + r5 ky), and n is the slice's normal (used for bounds only).
struct __align__(16) FftSlice {
    float r[6], n[3], pad[3];
};

constexpr int kGatherThreads = 128;
constexpr int kMerge = 4;  // lanes on one voxel from which a warp adds them up before the atomics
constexpr int kMaxCube = 1290;  // the largest m with m^3 below 2^31
constexpr size_t gather_smem(int m) { return sizeof(double) * 6 * (size_t)(2 * (m / 2) + 1); }

// Conversions between single and double by integer arithmetic, where the
// hardware's would issue on the FP64 pipe: exact widening, and narrowing rounded
// to nearest even; subnormal, infinite and NaN values take the instruction.
__device__ __forceinline__ double widen(float x)
{
    const uint32_t b = __float_as_uint(x), e = b & 0x7F800000u;
    if (e == 0u || e == 0x7F800000u) return (b << 1) ? (double)x : __hiloint2double((int)b, 0);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ float narrow(double x)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const uint32_t a = hi & 0x7FFFFFFFu;
    if ((a | lo) == 0u) return __uint_as_float(hi);
    if (a < 0x38100000u || a >= 0x47E00000u) return (float)x;  // below 2^-126, or 2^127 and above
    // the 23 significand bits kept, then half a unit less one plus the last kept bit
    const uint32_t keep = ((a - 0x38000000u) << 3) | (lo >> 29), rest = lo & 0x1FFFFFFFu;
    const uint32_t up = (rest + 0x0FFFFFFFu + (keep & 1u)) >> 29;
    return __uint_as_float((hi & 0x80000000u) | (keep + up));
}

// Gather of the samples near a row pair.  The samples of the row A = (k2, k3)
// and of its mate B = (-k2, -k3) mirror each other: projections are real, the
// slice coordinates, distances and weights of sample -s at -k are those of s at
// k (every FP32 step is odd or even in its arguments), so a test serves both:
// s adds to A's voxel k, and -s, with its own value, to B's voxel -k.  With an
// even m the last index has no mirror in the grid (-m/2 has no m/2): the loops
// run over -h .. h and each side counts only the samples and voxels it has.
//
// Bound: the FP64 pipe (2 operations per clock per SM; 75 % busy), with the sums
// and their compare-and-swap retries: 90 projections of 256 x 256, cutoff 0.7,
// 512^3 cube, 31 M pairs in 1.52 ms.  A scatter from the samples with FP64
// atomics into sums of the whole cube, cleared before and read back after (24
// bytes a voxel, 3.2 GB), took 5.1 ms for that gridding without recIFFT, 1.8 ms
// this way.
//
// A warp takes the projections in groups; each lane finds the interval of k1
// that can lie within reach of its slice, and the intervals of the group are
// dealt to the lanes candidate by candidate, so that long ones (slices nearly
// parallel to k1) cost no more than their candidates.  The pairs found go to a
// queue of the warp's in shared memory and are summed 32 at a time, one per
// lane: about one candidate in three yields a pair, and summing inside the test
// loop left each lane alone with its loads and atomics (3.56 ms).  One entry per
// candidate, its samples added in registers first, measured 1.67 ms; a second
// queue for a candidate's later pairs, which retry on the same voxel, 1.71.
//
// MERGE: where many of the 32 lie on one voxel (the axis of a tilt series, repeated
// angles), the retries are a serial chain, and the lanes add up their values first:
// 400 tilts of 48 x 48 (96^3 cube) 464 -> 301 us a call, one angle 100 times at 64 x
// 64 293 -> 153 (kMerge = 6: 310 and 155; 8: 333; 12: 385).  With random angles
// finding those lanes costs more than it saves (192^3 cube, 80 projections 228 -> 238).
template <typename T, bool MERGE>
__global__ void __launch_bounds__(kGatherThreads) k_fft_gather(const cplx<T> *__restrict__ X, const FftSlice *__restrict__ sl,
                                                               FftGridGeom g, unsigned long long *__restrict__ pairs,
                                                               cplx<T> *__restrict__ M)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *acc = reinterpret_cast<double *>(smem_raw);  // [row A / B][re, im, weight][2 h + 1], B indexed by A's k1
    __shared__ uint2 qpos[kGatherThreads / 32][64];   // {k1 + h | p << 16, i + h | (j + h) << 16}
    __shared__ float qw[kGatherThreads / 32][64];
    const int m = g.m, h = m / 2, hi = m - 1 - h, L = 2 * h + 1;  // indices -h .. hi are in the grid
    const int k2 = (int)blockIdx.x - h, k3 = blockIdx.y;
    if (k3 == 0 && k2 < 0) return;  // its mate's pair
    const bool inA = k2 <= hi && k3 <= hi, inB = -k2 <= hi;  // (k2 >= -h and -k3 <= 0 always)
    const bool self = k2 == 0 && k3 == 0;
    if (!inA && !inB) return;
    for (int i = threadIdx.x; i < 6 * L; i += kGatherThreads) acc[i] = 0.0;
    __syncthreads();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr int NW = kGatherThreads / 32;
    const int per = min(32, (g.P + NW - 1) / NW);  // projections of a warp's group
    const float K2 = (float)k2, K3 = (float)k3;
    unsigned cnt = 0;
    int queued = 0;  // pairs in the warp's queue (uniform)
    // sums the queue's first n (at most 32) pairs
    auto drain = [&](int n) {
        __syncwarp();
        int k1 = 0;
        double A[3] = {0.0, 0.0, 0.0}, B[3] = {0.0, 0.0, 0.0};  // MERGE: w re, w im, w of the pair's two samples
        if (lane < n) {
            const uint2 q = qpos[warp][lane];
            const double wgt = widen(qw[warp][lane]);
            k1 = (int)(q.x & 0xFFFFu) - h;
            const int p = (int)(q.x >> 16);
            const int i = (int)(q.y & 0xFFFFu) - h, j = (int)(q.y >> 16) - h;
            const cplx<T> *Xp = X + (size_t)p * m * m;
            const bool onA = inA && k1 <= hi && i <= hi && j <= hi;
            const bool onB = inB && !self && -k1 <= hi && -i <= hi && -j <= hi;
            cplx<T> va = mk((T)0, (T)0), vb = va;
            if (onA) va = Xp[(i < 0 ? i + m : i) + (size_t)m * (j < 0 ? j + m : j)];
            if (onB) vb = Xp[(i > 0 ? m - i : -i) + (size_t)m * (j > 0 ? m - j : -j)];
            auto add = [&](double *to, double (&v)[3], cplx<T> val) {
                if (val.x == (T)-999 && val.y == (T)0) return;  // the reference's flag of a bad value
                if constexpr (MERGE) {
                    v[0] = widen(val.x) * wgt;
                    v[1] = widen(val.y) * wgt;
                    v[2] = wgt;
                } else {
                    atomicAdd(to, widen(val.x) * wgt);
                    atomicAdd(to + L, widen(val.y) * wgt);
                    atomicAdd(to + 2 * L, wgt);
                }
                ++cnt;
            };
            if (onA) add(acc + k1 + h, A, va);
            if (onB) add(acc + 3 * L + k1 + h, B, vb);
        }
        if constexpr (MERGE) {
            // the lanes of one voxel as a list, which is summed into its first lane, and
            // that alone adds to the row (next: the lane whose partial sum continues this
            // one's, or itself at the end)
            const unsigned peers = __match_any_sync(0xffffffffu, lane < n ? k1 : m + lane);
            bool first = lane < n;
            if (__any_sync(0xffffffffu, __popc(peers) >= kMerge)) {
                first = first && lane == __ffs(peers) - 1;
                const unsigned above = lane == 31 ? 0u : peers & (0xffffffffu << (lane + 1));
                int next = above ? __ffs(above) - 1 : lane;
                while (__any_sync(0xffffffffu, next != lane)) {
                    const bool more = next != lane;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double a = __shfl_sync(0xffffffffu, A[c], next), b = __shfl_sync(0xffffffffu, B[c], next);
                        if (more) {
                            A[c] += a;
                            B[c] += b;
                        }
                    }
                    const int n2 = __shfl_sync(0xffffffffu, next, next);
                    next = more ? (n2 == next ? lane : n2) : lane;
                }
            }
            if (first) {
                double *to = acc + k1 + h;
                // (a weight is positive, and told by its bits: no FP64 compare)
                if (__double2hiint(A[2]))
                    for (int c = 0; c < 3; ++c) atomicAdd(to + c * L, A[c]);
                if (__double2hiint(B[2]))
                    for (int c = 0; c < 3; ++c) atomicAdd(to + (3 + c) * L, B[c]);
            }
        }
        __syncwarp();
        if (lane < queued - n) {  // the rest (fewer than 32) moves to the front
            qpos[warp][lane] = qpos[warp][n + lane];
            qw[warp][lane] = qw[warp][n + lane];
        }
        queued -= n;
        __syncwarp();
    };
    for (int p0 = warp * per; p0 < g.P; p0 += NW * per) {
        int lo = 0, len = 0;
        if (lane < per && p0 + lane < g.P) {
            const FftSlice &s = sl[p0 + lane];
            const float n1 = s.n[0], x = -(s.n[1] * K2 + s.n[2] * K3);
            int a = -h, b = h;
            if (fabsf(n1) >= 0.01f) {
                const float in = 1.0f / n1;
                float u = (x - g.reach) * in, v = (x + g.reach) * in;
                if (u > v) { const float t = u; u = v; v = t; }
                // (reach's 0.01 / |n1| covers the bounds' rounding)
                a = max(a, (int)ceilf(fmaxf(u, (float)-h - 4.f)));
                b = min(b, (int)floorf(fminf(v, (float)h + 4.f)));
            } else if (fabsf(x) > g.reach + fabsf(n1) * (float)h) {
                b = a - 1;
            }
            lo = a;
            len = max(0, b - a + 1);
        }
        int end = len;  // inclusive scan of the lengths
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += y;
        }
        const int total = __shfl_sync(0xffffffffu, end, 31);
        const int first = lo - (end - len);  // k1 = first + candidate number
        for (int c0 = 0; c0 < total; c0 += 32) {
            const int c = c0 + lane;
            // the interval holding candidate c: the first lane with end > c
            int at = 0;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const int y = __shfl_sync(0xffffffffu, end, at + o - 1);
                if (y <= c) at += o;
            }
            const int src = min(at, 31);
            const int k1 = __shfl_sync(0xffffffffu, first, src) + c;
            const int p = p0 + src;
            const FftSlice &s = sl[min(p, g.P - 1)];
            const float K1 = (float)k1;
            const float w = fmaf(s.n[0], K1, fmaf(s.n[1], K2, s.n[2] * K3));
            const float rest = g.reach * g.reach - w * w;
            int i0 = 0, j0 = 0, ni = 0, nj = 0;  // the samples that can be near: i0 .. i0 + ni - 1 by j0 .. j0 + nj - 1
            if (c < total && rest >= 0.f) {
                const float u = fmaf(s.r[0], K1, fmaf(s.r[2], K2, s.r[4] * K3));  // in-plane coordinates of the voxel
                const float v = fmaf(s.r[1], K1, fmaf(s.r[3], K2, s.r[5] * K3));
                const float rho = sqrtf(rest) + 0.01f;
                i0 = max(-h, (int)ceilf(u - rho));
                j0 = max(-h, (int)ceilf(v - rho));
                ni = max(0, min(h, (int)floorf(u + rho)) - i0 + 1);
                nj = max(0, min(h, (int)floorf(v + rho)) - j0 + 1);
            }
            const int most = __reduce_max_sync(0xffffffffu, ni * nj);
            int i = i0, j = j0;
            for (int t = 0; t < most; ++t) {
                bool hit = t < ni * nj;
                float wgt = 0.f;
                if (hit) {
                    const float kx = (float)i, ky = (float)j;
                    const float cx = __fadd_rn(__fmul_rn(s.r[0], kx), __fmul_rn(s.r[1], ky));
                    const float cy = __fadd_rn(__fmul_rn(s.r[2], kx), __fmul_rn(s.r[3], ky));
                    const float cz = __fadd_rn(__fmul_rn(s.r[4], kx), __fmul_rn(s.r[5], ky));
                    const float dx = __fsub_rn(cx, K1), dy = __fsub_rn(cy, K2), dz = __fsub_rn(cz, K3);
                    const float d = __fsqrt_rn(
                        __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
                    const float far = (float)g.s;  // the voxel is a shift of at most s from the nearest one
                    hit = d <= g.cut_le && fabsf(K1 - roundf(cx)) <= far && fabsf(K2 - roundf(cy)) <= far &&
                          fabsf(K3 - roundf(cz)) <= far;
                    wgt = __fdiv_rn(1.0f, __fadd_rn(d, 1e-5f));
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int o = queued + __popc(hits & ((1u << lane) - 1u));
                    qpos[warp][o] = make_uint2((uint32_t)(k1 + h) | (uint32_t)p << 16, (uint32_t)(i + h) | (uint32_t)(j + h) << 16);
                    qw[warp][o] = wgt;
                }
                queued += __popc(hits);
                if (queued >= 32) drain(32);
                if (++i == i0 + ni) {
                    i = i0;
                    ++j;
                }
            }
        }
    }
    if (queued) drain(queued);
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(pairs, (unsigned long long)cnt);
    __syncthreads();
    // FS = sum(w F) / sum(w) where sum(w) > 0, else 0: in FP64 for the FP64 output,
    // in FP32 from the FP64 sums for the single-precision output (no FP64
    // arithmetic).  The weight sum is >= 0, so it is positive iff its bits, as an
    // integer, are.
    auto average = [&](const double *q) -> cplx<T> {
        cplx<T> a = mk((T)0, (T)0);
        if (reinterpret_cast<const long long *>(q)[2 * L] > 0) {
            if constexpr (sizeof(T) == 8) {
                a = mk(q[0] / q[2 * L], q[L] / q[2 * L]);
            } else {
                const float w = narrow(q[2 * L]);
                a = mk(__fdiv_rn(narrow(q[0]), w), __fdiv_rn(narrow(q[L]), w));
            }
        }
        return a;
    };
    // hermitianSymmetrize: k and -k averaged over the number of non-zero ones, a
    // value outside the grid being zero
    cplx<T> *rowA = M + (size_t)m * ((k2 + h) + (size_t)m * (k3 + h)) + h;
    cplx<T> *rowB = M + (size_t)m * ((h - k2) + (size_t)m * (h - k3)) + h;
    for (int i = threadIdx.x; i < L; i += kGatherThreads) {
        const int k1 = i - h;
        const cplx<T> a = average(acc + i), b = average(self ? acc + (2 * h - i) : acc + 3 * L + i);
        const T half = (a.x != 0 || a.y != 0) && (b.x != 0 || b.y != 0) ? (T)0.5 : (T)1;
        const T re = (a.x + b.x) * half;
        if (inA && k1 <= hi) rowA[k1] = mk(re, (a.y - b.y) * half);
        if (inB && !self && -k1 <= hi) rowB[-k1] = mk(re, (b.y - a.y) * half);
    }
}

// The scatter: one thread per sample (x over the centred dim-1 index i, y = j, z =
// projection), FP64 atomics on sums of the whole cube in global memory, which
// k_fft_finalize averages and symmetrises.  Those atomics need no retries, but
// the cube's sums, 24 bytes a voxel, are cleared, updated and read back.
template <typename T>
__global__ void __launch_bounds__(128) k_fft_scatter(const cplx<T> *__restrict__ X, const FftSlice *__restrict__ sl,
                                                     FftGridGeom g, double2 *__restrict__ num,
                                                     double *__restrict__ ws, unsigned long long *__restrict__ pairs)
{
    const int m = g.m, h = m / 2;
    const int j = blockIdx.y, p = blockIdx.z;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned cnt = 0;
    if (i < m) {
        // centred (i, j) of my_fft = FFT index (i - h, j - h) mod m
        const cplx<T> val = X[(size_t)p * m * m + wrap(i - h, m) + (size_t)m * wrap(j - h, m)];
        if (!(val.x == (T)-999 && val.y == (T)0)) {
            const float *r = sl[p].r;
            const float kx = (float)(i - h), ky = (float)(j - h);
            const float cx = __fadd_rn(__fmul_rn(r[0], kx), __fmul_rn(r[1], ky));
            const float cy = __fadd_rn(__fmul_rn(r[2], kx), __fmul_rn(r[3], ky));
            const float cz = __fadd_rn(__fmul_rn(r[4], kx), __fmul_rn(r[5], ky));
            const float rx = roundf(cx), ry = roundf(cy), rz = roundf(cz);
            for (int ys = -g.s; ys <= g.s; ++ys)
                for (int xs = -g.s; xs <= g.s; ++xs)
                    for (int zs = -g.s; zs <= g.s; ++zs) {
                        const float tx = __fadd_rn(rx, (float)xs), ty = __fadd_rn(ry, (float)ys),
                                    tz = __fadd_rn(rz, (float)zs);
                        const int ix = (int)tx + h, iy = (int)ty + h, iz = (int)tz + h;
                        if (ix < 0 || ix >= m || iy < 0 || iy >= m || iz < 0 || iz >= m) continue;
                        const float dx = __fsub_rn(cx, tx), dy = __fsub_rn(cy, ty), dz = __fsub_rn(cz, tz);
                        const float d = __fsqrt_rn(
                            __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
                        if (!(d <= g.cut_le)) continue;
                        const double w = (double)__fdiv_rn(1.0f, __fadd_rn(d, 1e-5f));
                        const size_t v = (size_t)ix + (size_t)m * (iy + (size_t)m * iz);
                        atomicAdd(&num[v].x, (double)val.x * w);
                        atomicAdd(&num[v].y, (double)val.y * w);
                        atomicAdd(&ws[v], w);
                        ++cnt;
                    }
        }
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(pairs, (unsigned long long)cnt);
}

// sum(w F) / sum(w) where sum(w) > 0, else 0: in FP64 for the FP64 output,
// in FP32 from the FP64 sums for the single-precision output (no FP64
// arithmetic: this part's FP64 pipe issues 2 operations per clock per SM).
// The weight sum is >= 0, so it is positive iff its bits, as an integer, are.
template <typename TO>
__device__ __forceinline__ cplx<TO> fs_avg(const double2 *__restrict__ num, const double *__restrict__ ws, size_t v)
{
    cplx<TO> a = mk((TO)0, (TO)0);
    if (reinterpret_cast<const long long *>(ws)[v] > 0) {
        const double2 s = num[v];
        if constexpr (sizeof(TO) == 8) {
            const double w = ws[v];
            a = mk(s.x / w, s.y / w);
        } else {
            const float w = (float)ws[v];
            a = mk(__fdiv_rn((float)s.x, w), __fdiv_rn((float)s.y, w));
        }
    }
    return a;
}

// grid: x over dim 1, y = dim-2 index, z = dim-3 index of the m^3 cube.
// hermitianSymmetrize: mate of (i, j, k) is (e-1-i, e-1-j, e-1-k) on the
// odd-extended cube (e = m + 1 for even m), zero beyond the input; the two
// values are averaged over the number of non-zero ones.
template <typename TO>
__global__ void k_fft_finalize(const double2 *__restrict__ num, const double *__restrict__ ws, int m,
                               cplx<TO> *__restrict__ M)
{
    const int j = blockIdx.y, k = blockIdx.z;
    const int e = m + (m % 2 == 0);
    const int mj = e - 1 - j, mk_ = e - 1 - k;
    const size_t row = (size_t)m * (j + (size_t)m * k);
    const size_t mrow = (size_t)m * (mj + (size_t)m * mk_);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const int mi = e - 1 - i;
        const cplx<TO> a = fs_avg<TO>(num, ws, row + i);
        cplx<TO> b = mk((TO)0, (TO)0);
        if (mi < m && mj < m && mk_ < m) b = fs_avg<TO>(num, ws, mrow + mi);
        TO re = a.x + b.x, im = a.y - b.y;
        const int cnt = (a.x != 0 || a.y != 0) + (b.x != 0 || b.y != 0);
        if (cnt == 2) { re *= (TO)0.5; im *= (TO)0.5; }
        M[row + i] = mk(re, im);
    }
}

// Whether many samples of a voxel come from different slices: the slices share an
// axis or a plane.  With N the mean of n n' over the slices' unit normals, an
// eigenvalue of N is then near zero (its determinant), or two are (the sum of its
// principal 2 x 2 minors).  Of the first it takes many slices for the size of the cube
// to make up for MERGE, of the second few do.  us a call without MERGE / with it,
// complex64, tilt series: 100 on a 128^3 cube, cutoff 0.7 168 / 149, 0.2 92.6 / 92.3; 120 on
// 200^3 358 / 331, 170 / 175; 100 on 320^3 727 / 718, 341 / 356.
static bool shared_axis(const std::vector<FftSlice> &sl, int m)
{
    double N[6] = {0, 0, 0, 0, 0, 0};  // xx, yy, zz, xy, xz, yz
    for (const FftSlice &f : sl) {
        const double x = f.n[0], y = f.n[1], z = f.n[2];
        N[0] += x * x; N[1] += y * y; N[2] += z * z;
        N[3] += x * y; N[4] += x * z; N[5] += y * z;
    }
    for (double &v : N) v /= (double)sl.size();
    const double minors = N[0] * N[1] - N[3] * N[3] + N[0] * N[2] - N[4] * N[4] + N[1] * N[2] - N[5] * N[5];
    const double det = N[0] * (N[1] * N[2] - N[5] * N[5]) - N[3] * (N[3] * N[2] - N[5] * N[4]) + N[4] * (N[3] * N[5] - N[1] * N[4]);
    return (sl.size() >= 96 && 4 * sl.size() >= 3 * (size_t)m && det < 1e-3) || (sl.size() >= 16 && minors < 0.01);
}

// Scatter or gather.  The gather's sums cost more per pair (read, add, compare and
// swap in shared memory, and the rows near the origin, which every projection
// reaches, are few CTAs' work); the scatter's cost is the cube and the 27 or more
// shifts tested per sample.  So the scatter is for many pairs per sample, and
// for many projections of small ones.  us a call without recIFFT, complex64, random
// angles, gather / scatter:
//   cutoff 0.7, 100 projections: 64^3 103 / 88, 96^3 130 / 124, 128^3 142 / 178
//   cutoff 0.3, 400 projections: 16^3 113 / 93, 64^3 135 / 133
//   cutoff 1,    31 projections: 64^3 108 / 80, 128^3 137 / 141, 256^3 404 / 611
//   cutoff 1.5,  31 projections: 128^3 264 / 202, 256^3 827 / 739; one: 256^3 131 / 218
//   cutoff 3,    31 projections: 32^3 420 / 143, 128^3 1358 / 789; one: 32^3 105 / 124
// The rule: 100 pairs or more per sample position, all projections together, of
// cubes up to 48 + 16 times the pairs per sample (any size from 8 pairs on, which
// one to three projections make up for only from 128 points on).  Shifts beyond 8
// and windows wider than the cube stay with the gather, whose tests end at the
// cube's and the slices' edges.
static bool scatter_faster(int m, int P, int s, double cutoff)
{
    const double side = 2 * s + 1, c = std::max(cutoff, 0.0);
    const double pairs = std::min(4.18879 * c * c * c, side * side * side);  // per sample
    if (P * std::max(pairs, 0.5) < 100 || s > 8 || 2 * s >= m) return false;
    return pairs >= 8 ? P >= 4 || m >= 128 : m <= 48 + 16 * pairs;
}

template <typename T>
static void grid_fft_t(genfire_ctx *ctx, const genfire_params &p, const double *d_proj, const double *angles,
                       void *d_M, void *d_rec, int64_t *npairs)
{
    cudaStream_t st = ctx->stream;
    const int D1 = p.Dim1, D2 = p.Dim2, P = p.NumProjs;
    const int m = fft_grid_size(D2, p.oversamplingRatio);
    const size_t mm = (size_t)m * m;
    // 1-2: centred spectra of the padded projections (kept in FFT order)
    DevBuf X(sizeof(cplx<T>) * mm * P, st);
    GF_CUDA(cudaMemsetAsync(X.p, 0, X.bytes, st));
    k_pad_ishift<T><<<dim3(cdiv(D1, 128), D2, P), 128, 0, st>>>(d_proj, D1, D2, m, X.as<cplx<T>>());
    GF_CHECK_LAUNCH();
    fftn_device(ctx, sizeof(T) == 8 ? GENFIRE_PREC_FP64 : GENFIRE_PREC_MIXED, X.p, m, m, P, false, 3);
    // slice rotation: rotkCoords = R' [kx; ky; 0] with R of fillInFourierGrid.m:80-82,
    // which is the transpose of the projector's ZYZ matrix, so the rows are
    // (Rz(1,1), Rz(1,2)), (Rz(2,1), Rz(2,2)), (Rz(3,1), Rz(3,2)) in single precision
    std::vector<float> hr(6 * (size_t)P);
    for (int q = 0; q < P; ++q) {
        double R[9];
        rot_zyz(angles[q], angles[q + P], angles[q + 2 * P], R);
        float *r = &hr[6 * (size_t)q];
        r[0] = (float)R[0]; r[1] = (float)R[3];
        r[2] = (float)R[1]; r[3] = (float)R[4];
        r[4] = (float)R[2]; r[5] = (float)R[5];
    }
    std::vector<FftSlice> hs(P);
    for (int q = 0; q < P; ++q) {
        const float *r = &hr[6 * (size_t)q];
        FftSlice &f = hs[q];
        for (int k = 0; k < 6; ++k) f.r[k] = r[k];
        f.n[0] = r[2] * r[5] - r[4] * r[3];  // the first column times the second
        f.n[1] = r[4] * r[1] - r[0] * r[5];
        f.n[2] = r[0] * r[3] - r[2] * r[1];
        f.pad[0] = f.pad[1] = f.pad[2] = 0.f;
    }
    DevBuf dsl(sizeof(FftSlice) * hs.size(), st), dpairs(sizeof(unsigned long long), st);
    GF_CUDA(cudaMemcpyAsync(dsl.p, hs.data(), sizeof(FftSlice) * hs.size(), cudaMemcpyHostToDevice, st));
    GF_CUDA(cudaMemsetAsync(dpairs.p, 0, sizeof(unsigned long long), st));
    // 3: weighted averages and Hermitian symmetry
    FftGridGeom g;
    g.m = m;
    g.P = P;
    g.s = p.allowMultipleGridMatches ? (int)mround(p.interpolationCutoffDistance) : 0;
    g.cut_le = (float)p.interpolationCutoffDistance;
    if ((double)g.cut_le > p.interpolationCutoffDistance) g.cut_le = std::nextafter(g.cut_le, -INFINITY);
    // no pair is farther than its shift range and half a voxel allow
    const double reach = std::min(p.interpolationCutoffDistance, 1.7321 * (g.s + 0.5));
    g.reach = (float)reach + 0.01f;
    bool scatter = scatter_faster(m, P, g.s, p.interpolationCutoffDistance);
    DevBuf num, ws;
    if (scatter) {
        try {
            num.alloc(sizeof(double2) * mm * m, st);
            ws.alloc(sizeof(double) * mm * m, st);
        } catch (const Error &e) {
            if (e.st != GENFIRE_ERR_OOM) throw;
            num.release();
            scatter = false;  // the gather needs no sums of the cube
        }
    }
    if (scatter) {
        GF_CUDA(cudaMemsetAsync(num.p, 0, num.bytes, st));
        GF_CUDA(cudaMemsetAsync(ws.p, 0, ws.bytes, st));
        k_fft_scatter<T><<<dim3(cdiv(m, 128), m, P), 128, 0, st>>>(X.as<cplx<T>>(), dsl.as<FftSlice>(), g, num.as<double2>(),
                                                                   ws.as<double>(), dpairs.as<unsigned long long>());
        GF_CHECK_LAUNCH();
        k_fft_finalize<T><<<dim3(cdiv(m, 256), m, m), 256, 0, st>>>(num.as<double2>(), ws.as<double>(), m,
                                                                     reinterpret_cast<cplx<T> *>(d_M));
    } else {
        const int h = m / 2;
        const auto gather = shared_axis(hs, m) ? k_fft_gather<T, true> : k_fft_gather<T, false>;
        raise_smem_limit(ctx->device, (const void *)gather, gather_smem(kMaxCube));
        gather<<<dim3(2 * h + 1, h + 1), kGatherThreads, gather_smem(m), st>>>(
            X.as<cplx<T>>(), dsl.as<FftSlice>(), g, dpairs.as<unsigned long long>(), reinterpret_cast<cplx<T> *>(d_M));
    }
    GF_CHECK_LAUNCH();
    num.release();
    ws.release();
    X.release();
    // 4: recIFFT
    if (d_rec) rec_ifft(ctx, p.precision, d_M, m, m, D1, D2, d_rec);
    unsigned long long hp = 0;
    GF_CUDA(cudaMemcpyAsync(&hp, dpairs.p, sizeof(hp), cudaMemcpyDeviceToHost, st));
    GF_CUDA(cudaStreamSynchronize(st));
    if (npairs) *npairs = (int64_t)hp;
}

void grid_fft(genfire_ctx *ctx, const genfire_params &p, const double *d_proj, const double *angles, void *d_M,
              void *d_rec, int64_t *npairs)
{
    const int m = fft_grid_size(p.Dim2, p.oversamplingRatio);
    if (m < 0)
        fail(GENFIRE_ERR_ARG, "FFT gridding: Dim2 * oversamplingRatio (1 + (Dim2-1) * oversamplingRatio for odd "
                              "Dim2) must be an integer.");
    if (m < p.Dim1 || m < p.Dim2) fail(GENFIRE_ERR_ARG, "FFT gridding: the grid is smaller than the projections.");
    static_assert((long long)kMaxCube * kMaxCube * kMaxCube < (1LL << 31), "largest cube");
    if (m > kMaxCube) fail(GENFIRE_ERR_ARG, "FFT gridding: grid too large (m^3 must stay below 2^31).");
    if (p.NumProjs > 65535) fail(GENFIRE_ERR_ARG, "FFT gridding: at most 65535 projections.");
    if (p.precision == GENFIRE_PREC_FP64) grid_fft_t<double>(ctx, p, d_proj, angles, d_M, d_rec, npairs);
    else grid_fft_t<float>(ctx, p, d_proj, angles, d_M, d_rec, npairs);
}

}  // namespace gf
