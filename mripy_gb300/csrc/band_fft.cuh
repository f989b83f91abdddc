// Transforms between image and oversampled grid with pad, deapodisation and crop fused in:
// k_fft_rows_in (image -> transformed grid rows), k_fft_cols (a strided axis, in place) and
// k_fft_rows_out / k_fft_rows_sense (grid rows -> image).
//
// What bounds them: the bytes moved, through L1 and HBM.  An oversampled grid is zero outside the
// image band before the forward transform, and only the band is read after the inverse one.  A
// pad kernel, a library transform over the whole grid and a crop kernel move the grid 5 (2-D) to
// 7 (3-D) times; here an axis is transformed only on the band of the axes that come later, so
// type 2 reads the image once and moves 1/2 + 1/2 + 1 grids in 2-D (1/4 + 1/4 + 1/2 + 1/2 + 1
// in 3-D), and type 1 the same backwards.
//
// A line of N = R1 R2 cells is two register passes with one exchange through shared memory:
// a thread reads the R1 cells j + r R2 straight from the image or grid, transforms them,
// and writes them to shared memory; after one barrier it reads the R2 cells of output k,
// multiplies them by the twiddles W_N^{k r} (a table rounded from FP64), transforms them and
// writes the cells k + r R1 out.  A block of a strided pass takes fft_cols lines, adjacent cells
// of the inner axis (16: 128-byte rows; 8 where a radix is above 18), a block of a row pass
// kFftLines (row, coil) pairs, where the image side takes coils or pixels fastest, whichever is
// contiguous.  The transform in place is safe because a block's lines are its own and all of them
// are read before the barrier.
//
// Lengths: the products of two radices listed in band_fft_{a..f}.cu: 32 of the 42 even products of
// 2, 3 and 5 from 64 to 768 (not 90, 250, 450, 486, 500, 540, 600, 648, 720 and 750), and 112,
// 168, 224 and 336: one in ten of the even lengths there, the ones of the usual image sizes.  A plan
// with one other axis takes pad kernel, library transform and crop kernel.
//
// Measured (before: pad or crop kernel and cuFFT, band-pruned in 3-D): 64 x 12 images of
// 192^2 in 1.14 -> 0.49 ms and out 1.02 -> 0.48 ms; 8 images of 128^3 in 0.96 -> 0.56 ms, out
// 0.82 -> 0.55 ms.  The strided passes run at 69 to 77 % of the copy bandwidth with the L1/shared
// pipe at 73 to 78 %, two to four blocks per SM whose load, transform and store phases overlap
// only across blocks; the row passes at 3.3 TB/s wait for loads and barriers.  Error against 64
// bits: 1.3e-7 to 1.7e-7 (cuFFT 2.0e-7 to 2.6e-7).
//
// The inverse transform is the forward one with real and imaginary parts swapped on the way
// in and out.
#pragma once

#include <utility>

#include "common.cuh"

namespace gbn {

// ------------------------------------------------------------------ small transforms
namespace fft {

constexpr double kPi = 3.14159265358979323846;

// sine and cosine by their Taylor series on [0, pi/4]
constexpr double sin_small(double x) {
    double t = x, s = x;
    for (int n = 1; n < 12; ++n) {
        t *= -x * x / ((2 * n) * (2 * n + 1));
        s += t;
    }
    return s;
}
constexpr double cos_small(double x) {
    double t = 1, s = 1;
    for (int n = 1; n < 12; ++n) {
        t *= -x * x / ((2 * n - 1) * (2 * n));
        s += t;
    }
    return s;
}
constexpr double cos2pi(int k, int n) {  // cos(2 pi k / n)
    k %= n;
    double x = 2 * kPi * k / n;
    double sign = 1;
    if (x > kPi) x = 2 * kPi - x;
    if (x > kPi / 2) { x = kPi - x; sign = -1; }
    return sign * (x > kPi / 4 ? sin_small(kPi / 2 - x) : cos_small(x));
}
constexpr double sin2pi(int k, int n) {
    k %= n;
    double x = 2 * kPi * k / n;
    double sign = 1;
    if (x > kPi) { x = 2 * kPi - x; sign = -1; }
    if (x > kPi / 2) x = kPi - x;
    return sign * (x > kPi / 4 ? cos_small(kPi / 2 - x) : sin_small(x));
}

template <int... I, class F>
__device__ __forceinline__ void each_impl(std::integer_sequence<int, I...>, F f) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void each(F f) {  // f(0) .. f(N - 1) with constant arguments
    each_impl(std::make_integer_sequence<int, N>{}, f);
}

__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 mul(float2 a, float2 w) {
    return make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x));
}
// a exp(-2 pi i K / N)
template <int K0, int N>
__device__ __forceinline__ float2 turn(float2 a) {
    constexpr int K = K0 % N;
    if constexpr (K == 0) return a;
    else if constexpr (2 * K == N) return make_float2(-a.x, -a.y);
    else if constexpr (4 * K == N) return make_float2(a.y, -a.x);
    else if constexpr (4 * K == 3 * N) return make_float2(-a.y, a.x);
    else return mul(a, make_float2((float)cos2pi(K, N), (float)-sin2pi(K, N)));
}

template <int R> struct Dft;
template <> struct Dft<2> {
    static __device__ __forceinline__ void run(float2 (&v)[2]) {
        const float2 a = v[0];
        v[0] = add(a, v[1]);
        v[1] = sub(a, v[1]);
    }
};
template <> struct Dft<4> {
    static __device__ __forceinline__ void run(float2 (&v)[4]) {
        const float2 a = add(v[0], v[2]), b = sub(v[0], v[2]), c = add(v[1], v[3]), d = sub(v[1], v[3]);
        const float2 e = make_float2(d.y, -d.x);  // -i d
        v[0] = add(a, c);
        v[1] = add(b, e);
        v[2] = sub(a, c);
        v[3] = sub(b, e);
    }
};
// odd R: the sums and differences of the conjugate pairs (r, R - r)
template <int R>
__device__ __forceinline__ void dft_odd(float2 (&v)[R]) {
    constexpr int H = (R - 1) / 2;
    float2 s[H], d[H], x0 = v[0];
    each<H>([&](auto i) {
        s[i] = add(v[i + 1], v[R - 1 - i]);
        d[i] = sub(v[i + 1], v[R - 1 - i]);
        x0 = add(x0, s[i]);
    });
    float2 out[R];
    out[0] = x0;
    each<H>([&](auto k) {
        float2 e = v[0], o = make_float2(0.f, 0.f);
        each<H>([&](auto i) {
            constexpr int t = (k + 1) * (i + 1);
            constexpr float c = (float)cos2pi(t, R), w = (float)sin2pi(t, R);
            e = __ffma2_rn(make_float2(c, c), s[i], e);
            o = __ffma2_rn(make_float2(w, w), d[i], o);
        });
        out[k + 1] = make_float2(e.x + o.y, e.y - o.x);
        out[R - 1 - k] = make_float2(e.x - o.y, e.y + o.x);
    });
    each<R>([&](auto i) { v[i] = out[i]; });
}
template <> struct Dft<3> {
    static __device__ __forceinline__ void run(float2 (&v)[3]) { dft_odd<3>(v); }
};
template <> struct Dft<5> {
    static __device__ __forceinline__ void run(float2 (&v)[5]) { dft_odd<5>(v); }
};
template <> struct Dft<7> {
    static __device__ __forceinline__ void run(float2 (&v)[7]) { dft_odd<7>(v); }
};
// R = A B: n = B a + b, k = k1 + A k2
template <int A, int B>
__device__ __forceinline__ void dft_product(float2 (&v)[A * B]) {
    each<B>([&](auto b) {
        float2 c[A];
        each<A>([&](auto a) { c[a] = v[B * a + b]; });
        Dft<A>::run(c);
        each<A>([&](auto k) { v[B * k + b] = turn<b * k, A * B>(c[k]); });
    });
    float2 out[A * B];
    each<A>([&](auto k) {
        float2 c[B];
        each<B>([&](auto b) { c[b] = v[B * k + b]; });
        Dft<B>::run(c);
        each<B>([&](auto q) { out[k + A * q] = c[q]; });
    });
    each<A * B>([&](auto i) { v[i] = out[i]; });
}
#define GBN_DFT(R, A, B)                                                                         \
    template <> struct Dft<R> {                                                                  \
        static __device__ __forceinline__ void run(float2 (&v)[R]) { dft_product<A, B>(v); }     \
    }
GBN_DFT(8, 4, 2);
GBN_DFT(9, 3, 3);
GBN_DFT(10, 5, 2);
GBN_DFT(12, 4, 3);
GBN_DFT(14, 7, 2);
GBN_DFT(15, 5, 3);
GBN_DFT(16, 4, 4);
GBN_DFT(18, 9, 2);
GBN_DFT(20, 5, 4);
GBN_DFT(24, 8, 3);
GBN_DFT(32, 8, 4);
#undef GBN_DFT

}  // namespace fft

// ------------------------------------------------------------------ geometry

// Lines per block of a strided pass: 8 for the lengths with a radix above 18, whose cells take so
// many registers that only more, smaller blocks overlap their phases (384: 318 -> 285 us for
// 768 grids of 384^2); else 16 (with 8: 162 cells 81 -> 92 us, whose rows start off 64-byte
// boundaries; 256 unchanged).
constexpr int fft_cols(int r1, int r2) { return r1 > 18 || r2 > 18 ? 8 : 16; }

template <int R1, int R2, int LINES = kFftLines> struct FftLine {
    static constexpr int N = R1 * R2, LN = LINES;
    static constexpr int J = R1 < R2 ? R1 : R2;   // threads per line
    static constexpr int T = LINES * J;
    static constexpr int P = R1 + 1;              // exchange: output r of butterfly j at j P + r
    static constexpr int PITCH = (R2 * P) | 1;    // odd: adjacent lines on distinct banks
    static constexpr size_t SMEM = (size_t)LINES * PITCH * sizeof(float2);
    static constexpr int MAXR = R1 > R2 ? R1 : R2;
    // resident blocks the register budgets are set for.  Measured (256^3 grids, strided passes):
    // band in 3 blocks 0.46 ms against 2 blocks 0.57; band out 0.53 against 0.46.
    static constexpr int at_least_1(int b) { return b > 0 ? b : 1; }
    static constexpr int BLOCKS = at_least_1((MAXR <= 16 ? 768 : 512) / T);
    static constexpr int BLOCKS_IN = at_least_1((MAXR <= 16 && T >= 224 ? 768 : 512) / T);
    static constexpr int BLOCKS_OUT = at_least_1(512 / T);
};

__device__ __forceinline__ float2 swap_if(float2 v, int inv) { return inv ? make_float2(v.y, v.x) : v; }

// second pass: output k's R2 cells of line `line` of the exchange, twiddled and transformed
template <int R1, int R2>
__device__ __forceinline__ void fft_second(const float2 *line, int k, const float2 *__restrict__ tw, float2 (&v)[R2]) {
    using L = FftLine<R1, R2>;
    v[0] = line[k];
#pragma unroll
    for (int r = 1; r < R2; ++r) v[r] = fft::mul(line[r * L::P + k], __ldg(tw + k * r));
    fft::Dft<R2>::run(v);
}

// ------------------------------------------------------------------ strided axis, in place
// OUT: only the band's cells are written (before a crop); else only the band's cells are read
// and the others are zero (after a pad).
template <int R1, int R2, bool OUT>
__global__ void __launch_bounds__(FftLine<R1, R2, fft_cols(R1, R2)>::T,
                                  OUT ? FftLine<R1, R2, fft_cols(R1, R2)>::BLOCKS_OUT
                                      : FftLine<R1, R2, fft_cols(R1, R2)>::BLOCKS_IN)
    k_fft_cols(float2 *__restrict__ grid, FftCols a) {
    using L = FftLine<R1, R2, fft_cols(R1, R2)>;
    extern __shared__ float2 sm_fft[];
    const int ch = blockIdx.x % a.chunks, ob = blockIdx.x / a.chunks;
    const int inst = ob / a.n_sub, sub = ob - inst * a.n_sub;
    const int l = threadIdx.x % L::LN, jt = threadIdx.x / L::LN;
    const int col = ch * L::LN + l;
    const bool live = col < a.cols;
    // sub-volumes (the band planes of the axis in front) at the two ends of that axis
    const int64_t so = sub < a.sub_lo ? sub : sub + a.sub_skip;
    float2 *base = grid + (int64_t)inst * a.G + so * a.sub_stride + col;
    float2 *line = sm_fft + l * L::PITCH;
    const int hi0 = L::N - a.hi;
#pragma unroll
    for (int j = jt; j < R2; j += L::J) {
        float2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const int n = j + r * R2;
            v[r] = live && (OUT || n < a.lo || n >= hi0) ? base[n * a.stride] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = swap_if(v[r], a.inv);
        fft::Dft<R1>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) line[j * L::P + r] = v[r];
    }
    __syncthreads();
#pragma unroll
    for (int k = jt; k < R1; k += L::J) {
        float2 v[R2];
        fft_second<R1, R2>(line, k, a.tw, v);
        if (!live) continue;
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int n = k + r * R1;
            if (!OUT || n < a.lo || n >= hi0) base[n * a.stride] = swap_if(v[r], a.inv);
        }
    }
}

// ------------------------------------------------------------------ rows
// The block's line l: image row and coil; rows are (group, outer pixel) in order.  Worked out
// once per block (16 lines) and kept in shared memory.
struct FftLineId {
    int64_t grid;    // first cell of its grid row
    int64_t img;     // its image row
    int64_t sens;    // its row of the coil maps
    int i0, i1, grp; // outer pixel and group
    int live;
};
// table product of the line's outer axes (rows out: times the group's scale); loaded by every
// thread beside its cells, so that nothing waits for it at the barrier
__device__ __forceinline__ float fft_scale(const FftRows &a, const FftLineId &q, bool out) {
    const float s = a.tab0[q.i0] * (a.tab1 ? a.tab1[q.i1] : 1.f);
    return out ? s * a.grp_scale[q.grp] : s;
}
__device__ __forceinline__ void fft_lines(const FftRows &a, int rows0, int c0, FftLineId *sh) {
    if (threadIdx.x >= kFftLines) return;
    const int l = threadIdx.x, rl = l / a.cpc;
    const int coil = c0 + l - rl * a.cpc, gr = rows0 + rl;
    FftLineId q;
    q.live = rl < a.rpb && coil < a.n_coil && gr < a.n_rows;
    q.grid = q.img = q.sens = 0;
    q.i0 = q.i1 = q.grp = 0;
    if (q.live) {
        const int grp = gr / a.rows_per_grp, row = gr - grp * a.rows_per_grp;
        const int i0 = row / a.m1, i1 = row - i0 * a.m1;
        q.i0 = i0;
        q.i1 = i1;
        q.grp = grp;
        const int g0 = i0 - a.m0 / 2, g1 = i1 - a.m1 / 2;
        const int64_t x = g0 < 0 ? g0 + a.nf0 : g0;
        q.grid = (int64_t)(grp * a.n_coil + coil) * a.G +
                 (a.tab1 ? (x * a.nf1 + (g1 < 0 ? g1 + a.nf1 : g1)) : x) * a.nf;
        q.img = grp * a.IL.traj_stride + (int64_t)row * a.m * a.IL.elem_stride +
                (a.sens ? 0 : coil * a.IL.coil_stride);
        q.sens = (int64_t)row * a.m * a.SL.elem_stride + coil * a.SL.coil_stride;
    }
    sh[l] = q;
}

template <int R1, int R2, bool SENS>
__global__ void __launch_bounds__(FftLine<R1, R2>::T, FftLine<R1, R2>::BLOCKS)
    k_fft_rows_in(FftRows a, float2 *__restrict__ grid) {
    using L = FftLine<R1, R2>;
    extern __shared__ float2 sm_fft[];
    __shared__ FftLineId lines[kFftLines];
    const int hi0 = L::N - a.hi;
    fft_lines(a, (blockIdx.x / a.n_chunk) * a.rpb, (blockIdx.x % a.n_chunk) * a.cpc, lines);
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < kFftLines * R2; t += L::T) {
        const int l = a.lfast ? t % kFftLines : t / R2, j = a.lfast ? t / kFftLines : t % R2;
        const FftLineId &q = lines[l];
        const float2 *x = a.img + q.img;
        const bool live = q.live;
        const float s = fft_scale(a, q, false);
        float2 v[R1];
        if (SENS && live) {
            // coil maps: all loads of both arrays before the first use, without branches between
            // them (cells outside the band read the line's first pixel and are zeroed after); a
            // 2-D image's lines fill a part of the GPU, so a chain of loads is the kernel's time:
            // 256 lines of 4 and 8 coils 12.7 and 12.5 -> 9.3 and 8.7 us.  Without maps the
            // branches are the better: 64 frames of 12 coils, 192 lines, 208 against 238 us
            const float2 *sp = a.sens + q.sens;
            float2 w[R1];
            float f[R1];
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const int n = j + r * R2;
                const int i = n < a.lo ? n + a.hi : n - hi0;
                const bool in = i >= 0 && i < a.m;  // inside the band: [0, lo) or [hi0, N)
                const int ic = in ? i : 0;
                v[r] = x[ic * a.IL.elem_stride];
                w[r] = sp[ic * a.SL.elem_stride];
                f[r] = in ? s * a.tab[ic] : 0.f;
            }
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const int n = j + r * R2;
                const int i = n < a.lo ? n + a.hi : n - hi0;
                const float2 u = fft::mul(v[r], w[r]);
                v[r] = i >= 0 && i < a.m ? swap_if(make_float2(u.x * f[r], u.y * f[r]), a.inv) : make_float2(0.f, 0.f);
            }
        } else {
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const int n = j + r * R2;
                const int i = n < a.lo ? n + a.hi : n - hi0;
                v[r] = make_float2(0.f, 0.f);
                if (live && i >= 0 && i < a.m) {
                    const float2 u = x[i * a.IL.elem_stride];
                    const float f = s * a.tab[i];
                    v[r] = swap_if(make_float2(u.x * f, u.y * f), a.inv);
                }
            }
        }
        fft::Dft<R1>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) sm_fft[l * L::PITCH + j * L::P + r] = v[r];
    }
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < kFftLines * R1; t += L::T) {
        const int l = t / R1, k = t % R1;
        float2 v[R2];
        fft_second<R1, R2>(sm_fft + l * L::PITCH, k, a.tw, v);
        if (!lines[l].live) continue;
        float2 *g = grid + lines[l].grid + k;
#pragma unroll
        for (int r = 0; r < R2; ++r) g[r * R1] = swap_if(v[r], a.inv);
    }
}

// first pass of the row transforms that start from the grid
template <int R1, int R2>
__device__ __forceinline__ void fft_rows_load(const FftRows &a, const float2 *__restrict__ grid,
                                              const FftLineId *lines, float2 *sm) {
    using L = FftLine<R1, R2>;
#pragma unroll 1
    for (int t = threadIdx.x; t < kFftLines * R2; t += L::T) {
        const int l = t / R2, j = t % R2;
        const float2 *g = grid + lines[l].grid + j;
        const bool live = lines[l].live;
        float2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = live ? g[r * R2] : make_float2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = swap_if(v[r], a.inv);
        fft::Dft<R1>::run(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) sm[l * L::PITCH + j * L::P + r] = v[r];
    }
}

template <int R1, int R2>
__global__ void __launch_bounds__(FftLine<R1, R2>::T, FftLine<R1, R2>::BLOCKS)
    k_fft_rows_out(FftRows a, const float2 *__restrict__ grid) {
    using L = FftLine<R1, R2>;
    extern __shared__ float2 sm_fft[];
    __shared__ FftLineId lines[kFftLines];
    const int hi0 = L::N - a.hi;
    fft_lines(a, (blockIdx.x / a.n_chunk) * a.rpb, (blockIdx.x % a.n_chunk) * a.cpc, lines);
    __syncthreads();
    fft_rows_load<R1, R2>(a, grid, lines, sm_fft);
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < kFftLines * R1; t += L::T) {
        const int l = a.lfast ? t % kFftLines : t / R1, k = a.lfast ? t / kFftLines : t % R1;
        float2 v[R2];
        fft_second<R1, R2>(sm_fft + l * L::PITCH, k, a.tw, v);
        const FftLineId &q = lines[l];
        if (!q.live) continue;
        const float s = fft_scale(a, q, true);
        float2 *x = a.out + q.img;
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            const int n = k + r * R1;
            const int i = n < a.lo ? n + a.hi : n - hi0;
            if (i < 0 || i >= a.m) continue;
            const float f = s * a.tab[i];
            const float2 u = swap_if(v[r], a.inv);
            x[i * a.IL.elem_stride] = make_float2(u.x * f, u.y * f);
        }
    }
}

// grid rows -> sum over the coils of conj(S) times the image.  Up to kFftLines coils: the
// block holds all coils of its rows; more: one row, its coils in chunks, sums in registers.
template <int R1, int R2>
__global__ void __launch_bounds__(FftLine<R1, R2>::T, FftLine<R1, R2>::BLOCKS)
    k_fft_rows_sense(FftRows a, const float2 *__restrict__ grid) {
    using L = FftLine<R1, R2>;
    constexpr int U = (L::N + L::T - 1) / L::T;                     // pixels per thread of one row
    constexpr int B = (kFftLines * R1 + L::T - 1) / L::T;           // second-pass butterflies per thread
    extern __shared__ float2 sm_fft[];
    __shared__ FftLineId lines[kFftLines];
    const int hi0 = L::N - a.hi;
    float2 acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = make_float2(0.f, 0.f);
    for (int ck = 0; ck < a.n_chunk; ++ck) {
        const int c0 = ck * a.cpc;
        __syncthreads();  // the previous chunk is consumed
        fft_lines(a, blockIdx.x * a.rpb, c0, lines);
        __syncthreads();
        fft_rows_load<R1, R2>(a, grid, lines, sm_fft);
        __syncthreads();
        float2 w[B][R2];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int t = threadIdx.x + u * L::T;
            if (t < kFftLines * R1) fft_second<R1, R2>(sm_fft + (t / R1) * L::PITCH, t % R1, a.tw, w[u]);
        }
        __syncthreads();
        // the transformed lines, cell n at n (the exchange is consumed)
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int t = threadIdx.x + u * L::T;
            if (t >= kFftLines * R1) continue;
#pragma unroll
            for (int r = 0; r < R2; ++r) sm_fft[(t / R1) * L::PITCH + t % R1 + r * R1] = swap_if(w[u][r], a.inv);
        }
        __syncthreads();
        const int nc = min(a.cpc, a.n_coil - c0);
        const bool last = ck + 1 == a.n_chunk;
        auto pixel = [&](int rl, int i, float2 sum) {
            const FftLineId &q = lines[rl * a.cpc];
            if (!q.live) return sum;
            const int n = i >= a.hi ? i - a.hi : i + hi0;
            const float2 *sp = a.sens + q.sens + i * a.SL.elem_stride;
            const float2 *fp = sm_fft + rl * a.cpc * L::PITCH + n;
#pragma unroll 4
            for (int c = 0; c < nc; ++c) {
                const float2 s = sp[c * a.SL.coil_stride], f = fp[c * L::PITCH];
                sum.x += f.x * s.x + f.y * s.y;
                sum.y += f.y * s.x - f.x * s.y;
            }
            if (last) {
                const float f = fft_scale(a, q, true) * a.tab[i];
                a.out[q.img + i * a.IL.elem_stride] = make_float2(sum.x * f, sum.y * f);
            }
            return sum;
        };
        if (a.n_chunk == 1) {
            for (int t = threadIdx.x; t < a.rpb * a.m; t += L::T) {
                const int rl = t / a.m;
                pixel(rl, t - rl * a.m, make_float2(0.f, 0.f));
            }
        } else {  // one row per block
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = threadIdx.x + u * L::T;
                if (i < a.m) acc[u] = pixel(0, i, acc[u]);
            }
        }
    }
}

// ------------------------------------------------------------------ launchers of one length
// one table entry per supported length, filled by the band_fft_*.cu files
template <int R1, int R2>
struct FftLaunch {
    using L = FftLine<R1, R2>;
    template <typename K>
    static cudaError_t smem(K kern) {
        // raised once per kernel and process (the attribute does not change afterwards)
        if (L::SMEM <= 46 * 1024) return cudaSuccess;  // 48 KB less the static line records
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM);
    }
    static cudaError_t prepare() {
        cudaError_t e = smem(k_fft_cols<R1, R2, false>);
        if (e == cudaSuccess) e = smem(k_fft_cols<R1, R2, true>);
        if (e == cudaSuccess) e = smem(k_fft_rows_in<R1, R2, false>);
        if (e == cudaSuccess) e = smem(k_fft_rows_in<R1, R2, true>);
        if (e == cudaSuccess) e = smem(k_fft_rows_out<R1, R2>);
        if (e == cudaSuccess) e = smem(k_fft_rows_sense<R1, R2>);
        return e;
    }
    static cudaError_t cols(float2 *grid, const FftCols &a, int64_t blocks, bool out, cudaStream_t s) {
        using C = FftLine<R1, R2, fft_cols(R1, R2)>;
        if (out) k_fft_cols<R1, R2, true><<<(unsigned)blocks, C::T, C::SMEM, s>>>(grid, a);
        else k_fft_cols<R1, R2, false><<<(unsigned)blocks, C::T, C::SMEM, s>>>(grid, a);
        return cudaGetLastError();
    }
    static cudaError_t rows(float2 *grid, const FftRows &a, int64_t blocks, int kind, cudaStream_t s) {
        if (kind == kFftRowsIn && a.sens) k_fft_rows_in<R1, R2, true><<<(unsigned)blocks, L::T, L::SMEM, s>>>(a, grid);
        else if (kind == kFftRowsIn) k_fft_rows_in<R1, R2, false><<<(unsigned)blocks, L::T, L::SMEM, s>>>(a, grid);
        else if (kind == kFftRowsOut) k_fft_rows_out<R1, R2><<<(unsigned)blocks, L::T, L::SMEM, s>>>(a, grid);
        else k_fft_rows_sense<R1, R2><<<(unsigned)blocks, L::T, L::SMEM, s>>>(a, grid);
        return cudaGetLastError();
    }
    static FftEntry entry() { return FftEntry{R1 * R2, fft_cols(R1, R2), prepare, cols, rows}; }
};

}  // namespace gbn
