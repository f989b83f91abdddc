// Launchers of the fused image <-> grid transforms (band_fft.cuh) and the list of lengths.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"

namespace gbn {

// grid lengths with kernels: the products of two radices in band_fft_{a..f}.cu
extern const FftEntry *const fft_tables[];
extern const FftEntry fft_a[], fft_b[], fft_c[], fft_d[], fft_e[], fft_f[];
const FftEntry *const fft_tables[] = {fft_a, fft_b, fft_c, fft_d, fft_e, fft_f};

const FftEntry *fft_entry(int n) {
    for (const FftEntry *t : fft_tables)
        for (; t->n; ++t)
            if (t->n == n) return t;
    return nullptr;
}

cudaError_t fft_prepare(const FftEntry &e) {
    static std::mutex mu;
    static std::set<std::pair<int, int>> done;  // (device, length)
    int dev = 0;
    cudaError_t st = cudaGetDevice(&dev);
    if (st != cudaSuccess) return st;
    std::lock_guard<std::mutex> lock(mu);
    if (done.count({dev, e.n})) return cudaSuccess;
    st = e.prepare();
    if (st == cudaSuccess) done.insert({dev, e.n});
    return st;
}

namespace {
__global__ void k_fft_twiddles(int n, float2 *tw) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double s, c;
    sincospi(-2.0 * k / n, &s, &c);
    tw[k] = make_float2((float)c, (float)s);
}

struct Axis {
    int m, nf, lo, hi;
};
Axis axis(const DeapodArgs &a, int d) {
    return Axis{a.m[d], a.g.nf[d], a.m[d] - a.m[d] / 2, a.m[d] / 2};
}

cudaError_t strided(const BandFft &b, const DeapodArgs &a, int d, bool out, int inv, float2 *grid, cudaStream_t s) {
    const Geom &g = a.g;
    const Axis x = axis(a, d);
    FftCols c;
    c.G = g.G;
    c.lo = x.lo;
    c.hi = x.hi;
    c.tw = b.tw[d];
    c.inv = inv;
    if (d == 0) {
        c.stride = g.G / g.nf[0];
        c.cols = (int)c.stride;
        c.n_sub = c.sub_lo = 1;
        c.sub_skip = c.sub_stride = 0;
    } else {  // y of a 3-D grid, on the band's x planes
        const Axis p = axis(a, 0);
        c.stride = g.nf[2];
        c.cols = g.nf[2];
        c.n_sub = p.m;
        c.sub_lo = p.lo;
        c.sub_skip = p.nf - p.m;
        c.sub_stride = (int64_t)g.nf[1] * g.nf[2];
    }
    c.chunks = (c.cols + b.e[d]->lines - 1) / b.e[d]->lines;
    const int64_t blocks = (int64_t)g.n_coil * g.n_traj * c.n_sub * c.chunks;
    return b.e[d]->cols(grid, c, blocks, out, s);
}

bool coils_fastest(const gbn_layout &q) { return std::llabs(q.coil_stride) < std::llabs(q.elem_stride); }

FftRows rows_args(const BandFft &b, const DeapodArgs &a, int inv, gbn_layout L, const float2 *sens, gbn_layout SL,
                  bool coil_sum, int min_cpc) {
    const Geom &g = a.g;
    const int D = g.dim;
    const Axis x = axis(a, D - 1);
    FftRows r;
    r.G = g.G;
    r.rows_per_grp = a.m[0] * (D == 3 ? a.m[1] : 1);  // (fewer rows than grid cells: int)
    r.n_rows = r.rows_per_grp * g.n_traj;
    r.n_coil = g.n_coil;
    r.m0 = a.m[0];
    r.m1 = D == 3 ? a.m[1] : 1;
    r.nf0 = g.nf[0];
    r.nf1 = D == 3 ? g.nf[1] : 1;
    r.m = x.m;
    r.nf = x.nf;
    r.lo = x.lo;
    r.hi = x.hi;
    // a block's lines: coils x rows.  The coil sum needs all coils of a row (or one row and its
    // coils in chunks); otherwise the split that fills the block best, with chunks of at least
    // min_cpc coils (4: 32 bytes of a coil-last image; in host memory 8)
    const int n = g.n_coil;
    if (coil_sum) {
        r.n_chunk = (n + kFftLines - 1) / kFftLines;
        r.cpc = (n + r.n_chunk - 1) / r.n_chunk;
        r.rpb = r.n_chunk == 1 ? kFftLines / r.cpc : 1;
    } else {
        double best = 0;
        for (int k = (n + kFftLines - 1) / kFftLines; k <= n; ++k) {
            const int cpc = (n + k - 1) / k, rpb = kFftLines / cpc;
            if (best > 0 && cpc < min_cpc) break;
            const double used = (double)n * rpb / (k * kFftLines);
            if (used > best + 0.01) {
                best = used;
                r.cpc = cpc;
                r.rpb = rpb;
                r.n_chunk = (n + cpc - 1) / cpc;
            }
        }
    }
    r.tab0 = a.tab[0];
    r.tab1 = D == 3 ? a.tab[1] : nullptr;
    r.tab = a.tab[D - 1];
    r.grp_scale = a.grp_scale;
    r.tw = b.tw[D - 1];
    r.inv = inv;
    r.img = nullptr;
    r.out = nullptr;
    r.IL = L;
    r.sens = sens;
    r.SL = SL;
    r.lfast = r.cpc > 1 && coils_fastest(sens ? SL : L);
    return r;
}

int64_t row_blocks(const FftRows &r, bool coil_sum) {
    return (int64_t)((r.n_rows + r.rpb - 1) / r.rpb) * (coil_sum ? 1 : r.n_chunk);
}
}  // namespace

cudaError_t launch_fft_twiddles(int n, float2 *tw, cudaStream_t s) {
    k_fft_twiddles<<<(n + 127) / 128, 128, 0, s>>>(n, tw);
    return cudaGetLastError();
}

cudaError_t launch_band_fft_in(const BandFft &b, const DeapodArgs &a, int inv, const float2 *img, gbn_layout L,
                               const float2 *sens, gbn_layout SL, float2 *grid, cudaStream_t s) {
    NvtxRange range("gbn band fft in");
    const int D = a.g.dim;
    FftRows r = rows_args(b, a, inv, L, sens, SL, false,
                          sens ? 4 : std::max(4, host_min_cc(img, coils_fastest(L), a.g.n_coil, s)));
    r.img = img;
    cudaError_t e = b.e[D - 1]->rows(grid, r, row_blocks(r, false), kFftRowsIn, s);
    for (int d = D - 2; d >= 0 && e == cudaSuccess; --d) e = strided(b, a, d, false, inv, grid, s);
    return e;
}

cudaError_t launch_band_fft_out(const BandFft &b, const DeapodArgs &a, int inv, float2 *grid, float2 *img, gbn_layout L,
                                const float2 *sens, gbn_layout SL, cudaStream_t s) {
    NvtxRange range("gbn band fft out");
    const int D = a.g.dim;
    cudaError_t e = cudaSuccess;
    for (int d = 0; d <= D - 2 && e == cudaSuccess; ++d) e = strided(b, a, d, true, inv, grid, s);
    if (e != cudaSuccess) return e;
    FftRows r = rows_args(b, a, inv, L, sens, SL, sens != nullptr,
                          sens ? 4 : std::max(4, host_min_cc(img, coils_fastest(L), a.g.n_coil, s)));
    r.out = img;
    return b.e[D - 1]->rows(grid, r, row_blocks(r, sens != nullptr), sens ? kFftRowsSense : kFftRowsOut, s);
}

}  // namespace gbn
