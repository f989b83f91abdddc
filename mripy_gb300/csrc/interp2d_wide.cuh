// 2-D interp (type-2 gridding) with wide stencils (18 to 30 taps per axis): k_interp2d_wide, one
// coil per block.
//
// What bounds it: shared-memory reads, 8 bytes per tap and up to 900 taps a sample; the general
// kernel ran one thread per sample (52 us for 32,768 samples of 28 taps on a 384^2 grid; this one 27).
//
// As k_interp3d_one: a warp per sample, 16 lanes read a row's taps two cells (16 bytes) at a
// time from the even cell at or below the first, two rows a step; a cell outside the stencil
// is left out by a select, so that a value that is not finite there does not reach the
// sum (and one inside does, also where the weight has flushed to zero).
#pragma once

#include "grid2d_kernels.cuh"

namespace gbn {

// 16-byte units per staged row
__host__ __device__ inline int wide_row_units(const Geom &g) { return (g.tile[1] + g.W - 1 + 2) / 2; }
// One unit more than the window: the lane past a sample's last tap (its weights are zero) reads
// the unit behind the row where the sample is in the last cell of an even tile whose window
// starts on an odd cell.
inline size_t interp2d_wide_smem(const Geom &g) {
    if (g.dim != 2 || g.W < kWideMinW || g.W > kWideMaxW) return 0;
    return ((size_t)(g.tile[0] + g.W - 1) * wide_row_units(g) + 1) * sizeof(float4);
}

__global__ void __launch_bounds__(256) k_interp2d_wide(InterpArgs a, int vec, int coil0) {
    extern __shared__ float4 smem_iw[];  // [WX][R] pairs of y cells
    const Geom &g = a.g;
    const int4 sub = a.subs[blockIdx.x];
    const int coil = coil0 + blockIdx.y, grp = sub.x / g.ntiles;
    int o[3], e[3];
    tile_coords<2>(g, sub.x % g.ntiles, o, e);
    const int W = g.W, ns = g.ns;
    const int WX = g.tile[0] + W - 1, R = wide_row_units(g);
    const int nf0 = g.nf[0], nf1 = g.nf[1];
    const int ws0 = o[0] - (ns - 1), ws1 = o[1] - (ns - 1);
    const int ys = ws1 & ~1, offy = ws1 - ys;
    const float2 *gbase = a.grid + ((int64_t)grp * g.n_coil + coil) * g.G;
    const float rR = 1.f / (float)R;
#pragma unroll 4
    for (int i = threadIdx.x; i < WX * R; i += blockDim.x) {
        const int x = div_small(i, rR), p = i - x * R;
        const float2 *row = gbase + (int64_t)wrap_fast(ws0 + x, nf0) * nf1;
        if (vec) {
            smem_iw[i] = *reinterpret_cast<const float4 *>(row + wrap_fast(ys + 2 * p, nf1));
        } else {
            const float2 u = row[wrap_fast(ys + 2 * p, nf1)], w = row[wrap_fast(ys + 2 * p + 1, nf1)];
            smem_iw[i] = make_float4(u.x, u.y, w.x, w.y);
        }
    }
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int xo = lane >> 4, py = lane & 15;
    const bool live = py <= W / 2;
    for (int s = warp; s < sub.z; s += nw) {
        const float4 p = a.pts[(int64_t)sub.y + s];
        const uint32_t j = a.idx[(int64_t)sub.y + s];
        int c0[3], rel[2];
        unpack_cells(2, __float_as_uint(p.w), c0[0], c0[1], c0[2]);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            int cc = c0[d] + ns - 1;
            cc -= cc >= g.nf[d] ? g.nf[d] : 0;
            rel[d] = cc - o[d];
        }
        // lane k: the weight of x tap k; every lane its own two y weights
        const float dx = p.x + (float)(ns - 1 - lane);
        const float wxl = ex2_approx(-g.beta2[0] * dx * dx);
        const int yr = rel[1] + offy, ky = 2 * py - (yr & 1);
        float wy[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float d = p.y + (float)(ns - 1 - ky - t);
            const float ex = ex2_approx(-g.beta2[1] * d * d);
            wy[t] = live && (unsigned)(ky + t) < (unsigned)W ? ex : -1.f;  // -1: not a tap
        }
        const float4 *base = smem_iw + (rel[0] + xo) * R + (yr >> 1) + (live ? py : 0);
        float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
#pragma unroll 5
        for (int kx = 0; kx < W; kx += 2) {  // W is even: both rows are taps
            const float w = __shfl_sync(0xffffffffu, wxl, kx + xo);
            const float4 u = base[kx * R];
            const float2 w2 = make_float2(w, w);
            a0 = __ffma2_rn(w2, make_float2(u.x, u.y), a0);
            a1 = __ffma2_rn(w2, make_float2(u.z, u.w), a1);
        }
        float x = 0.f, y = 0.f;
        if (wy[0] >= 0.f) { x = wy[0] * a0.x; y = wy[0] * a0.y; }
        if (wy[1] >= 0.f) { x = fmaf(wy[1], a1.x, x); y = fmaf(wy[1], a1.y, y); }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, m);
            y += __shfl_xor_sync(0xffffffffu, y, m);
        }
        if (lane == 0) {
            const float sc = a.weight ? a.weight[j] : 1.f;
            a.c[(int64_t)j * a.c_elem + (int64_t)coil * a.c_coil] = make_float2(x * sc, y * sc);
        }
    }
}

}  // namespace gbn
