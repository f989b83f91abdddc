// 3-D interp (type-2 gridding) of one coil per block: k_interp3d_one<WT>, for plans of 1 to 6
// coils where that measured faster than groups of coils (interp_one_coil in api.cu).
//
// What bounds it: shared-memory reads (8 bytes per tap; W^3 taps a sample) and, behind them,
// issue.  With one coil the warp's lanes have to split a sample's own taps.  Here a lane reads
// two z cells at once (16 bytes) of one y row: W / 2 + 1 lanes cover a row's taps from the even
// cell below the first, and the warp takes several rows a step: 5 rows of 6 lanes for 10 taps
// (2 steps a plane), else 4 rows of 8 lanes (3 steps for 12 taps).  One 16-byte load and two
// packed FMAs then serve 60 (or 52) of 64 cells, against one 8-byte load and one FMA for 20 of
// 32 in the loop of k_interp3d.
//
// The window (tile + W - 1 cells per axis, periodic) is staged in rows of R 16-byte units
// whose first cell is even in the grid, so aligned grids are read 16 bytes at a time.  8-lane
// rows never conflict (a quarter warp reads 128 contiguous bytes).  For the 6-lane rows R = 1
// (mod 8), and a step takes the rows {0, 6, 4, 2, 8} + step: their 6-unit runs then start at
// units 0, 6, 12, 18, 24 (mod 8), i.e. the warp's units are consecutive mod 8 and no quarter
// warp conflicts.
// Lanes without taps (2 of 32 there, up to 3 of 8 in the 8-lane rows) repeat the first unit of
// their own row.  Sent to the sample's first unit instead they conflict with their quarter
// warp: 768,000 samples 0.385 -> 0.373 ms at 10 taps, 0.910 -> 0.571 at 12, 0.430 -> 0.308 at 8.
#pragma once

#include "grid2d_kernels.cuh"

namespace gbn {

constexpr int kOneMaxW = 14;  // W / 2 + 1 lanes a row, at most 8

// Bins of at most this many samples read their taps from the grid itself (through L1) instead
// of staging a window: a window is 5,000 to 6,900 cells however few the samples.  Measured
// against staging every bin: 256,000 samples of 12 taps on a 192^3 grid (35 a bin) 0.285 ->
// 0.262 ms; 115,000 of 10 taps (15 a bin) 0.132 -> 0.108; 768,000 of 10 taps (110 a bin) 0.378
// -> 0.372.  16 instead of 32 measures the same.
constexpr int kOneDirect = 32;

// 16-byte units per staged row
__host__ __device__ inline int one_row_units(const Geom &g) {
    int r = (g.tile[2] + g.W - 1 + 2) / 2;  // one cell more in front when the window starts odd
    if (g.W == 10) r = ((r + 6) & ~7) + 1;
    return r;
}
// One unit more than the window: a sample in the last cell of an even tile whose window starts
// on an odd cell has its W / 2 lanes end the row, and the lane past them (its weights are zero)
// reads the unit behind it.  (Sending that lane to the sample's first unit instead: 20 density
// iterations of 768,000 samples 16.1 ms against 15.1.)
inline size_t interp3d_one_smem_bytes(const Geom &g) {
    if (g.dim != 3 || g.W > kOneMaxW || (g.W & 1)) return 0;
    return ((size_t)(g.tile[0] + g.W - 1) * (g.tile[1] + g.W - 1) * one_row_units(g) + 1) * sizeof(float4);
}

template <int WT>
__global__ void __launch_bounds__(256) k_interp3d_one(InterpArgs a, int vec) {
    extern __shared__ float4 smem_i1[];  // [WX][WY][R] pairs of z cells
    const Geom &g = a.g;
    const int4 sub = a.subs[blockIdx.x];
    const int coil = blockIdx.y;
    const int grp = sub.x / g.ntiles;
    int o[3], e[3];
    tile_coords<3>(g, sub.x % g.ntiles, o, e);
    const int W = WT ? WT : g.W;
    const int ns = g.ns;
    const int WX = g.tile[0] + W - 1, WY = g.tile[1] + W - 1, R = one_row_units(g);
    const int nf0 = g.nf[0], nf1 = g.nf[1], nf2 = g.nf[2];
    const int ws0 = o[0] - (ns - 1), ws1 = o[1] - (ns - 1), ws2 = o[2] - (ns - 1);
    const int zs = ws2 & ~1, offz = ws2 - zs;  // even (also below zero)
    const float2 *gbase = a.grid + ((int64_t)grp * g.n_coil + coil) * g.G;
    const bool direct = vec && sub.z <= kOneDirect;
    if (!direct) {
        const int n = WX * WY * R;
        const float rR = 1.f / (float)R, rWY = 1.f / (float)WY;
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int xy = div_small(i, rR), p = i - xy * R;
            const int wx = div_small(xy, rWY), wy = xy - wx * WY;
            const int gx = wrap_fast(ws0 + wx, nf0), gy = wrap_fast(ws1 + wy, nf1);
            const float2 *row = gbase + ((int64_t)gx * nf1 + gy) * nf2;
            float4 v;
            if (vec) {  // nf2 even, 16-byte aligned grid: the pair lies within the row
                v = *reinterpret_cast<const float4 *>(row + wrap_fast(zs + 2 * p, nf2));
            } else {
                const float2 u = row[wrap_fast(zs + 2 * p, nf2)], w = row[wrap_fast(zs + 2 * p + 1, nf2)];
                v = make_float4(u.x, u.y, w.x, w.y);
            }
            smem_i1[i] = v;
        }
        __syncthreads();
    }

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    constexpr bool SIX = WT == 10;                      // 5 rows of 6 lanes; else 4 rows of 8
    constexpr int STEPS = SIX ? 2 : (WT ? (WT + 3) / 4 : (kOneMaxW + 3) / 4);
    const int grow = SIX ? lane / 6 : lane >> 3, pz = SIX ? lane % 6 : lane & 7;
    const int row0 = SIX ? (grow >= 4 ? 8 : (grow == 0 ? 0 : 8 - 2 * grow)) : grow;  // {0, 6, 4, 2, 8}
    const bool live = SIX ? lane < 30 : pz <= W / 2;
    const int rstep = SIX ? 1 : 4;
    const int kk = lane & 15;
    const float beta = lane < 16 ? g.beta2[0] : g.beta2[1];
    float4 p_next = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t j_next = 0;
    if (warp < sub.z) {
        p_next = a.pts[(int64_t)sub.y + warp];
        j_next = a.idx[(int64_t)sub.y + warp];
    }
    for (int s = warp; s < sub.z; s += nw) {
        const float4 p = p_next;
        const uint32_t j = j_next;
        if (s + nw < sub.z) {
            p_next = a.pts[(int64_t)sub.y + s + nw];
            j_next = a.idx[(int64_t)sub.y + s + nw];
        }
        int c0[3], rel[3];
        unpack_cells(3, __float_as_uint(p.w), c0[0], c0[1], c0[2]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            int cc = c0[d] + ns - 1;
            cc -= cc >= g.nf[d] ? g.nf[d] : 0;
            rel[d] = cc - o[d];
        }
        // lanes 0..15 the x weights, 16..31 the y weights, every lane its own two z weights
        float myw = 0.f;
        if (kk < W) {
            const float d = (lane < 16 ? p.x : p.y) + (float)(ns - 1 - kk);
            myw = ex2_approx(-beta * d * d);
        }
        const int zr = rel[2] + offz, kz = 2 * pz - (zr & 1);
        float wz[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float d = p.z + (float)(ns - 1 - kz - t);
            const float ex = ex2_approx(-g.beta2[2] * d * d);
            wz[t] = live && (unsigned)(kz + t) < (unsigned)W ? ex : -1.f;  // -1: not a tap
        }
        float wy[STEPS];
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int ky = row0 + rstep * i;
            const float v = __shfl_sync(0xffffffffu, myw, 16 + min(ky, 15));
            wy[i] = live && ky < W ? v : 0.f;
        }
        // a lane without taps repeats its row's first pair (its sums are not used), which a lane of
        // its quarter warp reads anyway: any other pair would be a bank conflict
        int off[STEPS];
        float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
        auto plane_sum = [&](const float4 *plane, float wx) {
#pragma unroll
            for (int i = 0; i < STEPS; ++i) {
                if ((WT == 0 || WT % 4) && !SIX && row0 + rstep * i >= W) continue;  // rows past the stencil
                const float4 v = plane[off[i]];
                const float w = wx * wy[i];
                const float2 w2 = make_float2(w, w);
                a0 = __ffma2_rn(w2, make_float2(v.x, v.y), a0);
                a1 = __ffma2_rn(w2, make_float2(v.z, v.w), a1);
            }
        };
        if (direct) {
            const int y0 = ws1 + rel[1], gz = wrap_fast(zs + (zr & ~1) + (live ? 2 * pz : 0), nf2) >> 1;
#pragma unroll
            for (int i = 0; i < STEPS; ++i)
                off[i] = wrap_fast(y0 + row0 + rstep * i, nf1) * (nf2 >> 1) + gz;
            const float4 *gb = reinterpret_cast<const float4 *>(gbase);
            const int64_t ps = (int64_t)nf1 * (nf2 >> 1);
            int gx = wrap_fast(ws0 + rel[0], nf0);
#pragma unroll(WT ? WT : 2)
            for (int kx = 0; kx < W; ++kx) {
                plane_sum(gb + gx * ps, __shfl_sync(0xffffffffu, myw, kx));
                gx = gx + 1 == nf0 ? 0 : gx + 1;
            }
        } else {
            const float4 *base = smem_i1 + ((size_t)rel[0] * WY + rel[1]) * R + (zr >> 1);
#pragma unroll
            for (int i = 0; i < STEPS; ++i) off[i] = (row0 + rstep * i) * R + (live ? pz : 0);
#pragma unroll(WT ? WT : 2)
            for (int kx = 0; kx < W; ++kx)
                plane_sum(base + (size_t)kx * WY * R, __shfl_sync(0xffffffffu, myw, kx));
        }
        // a grid value that is not finite must reach the sum from inside the stencil (also where
        // the weight has flushed to zero) and not from outside: select
        float x = 0.f, y = 0.f;
        if (wz[0] >= 0.f) { x = wz[0] * a0.x; y = wz[0] * a0.y; }
        if (wz[1] >= 0.f) { x = fmaf(wz[1], a1.x, x); y = fmaf(wz[1], a1.y, y); }
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
