// 2-D spread (type-1 gridding) with wide stencils (18 to 30 taps per axis; 28 at the functions'
// default accuracy eps = 1e-15), and with narrower ones for 1 to 3 coils: k_spread2d_wide, one
// coil per block.
//
// What bounds it: issue and latency.  A sample has up to 900 taps, so its 4 W^2 flops dwarf its
// bytes; the general kernel spent them on shared-memory float atomics (277 us for 32,768
// samples of 28 taps on a 384^2 grid; this kernel 18 us).
//
// As k_spread3d_few -- every warp holds the whole output tile, 32 x 32 cells: lane =
// x row, its 32 y cells as FP32x2 pairs, real and imaginary parts apart -- and takes its own
// 32-sample batches.  A (sample, tile) pair costs 8 packed FMAs per 8-cell y quarter that the
// stencil reaches (skipped otherwise, warp-uniform).  32 cells a side because a stencil nearly
// covers them: 3.4 pairs per sample, against 7.2 with 16-cell tiles.  The four partial tiles
// are added through shared memory in a fixed order.
//
// 1 to 3 coils below 18 taps, against the shared-memory rows of k_spread2d: 1 coil, 20 frames of
// 256^2 grids, 21,800 samples of 12 taps each 351 -> 90 us; 2 coils, 265,000 samples of 10 taps on
// a 1024^2 grid 210 -> 100; 3 coils, 20 frames of 256^2, 14,800 each 416 -> 164; only sparse random
// samples (15 a tile, 2 coils, 20 frames of 512^2) 79 -> 90.
//
// A value that is not finite reaches its own stencil and no other cells (guarded loop; by the
// taps in an instance of its own, as k_spread3d_few).
#pragma once

#include "grid2d_kernels.cuh"

namespace gbn {

constexpr int kWideTile = 32, kWideWarps = 4, kWideStride = 68;  // floats per staged sample: wx, wy, value
constexpr size_t kWideSmem = (size_t)kWideWarps * 32 * kWideStride * sizeof(float);
static_assert(kWideSmem >= 2 * 32 * 33 * sizeof(float2), "two partial tiles");

template <bool TAPS>
__global__ void __launch_bounds__(kWideWarps * 32, 4) k_spread2d_wide(SpreadArgs a, int coil0) {
    extern __shared__ float4 smem_wide[];
    const Geom &g = a.g;
    const int4 sub = a.subs[blockIdx.x];
    const int coil = coil0 + blockIdx.y, grp = sub.x / g.ntiles;
    int o[3], e[3];
    tile_coords<2>(g, sub.x % g.ntiles, o, e);
    // (tile_coords' axes 0, 1 of a 2-D grid)
    const int W = g.W, ns = g.ns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *st = reinterpret_cast<float *>(smem_wide) + warp * 32 * kWideStride;

    float2 re[16], im[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) re[i] = im[i] = make_float2(0.f, 0.f);

    auto fetch = [&](int base, float4 &p, float2 &v) {
        const int s = base + lane;
        p = make_float4(0.f, 0.f, 0.f, 0.f);
        v = make_float2(0.f, 0.f);
        if (s >= sub.z) return;
        p = a.pts[(int64_t)sub.y + s];
        const uint32_t j = a.idx[(int64_t)sub.y + s];
        v = a.c[(int64_t)j * a.c_elem + (int64_t)coil * a.c_coil];
        if (a.weight) {
            const float sw = a.weight[j];
            v = make_float2(v.x * sw, v.y * sw);
        }
    };

    float4 p;
    float2 v;
    if (warp * 32 < sub.z) fetch(warp * 32, p, v);
    for (int base = warp * 32; base < sub.z; base += kWideWarps * 32) {
        const int n = min(32, sub.z - base);
        int c0[3], r[2];
        unpack_cells(2, __float_as_uint(p.w), c0[0], c0[1], c0[2]);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            int rr = c0[d] - o[d];
            rr += rr < 0 ? g.nf[d] : 0;
            rr -= rr > g.nf[d] - W ? g.nf[d] : 0;
            r[d] = rr;
        }
        __syncwarp();  // the previous batch is consumed
        float4 *mine = reinterpret_cast<float4 *>(st + lane * kWideStride);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int d = q >> 3;
            const int t0 = 4 * (q & 7) - r[d];  // tap at the quad's first plane
            const float f = d ? p.y : p.x, k0 = (float)(ns - 1 - t0);
            float w4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float dd = f + (k0 - (float)i);
                const float ex = ex2_approx(-g.beta2[d] * dd * dd);
                w4[i] = (unsigned)(t0 + i) < (unsigned)W ? ex : 0.f;
            }
            mine[q] = make_float4(w4[0], w4[1], w4[2], w4[3]);
        }
        reinterpret_cast<float2 *>(mine + 16)[0] = v;
        unsigned hit[4];  // the y quarters each sample reaches
#pragma unroll
        for (int h = 0; h < 4; ++h) hit[h] = __ballot_sync(0xffffffffu, r[1] < 8 * h + 8 && r[1] + W > 8 * h);
        const unsigned bad = __ballot_sync(0xffffffffu, !(isfinite(v.x) && isfinite(v.y)));
        __syncwarp();
        if (base + kWideWarps * 32 < sub.z) fetch(base + kWideWarps * 32, p, v);
        if (TAPS && bad) {
            int r2[2];
            unpack_cells(2, __float_as_uint(a.pts[(int64_t)sub.y + min(base + lane, sub.z - 1)].w), c0[0], c0[1], c0[2]);
#pragma unroll
            for (int d = 0; d < 2; ++d) r2[d] = first_plane(c0[d], o[d], g.nf[d], W);
#pragma unroll 1
            for (int s = 0; s < n; ++s) {
                const float *w = st + s * kWideStride;
                const float wx = w[lane], vx = w[64], vy = w[65];
                const int sx = __shfl_sync(0xffffffffu, r2[0], s), sy = __shfl_sync(0xffffffffu, r2[1], s);
                if ((unsigned)(lane - sx) >= (unsigned)W) continue;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float ga = wx * w[32 + 2 * i], gb = wx * w[33 + 2 * i];
                    if ((unsigned)(2 * i - sy) < (unsigned)W) { re[i].x = fmaf(ga, vx, re[i].x); im[i].x = fmaf(ga, vy, im[i].x); }
                    if ((unsigned)(2 * i + 1 - sy) < (unsigned)W) { re[i].y = fmaf(gb, vx, re[i].y); im[i].y = fmaf(gb, vy, im[i].y); }
                }
            }
            continue;
        }
        if (bad) {  // guarded: only the cells inside the stencil
#pragma unroll 1
            for (int s = 0; s < n; ++s) {
                const float *w = st + s * kWideStride;
                const float wx = w[lane], vx = w[64], vy = w[65];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float ga = wx * w[32 + 2 * i], gb = wx * w[33 + 2 * i];
                    if (ga != 0.f) { re[i].x = fmaf(ga, vx, re[i].x); im[i].x = fmaf(ga, vy, im[i].x); }
                    if (gb != 0.f) { re[i].y = fmaf(gb, vx, re[i].y); im[i].y = fmaf(gb, vy, im[i].y); }
                }
            }
            continue;
        }
#pragma unroll 2
        for (int s = 0; s < n; ++s) {
            const float *w = st + s * kWideStride;
            const float2 vv = *reinterpret_cast<const float2 *>(w + 64);
            const float br = w[lane] * vv.x, bi = w[lane] * vv.y;
            const float2 b0 = make_float2(br, br), b1 = make_float2(bi, bi);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (!((hit[h] >> s) & 1u)) continue;
                const float4 ya = *reinterpret_cast<const float4 *>(w + 32 + 8 * h);
                const float4 yb = *reinterpret_cast<const float4 *>(w + 36 + 8 * h);
                const float2 wy[4] = {make_float2(ya.x, ya.y), make_float2(ya.z, ya.w), make_float2(yb.x, yb.y),
                                      make_float2(yb.z, yb.w)};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    re[4 * h + i] = __ffma2_rn(b0, wy[i], re[4 * h + i]);
                    im[4 * h + i] = __ffma2_rn(b1, wy[i], im[4 * h + i]);
                }
            }
        }
    }

    // (warp 0 + warp 2) + (warp 1 + warp 3), then out; cell (x, y) at y * 33 + x
    __syncthreads();
    float2 *red = reinterpret_cast<float2 *>(smem_wide) + (warp & 1) * 32 * 33;
    auto each = [&](auto f) {
#pragma unroll
        for (int y = 0; y < 32; ++y)
            f(red[y * 33 + lane], (y & 1) ? re[y / 2].y : re[y / 2].x, (y & 1) ? im[y / 2].y : im[y / 2].x);
    };
    if (warp >= 2) each([](float2 &m, float x, float y) { m = make_float2(x, y); });
    __syncthreads();
    if (warp < 2) each([](float2 &m, float x, float y) { m = make_float2(x + m.x, y + m.y); });
    __syncthreads();
    const float2 *p0 = reinterpret_cast<const float2 *>(smem_wide), *p1 = p0 + 32 * 33;
    const bool split = (sub.w & kSplitFlag) != 0;
    float2 *out = a.grid + ((int64_t)grp * g.n_coil + coil) * g.G;
    for (int i = threadIdx.x; i < 1024; i += kWideWarps * 32) {
        const int x = i >> 5, y = i & 31;
        if (x >= e[0] || y >= e[1]) continue;
        const float2 u = p0[y * 33 + x], w = p1[y * 33 + x];
        float2 *dst = out + (int64_t)(o[0] + x) * g.nf[1] + o[1] + y;
        if (split) {
            atomicAdd(&dst->x, u.x + w.x);
            atomicAdd(&dst->y, u.y + w.y);
        } else {
            *dst = make_float2(u.x + w.x, u.y + w.y);
        }
    }
}

}  // namespace gbn
