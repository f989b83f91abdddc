// 3-D interp of a real grid, one coil: k_interp3d_real<WT>, for the density compensation, whose
// weights and grid have imaginary part zero.
//
// What bounds it: shared-memory reads, as in k_interp3d_one, which reads 8 bytes a tap and here
// would read zeros in half of them.  The window is staged as real parts, so a lane reads four
// z cells at once (16 bytes): 4 lanes cover a row's taps from the 4-cell unit that holds the
// first, and the warp takes 8 rows a step.  The stencil's W * W rows are walked in one
// sequence over all planes (10 taps: 13 steps instead of 20), each lane with a fixed table of its
// rows in a period of Q planes = P whole steps.
//
// A quarter warp reads two rows of 4 units each; they do not conflict when the rows lie 4 units
// apart (mod 8).  R = 2 (mod 4) units a row makes that rows ky and ky + 2; where the row count
// of a plane leaves two over (10 and 6 taps) these pair with their own row in the next plane,
// the plane stride being 4 (mod 8).
//
// 20 density iterations (spread and interp), k_interp3d_one -> this kernel: 768,000 samples on a
// 192^3 grid, 10 taps 14.83 -> 13.81 ms, 8 taps 11.67 -> 9.73 ms; 2,560,000 samples on 256^3, 10
// taps 44.6 -> 41.3 ms; 192,000 on 128^3, 12 taps 6.28 -> 5.30 ms.  64 registers for four
// blocks an SM (74 and three blocks without the bound: 14.06 ms in the first case).
#pragma once

#include "grid2d_kernels.cuh"

namespace gbn {

__host__ __device__ inline int real_row_units(const Geom &g) {
    int r = (g.tile[2] >> 2) + 4;  // the last lane of a sample that starts in the tile's last unit
    while ((r & 3) != 2) ++r;
    return r;
}
__host__ __device__ inline int real_plane_units(const Geom &g) {
    int p = (g.tile[1] + g.W - 1) * real_row_units(g);
    while ((p & 7) != 4) p += 2;
    return p;
}
inline size_t interp3d_real_smem_bytes(const Geom &g) {
    if (g.dim != 3 || g.W < 6 || g.W > 12 || (g.W & 1)) return 0;
    return (size_t)(g.tile[0] + g.W - 1) * real_plane_units(g) * sizeof(float4);
}

// grid rows of an even length on a 16-byte boundary
template <int W>
__global__ void __launch_bounds__(256, 4) k_interp3d_real(InterpArgs a) {
    constexpr int Q = W % 8 == 0 ? 1 : (W % 4 == 0 ? 2 : 4);  // planes a period
    constexpr int P = Q * W / 8;                              // steps a period
    constexpr int PAIRS = W * W / 2, STEPS = (PAIRS + 3) / 4, REM = PAIRS % 4;
    extern __shared__ float4 smem_ir[];  // [WX][PS], rows of R units of 4 real z cells
    const Geom &g = a.g;
    const int4 sub = a.subs[blockIdx.x];
    const int coil = blockIdx.y;
    const int grp = sub.x / g.ntiles;
    int o[3], e[3];
    tile_coords<3>(g, sub.x % g.ntiles, o, e);
    const int ns = g.ns;
    const int WX = g.tile[0] + W - 1, WY = g.tile[1] + W - 1;
    const int R = real_row_units(g), PS = real_plane_units(g), NL = (g.tile[2] + W + 3) >> 2;
    const int nf0 = g.nf[0], nf1 = g.nf[1], nf2 = g.nf[2];
    const int ws0 = o[0] - (ns - 1), ws1 = o[1] - (ns - 1), ws2 = o[2] - (ns - 1);
    const int zs = ws2 & ~1, offz = ws2 - zs;  // even (also below zero)
    const float2 *gbase = a.grid + ((int64_t)grp * g.n_coil + coil) * g.G;
    {
        const int n = WX * WY * NL;
        const float rL = 1.f / (float)NL, rWY = 1.f / (float)WY;
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int xy = div_small(i, rL), p = i - xy * NL;
            const int wx = div_small(xy, rWY), wy = xy - wx * WY;
            const int gx = wrap_fast(ws0 + wx, nf0), gy = wrap_fast(ws1 + wy, nf1);
            const float2 *row = gbase + ((int64_t)gx * nf1 + gy) * nf2;
            const float4 u = *reinterpret_cast<const float4 *>(row + wrap_fast(zs + 4 * p, nf2));
            const float4 v = *reinterpret_cast<const float4 *>(row + wrap_fast(zs + 4 * p + 2, nf2));
            smem_ir[wx * PS + wy * R + p] = make_float4(u.x, u.z, v.x, v.z);
        }
        __syncthreads();
    }

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int q = lane >> 3, h = (lane >> 2) & 1, pz = lane & 3;
    int off[P], dx[P], dy[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int n = 4 * i + q;  // the lane's row pair in the period
        if (W % 4 == 0) {
            const int m = n % (W / 2);
            dx[i] = n / (W / 2);
            dy[i] = (m >> 1) * 4 + (m & 1) + 2 * h;
        } else {
            const int m = n % W, mm = m % ((W - 2) / 2);
            const bool cross = m >= W - 2;
            dx[i] = 2 * (n / W) + (cross ? h : m / ((W - 2) / 2));
            dy[i] = cross ? m : (mm >> 1) * 4 + (mm & 1) + 2 * h;
        }
        off[i] = dx[i] * PS + dy[i] * R + pz;
    }
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
        // lanes 0..15 the x weights, 16..31 the y weights, every lane its own four z weights
        float myw = 0.f;
        if (kk < W) {
            const float d = (lane < 16 ? p.x : p.y) + (float)(ns - 1 - kk);
            myw = ex2_approx(-beta * d * d);
        }
        const int zr = rel[2] + offz, kz = 4 * pz - (zr & 3);
        float wz[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float d = p.z + (float)(ns - 1 - kz - t);
            const float ex = ex2_approx(-g.beta2[2] * d * d);
            wz[t] = (unsigned)(kz + t) < (unsigned)W ? ex : 0.f;
        }
        float wy[P];
#pragma unroll
        for (int i = 0; i < P; ++i) wy[i] = __shfl_sync(0xffffffffu, myw, 16 + dy[i]);
        const float4 *base = smem_ir + ((size_t)rel[0] * PS + rel[1] * R + (zr >> 2));
        float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            const int per = st / P, i = st % P;
            const float w = __shfl_sync(0xffffffffu, myw, Q * per + dx[i]) * wy[i];
            if (REM && st == STEPS - 1 && q >= REM) continue;  // rows past the stencil
            const float4 v = base[per * Q * PS + off[i]];
            const float2 w2 = make_float2(w, w);
            a0 = __ffma2_rn(w2, make_float2(v.x, v.y), a0);
            a1 = __ffma2_rn(w2, make_float2(v.z, v.w), a1);
        }
        // select by tap, as in k_interp3d_one: cells outside the stencil may be anything
        float x = 0.f;
        if ((unsigned)kz < (unsigned)W) x = wz[0] * a0.x;
        if ((unsigned)(kz + 1) < (unsigned)W) x = fmaf(wz[1], a0.y, x);
        if ((unsigned)(kz + 2) < (unsigned)W) x = fmaf(wz[2], a1.x, x);
        if ((unsigned)(kz + 3) < (unsigned)W) x = fmaf(wz[3], a1.y, x);
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
        if (lane == 0) {
            const float sc = a.weight ? a.weight[j] : 1.f;
            a.c[(int64_t)j * a.c_elem + (int64_t)coil * a.c_coil] = make_float2(x * sc, 0.f);
        }
    }
}

}  // namespace gbn
