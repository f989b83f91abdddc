// 3-D spread (type-1 gridding) of 1 to 3 coils with the output tile in registers:
// k_spread3d_few<WT, NC, REAL, TAPS>.
//
// What bounds it: FP32 issue.  A sample's W^3 taps are 4 W^3 flops a coil against 16 + 8 NC
// bytes of input, so the cells have to stay out of shared memory: read-modify-write of a
// complex cell moves 16 shared-memory bytes per tap, which held the shared-memory kernel
// (k_spread3d) at 2.35 ms for 768,000 samples of 10 taps per axis on a 192^3 grid (1 coil).
// This kernel takes 0.47 ms there (0.49 of the issue slots).
//
// Every warp of a block holds the WHOLE tile -- 8 x 8 x TZ cells (TZ = 16 for one coil, 8 for
// more): lane (lx, yq) has the cells (x = lx, y = 2 yq + {0, 1}, all z) as FP32x2 pairs along
// z, real and imaginary parts apart -- and takes its own 32-sample batches of the work item
// (warp w: batches w, w + 4, ...).  A (sample, tile) pair costs a warp 16 packed FMAs per coil
// and touched 8-cell z half (a half that the stencil misses is skipped, warp-uniform).  There
// are no per-warp sample lists, no block barrier between batches, and the warps' loads are
// even whatever the samples' order.  Each lane stages one sample of the batch in shared
// memory: its 16 + TZ plane weights (zero outside the stencil) and coil values, read back as
// broadcasts.  At the end the four partial tiles are added through shared memory in a fixed
// order.
//
// REAL: the samples' imaginary parts are zero (density compensation): half the FMAs.
//
// A value that is not finite reaches the cells of its own stencil and no others, as with the
// kernels that walk the stencil: a batch with such a sample takes the guarded loop, which skips
// the zero weights instead of multiplying by them.  TAPS: the loop goes by the taps instead, for
// grids whose axes differ so much that weights inside the stencil are zero in FP32 (an instance of
// its own: with the comparisons of taps the others take up to 2.6 % longer, by their registers).
#pragma once

#include "grid2d_kernels.cuh"
#include "grid3d_kernels.cuh"

namespace gbn {

constexpr int kFewWarps = 4;
constexpr int kFewTile = 8;                     // x and y cells; z: few_tz
__host__ __device__ constexpr int few_tz(int nc) { return nc == 1 ? 16 : 8; }
// floats per staged sample: wx[8], wy[8], wz[TZ], the spread's coil values; a multiple of 4
// whose quarter is odd, so the lanes' 16-byte staging stores are free of bank conflicts
__host__ __device__ constexpr int few_stride(int nc) {
    int f = (16 + few_tz(nc) + 2 * nc + 3) / 4;
    return 4 * (f | 1);
}
__host__ __device__ constexpr int few_cells(int nc) { return kFewTile * kFewTile * few_tz(nc); }
constexpr size_t few_stage_bytes(int nc) { return (size_t)kFewWarps * 32 * few_stride(nc) * sizeof(float); }
// spread: staging and, afterwards, two partial tiles (33 cells per 32) share the same memory
constexpr size_t few_smem_bytes(int nc) {
    size_t red = 2 * (size_t)few_cells(nc) / 32 * 33 * nc * sizeof(float2);
    return few_stage_bytes(nc) > red ? few_stage_bytes(nc) : red;
}
// resident blocks per SM the register budget is set for
__host__ __device__ constexpr int few_blocks(int nc, bool real) { return real ? 6 : (nc <= 2 ? 4 : 3); }

// The lane's sample staged: first taps relative to the tile (signed), then the tile-plane
// weights.  Returns r[2] (z) for the half masks.
template <int WT, int TZ>
__device__ __forceinline__ int few_stage(const Geom &g, const int o[3], const float4 &p, float4 *mine) {
    const int W = WT ? WT : g.W, ns = g.ns;
    int c0[3], r[3];
    unpack_cells(3, __float_as_uint(p.w), c0[0], c0[1], c0[2]);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        int rr = c0[d] - o[d];
        rr += rr < 0 ? g.nf[d] : 0;
        rr -= rr > g.nf[d] - W ? g.nf[d] : 0;
        r[d] = rr;
    }
#pragma unroll
    for (int q = 0; q < (16 + TZ) / 4; ++q) {
        const int d = q < 2 ? 0 : (q < 4 ? 1 : 2);
        const int t0 = 4 * (q < 4 ? (q & 1) : q - 4) - r[d];  // tap at the quad's first plane
        const float f = d == 0 ? p.x : (d == 1 ? p.y : p.z);
        const float k0 = (float)(ns - 1 - t0);
        float w4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float dd = f + (k0 - (float)i);  // k0 - i is exact: as tap_weight's distance
            const float ex = ex2_approx(-g.beta2[d] * dd * dd);
            w4[i] = (unsigned)(t0 + i) < (unsigned)W ? ex : 0.f;
        }
        mine[q] = make_float4(w4[0], w4[1], w4[2], w4[3]);
    }
    return r[2];
}

__device__ __forceinline__ void few_load_z(const float *w, float2 (&wz)[4]) {
    const float4 a = *reinterpret_cast<const float4 *>(w), b = *reinterpret_cast<const float4 *>(w + 4);
    wz[0] = make_float2(a.x, a.y);
    wz[1] = make_float2(a.z, a.w);
    wz[2] = make_float2(b.x, b.y);
    wz[3] = make_float2(b.z, b.w);
}

// --------------------------------------------------------------------------------- spread
template <int WT, int NC, bool REAL, bool TAPS>
__global__ void __launch_bounds__(kFewWarps * 32, few_blocks(NC, REAL)) k_spread3d_few(SpreadArgs a) {
    constexpr int TZ = few_tz(NC), ZP = TZ / 2, ST = few_stride(NC), CELLS = few_cells(NC), RI = REAL ? 1 : 2;
    extern __shared__ float4 smem_few[];
    const Geom &g = a.g;
    const int4 sub = a.subs[blockIdx.x];
    const int grp = sub.x / g.ntiles;
    int o[3], e[3];
    tile_coords<3>(g, sub.x % g.ntiles, o, e);
    const int W = WT ? WT : g.W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lx = lane >> 2, yq = lane & 3;
    float *st = reinterpret_cast<float *>(smem_few) + warp * 32 * ST;

    float2 acc[NC][RI][2][ZP];  // [coil][re, im][row][z pair]
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < RI; ++k)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int z = 0; z < ZP; ++z) acc[c][k][r][z] = make_float2(0.f, 0.f);

    // the record and values of the lane's sample of a batch
    auto fetch = [&](int base, float4 &p, float (&v)[NC][RI]) {
        const int s = base + lane;
        p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int k = 0; k < RI; ++k) v[c][k] = 0.f;
        if (s >= sub.z) return;
        p = a.pts[(int64_t)sub.y + s];
        const uint32_t j = a.idx[(int64_t)sub.y + s];
        const float sw = a.weight ? a.weight[j] : 1.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float2 t = a.c[(int64_t)j * a.c_elem + (int64_t)c * a.c_coil];
            v[c][0] = t.x * sw;
            if constexpr (!REAL) v[c][1] = t.y * sw;
        }
    };

    float4 p;
    float v[NC][RI];
    if (warp * 32 < sub.z) fetch(warp * 32, p, v);
    for (int base = warp * 32; base < sub.z; base += kFewWarps * 32) {
        const int n = min(32, sub.z - base);
        __syncwarp();  // the previous batch is consumed
        const int rz = few_stage<WT, TZ>(g, o, p, reinterpret_cast<float4 *>(st + lane * ST));
        bool fin = true;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int k = 0; k < RI; ++k) {
                st[lane * ST + 16 + TZ + RI * c + k] = v[c][k];
                fin = fin && isfinite(v[c][k]);
            }
        // the z halves each sample reaches; samples with a value that is not finite
        const unsigned lo = __ballot_sync(0xffffffffu, rz < 8 && rz + W > 0);
        const unsigned hi = TZ > 8 ? __ballot_sync(0xffffffffu, rz < 16 && rz + W > 8) : 0u;
        const unsigned bad = __ballot_sync(0xffffffffu, !fin);
        __syncwarp();
        if (base + kFewWarps * 32 < sub.z) fetch(base + kFewWarps * 32, p, v);

        if (TAPS && bad) {
            int c0[3], r3[3];
            unpack_cells(3, __float_as_uint(a.pts[(int64_t)sub.y + min(base + lane, sub.z - 1)].w), c0[0], c0[1], c0[2]);
#pragma unroll
            for (int d = 0; d < 3; ++d) r3[d] = first_plane(c0[d], o[d], g.nf[d], W);
#pragma unroll 1
            for (int s = 0; s < n; ++s) {
                const float *w = st + s * ST;
                const float t[2] = {w[lx] * w[8 + 2 * yq], w[lx] * w[9 + 2 * yq]};
                const int sx = __shfl_sync(0xffffffffu, r3[0], s), sy = __shfl_sync(0xffffffffu, r3[1], s);
                const int sz = __shfl_sync(0xffffffffu, r3[2], s);
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int k = 0; k < RI; ++k) {
                        const float u = w[16 + TZ + RI * c + k];
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const bool in = (unsigned)(lx - sx) < (unsigned)W && (unsigned)(2 * yq + r - sy) < (unsigned)W;
#pragma unroll
                            for (int z = 0; z < ZP; ++z) {
                                float2 &m = acc[c][k][r][z];
                                if (in && (unsigned)(2 * z - sz) < (unsigned)W) m.x = fmaf(t[r] * w[16 + 2 * z], u, m.x);
                                if (in && (unsigned)(2 * z + 1 - sz) < (unsigned)W)
                                    m.y = fmaf(t[r] * w[17 + 2 * z], u, m.y);
                            }
                        }
                    }
            }
            continue;
        }
        if (bad) {  // guarded: only the cells inside the stencil
#pragma unroll 1
            for (int s = 0; s < n; ++s) {
                const float *w = st + s * ST;
                const float t[2] = {w[lx] * w[8 + 2 * yq], w[lx] * w[9 + 2 * yq]};
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int k = 0; k < RI; ++k) {
                        const float u = w[16 + TZ + RI * c + k];
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int z = 0; z < ZP; ++z) {
                                const float ga = t[r] * w[16 + 2 * z], gb = t[r] * w[17 + 2 * z];
                                float2 &m = acc[c][k][r][z];
                                if (ga != 0.f) m.x = fmaf(ga, u, m.x);
                                if (gb != 0.f) m.y = fmaf(gb, u, m.y);
                            }
                    }
            }
            continue;
        }
#pragma unroll 2
        for (int s = 0; s < n; ++s) {
            const float *w = st + s * ST;
            const float wx = w[lx];
            const float2 wy = *reinterpret_cast<const float2 *>(w + 8 + 2 * yq);
            const float t[2] = {wx * wy.x, wx * wy.y};
            float2 b[NC][RI][2];  // the row's x and y weights times the value, twice
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int k = 0; k < RI; ++k) {
                    const float u = w[16 + TZ + RI * c + k];
#pragma unroll
                    for (int r = 0; r < 2; ++r) b[c][k][r] = make_float2(t[r] * u, t[r] * u);
                }
#pragma unroll
            for (int h = 0; h < TZ / 8; ++h) {
                if (TZ > 8 && !(((h ? hi : lo) >> s) & 1u)) continue;
                float2 wz[4];
                few_load_z(w + 16 + 8 * h, wz);
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int k = 0; k < RI; ++k)
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int z = 0; z < 4; ++z)
                                acc[c][k][r][4 * h + z] = __ffma2_rn(b[c][k][r], wz[z], acc[c][k][r][4 * h + z]);
            }
        }
    }

    // (warp 0 + warp 2) + (warp 1 + warp 3), then out.  A lane's cells in shared memory:
    // [coil][slot][lane] with slot = row * TZ + z and 33 cells a slot: a warp's accesses are
    // 8-byte runs across lanes (here) or across slots (below), both free of bank conflicts.
    __syncthreads();
    constexpr int RED = CELLS / 32 * 33 * NC;
    float2 *red = reinterpret_cast<float2 *>(smem_few) + (size_t)(warp & 1) * RED;
    auto each = [&](auto f) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int z = 0; z < TZ; ++z) {
                    const float2 u = acc[c][0][r][z / 2], w = acc[c][RI - 1][r][z / 2];
                    f(red[((c * 2 + r) * TZ + z) * 33 + lane], (z & 1) ? u.y : u.x, (z & 1) ? w.y : w.x);
                }
    };
    if (warp >= 2) each([](float2 &m, float x, float y) { m = make_float2(x, y); });
    __syncthreads();
    if (warp < 2) each([](float2 &m, float x, float y) { m = make_float2(x + m.x, y + m.y); });
    __syncthreads();
    const float2 *p0 = reinterpret_cast<const float2 *>(smem_few), *p1 = p0 + RED;
    const bool split = (sub.w & kSplitFlag) != 0;
    for (int i = threadIdx.x; i < CELLS * NC; i += kFewWarps * 32) {
        const int c = i / CELLS, cell = i % CELLS;
        const int z = cell % TZ, y = (cell / TZ) % kFewTile, x = cell / (TZ * kFewTile);
        if (x >= e[0] || y >= e[1] || z >= e[2]) continue;
        const int m = ((c * 2 + (y & 1)) * TZ + z) * 33 + x * 4 + (y >> 1);
        const float2 u = p0[m], w = p1[m];
        const float2 val = make_float2(u.x + w.x, u.y + w.y);
        const int64_t at = ((int64_t)grp * g.n_coil + c) * g.G +
                           ((int64_t)(o[0] + x) * g.nf[1] + (o[1] + y)) * g.nf[2] + (o[2] + z);
        float2 *dst = a.grid + at;
        if (split) {
            atomicAdd(&dst->x, val.x);
            if (!REAL) atomicAdd(&dst->y, val.y);
        } else {
            *dst = REAL ? make_float2(val.x, 0.f) : val;
        }
    }
}

}  // namespace gbn
