// Sample preparation and bin sorting (the set_points stage).
//
// For every sample the FP64 coordinate reduction of the reference is applied once
// (xi = x*df mod 2pi, m = 1 + xi // h, fft/nufft_func.py:562-565), and the result is
// stored as the first tap cell (m - nspread) mod nf and the in-cell fraction in FP32.
// The spread and interp kernels only ever see these packed records.
#include "common.cuh"

namespace gbn {

namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;

// Python float semantics of a % b for b > 0 (CPython float_rem), so that the nearest-cell
// choice matches the reference.
__device__ inline double py_mod(double a, double b) {
    double m = fmod(a, b);
    if (m != 0.0) {
        if ((b < 0) != (m < 0)) m += b;
    } else {
        m = copysign(0.0, b);
    }
    return m;
}
__device__ inline int group_of(const int64_t *off, int n_traj, int64_t j) {
    int lo = 0, hi = n_traj;  // off[lo] <= j < off[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (off[mid] <= j) lo = mid; else hi = mid;
    }
    return lo;
}

// The nearest-cell choice of one coordinate: n = floor(xi / h) and the in-cell fraction, with
// xi = xs mod 2 pi, as Python's % and // give them.  FP64 runs at 1/64 of the FP32 rate here,
// and fmod and the divisions of the general form above took 129 of the 571 us that 256,000
// 3-D samples needed; within (-2 pi, 2 pi) the remainder is xs or xs + 2 pi (fmod is exact),
// and n follows from an estimate and the exact remainder xi - n h (one fused multiply-add,
// whose sign and size say whether the estimate was one off; Python's xi // h, (xi - xi % h) / h
// rounded to the nearest whole number, is that n).  12 FP64 instructions an axis.
__device__ __forceinline__ void nearest_cell(double xs, double h, double rh, bool wide, int &n, float &fr) {
    double xi = xs;
    if (xs < 0.0) xi = xs + kTwoPi;
    if (!(xi >= 0.0 && xs < kTwoPi)) xi = py_mod(xs, kTwoPi);  // outside (-2 pi, 2 pi)
    // `wide`: more cells than an FP32 estimate places within one
    int64_t k = wide ? (int64_t)(xi * rh) : (int64_t)(int)((float)xi * (float)rh);
    double r = fma(-(double)k, h, xi);
    if (r < 0.0) {
        k -= 1;
    } else if (r >= h) {
        k += 1;
    }
    n = (int)k;
    fr = (float)((xi - h * (double)k) * rh);
}

// one counter per key, keys of adjacent lanes often equal (samples along a spoke share tiles,
// and the k-space centre is one tile for all of them): one atomic per distinct key of a warp
__device__ __forceinline__ void count_key(uint32_t *count, uint32_t key) {
    const unsigned same = __match_any_sync(__activemask(), key);
    if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&count[key], (uint32_t)__popc(same));
}

template <typename T>
__global__ void __launch_bounds__(256) k_prep(PrepArgs a) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j == 0 && a.gs.n_traj == 1) {  // one group: its offsets and scale need no copy
        a.traj_off[0] = 0;
        a.traj_off[1] = a.M;
        a.grp_scale[0] = a.scale1;
    }
    if (j >= a.M) return;
    const Geom &gs = a.gs, &gi = a.gi;
    const int dim = gs.dim, ns = gs.ns;
    const T *src[3] = {(const T *)a.x, (const T *)a.y, (const T *)a.z};
    float f[3] = {0.f, 0.f, 0.f};
    int c0[3] = {0, 0, 0};
    bool bad = false;
    // loops over all three axes with a guard (not up to dim): unrolled, so the per-axis
    // arrays and the Geom fields are indexed by constants and stay out of local memory
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d >= dim) continue;
        const double xs = (double)src[d][j] * a.df;
        if (!isfinite(xs)) { bad = true; continue; }
        const int nf = gs.nf[d];
        int n;
        nearest_cell(xs, a.h[d], a.rh[d], nf > (1 << 20), n, f[d]);
        int first = (1 + n - ns) % nf;
        if (first < 0) first += nf;
        c0[d] = first;
    }
    if (bad) {
        atomicOr(a.status, 1u);
        for (int d = 0; d < 3; ++d) { f[d] = 0.f; c0[d] = 0; }
    }
    a.pts[j] = make_float4(f[0], f[1], f[2], __uint_as_float(pack_cells(dim, c0[0], c0[1], c0[2])));

    const int g = gs.n_traj == 1 ? 0 : group_of(a.traj_off, gs.n_traj, j);
    int t[3] = {0, 0, 0}, n[3] = {1, 1, 1}, t0[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d >= dim) continue;
        int cc = c0[d] + ns - 1;
        if (cc >= gi.nf[d]) cc -= gi.nf[d];
        t[d] = cc / gi.tile[d];
        n[d] = touched_tiles(c0[d], gs.W, gs.nf[d], gs.tile[d], gs.ntile[d]);
        t0[d] = c0[d] / gs.tile[d];
    }
    const uint32_t key = (uint32_t)g * (uint32_t)gi.ntiles +
                         (uint32_t)((t[0] * gi.ntile[1] + t[1]) * gi.ntile[2] + t[2]);
    a.home_key[j] = key;
    count_key(a.home_count, key);
    a.touch_count[j] = (uint32_t)(n[0] * n[1] * n[2]);
    const uint32_t base = (uint32_t)g * (uint32_t)gs.ntiles;
    for (int p = 0; p < n[0]; ++p) {
        const int tp = (t0[0] + p) % gs.ntile[0];
        for (int b = 0; b < n[1]; ++b) {
            const int tb = (t0[1] + b) % gs.ntile[1];
            for (int q = 0; q < n[2]; ++q) {
                const int tq = (t0[2] + q) % gs.ntile[2];
                count_key(a.tile_count, base + (uint32_t)((tp * gs.ntile[1] + tb) * gs.ntile[2] + tq));
            }
        }
    }
}

// The (sample, tile) entries, each sample's adjacent.  y_class: the key's low kYClassBits hold
// the stencil's first y row in the tile (+ W - 1: 0 is a stencil that reaches row 0 only), so
// that the sort leaves a tile's samples in the order of the rows they reach.  Before them, one
// entry per sample with its home bin's key above all of theirs: one sort makes both lists.
__global__ void k_dup_keys(const float4 *__restrict__ pts, int64_t M, const int64_t *__restrict__ traj_off,
                           Geom gs, const uint64_t *__restrict__ touch_off, uint32_t *__restrict__ keys,
                           uint32_t *__restrict__ vals, int y_class,
                           const uint32_t *__restrict__ home_key, uint32_t home_base) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= M) return;
    const int dim = gs.dim;
    int c0[3];
    unpack_cells(dim, __float_as_uint(pts[j].w), c0[0], c0[1], c0[2]);
    int n[3] = {1, 1, 1}, t0[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d >= dim) continue;
        n[d] = touched_tiles(c0[d], gs.W, gs.nf[d], gs.tile[d], gs.ntile[d]);
        t0[d] = c0[d] / gs.tile[d];
    }
    const uint32_t base = gs.n_traj == 1 ? 0u : (uint32_t)group_of(traj_off, gs.n_traj, j) * (uint32_t)gs.ntiles;
    keys[j] = home_base + home_key[j];
    vals[j] = (uint32_t)j;
    uint64_t pos = (uint64_t)M + touch_off[j];
    for (int a = 0; a < n[0]; ++a) {
        int ta = (t0[0] + a) % gs.ntile[0];
        for (int b = 0; b < n[1]; ++b) {
            int tb = (t0[1] + b) % gs.ntile[1];
            int r = c0[1] - tb * gs.tile[1];  // signed first row, as the kernels take it
            r += r < 0 ? gs.nf[1] : 0;
            r -= r > gs.nf[1] - gs.W ? gs.nf[1] : 0;
            for (int q = 0; q < n[2]; ++q) {
                int tq = (t0[2] + q) % gs.ntile[2];
                const uint32_t key = base + (uint32_t)((ta * gs.ntile[1] + tb) * gs.ntile[2] + tq);
                keys[pos] = y_class ? key << kYClassBits | (uint32_t)(r + gs.W - 1) : key;
                vals[pos] = (uint32_t)j;
                ++pos;
            }
        }
    }
}

// records in list order, for both lists
__global__ void k_gather_pts(const float4 *__restrict__ pts, const uint32_t *__restrict__ idx, int64_t n,
                             float4 *__restrict__ out, const uint32_t *__restrict__ idx2, int64_t n2,
                             float4 *__restrict__ out2) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = pts[idx[i]];
    else if (i - n < n2) out2[i - n] = pts[idx2[i - n]];
}

__device__ __forceinline__ uint32_t items_of(uint32_t c, const SubsJob &j) {
    const uint32_t s = (c + (uint32_t)j.max_sub - 1) / (uint32_t)j.max_sub;
    return j.every_tile && s == 0 ? 1u : s;
}

// sums of a block's 64-bit pairs, in thread 0 (sh: 64 words)
__device__ __forceinline__ void block_sum(uint64_t &c, uint64_t &s, uint64_t *sh) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        c += __shfl_down_sync(0xffffffffu, c, m);
        s += __shfl_down_sync(0xffffffffu, s, m);
    }
    if ((threadIdx.x & 31) == 0) {
        sh[2 * (threadIdx.x >> 5)] = c;
        sh[2 * (threadIdx.x >> 5) + 1] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 32; ++w) {
            c += sh[2 * w];
            s += sh[2 * w + 1];
        }
}

// entries and work items of each chunk of tiles, for k_tile_scan over several blocks
__global__ void __launch_bounds__(1024) k_tile_sums(SubsJob spread, SubsJob home, int64_t chunk, TileSums *part) {
    const SubsJob &j = blockIdx.y == 0 ? spread : home;
    __shared__ uint64_t sh[64];
    const int64_t t0 = blockIdx.x * chunk, t1 = min(t0 + chunk, j.T);
    uint64_t c = 0, s = 0;
#pragma unroll 4
    for (int64_t t = t0 + threadIdx.x; t < t1; t += 1024) {
        const uint32_t n = j.count[t];
        c += n;
        s += items_of(n, j);
    }
    block_sum(c, s, sh);
    if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = TileSums{c, s};
}

// Per tile, the exclusive sums of its entries (tile_off) and of its work items (sub_off), and
// the totals.  A block walks its chunk of tiles 4096 at a time.  Up to kScanOneBlock tiles one
// block per bin geometry does it all: it stands for two device scans and a count kernel per
// geometry, whose ten launches and separate read-backs took longer than the work.  A step is a
// chain of loads, shuffles and two barriers, 4.5 us, so more tiles (many groups, large 3-D grids)
// are cut into chunks, whose sums k_tile_sums leaves in `part` before.  set_points, one block ->
// chunks (device scans): 512 frames of 128^2, 262,144 bins 553 -> 266 us (467); 4096 frames,
// 2.1 M bins 3414 -> 1113 (1549); 384^3 image, 884,736 bins 1613 -> 645 (970).
__global__ void __launch_bounds__(1024) k_tile_scan(SubsJob spread, SubsJob home, int64_t chunk,
                                                    const TileSums *part, TileTotals *out) {
    const bool is_spread = blockIdx.y == 0, last = blockIdx.x + 1 == gridDim.x;
    const SubsJob &j = is_spread ? spread : home;
    __shared__ uint64_t sh_c[32];
    __shared__ uint32_t sh_s[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t base_c = 0;
    uint64_t base_s = 0;
    if (blockIdx.x > 0) {  // the chunks in front (at most 1024: one a thread)
        __shared__ uint64_t sh[64], base[2];
        if (threadIdx.x < blockIdx.x) {
            const TileSums p = part[blockIdx.y * gridDim.x + threadIdx.x];
            base_c = p.entries;
            base_s = p.items;
        }
        block_sum(base_c, base_s, sh);
        if (threadIdx.x == 0) {
            base[0] = base_c;
            base[1] = base_s;
        }
        __syncthreads();
        base_c = base[0];
        base_s = base[1];
    }
    uint32_t dense = 0, split = 0;
    const int64_t end = min((blockIdx.x + 1) * chunk, j.T);
    for (int64_t t0 = blockIdx.x * chunk; t0 < end; t0 += 4096) {
        const int64_t t = t0 + 4 * threadIdx.x;
        uint32_t c[4], s[4];
        uint64_t sum_c = 0;
        uint32_t sum_s = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            c[i] = t + i < j.T ? j.count[t + i] : 0u;
            s[i] = t + i < j.T ? items_of(c[i], j) : 0u;
            if (j.dense_min > 0 && c[i] >= j.dense_min) dense += s[i];
            if (s[i] > 1) split += 1;
            sum_c += c[i];
            sum_s += s[i];
        }
        uint64_t ic = sum_c;
        uint32_t is = sum_s;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint64_t vc = __shfl_up_sync(0xffffffffu, ic, m);
            const uint32_t vs = __shfl_up_sync(0xffffffffu, is, m);
            if (lane >= m) {
                ic += vc;
                is += vs;
            }
        }
        if (lane == 31) {
            sh_c[warp] = ic;
            sh_s[warp] = is;
        }
        __syncthreads();
        uint64_t wc = 0, tc = 0;
        uint64_t ws = 0, ts = 0;
#pragma unroll
        for (int w = 0; w < 32; ++w) {
            if (w < warp) {
                wc += sh_c[w];
                ws += sh_s[w];
            }
            tc += sh_c[w];
            ts += sh_s[w];
        }
        uint64_t ec = base_c + wc + ic - sum_c;
        uint64_t es = base_s + ws + is - sum_s;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (t + i < j.T) {
                j.tile_off[t + i] = (uint32_t)ec;
                j.sub_off[t + i] = (uint32_t)es;
                ec += c[i];
                es += s[i];
            }
        base_c += tc;
        base_s += ts;
        __syncthreads();  // sh_* are read
    }
    if (is_spread) {
        dense = __reduce_add_sync(0xffffffffu, dense);
        split = __reduce_add_sync(0xffffffffu, split);
        if (lane == 0) {
            atomicAdd(&out->n_dense, dense);
            atomicAdd(&out->n_split, split);
        }
    }
    if (threadIdx.x == 0 && last) {
        if (is_spread) out->entries = base_c;
        (is_spread ? out->spread_subs : out->interp_subs) = base_s;
    }
}

// interleave: the s > 1 items of a split tile take every s-th entry (item k: entries k,
// k + s, k + 2s, ...; stride s in the flags above kStrideShift) instead of consecutive runs,
// so that each item holds a spatially even share of the tile's samples
// (blockIdx.y 0: the spread's items, 1: the interp's)
__global__ void k_build_subs(SubsJob spread, SubsJob home) {
    const SubsJob &j = blockIdx.y == 0 ? spread : home;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= j.T) return;
    const uint32_t c = j.count[t], s = items_of(c, j), o = j.sub_off[t];
    const bool dense = j.dense_min > 0 && c >= j.dense_min;
    if (s > 1 && j.split_list) j.split_list[atomicAdd(j.split_cursor, 1u)] = (uint32_t)t;  // order is irrelevant
    if (dense && s > 0 && j.dense_list) {
        const uint32_t d = atomicAdd(j.dense_cursor, s);
        for (uint32_t k = 0; k < s; ++k) j.dense_list[d + k] = o + k;
    }
    for (uint32_t k = 0; k < s; ++k) {
        int flags = (s > 1 ? kSplitFlag : 0) | (k == 0 ? kFirstFlag : 0) | (dense ? kDenseFlag : 0);
        if (j.interleave && s > 1) {
            const uint32_t len = (c - k + s - 1) / s;  // entries k, k + s, ... below c
            j.subs[o + k] = make_int4((int)t, (int)(j.tile_off[t] + k), (int)len, flags | (int)(s << kStrideShift));
        } else {
            const uint32_t start = k * (uint32_t)j.max_sub;
            const uint32_t len = c > start ? min((uint32_t)j.max_sub, c - start) : 0u;
            j.subs[o + k] = make_int4((int)t, (int)(j.tile_off[t] + start), (int)len, flags);
        }
    }
}

inline unsigned blocks_for(int64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

cudaError_t launch_prep(int coord_dtype, PrepArgs a, cudaStream_t s) {
    if (a.M == 0) return cudaSuccess;
    for (int d = 0; d < 3; ++d) {
        a.h[d] = kTwoPi / a.gs.nf[d];
        a.rh[d] = 1.0 / a.h[d];
    }
    if (coord_dtype == GBN_COORD_F64)
        k_prep<double><<<blocks_for(a.M, 256), 256, 0, s>>>(a);
    else
        k_prep<float><<<blocks_for(a.M, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_dup_keys(const float4 *pts, int64_t M, const int64_t *d_traj_off, const Geom &gs,
                            const uint64_t *touch_off, uint32_t *keys, uint32_t *vals, bool y_class,
                            const uint32_t *home_key, uint32_t home_base, cudaStream_t s) {
    if (M == 0) return cudaSuccess;
    k_dup_keys<<<blocks_for(M, 256), 256, 0, s>>>(pts, M, d_traj_off, gs, touch_off, keys, vals, y_class ? 1 : 0,
                                                  home_key, home_base);
    return cudaGetLastError();
}

cudaError_t launch_gather_pts(const float4 *pts, const uint32_t *idx, int64_t n, float4 *out, const uint32_t *idx2,
                              int64_t n2, float4 *out2, cudaStream_t s) {
    if (n + n2 == 0) return cudaSuccess;
    k_gather_pts<<<blocks_for(n + n2, 256), 256, 0, s>>>(pts, idx, n, out, idx2, n2, out2);
    return cudaGetLastError();
}

cudaError_t launch_tile_scan(const SubsJob &spread, const SubsJob &home, TileSums *part, TileTotals *out,
                             cudaStream_t s) {
    const int64_t T = spread.T > home.T ? spread.T : home.T;
    int64_t chunk = T > 4096 ? (T + 4095) / 4096 * 4096 : 4096;
    if (T > kScanOneBlock) chunk = (T + 4096 * (int64_t)kScanChunks - 1) / (4096 * (int64_t)kScanChunks) * 4096;
    const dim3 blocks((unsigned)((T + chunk - 1) / chunk), 2);
    if (blocks.x > 1) {
        k_tile_sums<<<blocks, 1024, 0, s>>>(spread, home, chunk, part);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_tile_scan<<<blocks, 1024, 0, s>>>(spread, home, chunk, part, out);
    return cudaGetLastError();
}

cudaError_t launch_build_subs(const SubsJob &spread, const SubsJob &home, cudaStream_t s) {
    const int64_t T = spread.T > home.T ? spread.T : home.T;
    if (T == 0) return cudaSuccess;
    k_build_subs<<<dim3(blocks_for(T, 256), 2), 256, 0, s>>>(spread, home);
    return cudaGetLastError();
}

}  // namespace gbn
