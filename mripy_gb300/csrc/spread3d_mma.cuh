// Spread (type-1 gridding) of 8 coils on the tensor cores: k_spread_mma<D, WT, KAHAN>, 3-D
// (the default for 8 coils) and 2-D (selectable).
//
// The adjoint gridding of one tile is a sum of outer products over its samples s:
//     G[x, y, z, c] = sum_s wx_s[x] wy_s[y] wz_s[z] v_s[c]
// and with the separable weights split between the two operands it is a GEMM with the
// samples as its K dimension:
//     D[(y, z), (x, c, re/im)] = sum_s A[(y, z), s] * B[s, (x, c, re/im)]
//     A[(y, z), s] = wy_s[y] wz_s[z]                      (M = 8 x 16 = 128 cells)
//     B[s, (x, c, ri)] = wx_s[x] * (re, im)(v_s[c])       (N = 4 x 8 x 2 = 64)
// on tiles of 4 x 8 x 16 cells (2-D: tiles of 8 x 16 cells, the two grid axes in the roles
// of y and z, and B the coil values alone, N = 16).  The accumulator D lives in tensor memory
// (TMEM); A is built in TMEM (tcgen05.st), B in shared memory (K-major, 128-byte swizzle);
// one tcgen05.mma.kind::tf32 covers 8 samples.  Each FP32 operand is split as x = hi + lo
// with hi on the TF32 grid, and three MMAs (hi*hi + hi*lo + lo*hi) give products within
// ~1e-6 of FP32 (the lo*lo term, below 2^-22 relative, is left out).  The tensor core
// evaluates the whole tile for every sample (a 12-tap stencil covers ~22 % of a 4 x 8 x 16
// tile on average) but needs no per-cell instruction: the CUDA cores build 192 operand
// values per (sample, tile) pair instead of issuing the stencil's FMAs.
//
// One (work item, coil group) unit per block; 3 loader warps, NB builder warps (8 in the
// plain instance, 16 in the compensated one) and 1 MMA warp:
// * the loader warps fill a ring of 32-sample batches (loader l: batches l, l + 3, ...; the
//   sample indices of batch l are read before the block's set-up): per sample its tile-plane
//   weights ([plane][sample]) and the 8 coil values times the optional density weight
//   ([coil][sample]); `full` / `empty` mbarriers per slot.
// * the builder warps turn a batch into the MMA operands: a warp writes A's hi and lo parts
//   for the 32 TMEM lanes of its quarter and its share of the samples, and its share of B's
//   rows into shared memory; the operand buffer of batch t is reused by batch t + BUFS after
//   the MMAs of batch t completed (`done` mbarrier, signalled by tcgen05.commit).  In the
//   plain 3-D instance two groups of 4 warps build alternate batches, so that one group's
//   waits, fences and loads overlap the other's building.  After the last batch they read D
//   back (tcgen05.ld) and write the tile.
// * the MMA warp allocates TMEM, and its lane 0 issues 12 MMAs per batch once the builders
//   arrived on the buffer's `ops` mbarrier, then commits to the buffer's `done` mbarrier.
//
// What bounds it: the chain of waits per batch and the instructions of building, not the
// tensor pipe (36 % active).  2.56 M samples x 8 coils on 256^3, 12 taps, with the compensated
// instance: 5.36 ms with the weights computed by the builders behind a barrier of their own;
// 4.45 with the weights in the loaders; 4.12 with three operand buffers, two builder groups and
// 16-byte coil loads.  (16 builder warps: 4.94; 4 in one group: 4.69; 2 or 4 loaders: 4.98,
// 4.60; loaders prefetching a batch ahead: 4.51.)
// Summation: the tensor core's FP32 accumulation rounds less carefully than FP32 adds (its
// error grew with the number of accumulated MMAs: 1.6e-6 relative to the FP32 kernel with
// 1024-sample work items, 4.9e-6 with 8192, on the 3-D radial workload), so the plain
// instance sums groups of kMmaGroup batches (256 samples, 96 MMAs) only; the builders then
// add the accumulator into a running sum S (3-D: shared memory) with FP32 adds before the next group's
// first MMA overwrites it.  The compensated instance (KAHAN: the 3-D dense, k-space-centre
// units, one block per SM) drains every batch's accumulator (two of them alternate) into a
// group sum G with FP32 adds and folds G into a Kahan-compensated sum S, C in TMEM every
// kMmaGroup batches (measured against a Kahan add per batch: the same centre-cell error,
// 3.8e-7, in 1.5 % less time).  The order is fixed for a given trajectory and tiling.
//
// Every wait is bounded (kTmaWaitLimit probes); one that gives up sets kStatusSpreadTimeout
// in the plan's status word and goes on, so no launch can hang.  The plain instance runs a
// block per unit and leaves the dense ones at once; the compensated instance runs a block
// per dense unit only, through the plan's list of dense subproblems.
#pragma once

#include "common.cuh"
#include "grid2d_kernels.cuh"
#include "grid3d_kernels.cuh"
#include "spread3d_cube.cuh"
#include "tc.cuh"

namespace gbn {

constexpr int kMmaTX = 4, kMmaTY = 8, kMmaTZ = 16;  // the tile this kernel takes
constexpr int kMmaM = kMmaTY * kMmaTZ;              // 128 cells (y, z): one TMEM lane each
constexpr int kMmaN = kMmaTX * 16;                  // 64 columns (x, coil, re/im)
constexpr int kMmaBatch = 32;                       // samples per batch: one 128-byte K row
constexpr int kMmaLoaders = 3;
// builder warps: 8 in the plain instance (two blocks per SM, registers), 16 in the
// compensated one (one block per SM: more warps hide its latencies)
template <bool KAHAN> constexpr int mma_builders() { return KAHAN ? 16 : 8; }
// The plain 3-D instance's builders work as two groups of 4 warps on alternate batches, each
// with its own operand buffer
template <int D, bool KAHAN> constexpr int mma_groups() { return D == 3 && !KAHAN ? 2 : 1; }
template <bool KAHAN> constexpr int mma_threads() { return 32 * (mma_builders<KAHAN>() + kMmaLoaders + 1); }
// A (hi, lo) x 2 buffers: 0..127; D from 128; then A's third buffer (3-D) or the running sum S of
// the drained accumulators (2-D)
constexpr uint32_t kMmaTmemCols = 256;
constexpr uint32_t kMmaColD = 128;                  // the MMAs' accumulator
// the compensated instance: two accumulators D (batch k in D[k % 2]), the running sum S, its
// Kahan compensation C and the current group's FP32 sum G; one block per SM
constexpr uint32_t kMmaTmemColsK = 512;
constexpr uint32_t kMmaColSK = 256, kMmaColCK = 320, kMmaColGK = 384;
constexpr int kMmaGroup = 8;                        // batches the tensor core sums before a drain
constexpr int kMmaWS = 36;  // floats per staged [tap] row of 32 samples: 16-byte aligned, 4-bank skew

// shared memory, bytes from a 1024-byte aligned base
constexpr uint32_t kMmaBOp = kMmaN * 128;                               // one B operand: 64 rows x 128 B
constexpr uint32_t kMmaStWx = 0;                                        // [TX][kMmaWS] floats
constexpr uint32_t kMmaStWy = kMmaStWx + 4 * kMmaTX * kMmaWS;           // [TY][kMmaWS]
constexpr uint32_t kMmaStWz = kMmaStWy + 4 * kMmaTY * kMmaWS;           // [TZ][kMmaWS]
constexpr int kMmaVS = kMmaBatch + 2;  // float2 per staged coil row: the four 16-byte quarters of a
                                       // sample's coils are stored to distinct banks
constexpr uint32_t kMmaStV = kMmaStWz + 4 * kMmaTZ * kMmaWS;            // [8 coils][kMmaVS] float2
constexpr uint32_t kMmaStRow = kMmaStV + 8 * 8 * kMmaVS;                // int2: the y rows the batch reaches
constexpr uint32_t kMmaSlotBytes = kMmaStRow + 16;
static_assert(kMmaStV % 16 == 0 && kMmaSlotBytes % 16 == 0, "16-byte aligned staging");
// Per instance: operand buffers, staged batches, and the offsets after B's buffers.  The plain
// 3-D instance keeps three operand buffers -- A's third one takes the TMEM columns of the
// running sum S, which lives in shared memory there -- because a batch's chain (build, MMAs,
// commit, next build) takes longer than two batches of building: 8 % of its time.
template <int D, bool KAHAN> struct MmaCfg {
    static constexpr int BUFS = D == 3 && !KAHAN ? 3 : 2;
    static constexpr int SLOTS = D == 3 && !KAHAN ? 5 : 8;
    static constexpr uint32_t STAGE = 2 * BUFS * kMmaBOp;                 // B (hi, lo) x BUFS
    static constexpr uint32_t SUM = STAGE + SLOTS * kMmaSlotBytes;        // S: [64 columns][128 lanes] floats
    static constexpr uint32_t BAR = SUM + (BUFS == 3 ? 4 * kMmaN * kMmaM : 0);
    static constexpr uint32_t BARS = 2 * SLOTS + 2 * BUFS;                // full, empty, ops, done
    // + the TMEM address word and the alignment slack
    static constexpr size_t NEED = BAR + 8 * BARS + 16 + 1024;
    // The compensated instance asks for more than half the SM's shared memory: one block per SM
    // holds all 512 TMEM columns.  The others take more than a third, so at most two blocks
    // (2 x 256 TMEM columns) share an SM and tcgen05.alloc never waits.
    static constexpr size_t SMEM = KAHAN ? 116 * 1024 : (NEED > 77 * 1024 ? NEED : 77 * 1024);
    static_assert(SMEM >= NEED && SMEM > 228 * 1024 / 3, "shared memory");
    static_assert(KAHAN ? SMEM > 228 * 1024 / 2 : 2 * (SMEM + 1024) <= 228 * 1024, "blocks per SM");
    // A's TMEM columns of buffer b
    static __device__ __forceinline__ uint32_t a_col(int b) { return BUFS == 3 && b == 2 ? 192u : 64u * b; }
};

// The tile of each dimension: M = TY x TZ = 128 cells of grid dimensions (DY, DZ), N = NX
// planes along grid dimension 0 (3-D only) x 8 coils x re/im.  3-D: 4 x 8 x 16 cells,
// N = 64.  2-D: 8 x 16 cells, N = 16 (no plane weight: B is the coil values themselves).
template <int D> struct MmaTile;
template <> struct MmaTile<3> {
    static constexpr int NX = 4, DY = 1, DZ = 2, TAPS = kMmaTX + kMmaTY + kMmaTZ;
};
template <> struct MmaTile<2> {
    static constexpr int NX = 1, DY = 0, DZ = 1, TAPS = kMmaTY + kMmaTZ;
};
template <int D> constexpr int mma_n() { return MmaTile<D>::NX * 16; }


// Two products x = a * b (one packed FP32x2 multiply) split as x = hi + lo: hi rounded to
// the TF32 grid (11 significant bits; ties away from zero, by integer arithmetic on the bit
// pattern), lo = x - hi exactly (one packed subtraction).  The tensor core reads lo's top 11
// significant bits.  (Dekker's split t = x (2^13 + 1), hi = t - (t - x) in packed FP32x2
// arithmetic was measured on GB300 to return hi = x, lo = 0, so it is not used.)
__device__ __forceinline__ float tf32_round_bits(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}
// (Rounding lo to the TF32 grid as well and adding the lo * lo MMA left the compensated
// instance's centre-cell error unchanged, 3.9e-7 against 3.8e-7 on the 3-D radial test
// data, and cost 0.09 ms of 6.0 on the 3-D radial workload: the tensor core's own FP32
// accumulation within a batch dominates, so neither is done.)
__device__ __forceinline__ void tf32_split2(float2 a, float2 b, float2 &hi, float2 &lo) {
    const float2 x = __fmul2_rn(a, b);
    hi = make_float2(tf32_round_bits(x.x), tf32_round_bits(x.y));
    lo = __fadd2_rn(x, make_float2(-hi.x, -hi.y));
}

// S (+)= D over this thread's lane and the N / 2 columns of half hk; `first`: S = D.  D is
// at column kMmaColD, S right after it (N columns each).
// Where ssum is given (3-D), S is kept there: [column][128 lanes], this lane's at ssum.
template <int N, int DPW>
__device__ __forceinline__ void mma_drain(uint32_t tl, int hk, bool first, float *ssum = nullptr) {
    constexpr uint32_t kColS = kMmaColD + N;
    if constexpr (N == 64) {
#pragma unroll
        for (int h = 0; h < DPW / 16; ++h) {
            const uint32_t col = (uint32_t)DPW * hk + 16u * h;
            float d[16];
            tmem_ld_x16(tl + kMmaColD + col, d);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float &t = ssum[(col + i) * kMmaM];
                t = first ? d[i] : t + d[i];
            }
        }
    } else {
        static_assert(N == 16, "N is 64 (3-D) or 16 (2-D)");
        const uint32_t col = 8u * hk;
        float d[8], s[8];
        tmem_ld_x8(tl + kMmaColD + col, d);
        if (!first) {
            tmem_ld_x8(tl + kColS + col, s);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) d[i] += s[i];
        } else {
            tmem_wait_ld();
        }
        tmem_st_x8(tl + kColS + col, d);
    }
}

// S, C (+)= D[col_d] with Kahan compensation over this thread's lane and NCH 16-column
// chunks from column col0 (scalar FP32 operations); `first`: S = D, C = 0
template <int NCH>
__device__ __forceinline__ void mma_drain_kahan(uint32_t tl, uint32_t col0, uint32_t col_d, bool first) {
#pragma unroll
    for (int h = 0; h < NCH; ++h) {
        const uint32_t col = col0 + 16u * h;
        float d[16], s[16], c[16];
        tmem_ld_x16(tl + col_d + col, d);
        if (first) {
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) c[i] = 0.f;
            tmem_st_x16(tl + kMmaColSK + col, d);
        } else {
            tmem_ld_x16(tl + kMmaColSK + col, s);
            tmem_ld_x16(tl + kMmaColCK + col, c);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float y = d[i] - c[i];
                const float t = s[i] + y;
                c[i] = (t - s[i]) - y;
                s[i] = t;
            }
            tmem_st_x16(tl + kMmaColSK + col, s);
        }
        tmem_st_x16(tl + kMmaColCK + col, c);
    }
}

// G (+)= D[col_d] over this thread's lane and NCH 16-column chunks from column col0, G at
// kMmaColGK; `first`: G = D
template <int NCH>
__device__ __forceinline__ void mma_drain_group(uint32_t tl, uint32_t col0, uint32_t col_d, bool first) {
#pragma unroll
    for (int h = 0; h < NCH; ++h) {
        const uint32_t col = col0 + 16u * h;
        float d[16], gs[16];
        tmem_ld_x16(tl + col_d + col, d);
        if (!first) {
            tmem_ld_x16(tl + kMmaColGK + col, gs);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] += gs[i];
        } else {
            tmem_wait_ld();
        }
        tmem_st_x16(tl + kMmaColGK + col, d);
    }
}

// compensated instance: batch j's accumulator D[col_d] into the group sum G; when batch j
// starts a new group of kMmaGroup batches, the last group's G is first folded into the
// Kahan-compensated S, C
template <int NCH>
__device__ __forceinline__ void mma_drain_batch_k2(uint32_t tl, uint32_t col0, uint32_t col_d, int j) {
    if (j % kMmaGroup == 0 && j > 0) {
        mma_drain_kahan<NCH>(tl, col0, kMmaColGK, j == kMmaGroup);
        tmem_wait_st();
    }
    mma_drain_group<NCH>(tl, col0, col_d, j % kMmaGroup == 0);
}

// Dimension D (3: 4 x 8 x 16 tiles, N = 64; 2: 8 x 16 tiles, N = 16).  One kernel template
// rather than a device function behind per-dimension kernels: the arguments stay in the
// parameter space (an inlined copy of them cost registers and 4.5 % of the 3-D time).
template <int D, int WT, bool KAHAN>
__global__ void __launch_bounds__(mma_threads<KAHAN>(), KAHAN ? 1 : 2) k_spread_mma(SpreadArgs a, uint32_t *status, int n_cg) {
    constexpr int NB = mma_builders<KAHAN>();  // builder warps
    constexpr int WM = NB + kMmaLoaders;       // the MMA warp's index
    constexpr int NG = mma_groups<D, KAHAN>(); // builder groups: group b builds batches b, b + NG, ...
    constexpr int NBG = NB / NG;               // warps of a group
    constexpr int SPW = 128 / NBG;             // A: samples of the batch per builder warp (32 or 8)
    constexpr int RPW = mma_n<D>() / NBG;      // B: rows per builder warp
    constexpr int DPW = 256 / NBG;             // accumulator columns per builder warp and drain (3-D)
    constexpr int CPW = 256 / NB;              // accumulator columns per builder warp at the end (3-D)
    using T = MmaTile<D>;
    constexpr int N = mma_n<D>();
    constexpr uint32_t kBOp = N * 128;  // one B operand: N rows x 128 B
    constexpr uint32_t kCols = KAHAN ? kMmaTmemColsK : kMmaTmemCols;
    constexpr int B = kMmaBatch;
    constexpr int CG = 8;
    static_assert(!KAHAN || D == 3, "dense tiles are a 3-D notion");
    extern __shared__ unsigned char smem_mma_raw[];
    unsigned char *sm = smem_mma_raw + ((1024u - (smem_addr(smem_mma_raw) & 1023u)) & 1023u);
    unsigned char *opB = sm;  // [buf][hi, lo][N rows x 128 B], SW128
    using Cfg = MmaCfg<D, KAHAN>;
    constexpr int BUFS = Cfg::BUFS, SLOTS = Cfg::SLOTS;
    unsigned char *stage = sm + Cfg::STAGE;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + Cfg::BAR);
    uint64_t *empty = full + SLOTS;
    uint64_t *ops = empty + SLOTS;
    uint64_t *done = ops + BUFS;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + BUFS);

    const Geom &g = a.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = WT ? WT : g.W;

    // the plain instance runs a block per unit, the compensated one a block per dense unit
    // (through the list of dense subproblems); a block whose unit is of the other kind leaves
    // before it takes TMEM (all its threads alike)
    const int64_t unit = KAHAN ? (int64_t)a.dense_subs[blockIdx.x / n_cg] * n_cg + blockIdx.x % n_cg
                               : (int64_t)blockIdx.x;
    int4 sub;
    if (!cube_unit(a.subs, unit, n_cg, KAHAN, sub)) return;
    // a loader warp's first sample indices (its first batch: k = loader index), read before
    // the set-up below so that their latency overlaps it
    const int64_t stride = max(1, sub.w >> kStrideShift);  // interleaved item of a split tile
    uint32_t j0 = 0;
    if (warp >= NB && warp < WM && (warp - NB) * B + lane < sub.z)
        j0 = a.idx[(int64_t)sub.y + (int64_t)((warp - NB) * B + lane) * stride];

    if (warp == WM) {
        tmem_alloc(tslot, kCols);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < SLOTS; ++k) {
            mbar_init(&full[k], 32);                  // the loader warp, every lane
            mbar_init(&empty[k], NBG * 32);  // every builder lane of the batch's group
        }
        for (int b = 0; b < BUFS; ++b) {
            mbar_init(&ops[b], NBG * 32);
            mbar_init(&done[b], 1);                   // tcgen05.commit
        }
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;

    {
        const int nb = (sub.z + B - 1) / B;
        const int cg0 = (int)(unit % n_cg) * CG;

        if (warp >= NB && warp < WM) {
            // ------------------------------------------------------------ loader warp
            int o[3], e[3];
            tile_coords<D>(g, sub.x % g.ntiles, o, e);
            const int lw = warp - NB;
            const bool vec = a.c_coil == 1 && a.c_elem % 2 == 0 && cg0 + CG <= g.n_coil &&
                             (reinterpret_cast<uintptr_t>(a.c) & 15) == 0;
            const int ns = g.ns;
            for (int k = lw; k < nb; k += kMmaLoaders) {
                const int slot = k % SLOTS;
                const int n = min(B, sub.z - k * B);
                const bool ok = lane < n;
                float4 pt = make_float4(0.f, 0.f, 0.f, 0.f);
                uint32_t j = 0;
                if (ok) {
                    j = k == lw ? j0 : a.idx[(int64_t)sub.y + (int64_t)(k * B + lane) * stride];
                    pt = a.pts_by_sample[j];
                }
                float sw = 1.f;
                if (ok && a.weight) sw = a.weight[j];
                // the 8 coil values of each sample: where they are one aligned 64-byte run, four
                // lanes read a sample's together (16 bytes each, 8 samples an instruction: a
                // quarter of the sectors per request of a lane reading its own sample)
                float4 v4[4];
                float2 v[CG];
                if (vec) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int s8 = 8 * i + (lane >> 2);
                        const uint32_t js = __shfl_sync(0xffffffffu, j, s8);
                        v4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (s8 < n)
                            v4[i] = *reinterpret_cast<const float4 *>(a.c + (int64_t)js * a.c_elem + cg0 +
                                                                      2 * (lane & 3));
                    }
                } else {
#pragma unroll
                    for (int cc = 0; cc < CG; ++cc) {
                        v[cc] = make_float2(0.f, 0.f);
                        if (ok && cg0 + cc < g.n_coil)
                            v[cc] = a.c[(int64_t)j * a.c_elem + (int64_t)(cg0 + cc) * a.c_coil];
                    }
                }
                int r[3] = {0, 0, 0};
                if (ok) {
                    int c0[3];
                    unpack_cells(D, __float_as_uint(pt.w), c0[0], c0[1], c0[2]);
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        int rr = c0[d] - o[d];
                        rr += rr < 0 ? g.nf[d] : 0;
                        rr -= rr > g.nf[d] - W ? g.nf[d] : 0;
                        r[d] = rr;
                    }
                }
                // the slot's previous batch must be released by every builder lane
                if (k >= SLOTS &&
                    !mbar_wait_bounded(&empty[slot], (uint32_t)((k / SLOTS - 1) & 1)) && lane == 0)
                    atomicOr(status, kStatusSpreadTimeout);
                unsigned char *sl = stage + (size_t)slot * kMmaSlotBytes;
                // the sample's tile-plane weights (28 in 3-D, 24 in 2-D); a lane without a
                // sample gets a first tap no plane reaches, so all its weights are 0
                const float pf[3] = {pt.x, pt.y, pt.z};
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    constexpr int OFF = 3 - D;  // 2-D: the axes are the tile's y and z planes
                    const int planes = d + OFF == 0 ? kMmaTX : (d + OFF == 1 ? kMmaTY : kMmaTZ);
                    float *wp = reinterpret_cast<float *>(
                        sl + (d + OFF == 0 ? kMmaStWx : (d + OFF == 1 ? kMmaStWy : kMmaStWz)));
                    const float d0 = pf[d] + (float)(ns - 1 + r[d]);
                    const int rs = ok ? r[d] : -(1 << 20);
                    const float beta = g.beta2[d];
#pragma unroll
                    for (int t = 0; t < planes; ++t) {
                        const float dd = d0 - (float)t;
                        const float wv = ex2_approx(-beta * dd * dd);
                        wp[t * kMmaWS + lane] = (unsigned)(t - rs) < (unsigned)W ? wv : 0.f;
                    }
                }
                if constexpr (D == 3) {
                    // first and last y row that some sample of the batch reaches
                    const int lo = __reduce_min_sync(0xffffffffu, ok ? r[1] : kMmaTY);
                    const int hi = __reduce_max_sync(0xffffffffu, ok ? r[1] + W - 1 : -1);
                    if (lane == 0) *reinterpret_cast<int2 *>(sl + kMmaStRow) = make_int2(lo, hi);
                }
                float2 *vs = reinterpret_cast<float2 *>(sl + kMmaStV);
                if (vec) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int s8 = 8 * i + (lane >> 2);
                        const float ws = __shfl_sync(0xffffffffu, sw, s8);
                        float2 *vp = vs + 2 * (lane & 3) * kMmaVS + s8;
                        vp[0] = make_float2(v4[i].x * ws, v4[i].y * ws);
                        vp[kMmaVS] = make_float2(v4[i].z * ws, v4[i].w * ws);
                    }
                } else {
#pragma unroll
                    for (int cc = 0; cc < CG; ++cc) vs[cc * kMmaVS + lane] = make_float2(v[cc].x * sw, v[cc].y * sw);
                }
                mbar_arrive(&full[slot]);
            }
        } else if (warp == WM) {
            // ------------------------------------------------------------ MMA warp
            if (lane == 0) {
                constexpr uint32_t idesc = tc_idesc_tf32(kMmaM, N);
                const uint32_t b0 = smem_addr(opB);
                for (int k = 0; k < nb; ++k) {
                    const int buf = k % BUFS;
                    if (!mbar_wait_bounded(&ops[buf], (uint32_t)((k / BUFS) & 1))) atomicOr(status, kStatusSpreadTimeout);
                    tc_fence_after();
                    const uint32_t ah = tbase + Cfg::a_col(buf), al = ah + 32u;
                    const uint32_t d = tbase + kMmaColD + (KAHAN ? 64u * buf : 0u);
                    // K step jk starts 32 jk bytes further: + 2 jk in the descriptor's address
                    // field (16-byte units; shared addresses stay far below its 14-bit range)
                    const uint64_t dbh = tc_desc_sw128(b0 + 2u * buf * kBOp), dbl = tc_desc_sw128(b0 + (2u * buf + 1u) * kBOp);
                    // plain: a group's first MMA starts D afresh; compensated: every batch's
                    const uint32_t acc0 = KAHAN ? 0u : (uint32_t)((k % kMmaGroup) != 0);
#pragma unroll
                    for (int jk = 0; jk < B / 8; ++jk) {
                        const uint64_t xh = dbh + (uint64_t)(2 * jk), xl = dbl + (uint64_t)(2 * jk);
                        tc_mma_tf32_ts(d, ah + 8u * jk, xh, idesc, jk == 0 ? acc0 : 1u);
                        tc_mma_tf32_ts(d, ah + 8u * jk, xl, idesc, 1u);
                        tc_mma_tf32_ts(d, al + 8u * jk, xh, idesc, 1u);
                    }
                    tc_commit(&done[buf]);
                }
            }
            __syncwarp();
        } else {
            // ------------------------------------------------------------ builder warp
            // warp (q, hk): TMEM quarter q; A for samples SPW hk .. SPW hk + SPW - 1 of a batch;
            // B rows RPW warp .. (3-D: x plane bx, coils bc0 .. bc0 + RPW / 2 - 1); the
            // accumulator's columns CPW hk .. (3-D)
            const int wg = warp % NBG, grp_b = warp / NBG;
            const int q = wg & 3, hk = wg >> 2;
            const int m = 32 * q + lane, y = m >> 4, z = m & 15;  // tile cell (y, z) of TMEM lane m
            const uint32_t tl = tmem_lane_base(tbase, q);
            float *ssum = D == 3 && !KAHAN ? reinterpret_cast<float *>(sm + Cfg::SUM) + m : nullptr;
            for (int k = grp_b; k < nb; k += NG) {
                const int slot = k % SLOTS, buf = k % BUFS;
                if (!mbar_wait_bounded(&full[slot], (uint32_t)((k / SLOTS) & 1)) && lane == 0)
                    atomicOr(status, kStatusSpreadTimeout);
                // the MMAs of batch k - BUFS (same operand buffer) have completed
                if (k >= BUFS && !mbar_wait_bounded(&done[buf], (uint32_t)((k / BUFS - 1) & 1)) && lane == 0)
                    atomicOr(status, kStatusSpreadTimeout);
                if constexpr (KAHAN) {
                    if (k >= 2) {
                        // batch k - 2's accumulator D[k % 2] into the group sum before batch k
                        // overwrites it
                        tc_fence_after();
                        mma_drain_batch_k2<DPW / 16>(tl, DPW * hk, kMmaColD + 64u * buf, k - 2);
                    }
                }
                const unsigned char *sl = stage + (size_t)slot * kMmaSlotBytes;
                // A: cells (y, z) of this lane, samples SPW hk .. SPW hk + SPW - 1
                const float4 *wy4 = reinterpret_cast<const float4 *>(sl + kMmaStWy) + (y * kMmaWS + SPW * hk) / 4;
                const float4 *wz4 = reinterpret_cast<const float4 *>(sl + kMmaStWz) + (z * kMmaWS + SPW * hk) / 4;
                // (3-D) this quarter's rows 2 q, 2 q + 1 that no sample of the batch reaches are
                // zeros; the list's order by row makes that 32 % of all quarters
                bool reach = true;
                if constexpr (D == 3) {
                    const int2 rows = *reinterpret_cast<const int2 *>(sl + kMmaStRow);
                    reach = rows.x <= 2 * q + 1 && rows.y >= 2 * q;
                }
#pragma unroll
                for (int h = 0; h < SPW / 8; ++h) {  // 8 samples at a time: fewer live registers
                    float hi[8], lo[8];
                    if (!reach) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) hi[i] = 0.f;
                        tmem_st_x8(tl + Cfg::a_col(buf) + SPW * hk + 8u * h, hi);
                        tmem_st_x8(tl + Cfg::a_col(buf) + 32u + SPW * hk + 8u * h, hi);
                        continue;
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float4 p = wy4[2 * h + i], s = wz4[2 * h + i];
                        float2 h0, l0, h1, l1;
                        tf32_split2(make_float2(p.x, p.y), make_float2(s.x, s.y), h0, l0);
                        tf32_split2(make_float2(p.z, p.w), make_float2(s.z, s.w), h1, l1);
                        hi[4 * i] = h0.x;
                        hi[4 * i + 1] = h0.y;
                        hi[4 * i + 2] = h1.x;
                        hi[4 * i + 3] = h1.y;
                        lo[4 * i] = l0.x;
                        lo[4 * i + 1] = l0.y;
                        lo[4 * i + 2] = l1.x;
                        lo[4 * i + 3] = l1.y;
                    }
                    tmem_st_x8(tl + Cfg::a_col(buf) + SPW * hk + 8u * h, hi);
                    tmem_st_x8(tl + Cfg::a_col(buf) + 32u + SPW * hk + 8u * h, lo);
                }
                const float2 *vs = reinterpret_cast<const float2 *>(sl + kMmaStV);
                unsigned char *bh = opB + (size_t)(2 * buf) * kBOp, *bl = bh + kBOp;
                if constexpr (D == 3) {
                    // B: rows RPW wg .. (x plane, coil, re/im) for sample `lane`
#pragma unroll
                    for (int cc = 0; cc < RPW / 2; ++cc) {
                        const int nre = RPW * wg + 2 * cc;  // row: 16 x + 2 coil
                        const float wxk =
                            reinterpret_cast<const float *>(sl + kMmaStWx)[(nre >> 4) * kMmaWS + lane];
                        const float2 vv = vs[((nre & 15) >> 1) * kMmaVS + lane];
                        float2 h, l;
                        tf32_split2(make_float2(wxk, wxk), vv, h, l);
                        *reinterpret_cast<float *>(bh + sw128_offset(nre, lane)) = h.x;
                        *reinterpret_cast<float *>(bl + sw128_offset(nre, lane)) = l.x;
                        *reinterpret_cast<float *>(bh + sw128_offset(nre + 1, lane)) = h.y;
                        *reinterpret_cast<float *>(bl + sw128_offset(nre + 1, lane)) = l.y;
                    }
                } else {
                    // B: rows (coil = warp, re/im) for sample `lane`: the coil value itself
                    const float2 vv = vs[warp * kMmaVS + lane];
                    float2 h, l;
                    tf32_split2(make_float2(1.f, 1.f), vv, h, l);
                    *reinterpret_cast<float *>(bh + sw128_offset(2 * warp, lane)) = h.x;
                    *reinterpret_cast<float *>(bl + sw128_offset(2 * warp, lane)) = l.x;
                    *reinterpret_cast<float *>(bh + sw128_offset(2 * warp + 1, lane)) = h.y;
                    *reinterpret_cast<float *>(bl + sw128_offset(2 * warp + 1, lane)) = l.y;
                }
                mbar_arrive(&empty[slot]);
                if (!KAHAN && k % kMmaGroup == 0 && k > 0) {
                    // batch k starts a new group: once the previous group's MMAs are done,
                    // add its accumulator into S.  (The MMAs complete in order and batch k -
                    // BUFS was waited for above, so this barrier is in batch k - 1's phase.)
                    if (!mbar_wait_bounded(&done[(k - 1) % BUFS], (uint32_t)(((k - 1) / BUFS) & 1)) && lane == 0)
                        atomicOr(status, kStatusSpreadTimeout);
                    tc_fence_after();
                    mma_drain<N, DPW>(tl, hk, k == kMmaGroup, ssum);
                }
                // operands visible to the tensor core before the MMA warp proceeds
                tmem_wait_st();
                fence_proxy_async_smem();
                tc_fence_before();
                mbar_arrive(&ops[buf]);
            }

            // ---------------------------------------------------------------- epilogue
            if (nb > 0) {
                const int kl = nb - 1;
                // (two groups: the group's own last batch first, after which the other buffer's
                // barrier is in the phase of the block's last batch, so that its parity means
                // that phase and not the one before)
                const int ko = NG == 2 ? ((kl & 1) == grp_b ? kl : kl - 1) : kl;
                if (ko >= 0 && !mbar_wait_bounded(&done[ko % BUFS], (uint32_t)((ko / BUFS) & 1)) && lane == 0)
                    atomicOr(status, kStatusSpreadTimeout);
                if (NG == 2 && ko != kl && !mbar_wait_bounded(&done[kl % BUFS], (uint32_t)((kl / BUFS) & 1)) && lane == 0)
                    atomicOr(status, kStatusSpreadTimeout);
                if constexpr (NG == 2) {
                    // S, drained by group 0, is read by all builders below
                    asm volatile("bar.sync 1, %0;" ::"n"(NB * 32) : "memory");
                }
                tc_fence_after();
                if constexpr (KAHAN) {
                    // the last two batches' accumulators, in order
                    for (int j = max(0, nb - 2); j < nb; ++j) {
                        mma_drain_batch_k2<DPW / 16>(tl, DPW * hk, kMmaColD + 64u * (j & 1), j);
                        tmem_wait_st();  // G (and S, C) stored before the next drain reads them
                    }
                    // the last group's sum into S, C (S = G when there was one group)
                    mma_drain_kahan<DPW / 16>(tl, DPW * hk, kMmaColGK, nb <= kMmaGroup);
                    tmem_wait_st();
                }
            }
            // the tile's columns over all builder warps
            const int he = warp >> 2;
            // the unit's tile, read again here rather than kept in registers through the loop
            const int4 su = a.subs[unit / n_cg];
            int o[3], e[3];
            tile_coords<D>(g, su.x % g.ntiles, o, e);
            const int grp = su.x / g.ntiles;
            const bool split = (su.w & kSplitFlag) != 0;
            const bool inside = y < e[T::DY] && z < e[T::DZ];
            if constexpr (D == 3) {
                // this warp: lanes of quarter q, columns CPW he .. (x planes CPW he / 16 ..)
                const int64_t cell_yz = (int64_t)(o[1] + y) * g.nf[2] + (o[2] + z);
#pragma unroll
                for (int xi = 0; xi < CPW / 16; ++xi) {
                    // columns CPW he + 16 xi ..: cell x = (CPW / 16) he + xi, (coil, re/im) pairs
                    float dv[16];
                    if (nb > 0 && KAHAN) {
                        float cv[16];
                        tmem_ld_x16(tl + kMmaColSK + CPW * he + 16u * xi, dv);
                        tmem_ld_x16(tl + kMmaColCK + CPW * he + 16u * xi, cv);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) dv[i] -= cv[i];
                    } else if (nb > 0) {
                        tmem_ld_x16(tl + kMmaColD + CPW * he + 16u * xi, dv);
                        tmem_wait_ld();
                        if (nb > kMmaGroup) {  // plus the drained groups
#pragma unroll
                            for (int i = 0; i < 16; ++i) dv[i] += ssum[(CPW * he + 16 * xi + i) * kMmaM];
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) dv[i] = 0.f;
                    }
                    const int x = (CPW / 16) * he + xi;
                    if (!inside || x >= e[0]) continue;
                    const int64_t cell = (int64_t)(o[0] + x) * g.nf[1] * g.nf[2] + cell_yz;
#pragma unroll
                    for (int c = 0; c < CG; ++c) {
                        if (cg0 + c >= g.n_coil) break;
                        float2 *dst = a.grid + ((int64_t)grp * g.n_coil + cg0 + c) * g.G + cell;
                        if (split) {
                            atomicAdd(&dst->x, dv[2 * c]);
                            atomicAdd(&dst->y, dv[2 * c + 1]);
                        } else {
                            *dst = make_float2(dv[2 * c], dv[2 * c + 1]);
                        }
                    }
                }
            } else {
                // this warp: lanes of quarter q, columns 8 he .. 8 he + 7 (coils 4 he .. 4 he + 3)
                float dv[8];
                if (nb > 0) {
                    tmem_ld_x8(tl + kMmaColD + 8u * he, dv);
                    if (nb > kMmaGroup) {  // plus the drained groups
                        float sv[8];
                        tmem_ld_x8(tl + kMmaColD + N + 8u * he, sv);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; ++i) dv[i] += sv[i];
                    } else {
                        tmem_wait_ld();
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) dv[i] = 0.f;
                }
                if (inside) {
                    const int64_t cell = (int64_t)(o[0] + y) * g.nf[1] + (o[1] + z);
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) {
                        const int c = 4 * he + cc;
                        if (cg0 + c >= g.n_coil) break;
                        float2 *dst = a.grid + ((int64_t)grp * g.n_coil + cg0 + c) * g.G + cell;
                        if (split) {
                            atomicAdd(&dst->x, dv[2 * cc]);
                            atomicAdd(&dst->y, dv[2 * cc + 1]);
                        } else {
                            *dst = make_float2(dv[2 * cc], dv[2 * cc + 1]);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == WM) tmem_dealloc(tbase, kCols);
}


}  // namespace gbn
