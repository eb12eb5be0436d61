// tc_stream.cu - weights streamed once from HBM past the activation rows of a call on the 5th-generation
// tensor cores: the projections of two and more positions (up to the engine's pass of 2048), and the experts
// of two and more tokens.
//
// Three kernels: BF16 weights (tc_stream_bf16_kernel) and FP8 weights of up to 64 positions (tc_stream_fp8_kernel) go past
// one tile of at most 64 rows, each CTA an equal share of all columns; experts, and FP8 weights of more positions, past tiles of at most
// 32 rows, in pairs of 128 weight rows (tc_pair_kernel, described beside it). Further tiles of rows find the weights in L2.
//
// Reference: glm53f_mm_batch / matmul_f8_batch / matmul_bf16 (src/core/glm53f_ops.c:101-154,
// 378-444) and moe_chunk (:1144-1342), which decode each block of codes once for up to 64 inputs.
//
// One persistent CTA per SM. A row tile is 128 rows of W; its columns are cut into units of 32 KB of
// FP8 weights (256 codes per row) or 16 KB of BF16 (64 values). All units of the launch are numbered in a row and
// every CTA takes an equal, contiguous share, whatever the shapes: no last wave of tiles, no choice of a split.
// A tile that two or more CTAs worked on is put together by the one that finishes last (partial sums in
// an L2-resident buffer, added in the order of the columns, so the result does not depend on who that is). Where a
// projection's tile is cut depends on the launch, so the last bits of a row do too (its matrices, the number of positions, which
// tile of rows it is in): the ranks of a group agree because they run the same launch.
//
//   A operand  = 128 rows of W. BF16: the TMA tile in shared memory as stored. FP8: eight converter
//                warps turn the TMA tile's codes into F16 (exact) and put them into tensor memory, from
//                where the MMA takes them: through shared memory a 16 KB block would cross it six times (32 KB
//                written and 32 KB read beside the 16 KB in, 16 KB out and the activations), which
//                at 128 B per clock takes longer than HBM takes to deliver the block.
//   B operand  = the activations as exact sums of 16-bit terms (FP8 weights: x 2^e = hi + mid / 2048 in
//                F16; BF16 weights: hi + mid + lo in BF16), N = terms x rows; products are exact and
//                only the FP32 accumulation rounds. Terms lie in global memory (L2 resident) and are
//                loaded by TMA beside the weights.
//   D          = FP32 accumulators in tensor memory. FP8: one per 128 columns (they share one scale per
//                128 rows), multiplied by the scale and summed in registers. BF16: one per 512 columns, because
//                the tensor cores truncate when they accumulate (4096 columns in one accumulator come out 5e-6
//                off, in pieces of 512 6e-7).
//
// What the split of the work is about: a warp with a role of its own pays for every step of it - a wait on an
// mbarrier costs 100 to 200 cycles even when it has long been satisfied, a TMA load 150 to issue, an MMA of a few rows
// only 22 - and HBM delivers 32 KB to an SM in about 1400 cycles. So: FP8 units of 32 KB, not 16; one load
// instruction per unit for the weights and one for all terms; one barrier for both operands of an MMA; two warps that
// issue the MMAs of units in turn; and two groups of epilogue warps, which take units in turn while a tile has at
// most 32 rows and half of the rows each beyond. BF16 with 64 rows: 40 KB of shared memory a unit of 64 columns, five stages (in units of 128
// columns two, whose way from L2 showed: KDA projections of 64 positions 46.5 -> 42.7 us a launch); its products read 40 KB more
// there, 640 cycles in all of the 870 that it takes. The roles' code shares the SM's instruction cache: wait loops that the compiler
// had unrolled made it 96 KB, and every rarely run line cost its way from L2.
//
// Warps (FP8): 0-7 epilogue (tcgen05.ld: warp w reaches lanes 32 (w % 4) ..), 8-15 conversion, 16 weights, 17 terms,
// 18 and 19 MMA. BF16: 0-7 epilogue, 8 weights, 9 MMA, 10 terms. Every wait is bounded; one that runs out records a
// code in mapped host memory, lets every role drain its copies and MMAs, frees the tensor memory and returns.
#include <map>
#include <tuple>

#include "kernels.h"
#include "mma_stage.cuh"
#include "tc_ptx.cuh"

namespace g5b {

constexpr int TS_MAX_SEG = 8;              // matrices of one launch
constexpr int TS_N = 64;                   // activation rows per tile at most (of a pair of tiles: TP_ROWS)
constexpr int TS_EN = TS_N / 2;            // rows an epilogue thread holds
constexpr int TS_PARTS = 4;                 // partial results of a tile that are read at once
constexpr int TS_MAX_STAGES = 8, TS_MAX_XS = 3;    // FP8: activation stages at most
constexpr int TS_UNIT_BYTES = 32768, TS_EXCH = TS_EN * 128 * 4;
constexpr int TS_BF16_UNIT = TS_UNIT_BYTES / 2;    // BF16: units of 64 columns
constexpr int TS_SEG_UNITS = 8;            // BF16: units summed inside the tensor cores before the registers take over (512 columns)
enum { TS_DENSE = 0, TS_GATEUP = 1, TS_DOWN = 2 };
constexpr int TS_FP8_THREADS = 20 * 32, TS_BF16_THREADS = 11 * 32;

struct TsSeg {
    const float *S, *inv;      // FP8: block scales, 2^-e of each activation row
    float *y;
    int scols, R, ldy, tile0, xrow;
};
struct TsMaps { CUtensorMap w[TS_MAX_SEG], x[TS_N / 8]; };      // x: boxes of 8, 16, ... 64 rows
struct TsArgs {
    TsSeg seg[TS_MAX_SEG];
    int n_seg, tiles;          // projections: tiles of all matrices
    int KB;                    // units (pairs: steps of 128 columns) per tile
    int blocks;                // FP8: 128-column blocks per row (2 KB, or one less)
    int T, n, plane;           // rows, rows of the largest tile (a multiple of 8); rows between the terms' planes
    int nt;                    // projections: tiles of n rows that T rows make
    // experts
    const uint8_t *scales;     // expert 0's scales of the matrix (gate/up: of the gate); the up projection's lie up_off on
    size_t scale_stride, up_off;
    MoePlan p;
    int slots, RT, E, I;       // slots at most; 256-row tiles per expert
    const float *xinv;         // 2^-e of each pair's activation
    void *out;                 // gate/up: F16 terms, planes of [plane][I]; down: contribution rows [.][E]
    float limit, act_scale, act_inv;   // the scale of the SwiGLU output's terms, a power of two, and its reciprocal
    int *sched;                // work claimed, CTAs done (both zero between launches)
    float *part; int *cnt;     // partial results [CTA][2][row][128] (pairs: [claimed quarter][group][row][128]), units (quarters) done per tile (zero between launches)
    int xs;                    // FP8: activation stages
    int stages, x_stage;       // weight stages (BF16: of weights and terms); bytes of one stage's terms
    int *err;
};

// How a slot's cnt rows are cut into tiles: equal shares of at most `most` rows (a multiple of 8), rounded up to 8.
__device__ __forceinline__ int ts_tile_rows(int cnt, int most)
{
    if (cnt <= most) return (cnt + 7) & ~7;
    const int k = (cnt + most - 1) / most;
    return ((cnt + k - 1) / k + 7) & ~7;
}

// Walks the tiles of a CTA's share in order: matrix (or expert) `which`, its row tile rt, the np activation rows from
// row0 on, n = np rounded up to 8. An expert's row tile goes past its token tiles one after the other: its weights
// come from L2 then.
struct TsPlan { const int *tile0, *off, *cnt, *exp; int slots, rows; };
template <int MODE>
struct TsCursor {
    int which, rt, row0, np, n;
    int slot, tt, nt, rows, cnt;               // (projections: row0 = the matrix's first terms row + tt * n)
    __device__ __forceinline__ void rows_of_tile(const TsPlan &p)
    {
        const int left = cnt - tt * rows;
        row0 = p.off[slot] + tt * rows;
        np = left < rows ? left : rows;
        n = (np + 7) & ~7;
    }
    __device__ __forceinline__ void columns(const TsArgs &a)
    {
        const int left = a.T - tt * a.n;
        row0 = a.seg[which].xrow + tt * a.n;
        np = left < a.n ? left : a.n;
        n = (np + 7) & ~7;
    }
    __device__ __forceinline__ void enter(const TsPlan &p)
    {
        which = p.exp[slot]; cnt = p.cnt[slot]; rows = ts_tile_rows(cnt, p.rows); nt = p.tile0[slot + 1] - p.tile0[slot];
    }
    __device__ __forceinline__ void start(const TsArgs &a, const TsPlan &p, int tile)
    {
        if (MODE == TS_DENSE) {
            which = 0;
            for (int i = 1; i < a.n_seg; i++) if (tile >= a.seg[i].tile0) which = i;
            const int local = tile - a.seg[which].tile0;
            rt = local / a.nt; tt = local - rt * a.nt;
            columns(a);
        } else {
            int lo = 0, hi = p.slots - 1;                     // the last slot whose first tile is not beyond this one
            while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (p.tile0[mid] * a.RT <= tile) lo = mid; else hi = mid - 1; }
            slot = lo;
            enter(p);
            const int local = tile - p.tile0[lo] * a.RT;
            rt = local / nt; tt = local - rt * nt;
            rows_of_tile(p);
        }
    }
    __device__ __forceinline__ void next(const TsArgs &a, const TsPlan &p)      // (may step past the last tile: not used then)
    {
        if (MODE == TS_DENSE) {
            if (++tt == a.nt) { tt = 0; rt++; }
            if (tt == 0 && which + 1 < a.n_seg && rt * a.nt == a.seg[which + 1].tile0 - a.seg[which].tile0) { which++; rt = 0; }
            columns(a);
        } else {
            if (++tt == nt) { tt = 0; rt++; }
            if (rt == a.RT) {
                rt = 0;
                if (slot + 1 >= p.slots) return;
                slot++;
                enter(p);
                rows_of_tile(p);
            } else if (nt > 1) rows_of_tile(p);
        }
    }
};

// What the epilogue needs to know of a tile, fetched while the tile before it is multiplied.
template <bool FP8>
struct TsEpi {
    const float *srow;         // block scales of the tile's rows
    float2 s0;                 // lane i: those of unit i of the share's part of the tile (of the first 32)
    float inv0, inv1;          // lane i: 2^-e of rows i and i + 32
    __device__ __forceinline__ void fetch(const TsArgs &a, const TsCursor<TS_DENSE> &t, int kb, int lane)
    {
        if (!FP8) return;
        srow = a.seg[t.which].S + (size_t)t.rt * a.seg[t.which].scols;
        s0 = kb + lane < a.KB ? pair(a, kb + lane) : make_float2(0.f, 0.f);
        const float *iv = a.seg[t.which].inv + t.tt * a.n;
        inv0 = lane < t.np ? __ldcg(iv + lane) : 0.f;
        inv1 = lane + 32 < t.np ? __ldcg(iv + lane + 32) : 0.f;
    }
    __device__ __forceinline__ float2 pair(const TsArgs &a, int kb) const
    {
        return make_float2(__ldg(srow + 2 * kb), 2 * kb + 1 < a.blocks ? __ldg(srow + 2 * kb + 1) : 0.f);
    }
};

// Rows [r0, r0 + nr) of a finished tile, 256 threads: value(r, c) = the sum of activation row r and weight row c of
// the tile. The loops are rolled: this code runs once per tile, with a cold instruction cache, and everything
// unrolled over registers it kept the tensor cores waiting for 4500 cycles.
template <bool FP8, typename F>
__device__ __forceinline__ void ts_store(const TsArgs &a, const TsCursor<TS_DENSE> &t, const TsEpi<FP8> &ep, int r0, int nr, F &&value)
{
    const int tid = threadIdx.x, c = tid & 127;
    const TsSeg &sg = a.seg[t.which];
    float *y = sg.y + (size_t)t.tt * a.n * sg.ldy + t.rt * 128 + c;
    const bool live = t.rt * 128 + c < sg.R;              // (rows of a ragged last tile beyond R do not exist)
#pragma unroll 2
    for (int r = r0 + (tid >> 7); r < r0 + nr; r += 2) {
        const float inv = FP8 ? __shfl_sync(0xffffffffu, r < 32 ? ep.inv0 : ep.inv1, r & 31) : 1.0f;
        const float v = value(r, c);
        if (live) y[(size_t)r * sg.ldy] = FP8 ? v * inv : v;
    }
    __syncwarp();
}

// Projections: the 256 epilogue threads after a CTA's share kb0 .. kb1 of a tile. acc[i]: this thread's sums of weight row `row`. A
// tile of at most 32 rows (`small`): both groups of warps hold rows 0 .. 31, each the sums of its own units;
// otherwise group eg holds rows 32 eg .. The sums go through shared memory (exch: [32][128]), 32 rows at a time; a
// tile shared with other CTAs is put together by the one that finishes last.
__device__ __forceinline__ void ts_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// A CTA's partial results of a tile, `units` of it, are written: true (for all 256 threads) if they were the tile's last.
__device__ __forceinline__ bool ts_last(const TsArgs &a, int tile, int units, int *s_last)
{
    __threadfence();
    ts_bar();
    if (threadIdx.x == 0) {
        const int done = atomicAdd(a.cnt + tile, units) + units;
        *s_last = done == a.KB;
        if (done == a.KB) a.cnt[tile] = 0;
    }
    ts_bar();
    if (!*s_last) return false;
    __threadfence();
    return true;
}
template <bool FP8>
__device__ __forceinline__ void ts_finish(const TsArgs &a, const TsCursor<TS_DENSE> &t, const TsEpi<FP8> &ep, float (&acc)[TS_EN], int tile, bool first,
                                          int kb0, int kb1, long long U, bool small, int eg, int row, float *exch, int *s_last)
{
    const bool whole = kb0 == 0 && kb1 == a.KB;
    auto put = [&](int np, bool add) {
#pragma unroll
        for (int g = 0; g < TS_EN; g += 8)
            if (g < np) {
#pragma unroll
                for (int i = g; i < g + 8; i++) exch[i * 128 + row] = add ? __fadd_rn(acc[i], exch[i * 128 + row]) : acc[i];
            }
        __syncwarp();
    };
    float *pr = a.part + ((size_t)blockIdx.x * 2 + (first ? 0 : 1)) * (TS_N * 128);
    for (int r0 = 0; r0 < t.np; r0 += TS_EN) {
        const int nr = t.np - r0 < TS_EN ? t.np - r0 : TS_EN;
        if (r0) ts_bar();                                     // (the first time the barrier before this function did it)
        if (small) {
            if (eg) put(nr, false);
            ts_bar();
            if (!eg) put(nr, true);
        } else if (eg == (r0 != 0)) put(nr, false);
        ts_bar();
        if (whole) ts_store<FP8>(a, t, ep, r0, nr, [&](int r, int c) { return exch[(r - r0) * 128 + c]; });
        else
            for (int i = threadIdx.x * 4; i < nr * 128; i += 1024)
                __stcg(reinterpret_cast<float4 *>(pr + r0 * 128 + i), *reinterpret_cast<const float4 *>(exch + i));
    }
    if (whole) return;
    if (!ts_last(a, tile, kb1 - kb0, s_last)) return;
    const long long G = gridDim.x, ub = (long long)tile * a.KB;
    const int c0 = (int)(((ub + 1) * G - 1) / U), c1 = (int)(((ub + a.KB) * G - 1) / U);     // CTAs holding the first / last unit
    const int slot0 = (int)(U * c0 / G / a.KB) == tile ? 0 : 1;     // only the first of them began in an earlier tile
    // The parts are added in order, in 16-byte pieces and TS_PARTS at a time in flight, into the exchange buffer (element by
    // element with one load after the other this took 4 us for 8 rows in five parts, 25 for 64).
    for (int r0 = 0; r0 < t.np; r0 += TS_EN) {
        const int nr = t.np - r0 < TS_EN ? t.np - r0 : TS_EN;
        for (int i = threadIdx.x * 4; i < nr * 128; i += 1024) {
            const float *p0 = a.part + r0 * 128 + i;
            float4 v = __ldcg(reinterpret_cast<const float4 *>(p0 + ((size_t)c0 * 2 + slot0) * (TS_N * 128)));
            for (int k0 = c0 + 1; k0 <= c1; k0 += TS_PARTS) {
                float4 w[TS_PARTS];
#pragma unroll
                for (int k = 0; k < TS_PARTS; k++)               // (a CTA without units has no part)
                    w[k] = k0 + k <= c1 && U * (k0 + k) / G != U * (k0 + k + 1) / G
                               ? __ldcg(reinterpret_cast<const float4 *>(p0 + (size_t)(k0 + k) * 2 * (TS_N * 128))) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int k = 0; k < TS_PARTS; k++) {
                    v.x = __fadd_rn(v.x, w[k].x); v.y = __fadd_rn(v.y, w[k].y); v.z = __fadd_rn(v.z, w[k].z); v.w = __fadd_rn(v.w, w[k].w);
                }
            }
            *reinterpret_cast<float4 *>(exch + i) = v;
        }
        ts_bar();
        ts_store<FP8>(a, t, ep, r0, nr, [&](int r, int c) { return exch[(r - r0) * 128 + c]; });
        ts_bar();                                             // (the buffer is free again)
    }
}

// True when it is true for all 256 epilogue threads: they go on together or not at all (barriers follow).
__device__ __forceinline__ bool ts_all(bool ok)
{
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"((uint32_t)ok) : "memory");
    return all != 0;
}
__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, uint32_t n)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}

// A CTA's share of the units, tile by tile: f(cursor, tile, first unit, end).
#define TS_WALK(t, ...)                                                                            \
    do {                                                                                           \
        long long u_ = u0;                                                                         \
        TsCursor<MODE> t;                                                                          \
        if (u0 < u1) t.start(a, plan, tile_first);                                                 \
        _Pragma("unroll 1")                                                                        \
        for (int tile = tile_first; u_ < u1 && ok; tile++) {                                       \
            const int kb0 = (int)(u_ - (long long)tile * KB);                                      \
            const int kb1 = u1 - u_ < KB - kb0 ? kb0 + (int)(u1 - u_) : KB;                        \
            __VA_ARGS__                                                                            \
            u_ += kb1 - kb0;                                                                       \
            if (u_ < u1) t.next(a, plan);                                                          \
        }                                                                                          \
    } while (0)

__global__ void __launch_bounds__(TS_FP8_THREADS, 1) tc_stream_fp8_kernel(const __grid_constant__ TsMaps maps, const TsArgs a)
{
    constexpr int MODE = TS_DENSE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + (-smem_u32(smem_raw) & 1023u);      // (stays a shared-memory address: through an integer it becomes a generic one)
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int WS = a.stages, KB = a.KB, XB = a.x_stage, XS = a.xs;
    uint8_t *wst = smem;                                                   // [WS][32 KB]
    uint8_t *xst = wst + (size_t)WS * TS_UNIT_BYTES;                       // [XS][XB]
    float *exch = reinterpret_cast<float *>(xst + (size_t)XS * XB);        // 16 KB
    uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(exch) + TS_EXCH);
    // c_full: a unit's codes are converted (four warps), in one of two places of tensor memory
    uint64_t *w_full = bars, *w_empty = w_full + TS_MAX_STAGES, *x_full = w_empty + TS_MAX_STAGES, *x_empty = x_full + TS_MAX_XS;
    uint64_t *c_full = x_empty + TS_MAX_XS, *c_empty = c_full + 2, *acc_full = c_empty + 2, *acc_empty = acc_full + 2, *drained = acc_empty + 2;
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;

    pdl_trigger();
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < TS_MAX_STAGES; i++) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 4); }
#pragma unroll 1
        for (int i = 0; i < TS_MAX_XS; i++) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 2); }
        for (int i = 0; i < 2; i++) {
            mbar_init(&c_full[i], 4); mbar_init(&c_empty[i], 2);
            mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); mbar_init(&drained[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 18) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    // A projection's weights and their shares depend on nothing in front: they are under way while the kernel before this one
    // runs, and only the warps that read its results (the terms) or write (sums) wait.
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const TsPlan plan{};
    const long long U = (long long)a.tiles * KB;
    const long long u0 = U * blockIdx.x / gridDim.x, u1 = U * (blockIdx.x + 1) / gridDim.x;
    const int tile_first = (int)(u0 / KB);
    bool ok = true;

    if (warp == 16) {
        // ------------------------------------------------------------------- weights ----
        if (elect_one()) {
            int s = 0, ph = 1, issued = 0;                    // ph: parity that the stage's `empty` must have passed
            TS_WALK(t, {
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++) {
                    if (issued >= WS && !(ok = mbar_wait(&w_empty[s], (uint32_t)ph, a.err, 31))) break;
                    mbar_expect_tx(&w_full[s], TS_UNIT_BYTES);
                    uint8_t *dst = wst + (size_t)s * TS_UNIT_BYTES;
                    tma_load_3d(dst, &maps.w[t.which], 0, t.rt * 128, kb * 2, &w_full[s]);
                    issued++;
                    if (++s == WS) { s = 0; ph ^= 1; }
                }
            });
            if (!ok)                                          // copies in flight must land before shared memory goes away
#pragma unroll 1
                for (int j = issued - 1; j >= 0 && j >= issued - WS; j--) mbar_wait(&w_full[j % WS], (uint32_t)(j / WS) & 1, a.err, 33);
        }
        __syncwarp();
    } else if (warp == 17) {
        // ---------------------------------------------------------- activation terms ----
        pdl_wait();
        if (elect_one()) {
            int s = 0, ph = 1, issued = 0;
            TS_WALK(t, {
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++) {
                    if (issued >= XS && !(ok = mbar_wait(&x_empty[s], (uint32_t)ph, a.err, 32))) break;
                    mbar_expect_tx(&x_full[s], (uint32_t)(8 * t.n * 128));
                    tma_load_4d(xst + (size_t)s * XB, &maps.x[t.n / 8 - 1], 0, t.row0, 0, kb * 4, &x_full[s]);
                    issued++;
                    if (++s == XS) { s = 0; ph ^= 1; }
                }
            });
            if (!ok)
#pragma unroll 1
                for (int j = issued - 1; j >= 0 && j >= issued - XS; j--) mbar_wait(&x_full[j % XS], (uint32_t)(j / XS) & 1, a.err, 33);
        }
        __syncwarp();
    } else if (warp >= 18) {
        // ----------------------------------------------------------------------- MMA ----
        if (elect_one()) {
            // Each warp has an accumulator of its own. Up to 32 rows a unit's two blocks lie side by side in one and the
            // warps take units in turn; beyond, a unit's first block is the one warp's, the second the other's. Both wait for
            // every unit, so that neither loses count of the barrier's phases.
            const int mine = warp - 18;
            int it = 0, cp = 0, xs = 0, xp = 0, c = 0;        // c: uses of the own accumulator so far
            TS_WALK(t, {
                const uint32_t idesc = tc_idesc(0, 2 * t.n);
                const bool small = t.n <= TS_EN;
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++, it++) {
                    const int s = it & 1;
                    if (!(ok = mbar_wait(&x_full[xs], (uint32_t)xp, a.err, 36) && mbar_wait(&c_full[s], (uint32_t)cp, a.err, 35))) break;
                    if (!small || s == mine) {
                        if (c && !(ok = mbar_wait(&acc_empty[mine], (uint32_t)(c - 1) & 1, a.err, 34))) break;
                        c++;
                        tc_fence_after();
                        const uint32_t xb = smem_u32(xst) + (uint32_t)(xs * XB), ab = tmem + 256u + (uint32_t)s * 128u, d = tmem + (uint32_t)mine * 128u;
                        const int b0 = small ? 0 : mine, b1 = small ? 2 : mine + 1;
                        for (int b = b0; b < b1; b++)
#pragma unroll
                            for (int k = 0; k < 8; k++) {
                                const uint64_t bd = tc_smem_desc(xb + (uint32_t)((b * 2 + (k >> 2)) * 2 * t.n * 128)) + 2 * (k & 3);
                                tc_mma_f16_ts(d + (small ? (uint32_t)b * 64u : 0u), ab + (uint32_t)(b * 64 + k * 8), bd, idesc, k ? 1u : 0u);
                            }
                        tc_commit(&acc_full[mine]);
                        tc_commit(&x_empty[xs]);
                        tc_commit(&c_empty[s]);
                    } else { mbar_arrive(&x_empty[xs]); mbar_arrive(&c_empty[s]); }
                    if (s) cp ^= 1;
                    if (++xs == XS) { xs = 0; xp ^= 1; }
                }
            });
            // nothing of this thread is in flight, and no arrival still to come, when the CTA ends
            tc_commit(&drained[mine]);
            mbar_wait(&drained[mine], 0, a.err, 40);
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ---------------------------------- FP8 codes -> F16 in tensor memory, unit by unit ----
        // Two groups of four warps take the units in turn; a thread converts one row (lane of tensor memory).
        const int group = (warp - 8) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t dst = tmem + ((uint32_t)(quarter * 32) << 16) + 256u + (uint32_t)group * 128u;
        const int units = (int)(u1 - u0), x = r & 7;
        int ws = group % WS, wp = 0, xp = 1;
#pragma unroll 1
        for (int it = group; it < units; it += 2) {
            // In this order: with an odd number of stages the groups take turns at one, and only the unit two before having been
            // multiplied says that the stage's use in between is over (the old phase could be taken for this one).
            if (it >= 2 && !(ok = mbar_wait_all(&c_empty[group], (uint32_t)xp, a.err, 38))) break;
            if (!(ok = mbar_wait_all(&w_full[ws], (uint32_t)wp, a.err, 37))) break;
            tc_fence_after();
            const uint8_t *src = wst + (size_t)ws * TS_UNIT_BYTES + (size_t)r * 128;
#pragma unroll
            for (int half = 0; half < 4; half++) {
                uint32_t f[32];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(src + (half >> 1) * 16384 + ((((half & 1) * 4 + c) ^ x) << 4));
                    f[c * 8 + 0] = e4m3x2_to_f16x2(v.x); f[c * 8 + 1] = e4m3x2_to_f16x2(v.x >> 16);
                    f[c * 8 + 2] = e4m3x2_to_f16x2(v.y); f[c * 8 + 3] = e4m3x2_to_f16x2(v.y >> 16);
                    f[c * 8 + 4] = e4m3x2_to_f16x2(v.z); f[c * 8 + 5] = e4m3x2_to_f16x2(v.z >> 16);
                    f[c * 8 + 6] = e4m3x2_to_f16x2(v.w); f[c * 8 + 7] = e4m3x2_to_f16x2(v.w >> 16);
                }
                tmem_st32(dst + (uint32_t)(half * 32), f);
            }
            // the stage is handed back only here: the loads' values must have arrived, which only their use shows
            // (handed back right after the loads, a row of the next unit's codes was seen once in some 10^8)
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_empty[ws]);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&c_full[group]);
            xp ^= 1;
            ws += 2;
            if (ws >= WS) { ws -= WS; wp ^= 1; }
        }
    } else {
        // ------------------------------------------------- epilogue: scale, sum, finish, store ----
        pdl_wait();
        const int quarter = warp & 3, eg = warp >> 2;
        const int row = quarter * 32 + lane;                         // lane of tensor memory = weight row of the tile
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        int it = 0, c0 = 0, c1 = 0;
        TsCursor<MODE> nx;
        TsEpi<true> ep, ep_next;
        if (u0 < u1) {
            nx.start(a, plan, tile_first);
            ep_next.fetch(a, nx, (int)(u0 - (long long)tile_first * KB), lane);
        }
        long long u = u0;
#pragma unroll 1
        for (int tile = tile_first; u < u1; tile++) {
            const int kb0 = (int)(u - (long long)tile * KB);
            const int kb1 = u1 - u < KB - kb0 ? kb0 + (int)(u1 - u) : KB;
            const TsCursor<MODE> t = nx;
            ep = ep_next;
            u += kb1 - kb0;
            if (u < u1) {
                nx.next(a, plan);
                ep_next.fetch(a, nx, 0, lane);
            }
            const bool small = t.n <= TS_EN;
            const int e0 = small ? 0 : eg * TS_EN;                   // this thread's rows: e0 .. e0 + 31 of the tile
            const int np = t.np - e0 < 0 ? 0 : t.np - e0 < TS_EN ? t.np - e0 : TS_EN;
            float acc[TS_EN];
#pragma unroll
            for (int i = 0; i < TS_EN; i++) acc[i] = 0.f;
            // scale and add one block's products (columns past the rows hold nothing that is stored)
            auto take = [&](uint32_t base, float sc) {
#pragma unroll
                for (int g = 0; g < TS_EN; g += 16) {
                    if (g < np) {
                        uint32_t h[16], m[16];
                        tmem_ld16(base + e0 + g, h);
                        tmem_ld16(base + t.n + e0 + g, m);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            acc[g + i] = fmaf(fmaf(__uint_as_float(m[i]), 1.0f / 2048.0f, __uint_as_float(h[i])), sc, acc[g + i]);
                    }
                }
            };
            // lane i: the scales of unit kb0 + i, fetched 32 units at a time (one unit ahead, the copy into the next unit's registers waited
            // for their whole way from L2)
            float2 sl = ep.s0;
            auto scale_of = [&](int kb) {
                const int i = kb - kb0;
                if (i >= 32 && (i & 31) <= (small ? 1 : 0)) sl = kb - (i & 31) + lane < kb1 ? ep.pair(a, kb - (i & 31) + lane) : make_float2(0.f, 0.f);
                return make_float2(__shfl_sync(0xffffffffu, sl.x, i & 31), __shfl_sync(0xffffffffu, sl.y, i & 31));
            };
            if (small) {
                // (units of the other group's parity are its own)
                const int skip = (it & 1) != eg;
#pragma unroll 1
                for (int kb = kb0 + skip; kb < kb1; kb += 2) {
                    const float2 sc = scale_of(kb);
                    if (!(ok = mbar_wait_all(&acc_full[eg], (uint32_t)(eg ? c1 : c0) & 1, a.err, 39))) break;
                    tc_fence_after();
                    take(lane_addr + (uint32_t)(eg * 128), sc.x);
                    take(lane_addr + (uint32_t)(eg * 128 + 64), sc.y);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_n(&acc_empty[eg], 2);
                    if (eg) c1++; else c0++;
                }
                // the uses of the other accumulator in this tile
                const int n_units = kb1 - kb0, own = (n_units + ((it & 1) == eg)) >> 1;
                if (eg) c0 += n_units - own; else c1 += n_units - own;
                it += n_units;
            } else {
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++) {
                    const float2 sc = scale_of(kb);
                    if (!(ok = mbar_wait_all(&acc_full[0], (uint32_t)c0 & 1, a.err, 39))) break;
                    tc_fence_after();
                    take(lane_addr, sc.x);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[0]);
                    if (!(ok = mbar_wait_all(&acc_full[1], (uint32_t)c1 & 1, a.err, 39))) break;
                    tc_fence_after();
                    take(lane_addr + 128u, sc.y);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[1]);
                    c0++; c1++;
                }
                it += kb1 - kb0;
            }
            if (!(ok = ts_all(ok))) break;
            ts_finish<true>(a, t, ep, acc, tile, tile == tile_first, kb0, kb1, U, small, eg, row, exch, &s_last);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 18) { __syncwarp(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------- FP8 weights past tiles of up to 32 rows: experts, prompts ----
// The kernel above is at its best with one tile of rows per matrix and shares that come out of HBM at the same pace. Experts and
// prompts have many tiles, and what held them back there was (a unit of 128 x 256 weights and 32 rows took 2200 cycles from L2, its
// products 590) the way of an accumulator to the epilogue and back, paid for every unit, and (8 to 64 tokens) CTAs whose equal shares
// took 16 % longer than the average. So here
//   - a tile is 256 rows of W: a step multiplies two 128 x 128 blocks with the same terms, each block's products by a warp of its
//     own into two accumulators in turn (four in tensor memory), converted by four warps and drained by four;
//   - a warp group of the epilogue has 128 rows of W to itself and needs the other group nowhere;
//   - the first 4/5 of the tiles are dealt out evenly, whole and contiguous; the rest is claimed from a counter, a quarter of
//     a tile's columns at a time, so that CTAs end together whatever their pace;
//   - one warp walks the work and tells the others (a ring of items in shared memory).
// A sum has one order wherever its parts are computed: the blocks of a quarter in order from zero, then the quarters. So a row of an
// expert has the same bits wherever its tile lies, which CTAs work on it and what other rows are beside it: on every rank of an
// expert-parallel group (each computes the shared expert's rows itself, in a launch with other experts than its
// peers') and on one GPU, in every batch and in every run.
// Gate/up and down of 288 experts top-8, with the events around them, 2 / 8 / 64 / 333 / 2048 tokens: 67 + 38 / 147 + 84 / 323 + 167 /
// 637 + 299 / 2490 + 1126 us; in the kernel above, which had the experts before, 69 + 43 / 159 + 88 / 394 + 196 / 831 + 389 / 3399 + 1426. Up to
// 64 tokens HBM bounds them (5.9 TB/s at 64); a step of 32 rows takes 1550 cycles from L2, its shared memory traffic (48 KB in,
// 32 KB to the converters, 32 KB of terms read per product) 880, its products 590, at a clock that the power limit holds at 1.5 GHz. Tiles of 16 rows
// for batches of few rows per expert are no faster any more (64 tokens 327 + 168, 150: 480 + 226 against 427 + 208).
//
// Warps: 0-7 epilogue (two groups), 8-15 conversion, 16 weights and items, 17 terms, 18 and 19 MMA.
constexpr int TP_ROWS = TC_TILE_ROWS, TP_RING = 4, TP_MAX_WS = 6, TP_MAX_XS = 4, TP_PARTS = 4;
constexpr int TP_SLAB = TP_ROWS * 128;       // values of one quarter's sums of 128 rows of W
constexpr int TP_DYN = 3;                    // claimed tiles at most, per CTA
struct TpItem {
    int k0, k1;          // steps; k1 = 0: no more work
    int which, rt;       // matrix or expert; 256 rows of W from 256 rt on (gate/up: 128 channels from 128 rt on)
    int row0, np;        // rows of the terms
    int slab, t0;        // -1, or the place of a quarter's sums; projections: first position of the tile
};
// A tile's parts: of about eight steps, four at most; and where part q begins.
__device__ __forceinline__ int tp_parts(int KB) { return min(TP_PARTS, max(1, KB / 8)); }
__device__ __forceinline__ int tp_bound(int q, int KB, int parts) { return q * KB / parts; }

__device__ __forceinline__ void tp_bar(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

// The 128 threads of a group: rows 0 .. np of the finished sums sums[r][128]. iv: lane i has row i's factor, ds: its destination.
template <int MODE>
__device__ __forceinline__ void tp_store(const TsArgs &a, const TpItem &t, const float *sums, int eg, float iv, int ds)
{
    const int tid = threadIdx.x & 127;
    if (MODE == TS_DENSE) {
        const TsSeg &sg = a.seg[t.which];
        const int c = t.rt * 256 + eg * 128 + tid;
        float *y = sg.y + (size_t)t.t0 * sg.ldy + c;
        const bool live = c < sg.R;
#pragma unroll 8
        for (int r = 0; r < t.np; r++) {
            const float inv = __shfl_sync(0xffffffffu, iv, r);
            if (live) y[(size_t)r * sg.ldy] = sums[r * 128 + tid] * inv;
        }
    } else if (MODE == TS_DOWN) {
        const int c = t.rt * 256 + eg * 128 + tid;
        float *y = static_cast<float *>(a.out) + c;
        const bool live = c < a.E;
#pragma unroll 8
        for (int r = 0; r < t.np; r++) {
            const int dst = __shfl_sync(0xffffffffu, ds, r);
            if (live) y[(size_t)dst * a.E] = sums[r * 128 + tid] * a.act_inv;
        }
    } else {
        // weight rows 0..63 hold the gate, 64..127 the up product of the same 64 channels
        const int ch = tid & 63;
        __half *dst = static_cast<__half *>(a.out) + (size_t)t.row0 * a.I + t.rt * 128 + eg * 64 + ch;
#pragma unroll 4
        for (int r = tid >> 6; r < t.np; r += 2) {
            const float inv = __shfl_sync(0xffffffffu, iv, r);
            float gv = sums[r * 128 + ch] * inv, uv = sums[r * 128 + ch + 64] * inv;
            gv = gv > a.limit ? a.limit : gv;
            uv = uv > a.limit ? a.limit : (uv < -a.limit ? -a.limit : uv);
            __half hi, mid;
            split_f16(__fmul_rn(__fmul_rn(gv, sigmoid_near(gv)), uv) * a.act_scale, hi, mid);
            dst[(size_t)r * a.I] = hi;
            dst[((size_t)a.plane + r) * a.I] = mid;
        }
    }
    __syncwarp();
}

template <int MODE>
__global__ void __launch_bounds__(TS_FP8_THREADS, 1) tc_pair_kernel(const __grid_constant__ TsMaps maps, const TsArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + (-smem_u32(smem_raw) & 1023u);      // (stays a shared-memory address: through an integer it becomes a generic one)
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int WS = a.stages, KB = a.KB, XB = a.x_stage, XS = a.xs;
    uint8_t *wst = smem;                                                   // [WS][32 KB]
    uint8_t *xst = wst + (size_t)WS * TS_UNIT_BYTES;                       // [XS][XB]
    float *sums = reinterpret_cast<float *>(xst + (size_t)XS * XB);        // [group][a.n][128]
    uint64_t *bars = reinterpret_cast<uint64_t *>(sums + (size_t)2 * a.n * 128);
    // c_, acc_: [128 rows of W][one of two places]
    uint64_t *w_full = bars, *w_empty = w_full + TP_MAX_WS, *x_full = w_empty + TP_MAX_WS, *x_empty = x_full + TP_MAX_XS;
    uint64_t *c_full = x_empty + TP_MAX_XS, *c_empty = c_full + 4, *acc_full = c_empty + 4, *acc_empty = acc_full + 4;
    uint64_t *r_full = acc_empty + 4, *r_empty = r_full + TP_RING, *drained = r_empty + TP_RING;
    TpItem *ring = reinterpret_cast<TpItem *>(drained + 2);
    int *s_plan = reinterpret_cast<int *>(ring + TP_RING);                 // experts: per slot first token tile [slots + 1], first pair, pairs, expert
    __shared__ uint32_t s_tmem;
    __shared__ int s_last[2];

    pdl_trigger();
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < TP_MAX_WS; i++) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 8); }
#pragma unroll 1
        for (int i = 0; i < TP_MAX_XS; i++) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 2); }
        for (int i = 0; i < 4; i++) { mbar_init(&c_full[i], 4); mbar_init(&c_empty[i], 1); mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
        for (int i = 0; i < TP_RING; i++) { mbar_init(&r_full[i], 1); mbar_init(&r_empty[i], 1 + 2 + 8 + 8); }
        for (int i = 0; i < 2; i++) mbar_init(&drained[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 18) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    pdl_wait();                                                            // (the plan, the terms, the counters)
    int n_tiles = a.tiles;
    TsPlan plan{s_plan, s_plan + a.slots + 1, s_plan + 2 * a.slots + 1, s_plan + 3 * a.slots + 1, 0, a.n};
    if (MODE != TS_DENSE) {
        plan.slots = min(*a.p.n_slots, a.slots);
#pragma unroll 1
        for (int i = threadIdx.x; i < plan.slots; i += blockDim.x) {
            s_plan[i] = a.p.slot_tile0[i]; s_plan[a.slots + 1 + i] = a.p.slot_off[i];
            s_plan[2 * a.slots + 1 + i] = a.p.slot_cnt[i]; s_plan[3 * a.slots + 1 + i] = a.p.slot_expert[i];
        }
        const int tt = a.p.slot_tile0[plan.slots];
        if (threadIdx.x == 0) s_plan[plan.slots] = tt;
        n_tiles = tt * a.RT;
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int G = (int)gridDim.x, parts = tp_parts(KB);
    // whole tiles of each CTA: 4/5 of its share, and no more left to claim than there is room for quarters
    const int most_claimed = TP_DYN * G;
    const int whole = max((int)((long long)n_tiles * 4 / (5 * G)), (n_tiles - most_claimed + G - 1) / G);
    const int claimed = n_tiles - whole * G;                               // the tiles from whole * G on
    bool ok = true;

    if (warp == 16) {
        // ------------------------------------------------------------- items, weights ----
        if (elect_one()) {
            int s = 0, ph = 1, issued = 0, i = 0, next = 0;
#pragma unroll 1
            for (;; i++) {
                TpItem t{};
                int tile = -1, part = -1;
                if (i < whole) tile = (int)blockIdx.x * whole + i;
                else if (next < claimed * parts) {
                    if (i == whole) next = atomicAdd(a.sched, 1);
                    if (next < claimed * parts) { tile = whole * G + next / parts; part = next % parts; }
                }
                if (tile >= 0) {
                    t.k0 = part < 0 ? 0 : tp_bound(part, KB, parts); t.k1 = part < 0 ? KB : tp_bound(part + 1, KB, parts);
                    t.slab = part < 0 ? -1 : next;
                    TsCursor<MODE> c;
                    c.start(a, plan, tile);
                    t.which = c.which; t.rt = c.rt; t.row0 = c.row0; t.np = c.np; t.t0 = MODE == TS_DENSE ? c.tt * a.n : 0;
                }
                const int rs = i % TP_RING;
                if (i >= TP_RING && !(ok = mbar_wait(&r_empty[rs], (uint32_t)(i / TP_RING - 1) & 1, a.err, 47))) break;
                ring[rs] = t;
                mbar_arrive(&r_full[rs]);
                if (tile < 0) break;
                if (part >= 0) next = atomicAdd(a.sched, 1);               // (on its way while this one's weights are)
#pragma unroll 1
                for (int kb = t.k0; kb < t.k1; kb++) {
                    if (issued >= WS && !(ok = mbar_wait(&w_empty[s], (uint32_t)ph, a.err, 31))) break;
                    mbar_expect_tx(&w_full[s], TS_UNIT_BYTES);
                    uint8_t *dst = wst + (size_t)s * TS_UNIT_BYTES;
                    if (MODE == TS_DENSE)       tma_load_3d(dst, &maps.w[t.which], 0, t.rt * 256, kb, &w_full[s]);
                    else if (MODE == TS_GATEUP) tma_load_5d(dst, &maps.w[0], 0, t.rt * 128, 0, kb, t.which, &w_full[s]);
                    else                        tma_load_4d(dst, &maps.w[0], 0, t.rt * 256, kb, t.which, &w_full[s]);
                    issued++;
                    if (++s == WS) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
            }
            if (!ok)                                          // copies in flight must land before shared memory goes away
#pragma unroll 1
                for (int j = issued - 1; j >= 0 && j >= issued - WS; j--) mbar_wait(&w_full[j % WS], (uint32_t)(j / WS) & 1, a.err, 33);
        }
        __syncwarp();
    } else if (warp == 17) {
        // ---------------------------------------------------------- activation terms ----
        if (elect_one()) {
            int s = 0, ph = 1, issued = 0;
#pragma unroll 1
            for (int i = 0;; i++) {
                const int rs = i % TP_RING;
                if (!(ok = mbar_wait(&r_full[rs], (uint32_t)(i / TP_RING) & 1, a.err, 48))) break;
                const int k0 = ring[rs].k0, k1 = ring[rs].k1, row0 = ring[rs].row0, n = (ring[rs].np + 7) & ~7;
                mbar_arrive(&r_empty[rs]);
                if (!k1) break;
#pragma unroll 1
                for (int kb = k0; kb < k1; kb++) {
                    if (issued >= XS && !(ok = mbar_wait(&x_empty[s], (uint32_t)ph, a.err, 32))) break;
                    mbar_expect_tx(&x_full[s], (uint32_t)(4 * n * 128));
                    tma_load_4d(xst + (size_t)s * XB, &maps.x[n / 8 - 1], 0, row0, 0, kb * 2, &x_full[s]);
                    issued++;
                    if (++s == XS) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
            }
            if (!ok)
#pragma unroll 1
                for (int j = issued - 1; j >= 0 && j >= issued - XS; j--) mbar_wait(&x_full[j % XS], (uint32_t)(j / XS) & 1, a.err, 33);
        }
        __syncwarp();
    } else if (warp >= 18) {
        // ----------------------------------------------------------------------- MMA ----
        if (elect_one()) {
            const int m = warp - 18;
            int it = 0, xs = 0, xp = 0;
#pragma unroll 1
            for (int i = 0;; i++) {
                const int rs = i % TP_RING;
                if (!(ok = mbar_wait(&r_full[rs], (uint32_t)(i / TP_RING) & 1, a.err, 48))) break;
                const int steps = ring[rs].k1 - ring[rs].k0, n = (ring[rs].np + 7) & ~7;
                mbar_arrive(&r_empty[rs]);
                if (!steps) break;
                const uint32_t idesc = tc_idesc(0, 2 * n), atom = (uint32_t)(2 * n * 128) >> 4;
#pragma unroll 1
                for (int k = 0; k < steps; k++, it++) {
                    const int b = 2 * m + (it & 1);
                    const uint32_t use = (uint32_t)(it >> 1) & 1;
                    const bool x_in = mbar_test(&x_full[xs], (uint32_t)xp), free = it < 2 || mbar_test(&acc_empty[b], use ^ 1), codes = mbar_test(&c_full[b], use);
                    if (!x_in && !(ok = mbar_wait(&x_full[xs], (uint32_t)xp, a.err, 36))) break;
                    if (!free && !(ok = mbar_wait(&acc_empty[b], use ^ 1, a.err, 34))) break;
                    if (!codes && !(ok = mbar_wait(&c_full[b], use, a.err, 35))) break;
                    tc_fence_after();
                    uint64_t bd = tc_smem_desc(smem_u32(xst) + (uint32_t)(xs * XB));
                    uint32_t ad = tmem + 256u + (uint32_t)(b * 64);
                    const uint32_t d = tmem + (uint32_t)(b * 64);
                    // (a loop: this code runs alone, once per step, and waits for its instructions more than for anything else)
#pragma unroll 1
                    for (int h = 0; h < 2; h++) {
#pragma unroll
                        for (int j = 0; j < 4; j++) tc_mma_f16_ts(d, ad + (uint32_t)(j * 8), bd + 2 * j, idesc, h | j ? 1u : 0u);
                        bd += atom; ad += 32;
                    }
                    tc_commit(&c_empty[b]);
                    tc_commit(&acc_full[b]);
                    tc_commit(&x_empty[xs]);
                    if (++xs == XS) { xs = 0; xp ^= 1; }
                }
                if (!ok) break;
            }
            // nothing of this thread is in flight, and no arrival still to come, when the CTA ends
            tc_commit(&drained[m]);
            mbar_wait(&drained[m], 0, a.err, 40);
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ---------------------------------- FP8 codes -> F16 in tensor memory, step by step ----
        // Four warps have the step's first block, four the second; a thread converts one row (lane of tensor memory).
        const int m = (warp - 8) >> 2, quarter = warp & 3, r = quarter * 32 + lane, x = r & 7;
        const uint32_t dst = tmem + ((uint32_t)(quarter * 32) << 16) + 256u + (uint32_t)m * 128u;
        const int off = MODE == TS_GATEUP ? (r < 64 ? (m * 64 + r) * 128 : 16384 + (m * 64 + r - 64) * 128) : (m * 128 + r) * 128;
        int it = 0, ws = 0, wp = 0;
#pragma unroll 1
        for (int i = 0; ok; i++) {
            const int rs = i % TP_RING;
            if (!(ok = mbar_wait_all(&r_full[rs], (uint32_t)(i / TP_RING) & 1, a.err, 48))) break;
            const int steps = ring[rs].k1 - ring[rs].k0;
            __syncwarp();
            if (lane == 0) mbar_arrive(&r_empty[rs]);
            if (!steps) break;
#pragma unroll 1
            for (int k = 0; k < steps; k++, it++) {
                const int b = 2 * m + (it & 1);
                const uint32_t before = ((uint32_t)(it >> 1) & 1) ^ 1;
                const bool in = mbar_test(&w_full[ws], (uint32_t)wp), free = it < 2 || mbar_test(&c_empty[b], before);
                if (!__all_sync(0xffffffffu, in && free)) {
                    if (!(ok = mbar_wait_all(&w_full[ws], (uint32_t)wp, a.err, 37))) break;
                    if (it >= 2 && !(ok = mbar_wait_all(&c_empty[b], before, a.err, 38))) break;
                }
                tc_fence_after();
                const uint8_t *src = wst + (size_t)ws * TS_UNIT_BYTES + off;
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    uint32_t f[32];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint4 u = *reinterpret_cast<const uint4 *>(src + (((half * 4 + c) ^ x) << 4));
                        f[c * 8 + 0] = e4m3x2_to_f16x2(u.x); f[c * 8 + 1] = e4m3x2_to_f16x2(u.x >> 16);
                        f[c * 8 + 2] = e4m3x2_to_f16x2(u.y); f[c * 8 + 3] = e4m3x2_to_f16x2(u.y >> 16);
                        f[c * 8 + 4] = e4m3x2_to_f16x2(u.z); f[c * 8 + 5] = e4m3x2_to_f16x2(u.z >> 16);
                        f[c * 8 + 6] = e4m3x2_to_f16x2(u.w); f[c * 8 + 7] = e4m3x2_to_f16x2(u.w >> 16);
                    }
                    tmem_st32(dst + (uint32_t)((it & 1) * 64 + half * 32), f);
                }
                // the stage is handed back only here: the loads' values must have arrived, which only their use shows
                // (handed back right after the loads, a row of the next unit's codes was seen once in some 10^8)
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_empty[ws]);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&c_full[b]);
                if (++ws == WS) { ws = 0; wp ^= 1; }
            }
        }
    } else {
        // ------------------------------------------------- epilogue: scale, sum, finish, store ----
        const int eg = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;       // row: lane of tensor memory = weight row of the 128
        const uint32_t acc0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(eg * 128);
        float *mine = sums + (size_t)eg * a.n * 128;
        int it = 0;
#pragma unroll 1
        for (int i = 0; ok; i++) {
            const int rs = i % TP_RING;
            if (!(ok = mbar_wait_all(&r_full[rs], (uint32_t)(i / TP_RING) & 1, a.err, 48))) break;
            const TpItem t = ring[rs];
            __syncwarp();
            if (lane == 0) mbar_arrive(&r_empty[rs]);
            if (!t.k1) break;
            const int n = (t.np + 7) & ~7;
            // scales of this thread's 128 rows (gate/up: of its half of them), row factors or destinations
            const float *srow;
            float iv = 0.f;
            int ds = 0;
            if (MODE == TS_DENSE) {
                const TsSeg &sg = a.seg[t.which];
                srow = sg.S + (size_t)(t.rt * 256 + eg * 128 < sg.R ? t.rt * 2 + eg : t.rt * 2) * sg.scols;
                if (lane < t.np) iv = __ldcg(sg.inv + t.t0 + lane);
            } else if (MODE == TS_GATEUP) {
                srow = reinterpret_cast<const float *>(a.scales + (size_t)t.which * a.scale_stride + (quarter < 2 ? 0 : a.up_off)) + (size_t)t.rt * KB;
                if (lane < t.np) iv = __ldcg(a.xinv + t.row0 + lane);
            } else {
                srow = reinterpret_cast<const float *>(a.scales + (size_t)t.which * a.scale_stride) + (size_t)(t.rt * 256 + eg * 128 < a.E ? t.rt * 2 + eg : t.rt * 2) * KB;
                if (lane < t.np) ds = __ldcg(a.p.pair_dst + t.row0 + lane);
            }
            float acc[TP_ROWS];
#pragma unroll
            for (int j = 0; j < TP_ROWS; j++) acc[j] = 0.f;
            // lane i: the scale of step base + i. (Fetched a step ahead into a register, each scale cost its whole way from L2, 800 cycles
            // of a step's 1870: the copy to the next step's register waits for it.)
            float scales = 0.f;
            int part = 0, end = t.slab < 0 ? tp_bound(1, KB, parts) : t.k1;
#pragma unroll 1
            for (int kb = t.k0; kb < t.k1; kb++, it++) {
                if (((kb - t.k0) & 31) == 0) scales = kb + lane < t.k1 ? __ldg(srow + kb + lane) : 0.f;
                const int b = 2 * eg + (it & 1);
                if (!(ok = mbar_wait_all(&acc_full[b], (uint32_t)(it >> 1) & 1, a.err, 39))) break;
                tc_fence_after();
                const float sc = __shfl_sync(0xffffffffu, scales, (kb - t.k0) & 31);
                const uint32_t d = acc0 + (uint32_t)((it & 1) * 64);
#pragma unroll
                for (int g = 0; g < TP_ROWS; g += 16)
                    if (g < t.np) {
                        uint32_t h[16], md[16];
                        tmem_ld16(d + g, h);
                        tmem_ld16(d + n + g, md);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[g + j] = fmaf(fmaf(__uint_as_float(md[j]), 1.0f / 2048.0f, __uint_as_float(h[j])), sc, acc[g + j]);
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
                if (t.slab < 0 && kb + 1 == end) {
                    // a quarter of a whole tile: on to the others (loads first: one after the other each took its own way there and back)
#pragma unroll
                    for (int g = 0; g < TP_ROWS; g += 16)
                        if (g < t.np) {
                            float *q = mine + g * 128 + row, w[16];
#pragma unroll
                            for (int j = 0; j < 16; j++) w[j] = part && g + j < n ? q[j * 128] : 0.f;
#pragma unroll
                            for (int j = 0; j < 16; j++) {
                                if (g + j < n) q[j * 128] = part ? __fadd_rn(w[j], acc[g + j]) : acc[g + j];
                                acc[g + j] = 0.f;
                            }
                        }
                    part++;
                    end = tp_bound(part + 1, KB, parts);
                }
            }
            // a wait that ran out in one warp ends the group: barriers follow
            uint32_t all;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "=r"(all) : "r"((uint32_t)ok), "r"(eg + 1) : "memory");
            if (!(ok = all != 0)) break;
            if (t.slab >= 0) {
                float *own = a.part + ((size_t)t.slab * 2 + eg) * TP_SLAB + row;
#pragma unroll
                for (int g = 0; g < TP_ROWS; g += 8)
                    if (g < t.np) {
#pragma unroll
                        for (int j = g; j < g + 8; j++) __stcg(own + j * 128, acc[j]);
                    }
                __threadfence();
                tp_bar(eg);
                if ((threadIdx.x & 127) == 0) {
                    int *c = a.cnt + (t.slab / parts) * 2 + eg;
                    s_last[eg] = atomicAdd(c, 1) == parts - 1;
                    if (s_last[eg]) *c = 0;
                }
                tp_bar(eg);
                if (!s_last[eg]) continue;
                __threadfence();
                const float *first = a.part + ((size_t)(t.slab / parts * parts) * 2 + eg) * TP_SLAB;
#pragma unroll 1
                for (int j = (threadIdx.x & 127) * 4; j < t.np * 128; j += 512) {
                    float4 w[TP_PARTS];
#pragma unroll
                    for (int q = 0; q < TP_PARTS; q++) if (q < parts) w[q] = __ldcg(reinterpret_cast<const float4 *>(first + (size_t)q * 2 * TP_SLAB + j));
                    float4 v = w[0];
#pragma unroll
                    for (int q = 1; q < TP_PARTS; q++)
                        if (q < parts) { v.x = __fadd_rn(v.x, w[q].x); v.y = __fadd_rn(v.y, w[q].y); v.z = __fadd_rn(v.z, w[q].z); v.w = __fadd_rn(v.w, w[q].w); }
                    *reinterpret_cast<float4 *>(mine + j) = v;
                }
                tp_bar(eg);
            }
            tp_store<MODE>(a, t, mine, eg, iv, ds);
            tp_bar(eg);                                       // (the sums' place is free again)
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 18) { __syncwarp(); tmem_dealloc(tmem, 512); }
    if (threadIdx.x == 0) {
        // the counter starts at zero again once every CTA has made its last claim
        if (atomicAdd(a.sched + 1, 1) == G - 1) { a.sched[0] = 0; a.sched[1] = 0; }
    }
}

__global__ void __launch_bounds__(TS_BF16_THREADS, 1) tc_stream_bf16_kernel(const __grid_constant__ TsMaps maps, const TsArgs a)
{
    constexpr int MODE = TS_DENSE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + (-smem_u32(smem_raw) & 1023u);      // (stays a shared-memory address: through an integer it becomes a generic one)
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int WS = a.stages, KB = a.KB, SB = TS_BF16_UNIT + a.x_stage;     // stage: weights, then the terms
    float *exch = reinterpret_cast<float *>(smem + (size_t)WS * SB);
    uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<uint8_t *>(exch) + TS_EXCH);
    uint64_t *full = bars, *empty = full + TS_MAX_STAGES, *acc_full = empty + TS_MAX_STAGES, *acc_empty = acc_full + 2, *drained = acc_empty + 2;
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;
    pdl_trigger();
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int i = 0; i < TS_MAX_STAGES; i++) { mbar_init(&full[i], 2); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); mbar_init(&drained[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const TsPlan plan{};
    const long long U = (long long)a.tiles * KB;
    const long long u0 = U * blockIdx.x / gridDim.x, u1 = U * (blockIdx.x + 1) / gridDim.x;
    const int tile_first = (int)(u0 / KB);
    bool ok = true;

    if (warp == 8 || warp == 10) {
        // weights (which wait for nothing in front) and terms: a load takes 150 cycles to issue, so each has a warp
        const bool terms = warp == 10;
        if (terms) pdl_wait();
        if (elect_one()) {
            int s = 0, ph = 1, issued = 0;
            TS_WALK(t, {
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++) {
                    if (issued >= WS && !(ok = mbar_wait(&empty[s], (uint32_t)ph, a.err, 41))) break;
                    uint8_t *dst = smem + (size_t)s * SB;
                    mbar_expect_tx(&full[s], terms ? (uint32_t)(3 * t.n * 128) : (uint32_t)TS_BF16_UNIT);
                    if (terms) tma_load_4d(dst + TS_BF16_UNIT, &maps.x[t.n / 8 - 1], 0, t.row0, 0, kb, &full[s]);
                    else       tma_load_3d(dst, &maps.w[t.which], 0, t.rt * 128, kb, &full[s]);
                    issued++;
                    if (++s == WS) { s = 0; ph ^= 1; }
                }
            });
            if (!ok)
#pragma unroll 1
                for (int j = issued - 1; j >= 0 && j >= issued - WS; j--) mbar_wait(&full[j % WS], (uint32_t)(j / WS) & 1, a.err, 43);
        }
        __syncwarp();
    } else if (warp == 9) {
        if (elect_one()) {
            int s = 0, fp = 0, c = 0;
            TS_WALK(t, {
                const uint32_t idesc = tc_idesc(1, (3 * t.n + 15) & ~15);
#pragma unroll 1
                for (int kb = kb0; kb < kb1; kb++) {
                    const bool fresh = kb == kb0 || kb % TS_SEG_UNITS == 0;
                    if (fresh && c >= 2 && !(ok = mbar_wait(&acc_empty[c & 1], (uint32_t)(c / 2 - 1) & 1, a.err, 44))) break;
                    if (!(ok = mbar_wait(&full[s], (uint32_t)fp, a.err, 45))) break;
                    tc_fence_after();
                    const uint32_t wb = smem_u32(smem) + (uint32_t)(s * SB), xb = wb + TS_BF16_UNIT, d = tmem + (uint32_t)(c & 1) * 256u;
#pragma unroll
                    for (int k = 0; k < 4; k++) tc_mma_f16(d, tc_smem_desc(wb) + 2 * k, tc_smem_desc(xb) + 2 * k, idesc, fresh && k == 0 ? 0u : 1u);
                    tc_commit(&empty[s]);
                    if (kb + 1 == kb1 || (kb + 1) % TS_SEG_UNITS == 0) { tc_commit(&acc_full[c & 1]); c++; }
                    if (++s == WS) { s = 0; fp ^= 1; }
                }
            });
            tc_commit(&drained[0]);
            mbar_wait(&drained[0], 0, a.err, 40);
        }
        __syncwarp();
    } else {
        pdl_wait();
        const int quarter = warp & 3, eg = warp >> 2, e0 = eg * TS_EN, row = quarter * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        const TsEpi<false> ep{};
        int c = 0;
        TS_WALK(t, {
            const int np = t.np - e0 < 0 ? 0 : t.np - e0 < TS_EN ? t.np - e0 : TS_EN;
            float acc[TS_EN];
#pragma unroll
            for (int i = 0; i < TS_EN; i++) acc[i] = 0.f;
#pragma unroll 1
            for (int kb = kb0; kb < kb1; kb = (kb / TS_SEG_UNITS + 1) * TS_SEG_UNITS) {
                if (!(ok = mbar_wait_all(&acc_full[c & 1], (uint32_t)(c >> 1) & 1, a.err, 46))) break;
                tc_fence_after();
                const uint32_t base = lane_addr + (uint32_t)(c & 1) * 256u + (uint32_t)e0;
#pragma unroll
                for (int g = 0; g < TS_EN; g += 16) {
                    if (g < np) {
                        uint32_t h[16], m[16], l[16];
                        tmem_ld16(base + g, h);
                        tmem_ld16(base + t.n + g, m);
                        tmem_ld16(base + 2 * t.n + g, l);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            acc[g + i] = __fadd_rn(acc[g + i], __fadd_rn(__fadd_rn(__uint_as_float(h[i]), __uint_as_float(m[i])), __uint_as_float(l[i])));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[c & 1]);
                c++;
            }
            if (!(ok = ts_all(ok))) break;
            ts_finish<false>(a, t, ep, acc, tile, tile == tile_first, kb0, kb1, U, false, eg, row, exch, &s_last);
        });
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) { __syncwarp(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------- activation terms ----
// Row b of a launch is activation row rows[b] (or b): x' = x, or xw * (x * xinv) for a fused RMSNorm. F16: terms
// of x' 2^e with 2^e chosen per row so that the largest element sits near 2^14, inv = 2^-e. BF16: x' = hi +
// mid + lo exactly (24 bits), no scaling (BF16 has FP32's exponent range).
struct TsSplitIn { const float *x, *xinv, *xw; int ldx; };
struct TsSplit {
    TsSplitIn in[TS_MAX_SEG];
    const int *rows;            // optional: activation row of each output row
    const int *n_rows;          // optional: how many there are (device)
    void *terms;                // [in][term][plane][C]
    float *inv;                 // [in][plane]
    int C, plane;
};

template <bool FP8>
__global__ void __launch_bounds__(512) tc_split_kernel(const TsSplit s)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float wmax[16];
    const int b = blockIdx.x, C = s.C;
    if (s.n_rows && b >= *s.n_rows) return;
    const TsSplitIn &in = s.in[blockIdx.y];
    const float *xinv = in.xinv, *xw = in.xw;
    const int t = s.rows ? s.rows[b] : b;
    const float *xt = in.x + (size_t)t * in.ldx;
    const float rinv = xinv ? xinv[t] : 1.0f;
    auto value = [&](int c) {
        float4 v = *reinterpret_cast<const float4 *>(xt + c);
        if (xinv) {
            v.x = __fmul_rn(v.x, rinv); v.y = __fmul_rn(v.y, rinv); v.z = __fmul_rn(v.z, rinv); v.w = __fmul_rn(v.w, rinv);
            if (xw) {
                const float4 w = *reinterpret_cast<const float4 *>(xw + c);
                v.x = __fmul_rn(w.x, v.x); v.y = __fmul_rn(w.y, v.y); v.z = __fmul_rn(w.z, v.z); v.w = __fmul_rn(w.w, v.w);
            }
        }
        return v;
    };
    if (FP8) {
        float m = 0.f;
#pragma unroll 4
        for (int c = threadIdx.x * 4; c < C; c += 2048) {
            const float4 v = value(c);
            m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
        __syncthreads();
        m = wmax[threadIdx.x & 15];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        int ex = 0;
        if (m > 0.f && m < INFINITY) frexpf(m, &ex);
        const float sc = ldexpf(1.0f, 14 - ex);
        if (threadIdx.x == 0) s.inv[blockIdx.y * s.plane + b] = ldexpf(1.0f, ex - 14);
        __half *hi = static_cast<__half *>(s.terms) + ((size_t)blockIdx.y * 2 * s.plane + b) * C, *mid = hi + (size_t)s.plane * C;
#pragma unroll 4
        for (int c = threadIdx.x * 4; c < C; c += 2048) {
            const float4 v = value(c);
            __align__(8) __half h[4], l[4];
            split_f16(v.x * sc, h[0], l[0]); split_f16(v.y * sc, h[1], l[1]); split_f16(v.z * sc, h[2], l[2]); split_f16(v.w * sc, h[3], l[3]);
            *reinterpret_cast<uint2 *>(hi + c) = *reinterpret_cast<const uint2 *>(h);
            *reinterpret_cast<uint2 *>(mid + c) = *reinterpret_cast<const uint2 *>(l);
        }
    } else {
        __nv_bfloat16 *r0 = static_cast<__nv_bfloat16 *>(s.terms) + ((size_t)blockIdx.y * 3 * s.plane + b) * C;
        __nv_bfloat16 *r1 = r0 + (size_t)s.plane * C, *r2 = r1 + (size_t)s.plane * C;
#pragma unroll 4
        for (int c = threadIdx.x * 4; c < C; c += 2048) {
            const float4 f = value(c);
            const float v[4] = {f.x, f.y, f.z, f.w};
            __align__(8) __nv_bfloat16 h[4], m[4], l[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                h[i] = __float2bfloat16_rn(v[i]);
                const float e1 = v[i] - __bfloat162float(h[i]);              // exact
                m[i] = __float2bfloat16_rn(e1);
                l[i] = __float2bfloat16_rn(e1 - __bfloat162float(m[i]));     // exact
            }
            *reinterpret_cast<uint2 *>(r0 + c) = *reinterpret_cast<const uint2 *>(h);
            *reinterpret_cast<uint2 *>(r1 + c) = *reinterpret_cast<const uint2 *>(m);
            *reinterpret_cast<uint2 *>(r2 + c) = *reinterpret_cast<const uint2 *>(l);
        }
    }
}

// ------------------------------------------------------------------------- host ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// Row-major array of `elt`-byte elements, innermost dimension first; strides in bytes from dimension 1 on. Boxes
// are 128 bytes wide and stored with the 128-byte swizzle; what lies outside the array reads as zero.
bool tc_encode(CUtensorMap *m, const void *base, CUtensorMapDataType dt, int elt, int dims, const cuuint64_t *size,
               const cuuint64_t *stride, const cuuint32_t *box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint32_t box[5] = {(cuuint32_t)(128 / elt), 1, 1, 1, 1};
    const cuuint32_t one[5] = {1, 1, 1, 1, 1};
    for (int i = 1; i < dims; i++) box[i] = box_rows[i - 1];
    return fn(m, dt, (cuuint32_t)dims, const_cast<void *>(base), size, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct TcGemm {
    void *terms = nullptr;          // 16-bit values: [inputs][terms][plane][columns]
    size_t terms_n = 0;             // how many fit
    float *inv = nullptr;           // [inputs][plane]
    float *part = nullptr;          // partial results of the CTAs
    int *cnt = nullptr;             // units done per tile
    int max_c = 0, max_ec = 0, max_t = 0, ctas = 0;
    int *err = nullptr;
    // maps by (pointer, kind, rows, columns, pitch or inputs, box)
    std::map<std::tuple<const void *, int, size_t, size_t, size_t, int>, CUtensorMap> maps;
    std::map<const void *, std::pair<CUtensorMap, CUtensorMap>> experts;         // by slab: gate/up, down
};
constexpr int TS_CNT = 1 << 16;     // tiles of one launch at most (two more words: work claimed, CTAs done)

TcGemm *tc_gemm_create(int max_c, int max_ec, int max_t, int *err)
{
    if (!encode_fn()) return nullptr;
    TcGemm *g = new TcGemm;
    g->max_c = max_c; g->err = err; g->ctas = dev_sms();
    g->max_t = max_t > TS_N ? max_t : TS_N;
    g->max_ec = max_ec;
    // per CTA two partial results of a shared tile, or the quarters of the tiles that are claimed
    const size_t part = (size_t)g->ctas * (2 * TS_N * 128 > TP_DYN * TP_PARTS * 2 * TP_SLAB ? 2 * TS_N * 128 : TP_DYN * TP_PARTS * 2 * TP_SLAB);
    g->terms_n = (size_t)3 * (g->max_t > 2 * TS_N ? g->max_t : 2 * TS_N) * max_c;
    if (cudaMalloc(&g->terms, g->terms_n * 2) != cudaSuccess || cudaMalloc((void **)&g->inv, (size_t)TS_MAX_SEG * g->max_t * 4) != cudaSuccess ||
        cudaMalloc((void **)&g->part, part * 4) != cudaSuccess ||
        cudaMalloc((void **)&g->cnt, (TS_CNT + 2) * 4) != cudaSuccess) {
        cudaGetLastError();
        tc_gemm_free(g);
        return nullptr;
    }
    cudaMemset(g->terms, 0, g->terms_n * 2);
    cudaMemset(g->cnt, 0, (TS_CNT + 2) * 4);
    cudaStreamSynchronize(nullptr);      // the engine's streams do not wait for the default stream
    return g;
}

void tc_gemm_free(TcGemm *g)
{
    if (!g) return;
    if (g->terms) cudaFree(g->terms);
    if (g->inv) cudaFree(g->inv);
    if (g->part) cudaFree(g->part);
    if (g->cnt) cudaFree(g->cnt);
    delete g;
}

// A wait that ran out leaves counts of half-done tiles behind.
void tc_gemm_recover(TcGemm *g, cudaStream_t st) { if (g) cudaMemsetAsync(g->cnt, 0, (TS_CNT + 2) * 4, st); }

// A weight matrix: boxes of 128 rows of two 128-byte pieces of a row (a unit; of one: BF16), piece by piece, or (`pair`) of 256 rows of one.
static const CUtensorMap *w_map(TcGemm *g, const void *base, bool fp8, size_t rows, size_t cols, size_t pitch, bool pair)
{
    const auto key = std::make_tuple(base, (int)fp8 + 2 * (int)pair, rows, cols, pitch, 0);
    auto it = g->maps.find(key);
    if (it == g->maps.end()) {
        CUtensorMap m;
        const int elt = fp8 ? 1 : 2;
        const cuuint64_t size[3] = {(cuuint64_t)(128 / elt), (cuuint64_t)rows, (cuuint64_t)(cols * elt / 128)}, stride[2] = {(cuuint64_t)pitch * elt, 128};
        const cuuint32_t box[2] = {pair ? 256u : 128u, fp8 && !pair ? 2u : 1u};
        if (!tc_encode(&m, base, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, elt, 3, size, stride, box)) return nullptr;
        it = g->maps.emplace(key, m).first;
    }
    return &it->second;
}

// Terms in planes of `plane` rows of C 16-bit values. A box holds `atoms` * 64 columns of n rows: atoms of 64
// columns, in each the rows of the first term, then those of the second. Rows past the last input's plane read as
// zero (a tile's rows are rounded up to 8).
static bool x_maps(TcGemm *g, TsMaps &m, const void *base, bool fp8, size_t plane, size_t C, int inputs, int atoms)
{
    for (int b = 0; b < TS_N / 8; b++) {
        const auto key = std::make_tuple(base, 1000 + 10 * (int)fp8 + atoms, plane, C, (size_t)inputs, b);
        auto it = g->maps.find(key);
        if (it == g->maps.end()) {
            CUtensorMap x;
            const cuuint32_t terms = fp8 ? 2 : 3;
            const cuuint64_t size[4] = {64, (cuuint64_t)plane * ((inputs - 1) * terms + 1), terms, (cuuint64_t)C / 64};
            const cuuint64_t stride[3] = {(cuuint64_t)C * 2, (cuuint64_t)plane * C * 2, 128};
            const cuuint32_t box[3] = {(cuuint32_t)(8 * (b + 1)), terms, (cuuint32_t)atoms};
            if (!tc_encode(&x, base, fp8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 4, size, stride, box)) return false;
            it = g->maps.emplace(key, x).first;
        }
        m.x[b] = it->second;
    }
    return true;
}

// As many stages as fit the shared memory.
static size_t stage_plan(TsArgs &a, bool fp8)
{
    a.x_stage = (fp8 ? 8 : 3) * a.n * 128;                           // (a multiple of 1024 per 64-column atom)
    // A third activation stage in tiles of up to 32 rows: a stage is only refilled when its products are done, and with two the
    // way to L2 and back was part of every unit. The terms of larger tiles would leave
    // the weights too few stages.
    a.xs = a.n <= TS_EN ? TS_MAX_XS : 2;
    const size_t fixed = 1024 + 1024 + TS_EXCH + (fp8 ? (size_t)a.xs * a.x_stage : 0);
    const size_t stage = fp8 ? (size_t)TS_UNIT_BYTES : TS_BF16_UNIT + (size_t)a.x_stage;
    const size_t fit = (227 * 1024 - 512 - fixed) / stage;
    a.stages = (int)(fit < (size_t)TS_MAX_STAGES ? fit : (size_t)TS_MAX_STAGES);
    return fixed + a.stages * stage;
}
// The same for tc_pair_kernel; plan: what the experts' plan takes.
static size_t pair_plan(TsArgs &a, size_t plan)
{
    a.x_stage = 4 * a.n * 128;
    a.xs = a.n <= 16 ? TP_MAX_XS : 3;
    const size_t fixed = 1024 + 1024 + (size_t)2 * a.n * 128 * 4 + plan + (size_t)a.xs * a.x_stage;
    const size_t fit = (227 * 1024 - 512 - fixed) / TS_UNIT_BYTES;
    a.stages = (int)(fit < (size_t)TP_MAX_WS ? fit : (size_t)TP_MAX_WS);
    return fixed + (size_t)a.stages * TS_UNIT_BYTES;
}

template <typename K>
static int launch_stream(K kernel, SmemGrant &grant, cudaStream_t st, const TsMaps &m, const TsArgs &a, size_t smem, int grid, int threads)
{
    if (a.stages < 2 || !dev_opt_in_smem((const void *)kernel, smem, grant)) return -1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    ++g_launches;
    return cudaLaunchKernelEx(&cfg, kernel, m, a) == cudaSuccess ? 0 : -1;
}
// (what a kernel may use is kept by the device, not by one engine's TcGemm: one record per kernel)
static SmemGrant grant_dense, grant_pair, grant_gateup, grant_down, grant_bf16;

bool tc_gemm_takes(const TcGemm *g, const GemvSeg &s, int T)
{
    if (!g || T < 2 || T > g->max_t || s.C > g->max_c || s.R < 16) return false;
    if ((reinterpret_cast<uintptr_t>(s.W) & 15) || (((size_t)s.ldw * (s.dt == DT_FP8 ? 1 : 2)) & 15)) return false;
    if ((reinterpret_cast<uintptr_t>(s.x) & 15) || (s.ldx & 3) || (s.xw && (reinterpret_cast<uintptr_t>(s.xw) & 15))) return false;
    if ((s.R + 127) / 128 * ((T + 31) / 32) > TS_CNT / TS_MAX_SEG) return false;
    if (s.dt == DT_FP8) return s.C % 128 == 0 && s.br == 128 && s.bc == 128 && s.S != nullptr;
    if (s.dt == DT_BF16) return s.C % 64 == 0;
    return false;
}

int tc_gemm_run(TcGemm *g, cudaStream_t st, const GemvSeg *segs, int n, int T)
{
    bool done[GEMV_MAX_SEG] = {};
    for (int first = 0; first < n; first++) {
        if (done[first]) continue;
        // matrices of one format and width go out together, with as many different inputs as the terms buffer takes
        const bool fp8 = segs[first].dt == DT_FP8;
        const int C = segs[first].C, terms = fp8 ? 2 : 3;
        TsMaps m;
        TsArgs a{};
        TsSplit sp{};
        int ins = 0;
        const int plane = T <= TS_N ? TS_N : g->max_t;         // (two layouts only: the maps are kept)
        // FP8: one tile of up to 64 rows, or pairs of 128 rows of W past tiles of 32 (for calls of up to 64 positions those, which wait
        // for the kernel in front before their first load, are the slower ones: batch of 7 3.42 -> 3.83 ms, of 64 7.30 -> 7.59)
        const bool pair = fp8 && T > TS_N;
        const int most = pair ? TP_ROWS : TS_N, wr = pair ? 256 : 128;
        a.T = T; a.n = T < most ? (T + 7) & ~7 : most; a.nt = (T + a.n - 1) / a.n; a.plane = plane; a.KB = pair ? C / 128 : fp8 ? (C + 255) / 256 : C / 64; a.blocks = C / 128;
        for (int i = first; i < n && a.n_seg < TS_MAX_SEG; i++) {
            const GemvSeg &s = segs[i];
            if (done[i] || (s.dt == DT_FP8) != fp8 || s.C != C) continue;
            int k = 0;
            while (k < ins && !(sp.in[k].x == s.x && sp.in[k].xinv == s.xinv && sp.in[k].xw == s.xw && sp.in[k].ldx == s.ldx)) k++;
            if ((size_t)(k + 1) * terms * plane * C > g->terms_n) continue;
            if (k == ins) sp.in[ins++] = TsSplitIn{s.x, s.xinv, s.xw, s.ldx};
            const CUtensorMap *w = w_map(g, s.W, fp8, (size_t)s.R, (size_t)C, (size_t)s.ldw, pair);
            if (!w) return -1;
            m.w[a.n_seg] = *w;
            a.seg[a.n_seg++] = TsSeg{s.S, g->inv + (size_t)k * plane, s.y, s.scols, s.R, s.ldy, a.tiles, k * terms * plane};
            a.tiles += (s.R + wr - 1) / wr * a.nt;
            done[i] = true;
        }
        if (!x_maps(g, m, g->terms, fp8, (size_t)plane, (size_t)C, ins, fp8 ? (pair ? 2 : 4) : 1)) return -1;
        sp.terms = g->terms; sp.inv = g->inv; sp.C = C; sp.plane = plane;
        if (fp8) G5B_LAUNCH_PDL(tc_split_kernel<true>, dim3(T, ins), dim3(512), 0, st, sp);
        else     G5B_LAUNCH_PDL(tc_split_kernel<false>, dim3(T, ins), dim3(512), 0, st, sp);
        a.part = g->part; a.cnt = g->cnt; a.sched = g->cnt + TS_CNT; a.err = g->err;
        if (pair) {
            const size_t smem = pair_plan(a, 0);
            if (launch_stream(tc_pair_kernel<TS_DENSE>, grant_pair, st, m, a, smem, a.tiles < g->ctas ? a.tiles : g->ctas, TS_FP8_THREADS)) return -1;
            continue;
        }
        const size_t smem = stage_plan(a, fp8);
        // a CTA has at least two units of 32 KB: below that its fixed cost outweighs its share
        const long units = (long)a.tiles * a.KB;
        const long shares = units / (fp8 ? 2 : 4);
        const int grid = (int)(shares < 1 ? 1 : shares < g->ctas ? shares : g->ctas);
        if (fp8 ? launch_stream(tc_stream_fp8_kernel, grant_dense, st, m, a, smem, grid, TS_FP8_THREADS)
                : launch_stream(tc_stream_bf16_kernel, grant_bf16, st, m, a, smem, grid, TS_BF16_THREADS)) return -1;
    }
    return 0;
}

// ------------------------------------------------------------------ routed experts ----
bool tc_moe_takes(const TcGemm *g, const MoeShape &s, int T)
{
    if (!g || T < 1 || T > g->max_t || s.E > g->max_ec || s.I > g->max_ec || s.dt != DT_FP8 || s.br != 128 || s.bc != 128 || s.E % 128 || s.I % 128) return false;
    if (!(s.limit > 0.f) || s.limit * s.limit > 60000.f) return false;                  // activations must fit F16
    const int slots = (T * s.K < s.n_local ? T * s.K : s.n_local) + 1;
    return (long)(slots + (T * s.K + T) / tc_tile_rows(T)) * (s.I / 128 > (s.E + 255) / 256 ? s.I / 128 : (s.E + 255) / 256) <= (1 << 24);
}

static const std::pair<CUtensorMap, CUtensorMap> *expert_maps(TcGemm *g, const ExpertSlab &w, const MoeShape &s)
{
    auto it = g->experts.find(w.base);
    if (it == g->experts.end()) {
        std::pair<CUtensorMap, CUtensorMap> m;
        // 128 gate rows, then the up rows of the same channels: one step's two blocks of 64 + 64 rows
        const cuuint64_t gs[5] = {128, (cuuint64_t)s.I, 2, (cuuint64_t)s.E / 128, (cuuint64_t)w.count}, gt[4] = {(cuuint64_t)s.E, w.mat, 128, w.stride};
        const cuuint32_t gb[4] = {128, 2, 1, 1};
        const cuuint64_t ds[4] = {128, (cuuint64_t)s.E, (cuuint64_t)s.I / 128, (cuuint64_t)w.count}, dt[3] = {(cuuint64_t)s.I, 128, w.stride};
        const cuuint32_t db[3] = {256, 1, 1};
        if (!tc_encode(&m.first, w.base, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 5, gs, gt, gb) ||
            !tc_encode(&m.second, w.base + 2 * w.mat, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, 4, ds, dt, db)) return nullptr;
        it = g->experts.emplace(w.base, m).first;
    }
    return &it->second;
}

int tc_moe_run(TcGemm *g, cudaStream_t st, float *contrib, void *act, void *xterms, float *xinv, const float *x, int ldx,
               const ExpertSlab &w, const MoePlan &p, int T, const MoeShape &s, cudaEvent_t between)
{
    const std::pair<CUtensorMap, CUtensorMap> *em = expert_maps(g, w, s);
    if (!em) return -1;
    const int P = p.max_pairs, pairs = T * s.K + T;
    TsSplit sp{};
    sp.in[0] = TsSplitIn{x, nullptr, nullptr, ldx};
    sp.rows = p.pair_tok; sp.n_rows = p.n_pairs; sp.terms = xterms; sp.inv = xinv; sp.C = s.E; sp.plane = P;
    G5B_LAUNCH_PDL(tc_split_kernel<true>, dim3(pairs), dim3(512), 0, st, sp);
    TsMaps m;
    TsArgs a{};
    a.T = T; a.n = tc_tile_rows(T); a.plane = P; a.p = p; a.E = s.E; a.I = s.I; a.xinv = xinv; a.limit = s.limit; a.act_scale = act_term_scale(s.limit); a.act_inv = 1.0f / a.act_scale;
    a.slots = (T * s.K < s.n_local ? T * s.K : s.n_local) + 1;
    a.part = g->part; a.cnt = g->cnt; a.sched = g->cnt + TS_CNT; a.err = g->err;
    const size_t plan_bytes = (size_t)(4 * a.slots + 4) * sizeof(int);
    // gate/up with the clamped SwiGLU
    a.KB = s.E / 128; a.RT = s.I / 128; a.out = act;
    a.scales = w.base + 3 * w.mat; a.scale_stride = w.stride; a.up_off = w.scale_gate;
    m.w[0] = em->first;
    if (!x_maps(g, m, xterms, true, (size_t)P, (size_t)s.E, 1, 2)) return -1;
    size_t smem = pair_plan(a, plan_bytes);
    if (launch_stream(tc_pair_kernel<TS_GATEUP>, grant_gateup, st, m, a, smem, g->ctas, TS_FP8_THREADS)) return -1;
    if (between) cudaEventRecord(between, st);
    // down
    a.KB = s.I / 128; a.RT = (s.E + 255) / 256; a.out = contrib;
    a.scales = w.base + 3 * w.mat + 2 * w.scale_gate;
    m.w[0] = em->second;
    if (!x_maps(g, m, act, true, (size_t)P, (size_t)s.I, 1, 2)) return -1;
    return launch_stream(tc_pair_kernel<TS_DOWN>, grant_down, st, m, a, smem, g->ctas, TS_FP8_THREADS);
}

// ------------------------------------------------------------ instruction-rate probe ----
// What one tcgen05.mma costs when nothing else uses the SM: one thread issues `reps` groups of four
// instructions (the four K steps of a 128-byte swizzle row) on shared-memory tiles that never
// change, M = 128, N as given, rotating over `accs` accumulators; then one commit and a bounded
// wait. out[0] = cycles until the last instruction was issued, out[1] = until all had completed, of
// CTA 0.
__device__ __forceinline__ void tc_mma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__global__ void __launch_bounds__(64) tc_mma_rate_kernel(int N, int reps, int accs, int fp8, long long *out, int *err)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t bar;
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    for (int i = threadIdx.x; i < (16384 + 256 * 128) / 4; i += blockDim.x)       // A: 128 rows x 128 B; B: up to 256 rows x 128 B
        reinterpret_cast<uint32_t *>(base)[i] = fp8 ? 0x38383838u : 0x3c003c00u;      // ones
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_proxy_async();
    __syncthreads();
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = s_tmem;
    if (warp == 1 && elect_one()) {
        const uint32_t idesc = tc_idesc(0, N);                     // format code 0: F16, or E4M3 for the 8-bit kind
        const uint64_t ad = tc_smem_desc(smem_u32(base)), bd = tc_smem_desc(smem_u32(base) + 16384);
        const long long t0 = clock64();
        for (int r = 0; r < reps; r++) {
            const uint32_t d = tm + (uint32_t)((r % accs) * N);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (fp8) tc_mma_f8(d, ad + 2 * k, bd + 2 * k, idesc, (r >= accs || k) ? 1u : 0u);
                else     tc_mma_f16(d, ad + 2 * k, bd + 2 * k, idesc, (r >= accs || k) ? 1u : 0u);
            }
        }
        const long long t1 = clock64();
        tc_commit(&bar);
        const bool ok = mbar_wait(&bar, 0, err, 61);               // bounded; a wait that runs out records code 61
        const long long t2 = clock64();
        if (blockIdx.x == 0 && ok) { out[0] = t1 - t0; out[1] = t2 - t0; }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tm, 512);
}

}  // namespace g5b

// Cycles per tcgen05.mma (M = 128; K = 16 for kind::f16, 32 for kind::f8f6f4) with `ctas` CTAs
// running: cycles[0] until issued, cycles[1] until complete. Measurement aid, no counterpart in
// the reference.
extern "C" int g5b_debug_mma_rate(int n, int fp8, int accs, int ctas, int reps, double *cycles)
{
    using namespace g5b;
    if (n < 16 || n > 256 || (n & 15) || accs < 1 || accs * n > 512 || ctas < 1 || reps < 1) return -1;
    long long *out = nullptr;
    int *err = nullptr;
    if (cudaMalloc((void **)&out, 16) != cudaSuccess || cudaMalloc((void **)&err, 4) != cudaSuccess) { cudaFree(out); return -1; }
    cudaMemset(out, 0, 16); cudaMemset(err, 0, 4);
    const size_t smem = 16384 + 256 * 128 + 1024;
    static SmemGrant grant;
    int rc = -1;
    if (dev_opt_in_smem((const void *)tc_mma_rate_kernel, smem, grant)) {
        tc_mma_rate_kernel<<<ctas, 64, smem>>>(n, reps, accs, fp8, out, err);
        long long h[2] = {0, 0};
        int e = 0;
        if (cudaDeviceSynchronize() == cudaSuccess && cudaMemcpy(h, out, 16, cudaMemcpyDeviceToHost) == cudaSuccess &&
            cudaMemcpy(&e, err, 4, cudaMemcpyDeviceToHost) == cudaSuccess && e == 0) {
            cycles[0] = (double)h[0] / (4.0 * reps);
            cycles[1] = (double)h[1] / (4.0 * reps);
            rc = 0;
        }
    }
    cudaFree(out); cudaFree(err);
    return rc;
}
