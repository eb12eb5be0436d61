// mla.cu - multi-head latent attention over the compressed KV cache, and the DSA indexer that
// chooses which positions a query attends to.
//
// Reference: glm53f_mla, compressed-latent branch (src/core/glm53f_ops.c:828-911) and
// glm53f_dsa_append / glm53f_dsa_select (src/core/glm53f_dsa.c:74-171). The reference's GPU
// backend had neither: it expanded keys and values on the device, attended densely and refused
// sessions past 2051 positions (src/model/glm53f_model.c:337-349). Here the cache holds only the
// kv_lora latent per position (FP32, or BF16 when the engine is told so), kv_b is folded into
// the query (W_k^T q) and into the output (W_v applied once to the weighted latent sum), and the
// indexer runs on the device: pool scoring, an exact top-k by radix selection, and an ascending
// position list that the attention kernels gather through.
//
// Sums that decide indices (pool scores) repeat the reference's order in FP64, so equal inputs
// give bit-equal scores and therefore the same selection, ties included (lower pool wins).
#include "dot_rows.cuh"
#include "f64_tile.cuh"
#include "kernels.h"

namespace g5b {

// Indexer state, three consecutive arrays (src/core/glm53f_dsa.c:44-53).
__device__ __forceinline__ float *st_key(float *s, int ID, int pos) { return s + (size_t)pos * ID; }
__device__ __forceinline__ float *st_gate(float *s, int ID, int cap, int pos) { return s + ((size_t)cap + pos) * ID; }
__device__ __forceinline__ float *st_pool(float *s, int ID, int cap, int pool) { return s + ((size_t)2 * cap + pool) * ID; }

__device__ __forceinline__ float latent_at(const void *latent, int bf16, size_t i)
{
    return bf16 ? bf16_to_f32(static_cast<const uint16_t *>(latent)[i]) : static_cast<const float *>(latent)[i];
}

// Batch of sequences (MlaShape::batch): token t works on sequence t's caches, at position `cached`.
__device__ __forceinline__ int pos_of(const MlaShape &s, int cached, int t) { return s.batch ? cached : cached + t; }
__device__ __forceinline__ const void *seq_latent(const void *latent, const MlaShape &s, int t)
{
    if (!s.batch) return latent;
    return s.latent_bf16 ? static_cast<const void *>(static_cast<const uint16_t *>(latent) + (size_t)t * s.lat_seq)
                         : static_cast<const void *>(static_cast<const float *>(latent) + (size_t)t * s.lat_seq);
}
__device__ __forceinline__ float *seq_idx(float *idx_state, const MlaShape &s, int t)
{
    return s.batch ? idx_state + (size_t)t * s.idx_seq : idx_state;
}

// ------------------------------------------------------------------- append ----
// Per new position: latent = RMSNorm(kv_a x) into the cache; indexer key = LayerNorm(wk x)
// (biased variance, eps 1e-6, FP64) and gate = gate x into the indexer state.
__device__ void dsa_pool_one(float *idx_state, const float *ape, int pool, int i, const MlaShape &s);

// Blocks [0, T) write the latents, [T, 2T) the indexer's keys and gates, [2T, 3T) the RMSNorm factors of q_a's output: all of it waits,
// for memory, for sums over a block, for a root, and the three need nothing from each other (one block after the other did the
// first two: 10.0 us for one position with its inputs from memory, 7.6 so). With one new position, the second block also closes the
// pool that position completes (otherwise dsa_pool_kernel follows).
__global__ void __launch_bounds__(256) mla_store_kernel(
    void *latent, float *idx_state, const float *ct_raw, const float *kv_norm_w, const float *wk_raw,
    const float *gate_raw, const float *k_norm_w, const float *k_norm_b, int cached, MlaShape s,
    const float *q_raw, float *q_inv, int T, const float *ape, int pool_here)
{
    pdl_trigger();
    pdl_wait();
    __shared__ double red[32];
    const int part = blockIdx.x / T, t = blockIdx.x - part * T, pos = pos_of(s, cached, t);
    if (part != 1) {
        const int n = part ? s.q_lora : s.KL;
        const float *row = part ? q_raw + (size_t)t * n : ct_raw + (size_t)t * n;
        double ss = 0.0;
#pragma unroll 8
        for (int i = threadIdx.x; i < n; i += blockDim.x) ss += (double)row[i] * (double)row[i];
        ss = block_sum(ss, red);
        const float inv = (float)rsqrt_newton(ss / (double)n + (double)s.rms_eps);
        if (part) {
            if (threadIdx.x == 0) q_inv[t] = inv;
            return;
        }
        latent = const_cast<void *>(seq_latent(latent, s, t));
#pragma unroll 2
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float v = __fmul_rn(kv_norm_w[i], __fmul_rn(row[i], inv));
            if (s.latent_bf16) static_cast<uint16_t *>(latent)[(size_t)pos * n + i] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
            else               static_cast<float *>(latent)[(size_t)pos * n + i] = v;
        }
        return;
    }
    idx_state = seq_idx(idx_state, s, t);
    const float *raw = wk_raw + (size_t)t * s.ID;
    double sum = 0.0;
    for (int i = threadIdx.x; i < s.ID; i += blockDim.x) sum += (double)raw[i];
    const double mean = block_sum(sum, red) / (double)s.ID;
    double var = 0.0;
    for (int i = threadIdx.x; i < s.ID; i += blockDim.x) { const double d = (double)raw[i] - mean; var += d * d; }
    var = block_sum(var, red) / (double)s.ID;
    const double linv = 1.0 / sqrt(var + 1e-6);
    float *kp = st_key(idx_state, s.ID, pos), *gp = st_gate(idx_state, s.ID, s.cap, pos);
    for (int i = threadIdx.x; i < s.ID; i += blockDim.x) {
        kp[i] = mul_add_unfused((float)(((double)raw[i] - mean) * linv), k_norm_w[i], k_norm_b[i]);
        gp[i] = gate_raw[(size_t)t * s.ID + i];
    }
    if (pool_here >= 0) {                                     // this position completes a pool
        __syncthreads();                                      // its key and gate are written (same block)
        for (int i = threadIdx.x; i < s.ID; i += blockDim.x) dsa_pool_one(idx_state, ape, pool_here, i, s);
    }
}

// Pools closed by this call: per channel, softmax over the pool's (gate + ape) weights its keys.
__device__ void dsa_pool_one(float *idx_state, const float *ape, int pool, int i, const MlaShape &s)
{
    const int KP = s.KP;
    double top = -INFINITY, z = 0.0, acc = 0.0;
    for (int j = 0; j < KP; j++) {
        const double l = (double)st_gate(idx_state, s.ID, s.cap, pool * KP + j)[i] + (double)ape[j * s.ID + i];
        if (l > top) top = l;
    }
    for (int j = 0; j < KP; j++)
        z += exp((double)st_gate(idx_state, s.ID, s.cap, pool * KP + j)[i] + (double)ape[j * s.ID + i] - top);
    for (int j = 0; j < KP; j++) {
        const double p = exp((double)st_gate(idx_state, s.ID, s.cap, pool * KP + j)[i] + (double)ape[j * s.ID + i] - top) / z;
        acc = __dadd_rn(acc, __dmul_rn(p, (double)st_key(idx_state, s.ID, pool * KP + j)[i]));
    }
    st_pool(idx_state, s.ID, s.cap, pool)[i] = (float)acc;
}

__global__ void dsa_pool_kernel(float *idx_state, const float *ape, int pool0, MlaShape s)
{
    const int pool = pool0 + blockIdx.x, i = threadIdx.x;
    if (i >= s.ID) return;
    dsa_pool_one(idx_state, ape, pool, i, s);
}

void mla_store(cudaStream_t st, void *latent, float *idx_state, const float *ct_raw,
               const float *kv_norm_w, const float *wk_raw, const float *gate_raw,
               const float *k_norm_w, const float *k_norm_b, const float *ape, const float *q_raw, float *q_inv,
               int T, int cached, const MlaShape &s)
{
    const int pool0 = cached / s.KP;                                         // pools closed before this call
    const int pool1 = (cached + (s.batch ? 1 : T)) / s.KP;                   // pools closed after this call
    const int pool_here = ((T == 1 || s.batch) && pool1 > pool0) ? pool0 : -1;
    G5B_LAUNCH_PDL(mla_store_kernel, 3 * T, 256, 0, st, latent, idx_state, ct_raw, kv_norm_w, wk_raw, gate_raw,
               k_norm_w, k_norm_b, cached, s, q_raw, q_inv, T, ape, pool_here);
    if (pool1 > pool0 && pool_here < 0)
        G5B_LAUNCH(dsa_pool_kernel, pool1 - pool0, ((s.ID + 31) / 32) * 32, 0, st, idx_state, ape, pool0, s);
}

// ------------------------------------------------------------------- select ----
// score[pool] = (float) sum_h w[h]/sqrt(heads) * relu((q_h . P_pool)/sqrt(dim)), FP64, heads and
// dimensions in ascending order as the reference sums them (glm53f_dsa.c:141-157). A lane owns a
// head's dot products with DSA_POOLS pools; a lane per pool then adds the heads in order.
// Bound by the FP64 pipe, and with few pools per warp by the latency of its chains: both factors therefore become
// doubles once, not for every product, four pools share a chain, and what is not a sum (the weights' products) is
// taken out of the serial part. 8192 pools, 32 heads of 128: 35 us before, 13 now.
constexpr int DSA_WARPS = 8, DSA_POOLS = 4;
__global__ void __launch_bounds__(DSA_WARPS * 32) dsa_score_kernel(
    float *score, const float *idx_state, const float *qidx, const float *wproj, int cached, MlaShape s)
{
    pdl_trigger();
    extern __shared__ __align__(16) double dsa_smem[];
    double *qT = dsa_smem;                                                                   // [ID][IH]
    const int t = blockIdx.y, p = pos_of(s, cached, t);
    idx_state = seq_idx(const_cast<float *>(idx_state), s, t);
    const int np = (p + 1) / s.KP;
    if (np <= s.topk / s.KP || (int)blockIdx.x * DSA_WARPS * DSA_POOLS >= np) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double *mine = qT + (((size_t)s.ID * s.IH + 1) & ~(size_t)1) + (size_t)warp * DSA_POOLS * (s.IH + s.ID);   // [pools][IH]: the heads' terms
    double *pks = mine + (size_t)DSA_POOLS * s.IH;                                           // [ID][pools]: this warp's pooled keys
    const float *q = qidx + (size_t)t * s.IH * s.ID, *wt = wproj + (size_t)t * s.IH;
    for (int e = threadIdx.x; e < s.IH * s.ID; e += blockDim.x) {
        const int h = e % s.IH, i = e / s.IH;
        qT[e] = (double)q[(size_t)h * s.ID + i];
    }
    __syncthreads();
    const float hscale = 1.0f / sqrtf((float)s.IH), dscale = 1.0f / sqrtf((float)s.ID);
    for (int p0 = (blockIdx.x * DSA_WARPS + warp) * DSA_POOLS; p0 < np; p0 += gridDim.x * DSA_WARPS * DSA_POOLS) {
        const int n = min(DSA_POOLS, np - p0);
        const float *pk = idx_state + ((size_t)2 * s.cap + p0) * s.ID;
        for (int i = lane; i < s.ID; i += 32)
#pragma unroll
            for (int j = 0; j < DSA_POOLS; j++) pks[i * DSA_POOLS + j] = j < n ? (double)pk[(size_t)j * s.ID + i] : 0.0;
        __syncwarp();
        for (int h = lane; h < s.IH; h += 32) {
            double d[DSA_POOLS] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
            for (int i = 0; i < s.ID; i++) {
                const double qv = qT[i * s.IH + h];
                const double2 k0 = *reinterpret_cast<const double2 *>(pks + i * DSA_POOLS), k1 = *reinterpret_cast<const double2 *>(pks + i * DSA_POOLS + 2);
                d[0] = fma(qv, k0.x, d[0]); d[1] = fma(qv, k0.y, d[1]); d[2] = fma(qv, k1.x, d[2]); d[3] = fma(qv, k1.y, d[3]);
            }
            const double wh = __dmul_rn((double)wt[h], (double)hscale);
#pragma unroll
            for (int j = 0; j < DSA_POOLS; j++) {
                const double v = __dmul_rn(d[j], (double)dscale);
                mine[j * s.IH + h] = v > 0.0 ? __dmul_rn(wh, v) : 0.0;          // (a head that does not count adds nothing)
            }
        }
        __syncwarp();
        if (lane < n) {
            double acc = 0.0;
#pragma unroll 8
            for (int h = 0; h < s.IH; h++) acc = __dadd_rn(acc, mine[lane * s.IH + h]);
            score[(size_t)t * (s.cap / s.KP + 1) + p0 + lane] = (float)acc;
        }
        __syncwarp();
    }
}

// The same scores, bit for bit, with the FP64 matrix instruction: mma.sync.m8n8k4 on doubles is four fused multiply-adds in ascending
// k (equal in 12800 random sums of 256 products; a test compares both kernels' scores), so a sum over dimensions in steps of
// four is the chain above. A CTA takes all heads (a multiple of 8, up to 32) of one query and 64 pools, a warp 16 of the pools;
// a pooled key becomes a double once, as it is read. 64 queries of 1024 pools: 32 us, 110 before; one query of 8192: the layer
// takes 8 us less.
constexpr int DSM_POOLS = 64, DSM_WARPS = 4, DSM_HEADS = 32;
static size_t dsm_smem(int IH, int ID) 
{
    const size_t keys = (size_t)DSM_POOLS * (ID + 4) * 4, terms = (size_t)DSM_POOLS * (IH + 1) * 8;
    return (size_t)IH * (ID + 4) * 8 + (keys > terms ? keys : terms);
}
static bool dsm_takes(const MlaShape &s) { return s.IH % 8 == 0 && s.IH <= DSM_HEADS && s.ID % 16 == 0 && s.ID <= 256; }
__global__ void __launch_bounds__(DSM_WARPS * 32) dsa_score_tile_kernel(float *score, const float *idx_state, const float *qidx, const float *wproj, int cached, MlaShape s)
{
    pdl_trigger();
    extern __shared__ __align__(16) double dsa_smem[];
    const int t = blockIdx.y, p = pos_of(s, cached, t), QP = s.ID + 4, KP = s.ID + 4, MP = s.IH + 1;
    double *qs = dsa_smem;                                       // [IH][QP]
    float *ks = reinterpret_cast<float *>(qs + (size_t)s.IH * QP);           // [pools][KP]: pooled keys, and in their place
    double *terms = qs + (size_t)s.IH * QP;                      // [pools][MP]: the heads' terms
    idx_state = seq_idx(const_cast<float *>(idx_state), s, t);
    const int np = (p + 1) / s.KP, p0 = blockIdx.x * DSM_POOLS;
    if (np <= s.topk / s.KP || p0 >= np) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const float *pk = idx_state + ((size_t)2 * s.cap + p0) * s.ID;
    const int n = min(DSM_POOLS, np - p0), pieces = s.ID / 4;
    for (int i = tid; i < DSM_POOLS * pieces; i += DSM_WARPS * 32) {
        const int r = i / pieces, c = (i % pieces) * 4;
        if (r < n) cp_async16(ks + r * KP + c, pk + (size_t)r * s.ID + c);
        else       *reinterpret_cast<float4 *>(ks + r * KP + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float *qt = qidx + (size_t)t * s.IH * s.ID, *wt = wproj + (size_t)t * s.IH;
#pragma unroll 8
    for (int i = tid; i < s.IH * pieces; i += DSM_WARPS * 32) {
        const int h = i / pieces, c = (i % pieces) * 4;
        const float4 v = *reinterpret_cast<const float4 *>(qt + (size_t)h * s.ID + c);
        double2 *d = reinterpret_cast<double2 *>(qs + (size_t)h * QP + c);
        d[0] = make_double2((double)v.x, (double)v.y); d[1] = make_double2((double)v.z, (double)v.w);
    }
    cp_async_wait();
    __syncthreads();
    const int MT = s.IH / 8, w0 = warp * 16;
    double acc[DSM_HEADS / 8][2][2] = {};
#pragma unroll 4
    for (int k = 0; k < s.ID; k += 4) {
        const double b0 = (double)ks[(w0 + g) * KP + k + q], b1 = (double)ks[(w0 + 8 + g) * KP + k + q];
#pragma unroll
        for (int m = 0; m < DSM_HEADS / 8; m++)
            if (m < MT) {
                const double av = qs[(size_t)(m * 8 + g) * QP + k + q];
                mma_f64(acc[m][0], av, b0);
                mma_f64(acc[m][1], av, b1);
            }
    }
    __syncthreads();                                             // the keys have been read
    const float hscale = 1.0f / sqrtf((float)s.IH), dscale = 1.0f / sqrtf((float)s.ID);
#pragma unroll
    for (int m = 0; m < DSM_HEADS / 8; m++)
        if (m < MT) {
            const int h = m * 8 + g;
            const double wh = __dmul_rn((double)wt[h], (double)hscale);
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const double v = __dmul_rn(acc[m][j][i], (double)dscale);
                    terms[(w0 + j * 8 + 2 * q + i) * MP + h] = v > 0.0 ? __dmul_rn(wh, v) : 0.0;      // (a head that does not count adds nothing)
                }
        }
    __syncwarp();
    if (lane < 16 && w0 + lane < n) {
        double sum = 0.0;
#pragma unroll 8
        for (int h = 0; h < s.IH; h++) sum = __dadd_rn(sum, terms[(w0 + lane) * MP + h]);
        score[(size_t)t * (s.cap / s.KP + 1) + p0 + w0 + lane] = (float)sum;
    }
}

// Exact top-k of the pool scores (score descending, pool index ascending on ties, the order of
// the reference's qsort comparator, glm53f_dsa.c:111-116), by radix selection on a 64-bit key,
// then an order-preserving compaction: kept pools ascending, each expanded to its positions, then
// the incomplete tail pool.
constexpr int TOPK_THREADS = 1024, TOPK_KEEP = 8;      // scores a thread keeps in registers: 8192 pools, the rest is read again
__device__ __forceinline__ unsigned long long rank_key(float sc, int pool)
{
    if (sc == 0.0f) sc = 0.0f;                                    // -0 and +0 compare equal
    uint32_t b = __float_as_uint(sc);
    b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);               // ascending float order
    return ((unsigned long long)b << 32) | (unsigned long long)(0xffffffffu - (uint32_t)pool);
}

__global__ void __launch_bounds__(TOPK_THREADS) dsa_topk_kernel(int *sel, int *nsel, const float *score,
                                                                int cached, MlaShape s)
{
    pdl_trigger();
    pdl_wait();
    __shared__ int hist[256];
    __shared__ unsigned long long prefix_s;
    __shared__ int want_s, exact_s;
    __shared__ int scan[TOPK_KEEP * (TOPK_THREADS / 32)];
    const int t = blockIdx.x, p = pos_of(s, cached, t), tid = threadIdx.x;
    const int np = (p + 1) / s.KP, keep = s.topk / s.KP;
    int *out = sel + (size_t)t * (s.topk + s.KP);
    if (np <= keep) { if (tid == 0) nsel[t] = -1; return; }
    const float *sc = score + (size_t)t * (s.cap / s.KP + 1);

    float own[TOPK_KEEP];                                          // pool tid + 1024 k in place k
#pragma unroll
    for (int k = 0; k < TOPK_KEEP; k++) own[k] = tid + k * TOPK_THREADS < np ? sc[tid + k * TOPK_THREADS] : 0.f;

    // the keep-th largest key, one byte at a time from the top
    // (most scores share their upper bits: a warp counts equal ones before it touches the histogram. The other digits are spread, and
    // the lanes that still count few: 8192 pools 14.3 us with warps counting everywhere, 12.0 so. It holds when all scores are equal too, where five
    // more digits are one word that every lane adds to: the layer of one query 106.5 us so, 109.8 with warps counting, 112.5 with one vote of a
    // warp on its first lane's digit; 98.4, 100.3 and 100.3 with spread scores. The search ends as
    // soon as the digit's pools are just those still wanted, usually after the score's own four bytes: the other four
    // only tell equal scores apart)
    if (tid == 0) { prefix_s = 0ull; want_s = keep; exact_s = 0; }
    __syncthreads();
    for (int shift = 56; shift >= 0 && !exact_s; shift -= 8) {
        if (tid < 256) hist[tid] = 0;
        __syncthreads();
        const unsigned long long prefix = prefix_s;
        const unsigned long long mask = shift == 56 ? 0ull : (~0ull << (shift + 8));
        auto count = [&](int i, float v) {
            const unsigned long long k = rank_key(v, i);
            const int digit = i < np && (k & mask) == prefix ? (int)((k >> shift) & 0xff) : -1;
            if (shift == 56) {
                const unsigned same = __match_any_sync(0xffffffffu, digit);
                if (digit >= 0 && (tid & 31) == __ffs(same) - 1) atomicAdd(&hist[digit], __popc(same));
                __syncwarp();
            } else if (digit >= 0)
                atomicAdd(&hist[digit], 1);
        };
#pragma unroll
        for (int k = 0; k < TOPK_KEEP; k++)
            if (k * TOPK_THREADS < np) count(tid + k * TOPK_THREADS, own[k]);
        for (int i0 = TOPK_KEEP * TOPK_THREADS; i0 < np; i0 += TOPK_THREADS) count(i0 + tid, i0 + tid < np ? sc[i0 + tid] : 0.f);
        __syncthreads();
        if (tid < 32) {
            // the digit holding the want-th largest key: lane l owns digits 255 - 8l .. 248 - 8l; a warp
            // scan over the lanes' totals, then a walk over the owning lane's eight bins
            int c[8], tot = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) { c[k] = hist[255 - (8 * tid + k)]; tot += c[k]; }
            int incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            const int excl = incl - tot, want = want_s;
            __syncwarp();
            if (excl < want && want <= incl) {
                int w = want - excl, dgt = 255 - 8 * tid;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    if (c[k] >= w) { dgt = 255 - (8 * tid + k); break; }
                    w -= c[k];
                    dgt = 255 - (8 * tid + k) - 1;
                }
                if (dgt < 0) dgt = 0;
                prefix_s = prefix | ((unsigned long long)dgt << shift);
                want_s = w;
                exact_s = hist[dgt] == w;
            }
        }
        __syncthreads();
    }
    const unsigned long long threshold = prefix_s;     // exactly `keep` keys are >= it (keys are distinct)

    // order-preserving compaction over pool index, 8192 pools at a time: pool tid + 1024 k of them is the lane's in place
    // (k, warp); the places' counts are scanned
    constexpr int NW = TOPK_THREADS / 32, PLACES = TOPK_KEEP * NW;
    const int warp = tid >> 5, lane = tid & 31;
    int before = 0;                                                // kept so far
    for (int p0 = 0; p0 < np; p0 += TOPK_KEEP * TOPK_THREADS) {
        unsigned kept[TOPK_KEEP];
#pragma unroll
        for (int k = 0; k < TOPK_KEEP; k++) {
            const int i = p0 + tid + k * TOPK_THREADS;
            if (p0) own[k] = i < np ? sc[i] : 0.f;
            kept[k] = __ballot_sync(0xffffffffu, i < np && rank_key(own[k], i) >= threshold);
            if (lane == 0) scan[k * NW + warp] = __popc(kept[k]);
        }
        __syncthreads();
        if (warp == 0) {
            int c[PLACES / 32], tot = 0;
#pragma unroll
            for (int j = 0; j < PLACES / 32; j++) { c[j] = tot; tot += scan[lane * (PLACES / 32) + j]; }
            int incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
#pragma unroll
            for (int j = 0; j < PLACES / 32; j++) scan[lane * (PLACES / 32) + j] = incl - tot + c[j];
            if (lane == 31) want_s = incl;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TOPK_KEEP; k++) {
            const int i = p0 + tid + k * TOPK_THREADS, at = before + scan[k * NW + warp] + __popc(kept[k] & ((1u << lane) - 1u));
            if (kept[k] >> lane & 1u)
                for (int j = 0; j < s.KP; j++) out[at * s.KP + j] = i * s.KP + j;
        }
        before += want_s;
        __syncthreads();
    }
    const int base = keep * s.KP;
    for (int j = np * s.KP + tid; j <= p; j += TOPK_THREADS) out[base + (j - np * s.KP)] = j;
    if (tid == 0) nsel[t] = base + (p - np * s.KP + 1);
}

bool dsa_score_tile_takes(const MlaShape &s) { return dsm_takes(s); }
int dsa_scores(cudaStream_t st, float *score, const float *idx_state, const float *qidx, const float *wproj, int T, int cached, const MlaShape &s, bool tiled)
{
    const int np_max = (cached + (s.batch ? 1 : T)) / s.KP;
    if (tiled) {
        static SmemGrant grant;
        const size_t smem = dsm_smem(s.IH, s.ID);
        if (!dev_opt_in_smem((const void *)dsa_score_tile_kernel, smem, grant)) return -1;
        G5B_LAUNCH(dsa_score_tile_kernel, dim3((np_max + DSM_POOLS - 1) / DSM_POOLS, T), DSM_WARPS * 32, smem, st, score, idx_state, qidx, wproj, cached, s);
    } else {
        const size_t smem = ((((size_t)s.ID * s.IH + 1) & ~(size_t)1) + (size_t)DSA_WARPS * DSA_POOLS * (s.IH + s.ID)) * sizeof(double);
        static SmemGrant grant;
        if (!dev_opt_in_smem((const void *)dsa_score_kernel, smem, grant)) return -1;     // (many heads of many dimensions)
        const int want = (np_max + DSA_WARPS * DSA_POOLS - 1) / (DSA_WARPS * DSA_POOLS);
        int blocks = (444 + T - 1) / T > 32 ? (444 + T - 1) / T : 32;                        // (three fit an SM; each converts the query's heads first)
        if (blocks > want) blocks = want;
        G5B_LAUNCH(dsa_score_kernel, dim3(blocks, T), DSA_WARPS * 32, smem, st, score, idx_state, qidx, wproj, cached, s);
    }
    return 0;
}

int dsa_select(cudaStream_t st, int *sel, int *nsel, const float *idx_state, const float *qidx,
               const float *wproj, float *score, int T, int cached, const MlaShape &s)
{
    const int np_max = (cached + (s.batch ? 1 : T)) / s.KP;
    if (np_max > s.topk / s.KP && dsa_scores(st, score, idx_state, qidx, wproj, T, cached, s, dsm_takes(s))) return -1;
    G5B_LAUNCH_PDL(dsa_topk_kernel, T, TOPK_THREADS, 0, st, sel, nsel, score, cached, s);
    return 0;
}

// ---------------------------------------------------------------- attention ----
__device__ __forceinline__ double mat_elem(const DMat &m, int r, int c)
{
    if (m.dt == DT_BF16) return (double)bf16_to_f32(static_cast<const uint16_t *>(m.w)[(size_t)r * m.cols + c]);
    if (m.dt == DT_FP8)
        return __dmul_rn((double)e4m3_to_f32(static_cast<const uint8_t *>(m.w)[(size_t)r * m.cols + c]),
                         (double)m.s[(size_t)(r / m.br) * m.scols + c / m.bc]);
    return (double)static_cast<const float *>(m.w)[(size_t)r * m.cols + c];
}

// qa[t][h][c] = sum_i q[t][h][i] * W_k[h][i][c] in FP64, ascending i (matmul_transposed,
// glm53f_ops.c:793-814). A thread owns a latent column.
__global__ void mla_absorb_kernel(const QueryOut out, const float *q, const DMat kv_b, MlaShape s)
{
    const int h = blockIdx.x, t = blockIdx.y;
    const int kvd = s.qn + s.vh;
    const float *qt = q + ((size_t)t * s.H + h) * s.qn;
    for (int c = threadIdx.x; c < s.KL; c += blockDim.x) {
        double acc = 0.0;
        if (kv_b.dt == DT_BF16) {
            const uint16_t *w = static_cast<const uint16_t *>(kv_b.w) + (size_t)h * kvd * s.KL + c;
#pragma unroll 8
            for (int i = 0; i < s.qn; i++) acc = fma((double)qt[i], (double)bf16_to_f32(w[(size_t)i * s.KL]), acc);
        } else {
            for (int i = 0; i < s.qn; i++) acc = __dadd_rn(acc, __dmul_rn((double)qt[i], mat_elem(kv_b, h * kvd + i, c)));
        }
        out.put(t, h, c, acc);
    }
}

// The same sums with the GPU filled: a CTA takes 128 latent columns of one head, its eight row
// groups (32 rows each at qk_nope = 256) accumulate in FP64 and are added in ascending order.
constexpr int AB_COLS = 128, AB_GROUPS = 8;
__global__ void __launch_bounds__(AB_COLS * AB_GROUPS) mla_absorb_split_kernel(const QueryOut out, const float *q, const DMat kv_b, MlaShape s)
{
    __shared__ double part[AB_GROUPS][AB_COLS];
    extern __shared__ double ab_q[];                     // the head's query: converted once, not for every column
    const int h = blockIdx.x, t = blockIdx.y, c = blockIdx.z * AB_COLS + (threadIdx.x % AB_COLS), grp = threadIdx.x / AB_COLS;
    const int kvd = s.qn + s.vh, per = s.qn / AB_GROUPS;
    const float *qt = q + ((size_t)t * s.H + h) * s.qn;
    const uint16_t *w = static_cast<const uint16_t *>(kv_b.w) + ((size_t)h * kvd + (size_t)grp * per) * s.KL + c;
    for (int i = threadIdx.x; i < s.qn; i += AB_COLS * AB_GROUPS) ab_q[i] = (double)qt[i];
    __syncthreads();
    double acc = 0.0;
#pragma unroll 8
    for (int i = 0; i < per; i++) acc = fma(ab_q[grp * per + i], bf16_to_f64(w[(size_t)i * s.KL]), acc);
    part[grp][threadIdx.x % AB_COLS] = acc;
    __syncthreads();
    if (grp == 0) {
        double sum = part[0][threadIdx.x];
#pragma unroll
        for (int g = 1; g < AB_GROUPS; g++) sum += part[g][threadIdx.x];
        out.put(t, h, c, sum);
    }
}

void mla_absorb(cudaStream_t st, double *qa, void *terms, const float *q, const DMat &kv_b, int T, const MlaShape &s)
{
    const QueryOut out{qa, static_cast<__nv_bfloat16 *>(terms), (double)(1.0f / sqrtf((float)s.qn)), s.H, s.KL};
    // Several positions in tiles (64 positions of 64 heads: 230 -> 109 us, the FP64 pipe's own time; 7: 49 -> 42 us).
    if (T > 1 && kv_b.dt == DT_BF16 && s.KL % 8 == 0 && s.qn % F64_K == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(kv_b.w) & 15) == 0) {
        const size_t kvd = (size_t)(s.qn + s.vh);
        const F64Tile f{q, static_cast<const uint16_t *>(kv_b.w), nullptr, (size_t)s.H * s.qn, (size_t)s.KL, 0, (size_t)s.qn, kvd * s.KL, 0, T, s.KL, s.qn, out, nullptr};
        f64_tile<true>(st, f, s.H);
        return;
    }
    if (kv_b.dt == DT_BF16 && s.KL % AB_COLS == 0 && s.qn % (AB_GROUPS * 8) == 0 && s.qn <= 4096) {
        G5B_LAUNCH(mla_absorb_split_kernel, dim3(s.H, T, s.KL / AB_COLS), AB_COLS * AB_GROUPS, (size_t)s.qn * sizeof(double), st, out, q, kv_b, s);
        return;
    }
    G5B_LAUNCH(mla_absorb_kernel, dim3(s.H, T), s.KL >= 512 ? 512 : 128, 0, st, out, q, kv_b, s);
}

// d[t][h][jj] = (qa . c_j) * scale in FP64 for the visible positions (all, or the selection).
constexpr int ATT_WARPS = 8;
__global__ void __launch_bounds__(ATT_WARPS * 32) mla_score_kernel(
    double *dsc, const double *qa, const void *latent, const int *sel, const int *nsel, int cached,
    int stride, MlaShape s)
{
    extern __shared__ double qs[];                            // [KL]
    const int h = blockIdx.y, t = blockIdx.z, p = pos_of(s, cached, t);
    latent = seq_latent(latent, s, t);
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x * ATT_WARPS >= nvis) return;
    for (int i = threadIdx.x; i < s.KL; i += blockDim.x) qs[i] = qa[((size_t)t * s.H + h) * s.KL + i];
    __syncthreads();
    const float scale = 1.0f / sqrtf((float)s.qn);
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;
    for (int jj = blockIdx.x * ATT_WARPS + warp; jj < nvis; jj += gridDim.x * ATT_WARPS) {
        const int j = ns < 0 ? jj : sl[jj];
        double d = 0.0;
        for (int i = lane; i < s.KL; i += 32) d = fma(qs[i], (double)latent_at(latent, s.latent_bf16, (size_t)j * s.KL + i), d);
        d = warp_sum(d);
        if (lane == 0) dsc[((size_t)t * s.H + h) * stride + jj] = d * (double)scale;
    }
}

// The same scores for kv_lora = 512 with four heads per CTA: the absorbed queries of the four
// heads stay in registers (lane l holds elements 2l, 2l+1 of every 64), a latent row is loaded
// once for the four of them, and the four sums cross the warp in six exchanges instead of twenty.
constexpr int SC_HEADS = 4, SC_CHUNK = 64;
// The chunk CTA that finishes a (token, head group) last - a counter, no spinning - also takes the
// softmax statistics of its four heads (max of the unrounded scores, z of the float-rounded ones:
// src/core/glm53f_ops.c:890-903), which saves the launch that did only that.
__global__ void __launch_bounds__(256) mla_score4_kernel(double *dsc, const double *qa, const void *latent, const int *sel,
                                                         const int *nsel, int cached, int stride, MlaShape s,
                                                         double *stats, int *counters, int chunk)
{
    pdl_trigger();
    pdl_wait();
    __shared__ double ptop[8], pz[8];
    __shared__ int is_last;
    const int h0 = blockIdx.y * SC_HEADS, t = blockIdx.z, p = pos_of(s, cached, t);
    latent = seq_latent(latent, s, t);
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const int j0 = blockIdx.x * chunk;                         // chunk = 64 or 256 positions (<= 32 per warp)
    if (j0 >= nvis) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double q[SC_HEADS][16];
#pragma unroll
    for (int hh = 0; hh < SC_HEADS; hh++)
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const double2 v = *reinterpret_cast<const double2 *>(qa + ((size_t)t * s.H + h0 + hh) * s.KL + 64 * k + 2 * lane);
            q[hh][2 * k] = v.x;
            q[hh][2 * k + 1] = v.y;
        }
    const double scale = (double)(1.0f / sqrtf((float)s.qn));
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;
    const int jend = min(j0 + chunk, nvis);
    // this warp's positions are j0 + warp + 8k; their cache rows are looked up first (lane k holds
    // row k), and four positions' latent rows are in flight at a time
    int myrow = 0;
    {
        const int jj = j0 + warp + 8 * lane;
        if (lane < chunk / 8 && jj < jend) myrow = ns < 0 ? jj : sl[jj];
    }
    auto load_row = [&](float (&c)[16], int j) {
        if (s.latent_bf16) {
            const uint32_t *row = reinterpret_cast<const uint32_t *>(static_cast<const uint16_t *>(latent) + (size_t)j * s.KL);
#pragma unroll
            for (int k = 0; k < 8; k++) bf16x2_to_f32(row[32 * k + lane], c[2 * k], c[2 * k + 1]);
        } else {
            const float2 *row = reinterpret_cast<const float2 *>(static_cast<const float *>(latent) + (size_t)j * s.KL);
#pragma unroll
            for (int k = 0; k < 8; k++) { const float2 v = row[32 * k + lane]; c[2 * k] = v.x; c[2 * k + 1] = v.y; }
        }
    };
    auto finish = [&](const float (&c)[16], int jj) {
        double a[SC_HEADS] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double cd = (double)c[k];
#pragma unroll
            for (int hh = 0; hh < SC_HEADS; hh++) a[hh] = fma(q[hh][k], cd, a[hh]);
        }
        // four sums across 32 lanes: halve the values a lane carries, twice, then a plain butterfly
        const bool up16 = lane & 16, up8 = lane & 8;
        const double r0 = (up16 ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, up16 ? a[0] : a[2], 16);
        const double r1 = (up16 ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, up16 ? a[1] : a[3], 16);
        double v = (up8 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, up8 ? r0 : r1, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if ((lane & 7) == 0) {
            const int hh = ((lane >> 4) << 1) | ((lane >> 3) & 1);
            dsc[((size_t)t * s.H + h0 + hh) * stride + jj] = v * scale;
        }
    };
    for (int k = 0; k < chunk / 8; k += 4) {                     // four latent rows in flight per warp
        const int jj0 = j0 + warp + 8 * k, jj1 = jj0 + 8, jj2 = jj0 + 16, jj3 = jj0 + 24;
        if (jj0 >= jend) break;
        const int row0 = __shfl_sync(0xffffffffu, myrow, k), row1 = __shfl_sync(0xffffffffu, myrow, k + 1);
        const int row2 = __shfl_sync(0xffffffffu, myrow, k + 2), row3 = __shfl_sync(0xffffffffu, myrow, k + 3);
        float c0[16], c1[16], c2[16], c3[16];
        load_row(c0, row0);
        if (jj1 < jend) load_row(c1, row1);
        if (jj2 < jend) load_row(c2, row2);
        if (jj3 < jend) load_row(c3, row3);
        finish(c0, jj0);
        if (jj1 < jend) finish(c1, jj1);
        if (jj2 < jend) finish(c2, jj2);
        if (jj3 < jend) finish(c3, jj3);
    }
    // ---- statistics by the last chunk of this (token, head group)
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int *cnt = counters + (size_t)t * gridDim.y + blockIdx.y;
        const int active = (nvis + chunk - 1) / chunk;
        const int prev = atomicAdd(cnt, 1);
        is_last = prev == active - 1;
        if (is_last) *cnt = 0;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const int hh = warp >> 1, half = warp & 1;                 // two warps per head
    const double *d = dsc + ((size_t)t * s.H + h0 + hh) * stride;
    double top = -INFINITY;
    for (int jj = half * 32 + lane; jj < nvis; jj += 64) top = fmax(top, __ldcg(d + jj));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) ptop[warp] = top;
    __syncthreads();
    top = fmax(ptop[2 * hh], ptop[2 * hh + 1]);
    double z = 0.0;
    for (int jj = half * 32 + lane; jj < nvis; jj += 64) z += exp((double)(float)__ldcg(d + jj) - top);
    z = warp_sum(z);
    if (lane == 0) pz[warp] = z;
    __syncthreads();
    if (half == 0 && lane == 0) {
        stats[((size_t)t * s.H + h0 + hh) * 2] = top;
        stats[((size_t)t * s.H + h0 + hh) * 2 + 1] = pz[2 * hh] + pz[2 * hh + 1];
    }
}

// Softmax as the reference takes it (glm53f_ops.c:890-903): max over the unrounded scores, the
// exponent of the score rounded to float, probabilities in FP64; then cb = sum_j p_j c_j with a
// thread per latent column walking the positions in ascending order.
__global__ void __launch_bounds__(512) mla_wsum_kernel(
    float *cb, double *dsc, const void *latent, const int *sel, const int *nsel, int cached,
    int stride, MlaShape s)
{
    __shared__ double red[32];
    __shared__ double zs;
    const int h = blockIdx.x, t = blockIdx.y, p = pos_of(s, cached, t);
    latent = seq_latent(latent, s, t);
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    double *d = dsc + ((size_t)t * s.H + h) * stride;
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;

    double top = -INFINITY;
    for (int jj = threadIdx.x; jj < nvis; jj += blockDim.x) top = fmax(top, d[jj]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = top;
    __syncthreads();
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) top = fmax(top, red[w]);
    __syncthreads();

    double z = 0.0;
    for (int jj = threadIdx.x; jj < nvis; jj += blockDim.x) {
        const double e = exp((double)(float)d[jj] - top);
        d[jj] = e;                                         // keep the numerator
        z += e;
    }
    z = block_sum(z, red);
    if (threadIdx.x == 0) zs = z;
    __syncthreads();
    z = zs;
    for (int jj = threadIdx.x; jj < nvis; jj += blockDim.x) d[jj] = d[jj] / z;
    __syncthreads();
    for (int i = threadIdx.x; i < s.KL; i += blockDim.x) {
        double acc = 0.0;
        for (int jj = 0; jj < nvis; jj++) {
            const int j = ns < 0 ? jj : sl[jj];
            acc = fma(d[jj], (double)latent_at(latent, s.latent_bf16, (size_t)j * s.KL + i), acc);
        }
        cb[((size_t)t * s.H + h) * s.KL + i] = (float)acc;
    }
}

// The same softmax and weighted sum spread over the whole GPU (the kernel above walks all positions
// with one CTA per head: 0.44 ms at 2051 positions). Three small launches:
//   stats   per (head, token): max of the unrounded scores and z = sum exp((double)(float)s - max)
//   chunk   per (32 positions, 8 heads, token): p_j = exp(.) / z, partial sums of p_j c_j in FP64,
//           positions ascending; the eight heads share every latent row they load
//   reduce  per (head, token, column): the chunks' partial sums added in ascending order
// The association of the FP64 sum differs from the reference's single ascending walk by the chunk
// boundaries only; the result is rounded to float once, at the end, like the reference's.
constexpr int WS_CHUNK = 32, WS_HEADS = 8, WS_THREADS = 256;

__global__ void __launch_bounds__(256) mla_softmax_stats_kernel(double *stats, const double *dsc, const int *nsel,
                                                                int cached, int stride, MlaShape s)
{
    __shared__ double red[32];
    const int h = blockIdx.x, t = blockIdx.y, p = pos_of(s, cached, t);
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const double *d = dsc + ((size_t)t * s.H + h) * stride;
    double top = -INFINITY;
    for (int jj = threadIdx.x; jj < nvis; jj += blockDim.x) top = fmax(top, d[jj]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = top;
    __syncthreads();
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) top = fmax(top, red[w]);
    __syncthreads();
    double z = 0.0;
    for (int jj = threadIdx.x; jj < nvis; jj += blockDim.x) z += exp((double)(float)d[jj] - top);
    z = block_sum(z, red);
    if (threadIdx.x == 0) {
        stats[((size_t)t * s.H + h) * 2] = top;
        stats[((size_t)t * s.H + h) * 2 + 1] = z;
    }
}

__global__ void __launch_bounds__(WS_THREADS) mla_wsum_chunk_kernel(
    double *part, const double *dsc, const double *stats, const void *latent, const int *sel, const int *nsel,
    int cached, int stride, int nchunks, MlaShape s)
{
    pdl_trigger();
    pdl_wait();
    __shared__ double pj[WS_HEADS][WS_CHUNK];
    __shared__ int idx[WS_CHUNK];
    const int chunk = blockIdx.x, h0 = blockIdx.y * WS_HEADS, t = blockIdx.z, p = pos_of(s, cached, t);
    latent = seq_latent(latent, s, t);
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const int j0 = chunk * WS_CHUNK;
    const int cnt = min(WS_CHUNK, nvis - j0);
    const int i0 = threadIdx.x, i1 = threadIdx.x + WS_THREADS;         // this thread's two latent columns
    double acc0[WS_HEADS], acc1[WS_HEADS];
#pragma unroll
    for (int q = 0; q < WS_HEADS; q++) { acc0[q] = 0.0; acc1[q] = 0.0; }
    if (cnt > 0) {
        const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;
        for (int k = threadIdx.x; k < WS_HEADS * WS_CHUNK; k += WS_THREADS) {
            const int q = k / WS_CHUNK, jj = k % WS_CHUNK;
            double v = 0.0;
            if (jj < cnt) {
                const size_t hs = (size_t)t * s.H + h0 + q;
                v = exp((double)(float)dsc[hs * stride + j0 + jj] - stats[hs * 2]) / stats[hs * 2 + 1];
            }
            pj[q][jj] = v;
        }
        for (int jj = threadIdx.x; jj < WS_CHUNK; jj += WS_THREADS) idx[jj] = jj < cnt ? (ns < 0 ? j0 + jj : sl[j0 + jj]) : 0;
        __syncthreads();
#pragma unroll 8
        for (int jj = 0; jj < cnt; jj++) {
            const size_t row = (size_t)idx[jj] * s.KL;
            const double c0 = (double)latent_at(latent, s.latent_bf16, row + i0);
            const double c1 = (double)latent_at(latent, s.latent_bf16, row + i1);
#pragma unroll
            for (int q = 0; q < WS_HEADS; q++) {
                const double pv = pj[q][jj];
                acc0[q] = fma(pv, c0, acc0[q]);
                acc1[q] = fma(pv, c1, acc1[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < WS_HEADS; q++) {
        double *dst = part + (((size_t)t * s.H + h0 + q) * nchunks + chunk) * s.KL;
        dst[i0] = acc0[q];
        dst[i1] = acc1[q];
    }
}

__global__ void __launch_bounds__(256) mla_wsum_reduce_kernel(float *cb, const double *part, int nchunks, int used,
                                                              int n, int KL)
{
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;                // (t, h, column)
    if (i >= n) return;
    const int th = i / KL, col = i % KL;
    const double *src = part + (size_t)th * nchunks * KL + col;
    double acc = 0.0;
    for (int c = 0; c < used; c++) acc += src[(size_t)c * KL];
    cb[i] = (float)acc;
}

// ---- the FP64 core for several queries and the FP32 cache: both contractions with the FP64 matrix instruction (f64_tile.cuh).
// A thread or a warp per sum, as above, reads a factor from memory or shared memory for every product or four of them and
// converts it; a tile of 64 heads x 64 positions (or latent columns) converts and reads each once for 64, and the pipe's 64 FMA
// per clock and SM are what is left. Three launches, sums in FP64 throughout, positions ascending:
//   score   d[t][h][j] = (q~ . c_j) * scale
//   prob    p_j = exp((double)(float) d_j - max) / z in place (the reference's softmax, src/core/glm53f_ops.c:890-903)
//   sum     sum_j p_j c_j in stretches of AT_SPAN positions, added in order by mla_wsum_reduce_kernel if there are several
// A prompt of 333: 0.6 ms a layer, 2.1 before.
constexpr int AT_TILE = 64, AT_SPAN = 512, AT_MIN_T = 6;

// visible position jj of the query: a row of the cache
__device__ __forceinline__ int vis_row(const int *sl, int ns, int jj) { return ns < 0 ? jj : sl[jj]; }

__global__ void __launch_bounds__(F64_THREADS, 3) mla_score_tile_kernel(double *dsc, const double *qa, const float *latent, const int *sel, const int *nsel,
                                                                       int cached, int stride, MlaShape s)
{
    __shared__ __align__(16) double sa[AT_TILE][F64_KPITCH], sb[AT_TILE][F64_KPITCH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int h0 = blockIdx.y * AT_TILE, t = blockIdx.z, pos = pos_of(s, cached, t), j0 = blockIdx.x * AT_TILE;
    const int ns = nsel ? nsel[t] : -1, nvis = ns < 0 ? pos + 1 : ns;
    if (j0 >= nvis) return;
    latent = static_cast<const float *>(seq_latent(latent, s, t));
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;
    // eight lanes take 32 columns of a row, 16 rows at a time
    const int lr = tid >> 3, lk = (tid & 7) * 4;
    const double *A = qa + ((size_t)t * s.H + h0 + lr) * s.KL + lk;
    const float *B[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int jj = j0 + lr + 16 * i;
        B[i] = jj < nvis ? latent + (size_t)vis_row(sl, ns, jj) * s.KL + lk : nullptr;
    }
    double2 ra[4][2];
    float4 rb[4];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ra[i][0] = *reinterpret_cast<const double2 *>(A + (size_t)(16 * i) * s.KL + k0);
            ra[i][1] = *reinterpret_cast<const double2 *>(A + (size_t)(16 * i) * s.KL + k0 + 2);
            rb[i] = B[i] ? *reinterpret_cast<const float4 *>(B[i] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    double acc[4][4][2] = {};
    load(0);
    for (int k0 = 0; k0 < s.KL; k0 += F64_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            double2 *da = reinterpret_cast<double2 *>(&sa[lr + 16 * i][lk]), *db = reinterpret_cast<double2 *>(&sb[lr + 16 * i][lk]);
            da[0] = ra[i][0]; da[1] = ra[i][1];
            db[0] = make_double2((double)rb[i].x, (double)rb[i].y); db[1] = make_double2((double)rb[i].z, (double)rb[i].w);
        }
        __syncthreads();
        if (k0 + F64_K < s.KL) load(k0 + F64_K);
#pragma unroll
        for (int k = 0; k < F64_K; k += 4) {
            double av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { av[i] = sa[wm + i * 8 + g][k + q]; bv[i] = sb[wn + i * 8 + g][k + q]; }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f64(acc[i][j], av[i], bv[j]);
        }
    }
    const double scale = (double)(1.0f / sqrtf((float)s.qn));
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int jj = j0 + wn + j * 8 + 2 * q;
            double *d = dsc + ((size_t)t * s.H + h0 + wm + i * 8 + g) * stride + jj;
            if (jj < nvis) d[0] = acc[i][j][0] * scale;
            if (jj + 1 < nvis) d[1] = acc[i][j][1] * scale;
        }
}

// A warp per (query, head); `rows` of them.
__global__ void __launch_bounds__(256) mla_prob_kernel(double *dsc, const int *nsel, int cached, int stride, int rows, MlaShape s)
{
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    const int t = r / s.H, ns = nsel ? nsel[t] : -1, nvis = ns < 0 ? pos_of(s, cached, t) + 1 : ns;
    double *d = dsc + (size_t)r * stride;
    double top = -INFINITY, z = 0.0;
    for (int j = lane; j < nvis; j += 32) top = fmax(top, d[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    for (int j = lane; j < nvis; j += 32) {
        const double e = exp((double)(float)d[j] - top);
        d[j] = e;
        z += e;
    }
    z = warp_sum(z);
    for (int j = lane; j < nvis; j += 32) d[j] = d[j] / z;
}

// 64 heads x 64 latent columns over the positions [AT_SPAN blockIdx.y % spans ..) of a query; one stretch: the sums go to cb.
__global__ void __launch_bounds__(F64_THREADS, 3) mla_sum_tile_kernel(float *cb, double *part, const double *dsc, const float *latent, const int *sel, const int *nsel,
                                                                     int cached, int stride, int spans, MlaShape s)
{
    __shared__ __align__(16) double sa[AT_TILE][F64_KPITCH], sb[F64_K][F64_NPITCH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int n0 = blockIdx.x * AT_TILE, h0 = (int)blockIdx.y / spans * AT_TILE, span = (int)blockIdx.y % spans, t = blockIdx.z, pos = pos_of(s, cached, t);
    const int ns = nsel ? nsel[t] : -1, nvis = ns < 0 ? pos + 1 : ns;
    const int j0 = span * AT_SPAN, j1 = min(nvis, j0 + AT_SPAN);
    latent = static_cast<const float *>(seq_latent(latent, s, t));
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;
    const int lr = tid >> 3, lk = (tid & 7) * 4;                  // probabilities: eight lanes take 32 positions of a head
    const int br = tid >> 4, bc = (tid & 15) * 4;                 // latents: 16 lanes take 64 columns of a position
    const double *A = dsc + ((size_t)t * s.H + h0 + lr) * stride;
    double ra[4][4];
    float4 rb[4];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int jb = k0 + br + 8 * i;
#pragma unroll
            for (int k = 0; k < 4; k++) ra[i][k] = k0 + lk + k < j1 ? A[(size_t)(16 * i) * stride + k0 + lk + k] : 0.0;
            rb[i] = jb < j1 ? *reinterpret_cast<const float4 *>(latent + (size_t)vis_row(sl, ns, jb) * s.KL + n0 + bc) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    double acc[4][4][2] = {};
    if (j0 < j1) load(j0);
    for (int k0 = j0; k0 < j1; k0 += F64_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++) {
            double2 *da = reinterpret_cast<double2 *>(&sa[lr + 16 * i][lk]), *db = reinterpret_cast<double2 *>(&sb[br + 8 * i][bc]);
            da[0] = make_double2(ra[i][0], ra[i][1]); da[1] = make_double2(ra[i][2], ra[i][3]);
            db[0] = make_double2((double)rb[i].x, (double)rb[i].y); db[1] = make_double2((double)rb[i].z, (double)rb[i].w);
        }
        __syncthreads();
        if (k0 + F64_K < j1) load(k0 + F64_K);
#pragma unroll
        for (int k = 0; k < F64_K; k += 4) {
            double av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { av[i] = sa[wm + i * 8 + g][k + q]; bv[i] = sb[k + q][wn + i * 8 + g]; }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_f64(acc[i][j], av[i], bv[j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const size_t th = (size_t)t * s.H + h0 + wm + i * 8 + g;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + wn + j * 8 + 2 * q;
            if (spans == 1) *reinterpret_cast<float2 *>(cb + th * s.KL + n) = make_float2((float)acc[i][j][0], (float)acc[i][j][1]);
            else            *reinterpret_cast<double2 *>(part + (th * spans + span) * s.KL + n) = make_double2(acc[i][j][0], acc[i][j][1]);
        }
    }
}

void mla_attend(cudaStream_t st, float *cb, const double *qa, const void *latent, const int *sel,
                const int *nsel, double *dsc, double *part, double *stats, int *counters, int part_tokens, int T,
                int cached, const MlaShape &s)
{
    const int span = s.batch ? 1 : T;                                      // positions this call adds to a sequence
    const int nvis_max = cached + span < s.topk + s.KP ? cached + span : s.topk + s.KP;
    const int stride = s.topk + s.KP;
    // few queries do not fill the GPU with tiles (layer, us, one head after the other / in tiles: 4 queries at 300 positions 228 / 240, 6 at
    // 64 240 / 226, 3 at 1000 252 / 266, 3 at 2000 304 / 272, 12 at 8000 687 / 408)
    const int spans = (nvis_max + AT_SPAN - 1) / AT_SPAN;
    if ((T >= AT_MIN_T || (T >= 3 && nvis_max >= 1500)) && !s.latent_bf16 && s.H % AT_TILE == 0 && s.KL % AT_TILE == 0 && part && part_tokens > 0) {
        const float *lat = static_cast<const float *>(latent);
        G5B_LAUNCH(mla_score_tile_kernel, dim3((nvis_max + AT_TILE - 1) / AT_TILE, s.H / AT_TILE, T), F64_THREADS, 0, st, dsc, qa, lat, sel, nsel, cached, stride, s);
        G5B_LAUNCH(mla_prob_kernel, (T * s.H + 7) / 8, 256, 0, st, dsc, nsel, cached, stride, T * s.H, s);
        const int most = part_tokens * ((stride + WS_CHUNK - 1) / WS_CHUNK) / spans;      // queries whose stretches fit
        for (int t0 = 0; t0 < T; t0 += spans > 1 ? most : T) {
            const int n = spans > 1 && T - t0 > most ? most : T - t0;
            const size_t d0 = (size_t)t0 * s.H;
            G5B_LAUNCH(mla_sum_tile_kernel, dim3(s.KL / AT_TILE, s.H / AT_TILE * spans, n), F64_THREADS, 0, st, cb + d0 * s.KL, part, dsc + d0 * stride,
                       s.batch ? lat + (size_t)t0 * s.lat_seq : lat, sel ? sel + (size_t)t0 * stride : nullptr, nsel ? nsel + t0 : nullptr, s.batch ? cached : cached + t0, stride, spans, s);
            if (spans > 1) G5B_LAUNCH(mla_wsum_reduce_kernel, (n * s.H * s.KL + 255) / 256, 256, 0, st, cb + d0 * s.KL, part, spans, spans, n * s.H * s.KL, s.KL);
        }
        return;
    }
    int blocks = (nvis_max + ATT_WARPS - 1) / ATT_WARPS;
    if (blocks > 32) blocks = 32;
    const bool fast_score = s.KL == 512 && s.H % SC_HEADS == 0 && stats && counters;
    if (fast_score) {
        // many tokens: fewer, longer CTAs, so that loading the four absorbed queries (16 KB) is a small
        // part of a CTA's work; one token: many short CTAs, for the latency
        const int chunk = T >= 8 ? 4 * SC_CHUNK : SC_CHUNK;
        G5B_LAUNCH_PDL(mla_score4_kernel, dim3((nvis_max + chunk - 1) / chunk, s.H / SC_HEADS, T), 256, 0, st, dsc, qa,
                   latent, sel, nsel, cached, stride, s, stats, counters, chunk);
    }
    else
        G5B_LAUNCH(mla_score_kernel, dim3(blocks, s.H, T), ATT_WARPS * 32, (size_t)s.KL * sizeof(double), st, dsc, qa,
                   latent, sel, nsel, cached, stride, s);
    if (s.KL != 2 * WS_THREADS || s.H % WS_HEADS != 0 || !part || part_tokens < 1) {
        G5B_LAUNCH(mla_wsum_kernel, dim3(s.H, T), s.KL >= 512 ? 512 : 128, 0, st, cb, dsc, latent, sel, nsel, cached,
                   stride, s);
        return;
    }
    const int nchunks = (stride + WS_CHUNK - 1) / WS_CHUNK;             // the partial buffer is laid out for this many
    if (!fast_score) G5B_LAUNCH(mla_softmax_stats_kernel, dim3(s.H, T), 256, 0, st, stats, dsc, nsel, cached, stride, s);
    for (int t0 = 0; t0 < T; t0 += part_tokens) {
        const int n = T - t0 < part_tokens ? T - t0 : part_tokens;
        const int reach = s.batch ? cached + 1 : cached + t0 + n;
        const void *lat0 = latent;                                 // the kernel's token 0 is sequence t0 of a batch
        if (s.batch)
            lat0 = s.latent_bf16 ? static_cast<const void *>(static_cast<const uint16_t *>(latent) + (size_t)t0 * s.lat_seq)
                                 : static_cast<const void *>(static_cast<const float *>(latent) + (size_t)t0 * s.lat_seq);
        const int used = (((reach < stride) ? reach : stride) + WS_CHUNK - 1) / WS_CHUNK;
        G5B_LAUNCH_PDL(mla_wsum_chunk_kernel, dim3(used, s.H / WS_HEADS, n), WS_THREADS, 0, st, part,
                   dsc + (size_t)t0 * s.H * stride, stats + (size_t)t0 * s.H * 2, lat0,
                   sel ? sel + (size_t)t0 * stride : nullptr, nsel ? nsel + t0 : nullptr, s.batch ? cached : cached + t0, stride, nchunks,
                   s);
        // chunks beyond `used` were not written: reduce over the used ones only
        G5B_LAUNCH_PDL(mla_wsum_reduce_kernel, dim3((n * s.H * s.KL + 255) / 256), 256, 0, st,
                   cb + (size_t)t0 * s.H * s.KL, part, nchunks, used, n * s.H * s.KL, s.KL);
    }
}

// ------------------------------------------------- attention core on the tensor cores ----
// With the latent cache in BF16 the two contractions of the attention core - scores q~ . c_j over
// the 512 latent columns, and the weighted sum of the latent rows - are small GEMMs whose one
// operand (the cache) is already exact in BF16. The other operand is split into three BF16 terms
// (24 significant bits: the absorbed query after the 1/sqrt(d) scaling, the probabilities), so the
// products are exact and only the FP32 accumulation of mma.sync rounds (about 4e-7 relative; the
// reference, src/core/glm53f_ops.c:879-911, accumulates in FP64 and rounds the score to float).
// A CTA takes FL_HEADS heads of one query and a stretch of its visible positions, FL_POS of them at a time: it gathers the latent
// rows into shared memory (the DSA selection is a list of row numbers), multiplies scores, takes exponentials, multiplies the weighted
// sum and adds it to its own, in registers. Those additions are Kahan's: what one rounds away is where the next chunk's products begin
// to be added up, so that as many chunks as there are lose no more than two roundings (plain FP32 additions let go of everything that is small
// beside the sum: 1800 positions of 2^-22 behind one of 256 were 2e-6 of the result). It is kept to eight bits, two to a register: sums and whole
// remainders together do not fit the registers of two CTAs per SM. (64 queries of 2051 positions, the layer: 557 us with plain
// additions, 575 so, 604 with remainders added up by Knuth's two-sum beside the sums, 618 before the loops were cut down to the registers.)
// A query's reference R for the exponents is its first chunk's maximum, and rises by a multiple of ln 2 when a later
// one exceeds it by 16 (the reference takes the maximum of all scores first; e^16 more is nothing to a float's range): so the sums
// are hardly ever rescaled, and then without rounding. Few queries are split
// into stretches, which a second kernel puts together.
// Bound by mma.sync (1024 products per clock and SM, measured: a quarter of the tcgen05 rate) and nearly as much by shared memory: per chunk of
// 48 positions x 16 heads 2300 cycles of products, 2350 of ldmatrix and the rest. A CTA is a chain of phases, so two of them share an SM: rows are kept
// without padding (16-byte pieces of row r at place piece ^ (r & 7), which ldmatrix reads without conflicts) and probabilities
// take the place of the scores' parts, 113 KB in all. Scores are dealt out as two groups of positions x four quarters of the columns: all
// warps at all 512 columns of eight positions each read the query's 48 KB eight times over.
// Measured, with the reduction: 64 queries of 2051 positions 437 -> 256 us (274 with the remainders), a prompt of 2048 6.9 -> 3.2 ms a layer (a chunk of 64
// positions per CTA, its sums in memory, before); one query 15.6 -> 19.5. Against the FP64 core on the same cache 1.3e-6 -> 3.5e-7: fewer and better ordered
// truncations of the tensor cores' sums.
constexpr int FL_POS = 48, FL_HEADS = 16, FL_KL = 512, FL_PPITCH = FL_POS + 8, FL_SPITCH = FL_POS + 8;
constexpr int FL_THREADS = 256, FL_KQ = 4;
constexpr size_t FL_SMEM = (size_t)3 * FL_HEADS * FL_KL * 2 + (size_t)FL_POS * FL_KL * 2 + (size_t)FL_KQ * FL_HEADS * FL_SPITCH * 4;
static_assert((size_t)3 * FL_HEADS * FL_PPITCH * 2 <= (size_t)FL_KQ * FL_HEADS * FL_SPITCH * 4, "probabilities fit where the scores' parts were");
// element (row, 8 * piece) of rows of FL_KL 16-bit values
__device__ __forceinline__ int fl_at(int row, int piece) { return row * FL_KL + ((piece ^ (row & 7)) << 3); }

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], const void *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x and y cut off to BF16
__device__ __forceinline__ __nv_bfloat162 upper_halves(float x, float y)
{
    const uint32_t v = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    return *reinterpret_cast<const __nv_bfloat162 *>(&v);
}
// part: [T][H][splits][KL] floats (unnormalised rows of a stretch), cstat: [T][H][splits][2] doubles (its reference, its sum of exponentials);
// one stretch: the finished rows go to cb. span: chunks per stretch.
__global__ void __launch_bounds__(FL_THREADS, 2) mla_flash_kernel(float *cb, float *part, double *cstat, const __nv_bfloat16 *qterms, const void *latent,
                                                               const int *sel, const int *nsel, int cached, int splits, int span, MlaShape s)
{
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) uint8_t fl_smem[];
    __shared__ float s_scale[FL_HEADS];
    __shared__ double s_z[FL_HEADS];
    __shared__ int s_rows[FL_POS];                                 // cache rows of the next chunk to fetch
    __nv_bfloat16 *qs = reinterpret_cast<__nv_bfloat16 *>(fl_smem);                          // [3][16][512]
    __nv_bfloat16 *cs = qs + 3 * FL_HEADS * FL_KL;                                          // [48][512]
    float *ss = reinterpret_cast<float *>(cs + FL_POS * FL_KL);                             // [4][16][FL_SPITCH], then
    __nv_bfloat16 *ps = reinterpret_cast<__nv_bfloat16 *>(ss);                              // [3][16][FL_PPITCH]
    const int split = blockIdx.x, h0 = blockIdx.y * FL_HEADS, t = blockIdx.z, p = pos_of(s, cached, t);
    const uint16_t *lat = static_cast<const uint16_t *>(seq_latent(latent, s, t));
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const int first = split * span * FL_POS, end = min(nvis, first + span * FL_POS);
    if (first >= nvis) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int *sl = sel ? sel + (size_t)t * (s.topk + s.KP) : nullptr;

    // a chunk's rows; those past the last visible position are zero so that nothing undefined enters a product
    constexpr int PIECES = FL_KL / 8, PER = FL_POS * PIECES / FL_THREADS, QPER = 3 * FL_HEADS * PIECES / FL_THREADS;
    static_assert(FL_POS * PIECES % FL_THREADS == 0 && 3 * FL_HEADS * PIECES % FL_THREADS == 0, "pieces per thread");
    auto row_of = [&](int jj) { return jj < end ? (ns < 0 ? jj : sl[jj]) : -1; };
    // this thread's rows are grow + 4 k: every second one has its pieces four places on (fl_at)
    static_assert(FL_THREADS == 4 * PIECES, "rows per round of the gather");
    const int grow = tid / PIECES, gpiece = tid % PIECES, gat = fl_at(grow, gpiece);
    auto gather = [&]() {
#pragma unroll 6
        for (int k = 0; k < PER; k++) {
            const int j = s_rows[grow + 4 * k];
            __nv_bfloat16 *o = cs + (gat ^ ((k & 1) * 32)) + 4 * k * FL_KL;
            if (j >= 0) cp_async16(o, lat + (size_t)j * FL_KL + gpiece * 8);
            else        *reinterpret_cast<uint4 *>(o) = make_uint4(0u, 0u, 0u, 0u);
        }
    };
    if (tid < FL_POS) s_rows[tid] = row_of(first + tid);
    {
        const __nv_bfloat16 *qt = qterms + ((size_t)t * s.H + h0) * 3 * FL_KL;               // [head][term][512]
#pragma unroll
        for (int k = 0; k < QPER; k++) {
            const int i = tid + k * FL_THREADS, row = i / PIECES, piece = i % PIECES;
            cp_async16(qs + fl_at((row % 3) * FL_HEADS + row / 3, piece), qt + (size_t)row * FL_KL + piece * 8);
        }
    }
    __syncthreads();
    gather();

    const int pg = warp >> 2, kq = warp & 3;                        // scores: positions 24 pg .., columns 128 kq ..
    const int row = 2 * warp + (lane >> 4), l16 = lane & 15;        // exponentials: this lane's head, positions l16, l16 + 16, l16 + 32
    const int arow = (lane & 7) + 8 * ((lane >> 3) & 1), ahalf = lane >> 4;
    double z = 0.0, ref = -INFINITY;
    float2 sum[8][2];                                               // weighted sums: columns 64 warp + 8 n + 2 (lane % 4) and the next, heads lane / 4 and + 8
    __nv_bfloat162 rest[8][2];                                      // what the last addition to them rounded away, to eight bits
#pragma unroll
    for (int n = 0; n < 8; n++)
#pragma unroll
        for (int i = 0; i < 2; i++) { sum[n][i] = make_float2(0.f, 0.f); rest[n][i] = __floats2bfloat162_rn(0.f, 0.f); }

#pragma unroll 1
    for (int j0 = first; j0 < end; j0 += FL_POS) {
        cp_async_wait();
        __syncthreads();
        const int next = tid < FL_POS ? row_of(j0 + FL_POS + tid) : -1;   // (on its way while the scores are multiplied)
        // ---- scores
        {
            float c[3][4];
#pragma unroll
            for (int n = 0; n < 3; n++) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
            const int b4 = pg * 24 + (lane & 7) + 8 * (lane >> 4), b2 = pg * 24 + 16 + (lane & 7), bhalf = (lane >> 3) & 1;
#pragma unroll 1
            for (int k = 0; k < 8; k++) {
                const int piece = kq * 16 + k * 2;
                uint32_t b[4], d[2];
                ldsm_x4(b, cs + fl_at(b4, piece + bhalf));
                ldsm_x2(d, cs + fl_at(b2, piece + bhalf));
#pragma unroll
                for (int term = 2; term >= 0; term--) {
                    uint32_t a[4];
                    ldsm_x4(a, qs + fl_at(term * FL_HEADS + arow, piece + ahalf));
                    mma_bf16(c[0], a, b[0], b[1]);
                    mma_bf16(c[1], a, b[2], b[3]);
                    mma_bf16(c[2], a, d[0], d[1]);
                }
            }
            float *o = ss + (kq * FL_HEADS + (lane >> 2)) * FL_SPITCH + pg * 24 + 2 * (lane & 3);
#pragma unroll
            for (int n = 0; n < 3; n++) {
                *reinterpret_cast<float2 *>(o + 8 * n) = make_float2(c[n][0], c[n][1]);
                *reinterpret_cast<float2 *>(o + 8 * FL_SPITCH + 8 * n) = make_float2(c[n][2], c[n][3]);
            }
        }
        if (tid < FL_POS) s_rows[tid] = next;
        __syncthreads();
        // ---- exponentials
        float e[3], scale = 1.f;
        {
            float m = -INFINITY, v[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float *o = ss + row * FL_SPITCH + l16 + 16 * k;
                const float x = __fadd_rn(__fadd_rn(o[0], o[FL_HEADS * FL_SPITCH]), __fadd_rn(o[2 * FL_HEADS * FL_SPITCH], o[3 * FL_HEADS * FL_SPITCH]));
                v[k] = j0 + l16 + 16 * k < end ? x : -INFINITY;
                m = fmaxf(m, v[k]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (!((double)m <= ref + 16.0)) {                       // (the first chunk, a score much larger, NaN)
                const double d = (double)m - ref;
                if (d < 80.0) {                                     // by a power of two, which takes nothing from the sums
                    const double k = rint(d * 1.4426950408889634);
                    scale = __int_as_float((127 - (int)k) << 23);
                    ref = fma(k, 0.6931471805599453, ref);
                } else {                                            // the first chunk, whose sums are zero; or nothing of the others is left
                    scale = ref == -INFINITY ? 1.f : 0.f;
                    ref = (double)m;
                }
                z *= (double)scale;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double x = j0 + l16 + 16 * k < end ? exp((double)v[k] - ref) : 0.0;
                z += x;
                e[k] = (float)x;
            }
            if (l16 == 0) s_scale[row] = scale;
        }
        __syncthreads();                                            // the scores have been read: probabilities go there
#pragma unroll
        for (int k = 0; k < 3; k++) {
            __nv_bfloat16 a, b, d;
            split3_bf16(e[k], a, b, d);
            __nv_bfloat16 *o = ps + row * FL_PPITCH + l16 + 16 * k;
            o[0] = a; o[FL_HEADS * FL_PPITCH] = b; o[2 * FL_HEADS * FL_PPITCH] = d;
        }
        if (__syncthreads_or(scale != 1.f)) {
            const float f0 = s_scale[lane >> 2], f1 = s_scale[(lane >> 2) + 8];
#pragma unroll
            for (int n = 0; n < 8; n++) {
                sum[n][0].x *= f0; sum[n][0].y *= f0; rest[n][0] = __hmul2(rest[n][0], __floats2bfloat162_rn(f0, f0));
                sum[n][1].x *= f1; sum[n][1].y *= f1; rest[n][1] = __hmul2(rest[n][1], __floats2bfloat162_rn(f1, f1));
            }
        }
        // ---- weighted sum of the rows: this warp's 64 columns for the 16 heads, 16 of them at a time
#pragma unroll
        for (int quarter = 0; quarter < 4; quarter++) {
            float acc[2][4];
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 2; i++) { const float2 r = __bfloat1622float2(rest[quarter * 2 + n][i]); acc[n][2 * i] = r.x; acc[n][2 * i + 1] = r.y; }
            uint32_t b[FL_POS / 16][4];
#pragma unroll
            for (int k = 0; k < FL_POS / 16; k++)
                ldsm_x4_trans(b[k], cs + fl_at(k * 16 + (lane & 15), warp * 8 + quarter * 2 + (lane >> 4)));
#pragma unroll
            for (int term = 2; term >= 0; term--)                   // (the small terms first: the tensor cores truncate to the sum's last place)
#pragma unroll
                for (int k = 0; k < FL_POS / 16; k++) {
                    uint32_t a[4];
                    ldsm_x4(a, ps + (size_t)(term * FL_HEADS + arow) * FL_PPITCH + k * 16 + 8 * ahalf);
                    mma_bf16(acc[0], a, b[k][0], b[k][1]); mma_bf16(acc[1], a, b[k][2], b[k][3]);
                }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    float2 &u = sum[quarter * 2 + n][i];
                    const float x0 = acc[n][2 * i], x1 = acc[n][2 * i + 1], t0 = __fadd_rn(u.x, x0), t1 = __fadd_rn(u.y, x1), y0 = __fsub_rn(t0, u.x), y1 = __fsub_rn(t1, u.y);
                    rest[quarter * 2 + n][i] = upper_halves(__fsub_rn(x0, y0), __fsub_rn(x1, y1));
                    u.x = t0; u.y = t1;
                }
        }
        __syncthreads();                                            // the rows have been read
        if (j0 + FL_POS < end) gather();
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (l16 == 0) {
        s_z[row] = z;
        if (splits > 1) {
            double *st = cstat + (((size_t)t * s.H + h0 + row) * splits + split) * 2;
            st[0] = ref;
            st[1] = z;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int r = (lane >> 2) + 8 * i;
        const double inv = splits > 1 ? 1.0 : 1.0 / s_z[r];
        float *o = (splits > 1 ? part + (((size_t)t * s.H + h0 + r) * splits + split) * FL_KL : cb + ((size_t)t * s.H + h0 + r) * FL_KL) + warp * 64 + 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < 8; n++) {
            const float a = sum[n][i].x, b = sum[n][i].y;
            const float2 c = __bfloat1622float2(rest[n][i]);       // (not a number where the sum is infinite)
            const double da = (double)a + (c.x == c.x ? (double)c.x : 0.0), db = (double)b + (c.y == c.y ? (double)c.y : 0.0);
            *reinterpret_cast<float2 *>(o + n * 8) = make_float2((float)(da * inv), (float)(db * inv));
        }
    }
}

// cb[t][h][c] = sum_s e^(R_s - M) part_s[c] / sum_s e^(R_s - M) z_s over the stretches s, ascending, FP64.
// A thread owns a latent column. Everything is asked for before anything is used (the rows do not depend on the weights), the weights are
// computed by the first two warps, one exponential per stretch. FL_AHEAD: rows asked for, 48 for a query in many stretches (43: 10.7 -> 8.2 us), 8 for many
// queries in few (64 queries in five: 98 us with the registers of 48, 27 so).
constexpr int FL_MAX_SPLITS = 64;
template <int FL_AHEAD>
__device__ __forceinline__ float flash_column(const float *part, const double *cstat, const int *nsel, int cached, int splits, int span, const MlaShape &s, int h, int t)
{
    __shared__ double s_m[FL_MAX_SPLITS], s_w[FL_MAX_SPLITS], s_z[2];
    const int p = pos_of(s, cached, t), tid = threadIdx.x;
    const float *pr = part + ((size_t)t * s.H + h) * splits * FL_KL + tid;
    float v[FL_AHEAD];
#pragma unroll
    for (int i = 0; i < FL_AHEAD; i++) v[i] = i < splits ? __ldcg(pr + (size_t)i * FL_KL) : 0.f;      // (unused stretches too: they are not multiplied)
    const int ns = nsel ? nsel[t] : -1;
    const int nvis = ns < 0 ? p + 1 : ns;
    const int used = (nvis + span * FL_POS - 1) / (span * FL_POS);
    if (tid < FL_MAX_SPLITS) {
        const double *st = cstat + ((size_t)t * s.H + h) * splits * 2;
        double m = -INFINITY, zc = 0.0;
        if (tid < used) { m = st[2 * tid]; zc = st[2 * tid + 1]; }
        s_m[tid] = m;
        asm volatile("bar.sync 1, 64;" ::: "memory");
        double M = fmax(s_m[tid & 31], s_m[(tid & 31) + 32]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) M = fmax(M, __shfl_xor_sync(0xffffffffu, M, o));
        const double w = tid < used ? exp(m - M) : 0.0;
        s_w[tid] = w;
        const double z = warp_sum(w * zc);
        if ((tid & 31) == 0) s_z[tid >> 5] = z;
    }
    __syncthreads();
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < FL_AHEAD; i++) if (i < used) acc = fma(s_w[i], (double)v[i], acc);
    for (int i = FL_AHEAD; i < used; i++) acc = fma(s_w[i], (double)__ldcg(pr + (size_t)i * FL_KL), acc);
    return (float)(acc / (s_z[0] + s_z[1]));
}

template <int FL_AHEAD>
__global__ void __launch_bounds__(FL_KL) mla_flash_reduce_kernel(float *cb, const float *part, const double *cstat, const int *nsel,
                                                               int cached, int splits, int span, MlaShape s)
{
    pdl_trigger();
    pdl_wait();
    cb[((size_t)blockIdx.y * s.H + blockIdx.x) * FL_KL + threadIdx.x] = flash_column<FL_AHEAD>(part, cstat, nsel, cached, splits, span, s, blockIdx.x, blockIdx.y);
}

// The same sum and, for the few queries of a decode step, the value rows of kv_b behind it: a CTA takes FL_VROWS of a head's rows, whose
// weights are asked for with the stretches' columns, and sums the stretches for itself (88 KB out of L2, twice a head). One launch and one way to
// memory less: reduction and mla_vout_kernel one after the other 8.2 + 7.4 us for 43 stretches, 10.8 so; the layer of one query 130.7 -> 127.2 us. (48
// columns at a time spill beside the weights: 128.8; four rows to a warp: 131.) From four queries on mla_vout's FP64 tiles take the
// rows of all of them at once.
constexpr int FL_VOUT_T = 4, FL_VWARP = 8, FL_VROWS = FL_KL / 32 * FL_VWARP;
template <int FL_AHEAD>
__global__ void __launch_bounds__(FL_KL) mla_flash_vout_kernel(float *acc_out, const uint16_t *w, const float *part, const double *cstat, const int *nsel,
                                                             int cached, int splits, int span, MlaShape s)
{
    pdl_trigger();
    __shared__ __align__(16) float x[FL_KL];
    const int h = blockIdx.y, t = blockIdx.z, lane = threadIdx.x & 31, r0 = blockIdx.x * FL_VROWS + (threadIdx.x >> 5) * FL_VWARP;
    uint4 wv[FL_VWARP][2];
#pragma unroll
    for (int r = 0; r < FL_VWARP; r++) {
        const uint16_t *row = w + ((size_t)h * (s.qn + s.vh) + s.qn + min(r0 + r, s.vh - 1)) * FL_KL;
        wv[r][0] = ld_stream16(row + lane * 8);
        wv[r][1] = ld_stream16(row + 256 + lane * 8);
    }
    pdl_wait();
    x[threadIdx.x] = flash_column<FL_AHEAD>(part, cstat, nsel, cached, splits, span, s, h, t);
    __syncthreads();
    float acc[FL_VWARP];
#pragma unroll
    for (int r = 0; r < FL_VWARP; r++) acc[r] = 0.f;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const float4 xa = *reinterpret_cast<const float4 *>(x + g * 256 + lane * 8), xb = *reinterpret_cast<const float4 *>(x + g * 256 + lane * 8 + 4);
#pragma unroll
        for (int r = 0; r < FL_VWARP; r++) {
            float v[8];
            bf16x2_to_f32(wv[r][g].x, v[0], v[1]); bf16x2_to_f32(wv[r][g].y, v[2], v[3]);
            bf16x2_to_f32(wv[r][g].z, v[4], v[5]); bf16x2_to_f32(wv[r][g].w, v[6], v[7]);
            const float s0 = fmaf(v[6], xb.z, fmaf(v[4], xb.x, fmaf(v[2], xa.z, v[0] * xa.x))), s1 = fmaf(v[7], xb.w, fmaf(v[5], xb.y, fmaf(v[3], xa.w, v[1] * xa.y)));
            acc[r] += s0 + s1;
        }
    }
#pragma unroll
    for (int r = 0; r < FL_VWARP; r++) {
        acc[r] = warp_sum(acc[r]);
        if (lane == r && r0 + r < s.vh) acc_out[((size_t)t * s.H + h) * s.vh + r0 + r] = acc[r];
    }
}

// The kernels know no limit of positions; a layer that looks at more than this stays with the FP64 core, whose results it has always had.
// (4096 positions, the layer of one / of 64 queries: 65 / 730 us here, 145 / 4334 with the FP64 core.)
constexpr int FL_MAX_POSITIONS = 4096;
bool mla_flash_takes(const MlaShape &s)
{
    return s.latent_bf16 && s.KL == FL_KL && s.H % FL_HEADS == 0 && s.topk + s.KP <= FL_MAX_POSITIONS;
}

// Returns 1 when the value projection into acc_out (kv_b's value rows) is done too, 0 when cb is what there is, -1 on failure.
// scratch: `part_bytes` bytes for the stretches' rows; `cstat` room for [T][H][splits][2] doubles.
int mla_attend_flash(cudaStream_t st, float *cb, const void *qterms, const void *latent, const int *sel, const int *nsel,
                     void *part, size_t part_bytes, double *cstat, int T, int cached, const MlaShape &s, float *acc_out, const DMat &kv_b)
{
    static SmemGrant grant;
    if (!dev_opt_in_smem((const void *)mla_flash_kernel, FL_SMEM, grant)) return -1;
    const int stride = s.topk + s.KP;
    const int last = s.batch ? cached + 1 : cached + T, chunks = ((last < stride ? last : stride) + FL_POS - 1) / FL_POS;
    // As many stretches as give every SM two CTAs four times over, so that the last ones to end are a small part: a stretch reads the
    // query's 48 KB once more. Queries of a long prompt are enough by themselves, and need no second kernel.
    const int ctas = T * (s.H / FL_HEADS), room = (int)(part_bytes / ((size_t)T * s.H * FL_KL * sizeof(float)));
    int splits = (8 * dev_sms() + ctas - 1) / ctas;
    if (ctas >= 4 * dev_sms()) splits = 1;
    if (splits > chunks) splits = chunks;
    if (splits > FL_MAX_SPLITS) splits = FL_MAX_SPLITS;             // (places of the second kernel)
    if (splits > room) splits = room < 1 ? 1 : room;
    const int span = (chunks + splits - 1) / splits;
    splits = (chunks + span - 1) / span;
    G5B_LAUNCH_PDL(mla_flash_kernel, dim3(splits, s.H / FL_HEADS, T), FL_THREADS, FL_SMEM, st, cb, static_cast<float *>(part), cstat,
                   static_cast<const __nv_bfloat16 *>(qterms), latent, sel, nsel, cached, splits, span, s);
    // (launched the ordinary way: launched early, its CTAs crowd the SMs beside the core's, of which two fit an SM - one
    // token at 2048 / 8192 / 32768 positions: MLA layer 102.4 / 112.6 / 120.9 us, 96.3 / 106.6 / 114.8 so)
    if (splits > 1 && acc_out && T < FL_VOUT_T && kv_b.dt == DT_BF16 && (reinterpret_cast<uintptr_t>(kv_b.w) & 15) == 0) {
        auto sum = splits > 8 ? mla_flash_vout_kernel<24> : mla_flash_vout_kernel<8>;
        G5B_LAUNCH(sum, dim3((s.vh + FL_VROWS - 1) / FL_VROWS, s.H, T), FL_KL, 0, st, acc_out, static_cast<const uint16_t *>(kv_b.w), static_cast<const float *>(part), cstat, nsel,
                   cached, splits, span, s);
        return 1;
    }
    if (splits > 1) {
        auto reduce = splits > 8 ? mla_flash_reduce_kernel<48> : mla_flash_reduce_kernel<8>;
        G5B_LAUNCH(reduce, dim3(s.H, T), FL_KL, 0, st, cb, static_cast<const float *>(part), cstat, nsel, cached, splits, span, s);
    }
    return 0;
}


// o[t][h][r] = W_v[h][r] . cb[t][h]: the value half of kv_b applied once per query and head
// (glm53f_ops.c:904-909). A warp takes RW rows of one head.
// TT queries per block (blockIdx.z = group of TT): the head's rows are read once for all of them.
template <int TT>
__global__ void __launch_bounds__(256) mla_vout_kernel(float *acc_out, const float *cb, const DMat kv_b, MlaShape s, int T)
{
    pdl_trigger();
    pdl_wait();
    const int h = blockIdx.y, t0 = blockIdx.z * TT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (blockIdx.x * 8 + warp) * RW;
    if (r >= s.vh) return;
    const int kvd = s.qn + s.vh;
    const size_t rb = (size_t)s.KL * (kv_b.dt == DT_FP8 ? 1 : kv_b.dt == DT_BF16 ? 2 : 4);
    const void *wrow[RW];
    const float *srow[RW];
#pragma unroll
    for (int q = 0; q < RW; q++) {
        const int row = h * kvd + s.qn + min(r + q, s.vh - 1);
        wrow[q] = static_cast<const uint8_t *>(kv_b.w) + (size_t)row * rb;
        srow[q] = kv_b.dt == DT_FP8 ? kv_b.s + (size_t)(row / kv_b.br) * kv_b.scols : nullptr;
    }
    const float *xp[TT];
    float xinv[TT];
#pragma unroll
    for (int i = 0; i < TT; i++) {
        xp[i] = cb + ((size_t)min(t0 + i, T - 1) * s.H + h) * s.KL;       // queries past the last one repeat it, unused
        xinv[i] = 1.f;
    }
    float acc[RW][TT];
#pragma unroll
    for (int q = 0; q < RW; q++)
#pragma unroll
        for (int i = 0; i < TT; i++) acc[q][i] = 0.f;
    dot_rows<TT>(acc, kv_b.dt, wrow, srow, kv_b.bc, xp, xinv, nullptr, false, 0, s.KL / piece_elems(kv_b.dt), lane);
#pragma unroll
    for (int q = 0; q < RW; q++)
#pragma unroll
        for (int i = 0; i < TT; i++) {
            const float v = warp_sum(acc[q][i]);
            if (lane == 0 && r + q < s.vh && t0 + i < T) acc_out[((size_t)(t0 + i) * s.H + h) * s.vh + r + q] = v;
        }
}

// Same product for shapes the streaming loop cannot take (ragged columns, tiny FP8 blocks).
__global__ void mla_vout_any_kernel(float *acc_out, const float *cb, const DMat kv_b, MlaShape s)
{
    const int h = blockIdx.y, t = blockIdx.z;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= s.vh) return;
    const int row = h * (s.qn + s.vh) + s.qn + r;
    const float *x = cb + ((size_t)t * s.H + h) * s.KL;
    double acc = 0.0;
    for (int c = 0; c < s.KL; c++) acc += mat_elem(kv_b, row, c) * (double)x[c];
    acc_out[((size_t)t * s.H + h) * s.vh + r] = (float)acc;
}

void mla_vout(cudaStream_t st, float *acc_out, const float *cb, const DMat &kv_b, int T, const MlaShape &s)
{
    // Four queries and more in FP64 tiles: a head's rows become doubles once for eight to 64 queries (64 queries of 64 heads: 47 us, 145 with a warp per
    // four rows and four queries at a time; 7: 17.6 and 21)
    if (T >= 4 && kv_b.dt == DT_BF16 && s.KL % F64_K == 0 && s.vh % 2 == 0 && (reinterpret_cast<uintptr_t>(cb) & 15) == 0 && (reinterpret_cast<uintptr_t>(kv_b.w) & 15) == 0) {
        const size_t kvd = (size_t)(s.qn + s.vh);
        f64_tile<false>(st, F64Tile{cb, static_cast<const uint16_t *>(kv_b.w) + (size_t)s.qn * s.KL, nullptr, (size_t)s.H * s.KL, (size_t)s.KL, (size_t)s.H * s.vh, (size_t)s.KL,
                                    kvd * s.KL, (size_t)s.vh, T, s.vh, s.KL, {}, acc_out}, s.H);
        return;
    }
    const bool fast = s.KL % piece_elems(kv_b.dt) == 0 && (kv_b.dt != DT_FP8 || kv_b.bc % 16 == 0);
    if (fast && T >= 4) G5B_LAUNCH_PDL(mla_vout_kernel<4>, dim3((s.vh + 8 * RW - 1) / (8 * RW), s.H, (T + 3) / 4), 256, 0, st, acc_out, cb, kv_b, s, T);
    else if (fast)      G5B_LAUNCH_PDL(mla_vout_kernel<1>, dim3((s.vh + 8 * RW - 1) / (8 * RW), s.H, T), 256, 0, st, acc_out, cb, kv_b, s, T);
    else      G5B_LAUNCH(mla_vout_any_kernel, dim3((s.vh + 63) / 64, s.H, T), 64, 0, st, acc_out, cb, kv_b, s);
}

}  // namespace g5b
