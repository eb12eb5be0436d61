// mhc.cu - manifold-constrained hyper-connections: the 4-stream residual of the architecture.
//
// Reference: glm53f_hc_pre / glm53f_hc_post (src/core/glm53f_ops.c:560-625) and the device
// kernels k_hc_mix / k_hc_collapse / k_hc_post (src/gpu/glm53f_gpu_kernels.cu:455-535), where one
// thread per token ran the whole Sinkhorn normalisation and two more launches collapsed and
// expanded the streams. Here one launch per site does gates, Sinkhorn and the collapse: warp 0
// normalises the mixer while the other warps collapse the streams, which only need `pre`.
#include "acc2.cuh"
#include "common.cuh"
#include "f64_tile.cuh"
#include "kernels.h"

namespace g5b {

constexpr int HC_THREADS = 256;

__global__ void __launch_bounds__(HC_THREADS) hc_finish_kernel(
    float *x, float *post, float *comb, const float *h, const float *mix, const float *base,
    const float *scale, int M, int E, int iters, float epsf)
{
    __shared__ double pre[G5B_MAX_HC];
    __shared__ double cm[G5B_MAX_HC * G5B_MAX_HC];
    const int t = blockIdx.x, tid = threadIdx.x;
    const int MIX = (2 + M) * M;
    const float *mx = mix + (size_t)t * MIX;
    const double eps = (double)epsf;

    if (tid >= 32 && tid < 32 + M) {
        const int i = tid - 32;
        pre[i] = (double)sigmoid_host(mul_add_unfused(mx[i], scale[0], base[i])) + eps;
        post[(size_t)t * M + i] = __fmul_rn(2.0f, sigmoid_host(mul_add_unfused(mx[M + i], scale[1], base[M + i])));
    }
    __syncthreads();

    if (tid < 32) {
        // Row softmax + eps, then column / row normalisations, each dividing by (sum + eps) with
        // the sum taken in index order (src/core/glm53f_ops.c:577-598).
        const int MM = M * M;
        for (int e = tid; e < MM; e += 32) {
            const int i = e / M, j = e % M;
            double top = -INFINITY, z = 0.0, mine = 0.0;
            for (int jj = 0; jj < M; jj++) {
                const int k = 2 * M + i * M + jj;
                const double l = (double)mul_add_unfused(mx[k], scale[2], base[k]);
                if (l > top) top = l;
            }
            for (int jj = 0; jj < M; jj++) {
                const int k = 2 * M + i * M + jj;
                const double l = (double)mul_add_unfused(mx[k], scale[2], base[k]);
                const double ex = exp(l - top);
                z += ex;
                if (jj == j) mine = ex;
            }
            cm[e] = mine / z + eps;
        }
        __syncwarp();
        for (int pass = 0; pass < 2 * iters - 1; pass++) {
            const bool by_col = (pass & 1) == 0;
            double nv[2];
            int n = 0;
            for (int e = tid; e < MM; e += 32, n++) {
                const int i = e / M, j = e % M;
                double s = 0.0;
                for (int b = 0; b < M; b++) s += by_col ? cm[b * M + j] : cm[i * M + b];
                nv[n] = cm[e] / (s + eps);
            }
            __syncwarp();
            n = 0;
            for (int e = tid; e < MM; e += 32, n++) cm[e] = nv[n];
            __syncwarp();
        }
        for (int e = tid; e < MM; e += 32) comb[(size_t)t * MM + e] = (float)cm[e];
    } else {
        // x[d] = sum_i pre[i] * h[i][d] in FP64 (src/core/glm53f_ops.c:603-607)
        const float *ht = h + (size_t)t * M * E;
        for (int d = tid - 32; d < E; d += HC_THREADS - 32) {
            double s = 0.0;
            for (int i = 0; i < M; i++) s += pre[i] * (double)ht[(size_t)i * E + d];
            x[(size_t)t * E + d] = (float)s;
        }
    }
}

void hc_finish(cudaStream_t st, float *x, float *post, float *comb, const float *h, const float *mix,
               const HcW &w, int T, int M, int E, int iters, float eps)
{
    G5B_LAUNCH(hc_finish_kernel, T, HC_THREADS, 0, st, x, post, comb, h, mix, w.base, w.scale, M, E, iters, eps);
}

// ---- one launch per site for the decoder layer: RMSNorm0 factor + mixer product + gates + Sinkhorn
// + collapse + the sub-block's input RMSNorm.
// As separate launches these were six kernels of one to six CTAs each, about 60 us per site and
// two sites per layer - more than the attention or the MoE block they wrap. Here HCF_SLICES CTAs
// per token each take a slice of the flattened streams: the slice's sum of squares and its part
// of the (2+M)M mixer dot products, in FP64. The CTA that finishes a token last (a counter, no
// spinning) adds the parts in slice order, applies the norm factor to the dots (the mixer's input
// is RMSNorm0(h) = h * inv without a weight, src/core/glm53f_ops.c:563-569), then runs the code of
// hc_finish_kernel above and finally normalises the collapsed vector with the layer's norm weight
// (glm53f_rmsnorm, src/core/glm53f_ops.c:473-480), so the sub-block reads its input directly.
// 1 / d for d > 0 to within an ulp or two: the hardware's 20-bit estimate and two Newton steps.
// The Sinkhorn passes below are a chain of 39 dependent divisions per site; the exact division
// sequence made that chain 7 us long, and the mixer is rounded to float at the end anyway.
__device__ __forceinline__ double recip_newton(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    r = fma(r, fma(-d, r, 1.0), r);
    return r;
}

constexpr int HCF_SLICES = 32, HCF_MAX_E = 8192, HCF_MAX_MIX = (2 + G5B_MAX_HC) * G5B_MAX_HC;

struct HcFused {
    float *xn, *post, *comb;
    float *h;                       // [T][M][E]; rewritten in place when y is given
    const float *y;                 // optional: the previous sub-block's output [T][E] - its hc_post
                                    // (with the post / comb still in the arrays above) is applied first
    const uint16_t *fn;             // BF16 [(2+M)M][M*E]
    const float *base, *scale, *norm_w;
    double *part;                   // [T][HCF_SLICES][(2+M)M + 1]
    int *counters;                  // [T], zero between launches
    int M, E, iters;
    float hc_eps, rms_eps;
};

__global__ void __launch_bounds__(HC_THREADS) hc_pre_fused_kernel(const HcFused a)
{
    __shared__ float hs[HCF_MAX_E * G5B_MAX_HC / HCF_SLICES];   // this CTA's slice of the streams; later reused
    __shared__ float xs[HCF_MAX_E];                              // collapsed vector (last CTA)
    __shared__ double red[32];
    __shared__ double dots[HCF_MAX_MIX + 1];
    __shared__ float mx[HCF_MAX_MIX];
    __shared__ double pre[G5B_MAX_HC];
    __shared__ double cm[G5B_MAX_HC * G5B_MAX_HC];
    __shared__ int is_last;
    const int t = blockIdx.y, cta = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int M = a.M, E = a.E, ME = M * E, MIX = (2 + M) * M;
    const int W = E / HCF_SLICES, d0 = cta * W;                 // this CTA's columns, of every stream
    float *ht = a.h + (size_t)t * ME;

    // ---- every CTA: its columns of the M streams
    for (int i = tid; i < M * W; i += HC_THREADS) hs[i] = ht[(size_t)(i / W) * E + d0 + (i % W)];
    __syncthreads();
    if (a.y) {
        // the pending hc_post of the previous site: h'[j][d] = post[j] y[d] + sum_i comb[i][j] h[i][d]
        // in FP64 (src/core/glm53f_ops.c:612-625), written back and used below
        float nv[G5B_MAX_HC];
        if (tid < W) {
            const double yv = (double)a.y[(size_t)t * E + d0 + tid];
            const float *cb = a.comb + (size_t)t * M * M, *po = a.post + (size_t)t * M;
            for (int j = 0; j < M; j++) {
                double sj = (double)po[j] * yv;
                for (int i = 0; i < M; i++) sj += (double)cb[i * M + j] * (double)hs[i * W + tid];
                nv[j] = (float)sj;
            }
        }
        __syncthreads();
        if (tid < W)
            for (int j = 0; j < M; j++) {
                hs[j * W + tid] = nv[j];
                ht[(size_t)j * E + d0 + tid] = nv[j];
            }
        __syncthreads();
    }
    double ss = 0.0;
    for (int i = tid; i < M * W; i += HC_THREADS) ss += (double)hs[i] * (double)hs[i];
    ss = block_sum(ss, red);
    double *mine = a.part + ((size_t)t * HCF_SLICES + cta) * (MIX + 1);
    if (tid == 0) mine[MIX] = ss;
    const int per_seg = W / 8;                                     // 16-byte pieces per stream segment
    for (int k = warp; k < MIX; k += HC_THREADS / 32) {
        const uint16_t *row = a.fn + (size_t)k * ME + d0;
        double acc = 0.0;
        for (int piece = lane; piece < M * per_seg; piece += 32) {
            const int i = piece / per_seg, off = (piece % per_seg) * 8;
            const uint4 wv = ld_stream16(row + (size_t)i * E + off);
            float w[8];
            bf16x2_to_f32(wv.x, w[0], w[1]); bf16x2_to_f32(wv.y, w[2], w[3]);
            bf16x2_to_f32(wv.z, w[4], w[5]); bf16x2_to_f32(wv.w, w[6], w[7]);
#pragma unroll
            for (int j = 0; j < 8; j++) acc = fma((double)w[j], (double)hs[i * W + off + j], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) mine[k] = acc;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int prev = atomicAdd(a.counters + t, 1);
        is_last = prev == HCF_SLICES - 1;
        if (is_last) a.counters[t] = 0;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();

    // ---- the token's last CTA: parts in slice order, factor, gates
    if (tid <= MIX) {
        double s = 0.0;
        for (int cc = 0; cc < HCF_SLICES; cc++) s += __ldcg(a.part + ((size_t)t * HCF_SLICES + cc) * (MIX + 1) + tid);
        dots[tid] = s;
    }
    __syncthreads();
    if (tid < MIX) {
        const float inv = (float)(1.0 / sqrt(dots[MIX] / (double)ME + (double)a.rms_eps));
        mx[tid] = (float)(dots[tid] * (double)inv);
    }
    __syncthreads();
    const double eps = (double)a.hc_eps;
    if (tid >= 32 && tid < 32 + M) {
        const int i = tid - 32;
        pre[i] = (double)sigmoid_host(mul_add_unfused(mx[i], a.scale[0], a.base[i])) + eps;
        a.post[(size_t)t * M + i] = __fmul_rn(2.0f, sigmoid_host(mul_add_unfused(mx[M + i], a.scale[1], a.base[M + i])));
    }
    __syncthreads();
    if (tid < 32) {
        // row softmax + eps, then column / row normalisations (src/core/glm53f_ops.c:577-598)
        const int MM = M * M;
        for (int e = tid; e < MM; e += 32) {
            const int i = e / M, j = e % M;
            double top = -INFINITY, z = 0.0, own = 0.0;
            for (int jj = 0; jj < M; jj++) {
                const int k = 2 * M + i * M + jj;
                const double l = (double)mul_add_unfused(mx[k], a.scale[2], a.base[k]);
                if (l > top) top = l;
            }
            for (int jj = 0; jj < M; jj++) {
                const int k = 2 * M + i * M + jj;
                const double l = (double)mul_add_unfused(mx[k], a.scale[2], a.base[k]);
                const double ex = exp(l - top);
                z += ex;
                if (jj == j) own = ex;
            }
            cm[e] = own / z + eps;
        }
        __syncwarp();
        if (MM <= 32) {
            // a lane per matrix element, sums gathered with shuffles in the reference's index order
            const int i = tid / M, j = tid % M;
            double v = tid < MM ? cm[tid] : 0.0;
            for (int pass = 0; pass < 2 * a.iters - 1; pass++) {
                const bool by_col = (pass & 1) == 0;
                double sum = 0.0;
                for (int b = 0; b < M; b++) {
                    const int src = by_col ? b * M + j : i * M + b;
                    sum += __shfl_sync(0xffffffffu, v, src < 32 ? src : 0);
                }
                if (tid < MM) v = v * recip_newton(sum + eps);
            }
            if (tid < MM) a.comb[(size_t)t * MM + tid] = (float)v;
        } else {
            for (int pass = 0; pass < 2 * a.iters - 1; pass++) {
                const bool by_col = (pass & 1) == 0;
                double nv[2];
                int n = 0;
                for (int e = tid; e < MM; e += 32, n++) {
                    const int i = e / M, j = e % M;
                    double s = 0.0;
                    for (int b = 0; b < M; b++) s += by_col ? cm[b * M + j] : cm[i * M + b];
                    nv[n] = cm[e] / (s + eps);
                }
                __syncwarp();
                n = 0;
                for (int e = tid; e < MM; e += 32, n++) cm[e] = nv[n];
                __syncwarp();
            }
            for (int e = tid; e < MM; e += 32) a.comb[(size_t)t * MM + e] = (float)cm[e];
        }
    } else {
        // x[d] = sum_i pre[i] * h[i][d] in FP64 (src/core/glm53f_ops.c:603-607), kept in shared memory.
        // Four columns per thread and all of a thread's loads issued before the sums: one CTA walks
        // the whole token here, so the loads must overlap (they hit L2: the slices were just read).
        for (int d0 = (tid - 32) * 4; d0 < E; d0 += (HC_THREADS - 32) * 4 * 2) {
            const int d1 = d0 + (HC_THREADS - 32) * 4;
            float4 va[G5B_MAX_HC], vb[G5B_MAX_HC];
#pragma unroll
            for (int i = 0; i < G5B_MAX_HC; i++)
                if (i < M) {
                    va[i] = *reinterpret_cast<const float4 *>(ht + (size_t)i * E + d0);
                    if (d1 < E) vb[i] = *reinterpret_cast<const float4 *>(ht + (size_t)i * E + d1);
                }
            double sa[4] = {0.0, 0.0, 0.0, 0.0}, sb[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int i = 0; i < G5B_MAX_HC; i++)
                if (i < M) {
                    const double p = pre[i];
                    sa[0] += p * (double)va[i].x; sa[1] += p * (double)va[i].y; sa[2] += p * (double)va[i].z; sa[3] += p * (double)va[i].w;
                    if (d1 < E) { sb[0] += p * (double)vb[i].x; sb[1] += p * (double)vb[i].y; sb[2] += p * (double)vb[i].z; sb[3] += p * (double)vb[i].w; }
                }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                xs[d0 + q] = (float)sa[q];
                if (d1 < E) xs[d1 + q] = (float)sb[q];
            }
        }
    }
    __syncthreads();
    // ---- the sub-block's input: RMSNorm(x) * w
    double s2 = 0.0;
    for (int d = tid; d < E; d += HC_THREADS) s2 += (double)xs[d] * (double)xs[d];
    s2 = block_sum(s2, red);
    __shared__ float inv2;
    if (tid == 0) inv2 = (float)(1.0 / sqrt(s2 / (double)E + (double)a.rms_eps));
    __syncthreads();
    const float f = inv2;
    for (int d = tid; d < E; d += HC_THREADS) a.xn[(size_t)t * E + d] = __fmul_rn(a.norm_w[d], __fmul_rn(xs[d], f));
}

// ---- the same site as one thread-block cluster per token.
// The kernel above hands a token to whichever CTA finishes last: a fence, an atomic, a reload of
// 32 x 25 partial sums and then ONE CTA walking the whole token for the collapse and the norm
// (about 21 us per site, two sites per layer: a quarter of a batch-1 decoder layer). Here the
// HCC_CTAS CTAs of a cluster each keep their columns of the streams in shared memory from the
// first load to the last store; the partial sums (mixer dots, then the collapsed vector's sum of
// squares) are exchanged through distributed shared memory at two cluster barriers, every CTA
// derives the gates for itself and collapses and normalises its own columns. The Sinkhorn chain
// (39 dependent normalisations, needed only for the NEXT stream expansion) runs in warp 0 of CTA 0
// beside all that: warp 0 arrives at the second barrier before it starts and waits after.
constexpr int HCC_CTAS = 8, HCC_THREADS = 512, HCC_WARPS = HCC_THREADS / 32, HCC_MAX_W = 1024, HCC_MAX_HS = 4096;
constexpr int HCC_ROWS = 3, HCC_ROW_WARPS = 8, HCC_SPLITS = HCC_WARPS / HCC_ROW_WARPS;

// v / d for d > 0 to a relative 2^-40: the hardware's reciprocal estimate r (20 bits), its error
// e = 1 - d r, and v r (1 + e). An FP64 instruction occupies its pipe for 32 cycles per warp here
// and a Sinkhorn pass is a chain of nothing else, so every instruction less is 0.6 us per site; the
// mixer is rounded to float (2^-24) after the last pass.
__device__ __forceinline__ double div_chain(double v, double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double q = v * r;
    return fma(q, fma(-d, r, 1.0), q);
}

// The 2 iters - 1 alternating column / row normalisations v <- v / (sum + eps) of the mixer
// (src/core/glm53f_ops.c:583-598) for the lane that holds element (i, j); all 32 lanes call it. One
// warp runs this chain while the rest of the cluster waits for nothing else, so the M = 4 case is
// written without a loop or a branch inside a pass: four shuffles, the members' sum as a two-level
// tree (the reference keeps a running sum: a few ulps of FP64 apart), one division.
template <int MT>
__device__ __forceinline__ double sinkhorn_passes(double v, int M, int i, int j, int passes, double eps)
{
    if constexpr (MT == 4) {
        for (int pass = 0; pass < passes; pass++) {
            const bool by_col = (pass & 1) == 0;
            const int s0 = by_col ? j : i * 4, st = by_col ? 4 : 1;
            const double p0 = __shfl_sync(0xffffffffu, v, s0), p1 = __shfl_sync(0xffffffffu, v, s0 + st);
            const double p2 = __shfl_sync(0xffffffffu, v, s0 + 2 * st), p3 = __shfl_sync(0xffffffffu, v, s0 + 3 * st);
            v = div_chain(v, ((p0 + p1) + (p2 + p3)) + eps);
        }
    } else {
        for (int pass = 0; pass < passes; pass++) {
            const bool by_col = (pass & 1) == 0;
            double sum = 0.0;
            for (int m = 0; m < M; m++) sum += __shfl_sync(0xffffffffu, v, by_col ? m * M + j : i * M + m);
            v = div_chain(v, sum + eps);
        }
    }
    return v;
}

__global__ void __cluster_dims__(HCC_CTAS, 1, 1) __launch_bounds__(HCC_THREADS) hc_pre_cluster_kernel(const HcFused a)
{
    __shared__ __align__(16) float hs[HCC_MAX_HS];     // this CTA's columns of the M streams
    __shared__ float xs[HCC_MAX_W];                     // its columns of the collapsed vector
    __shared__ double red[32];
    __shared__ double mine[HCC_SPLITS][HCF_MAX_MIX + 1];   // this CTA's parts of the dots; [0][MIX] = sum h^2
    __shared__ double mine_s2;                          // its part of sum x^2
    __shared__ double dots[HCF_MAX_MIX + 1];
    __shared__ float mx[HCF_MAX_MIX];
    __shared__ double pre[G5B_MAX_HC];
    const int t = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_cta_rank();
    const int M = a.M, E = a.E, ME = M * E, MIX = (2 + M) * M, MM = M * M;
    const int W = E / HCC_CTAS, d0 = (int)rank * W;
    float *ht = a.h + (size_t)t * ME;
    const double eps = (double)a.hc_eps;

    // Warp (q, b) takes the mixer rows b, b + 8, ... HCC_ROWS at a time and every HCC_SPLITS-th group of
    // 32 16-byte pieces of each. The rows depend on nothing computed here: the first piece is
    // requested before anything else; after that the piece for the next turn of the loop is
    // requested before the current one is summed. (The loop is kept rolled on purpose: this kernel
    // runs once per site with a cold instruction cache, and with the twelve pieces of a warp
    // unrolled - 17 KB of straight-line code - it waited for instruction fetch more than for data.)
    const int per_seg = W / 8, n_pieces = M * per_seg;            // pieces per stream segment / per row
    const int q = warp / HCC_ROW_WARPS, b = warp % HCC_ROW_WARPS;
    const int p_first = lane + 32 * q, p_step = 32 * HCC_SPLITS;
    uint4 wnext[HCC_ROWS];
    auto load_piece = [&](int k0, int piece) {
#pragma unroll
        for (int r = 0; r < HCC_ROWS; r++) {
            const int k = k0 + r * HCC_ROW_WARPS;
            if (k < MIX && piece < n_pieces)
                wnext[r] = ld_stream16(a.fn + (size_t)k * ME + (size_t)(piece / per_seg) * E + d0 + (piece % per_seg) * 8);
        }
    };
    load_piece(b, p_first);
    pdl_wait();                  // the streams and y come from earlier kernels; the mixer rows do not

    for (int i = tid * 4; i < M * W; i += HCC_THREADS * 4)
        *reinterpret_cast<float4 *>(hs + i) = *reinterpret_cast<const float4 *>(ht + (size_t)(i / W) * E + d0 + (i % W));
    __syncthreads();
    if (a.y) {
        // the pending hc_post of the previous site: h'[j][d] = post[j] y[d] + sum_i comb[i][j] h[i][d]
        // (src/core/glm53f_ops.c:612-625, FP64 there, compensated FP32 here); a thread owns a column,
        // so no barrier inside
        const float *cb = a.comb + (size_t)t * MM, *po = a.post + (size_t)t * M;
        for (int d = tid; d < W; d += HCC_THREADS) {
            const float yv = a.y[(size_t)t * E + d0 + d];
            float hv[G5B_MAX_HC];
#pragma unroll
            for (int i = 0; i < G5B_MAX_HC; i++) hv[i] = i < M ? hs[i * W + d] : 0.f;
#pragma unroll 1
            for (int j = 0; j < M; j++) {                // rolled: cold instruction cache, see above
                Acc2 sj;
                acc2_fma(sj, po[j], yv);
#pragma unroll
                for (int i = 0; i < G5B_MAX_HC; i++)
                    if (i < M) acc2_fma(sj, cb[i * M + j], hv[i]);
                const float nv = acc2_f32(sj);
                hs[j * W + d] = nv;
                ht[(size_t)j * E + d0 + d] = nv;
            }
        }
        __syncthreads();
    }
    Acc2 sq;
    for (int i = tid; i < M * W; i += HCC_THREADS) acc2_fma(sq, hs[i], hs[i]);
    const double ss = block_sum(acc2_f64(sq), red);
    if (tid == 0) mine[0][MIX] = ss;

    // mixer rows (compensated FP32 sums; the reference's are FP64)
    for (int k0 = b; k0 < MIX; k0 += HCC_ROW_WARPS * HCC_ROWS) {
        Acc2 acc[HCC_ROWS];
        if (k0 != b) load_piece(k0, p_first);
#pragma unroll 1
        for (int piece = p_first; piece < n_pieces; piece += p_step) {
            uint4 wv[HCC_ROWS];
#pragma unroll
            for (int r = 0; r < HCC_ROWS; r++) wv[r] = wnext[r];
            load_piece(k0, piece + p_step);
            const float *hv = hs + (piece / per_seg) * W + (piece % per_seg) * 8;
            const float4 h0 = *reinterpret_cast<const float4 *>(hv), h1 = *reinterpret_cast<const float4 *>(hv + 4);
            const float hd[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
            for (int r = 0; r < HCC_ROWS; r++) {
                if (k0 + r * HCC_ROW_WARPS >= MIX) continue;
                const uint32_t wr[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc2_fma(acc[r], __uint_as_float(wr[j] << 16), hd[2 * j]);
                    acc2_fma(acc[r], __uint_as_float(wr[j] & 0xffff0000u), hd[2 * j + 1]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < HCC_ROWS; r++) {
            const int k = k0 + r * HCC_ROW_WARPS;
            const double s = warp_sum(acc2_f64(acc[r]));
            if (lane == 0 && k < MIX) mine[q][k] = s;
        }
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();

    // ---- every CTA: the token's sums in CTA order, the norm factor, the gates
    if (tid <= MIX) {
        double s = 0.0;
        for (uint32_t r = 0; r < HCC_CTAS; r++) {
            double part = ld_cluster_f64(&mine[0][tid], r);
            if (tid < MIX)
                for (int qq = 1; qq < HCC_SPLITS; qq++) part += ld_cluster_f64(&mine[qq][tid], r);
            s += part;
        }
        dots[tid] = s;
    }
    __syncthreads();
    if (tid < MIX) {
        const float inv = (float)(1.0 / sqrt(dots[MIX] / (double)ME + (double)a.rms_eps));
        mx[tid] = (float)(dots[tid] * (double)inv);
    }
    __syncthreads();
    if (tid >= 32 && tid < 32 + M) {
        const int i = tid - 32;
        pre[i] = (double)sigmoid_host(mul_add_unfused(mx[i], a.scale[0], a.base[i])) + eps;
        if (rank == 0)
            a.post[(size_t)t * M + i] = __fmul_rn(2.0f, sigmoid_host(mul_add_unfused(mx[M + i], a.scale[1], a.base[M + i])));
    }
    if (warp == 0) {
        cluster_arrive();                                // nothing of this warp goes into sum x^2
        if (rank == 0) {
            // row softmax + eps, then column / row normalisations (src/core/glm53f_ops.c:577-598): a
            // lane per matrix element, the row's / column's members gathered with shuffles
            const int el = lane < MM ? lane : 0, i = el / M, j = el % M;
            const int k = 2 * M + el;
            const double l = (double)mul_add_unfused(mx[k], a.scale[2], a.base[k]);
            double top = -INFINITY;
            for (int jj = 0; jj < M; jj++) top = fmax(top, __shfl_sync(0xffffffffu, l, i * M + jj));
            const double ex = exp(l - top);
            double z = 0.0;
            for (int jj = 0; jj < M; jj++) z += __shfl_sync(0xffffffffu, ex, i * M + jj);
            double v = ex / z + eps;
            v = M == 4 ? sinkhorn_passes<4>(v, M, i, j, 2 * a.iters - 1, eps) : sinkhorn_passes<0>(v, M, i, j, 2 * a.iters - 1, eps);
            if (lane < MM) a.comb[(size_t)t * MM + lane] = (float)v;
            __syncwarp();
        }
        cluster_wait();
    } else {
        // x[d] = sum_i pre[i] * h[i][d] in FP64 (src/core/glm53f_ops.c:603-607) for this CTA's columns
        constexpr int NW = HCC_THREADS - 32;
        const int wt = tid - 32;
        asm volatile("bar.sync 1, %0;" ::"n"(NW) : "memory");     // `pre` comes from threads of these warps
        double s2 = 0.0;
        for (int d = wt; d < W; d += NW) {
            double s = 0.0;
            for (int i = 0; i < M; i++) s += pre[i] * (double)hs[i * W + d];
            const float xv = (float)s;
            xs[d] = xv;
            s2 += (double)xv * (double)xv;
        }
        s2 = warp_sum(s2);
        if (lane == 0) red[warp] = s2;
        asm volatile("bar.sync 1, %0;" ::"n"(NW) : "memory");
        if (wt == 0) {
            double s = 0.0;
            for (int w = 1; w < HCC_WARPS; w++) s += red[w];
            mine_s2 = s;
        }
        cluster_arrive();
        cluster_wait();
        // ---- the sub-block's input: RMSNorm(x) * w (glm53f_rmsnorm, src/core/glm53f_ops.c:473-480)
        double tot = 0.0;
        for (uint32_t r = 0; r < HCC_CTAS; r++) tot += ld_cluster_f64(&mine_s2, r);
        const float f = (float)(1.0 / sqrt(tot / (double)E + (double)a.rms_eps));
        for (int d = wt; d < W; d += NW)
            a.xn[(size_t)t * E + d0 + d] = __fmul_rn(a.norm_w[d0 + d], __fmul_rn(xs[d], f));
    }
    // no CTA leaves while another may still read its shared memory
    cluster_arrive();
    cluster_wait();
}

// ---- the same site for one position and four streams, what a decode step runs twice per layer: a chain of latencies.
// In the kernel above (28,600 cycles from its first instruction to its last, cold) the mixer product took 9800 of them - ten FP32
// instructions a term - and the pending expansion 4400, most of them the way of y, post and comb from L2, one after the other. Here
// everything that comes from memory is asked for at once: the mixer rows and norm weights before the wait for the kernel in front, the
// rest after it; streams become doubles once, in shared memory; and the products are FP64 FMA (64 per clock and SM) whose BF16 factor is
// its bits put where a double has them, two instructions and a value 2^896 times too small (bf16_bits_f64). 20,500 cycles cold; under ncu
// 16.6 -> 12.5 us, one token of eight layers 1617 -> 1550 us. What is left: one round trip to memory, two cluster barriers, the Sinkhorn chain.
constexpr int HCO_M = 4, HCO_MIX = (2 + HCO_M) * HCO_M;
static size_t hco_smem(int W) { return (size_t)HCO_M * 4 * (W / 8 + 1) * sizeof(double2) + (size_t)HCO_MIX * HCO_M * W * 2; }

__global__ void __cluster_dims__(HCC_CTAS, 1, 1) __launch_bounds__(HCC_THREADS, 1) hc_pre_one_kernel(const HcFused a)
{
    // piece p's elements 2 e2, 2 e2 + 1 of stream i: double2 at [i][e2][p], so that lanes with consecutive pieces read side by side
    extern __shared__ __align__(16) double2 hd[];
    __shared__ float xs[HCC_MAX_W];                     // this CTA's columns of the collapsed vector
    __shared__ double red[HCC_WARPS], mine[HCC_SPLITS][HCO_MIX + 1], dots[HCO_MIX + 1], pre[HCO_M], mine_s2;
    __shared__ float mx[HCO_MIX];
    constexpr int M = HCO_M, MM = M * M, MIX = HCO_MIX;
    pdl_trigger();
    const int t = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_cta_rank();
    const int E = a.E, ME = M * E, W = E / HCC_CTAS, d0 = (int)rank * W, per = W / 8, pitch = per + 1;
    float *ht = a.h + (size_t)t * ME + d0;
    const double eps = (double)a.hc_eps;
    auto at = [&](int i, int d) -> double & { return reinterpret_cast<double *>(hd + (i * 4 + ((d & 7) >> 1)) * pitch + (d >> 3))[d & 1]; };

    // warp (q, b): mixer rows b, b + 8, b + 16, every HCC_SPLITS-th group of 32 pieces of each
    const int q = warp / HCC_ROW_WARPS, b = warp % HCC_ROW_WARPS, pieces = M * per;
    uint4 *wm = reinterpret_cast<uint4 *>(hd + M * 4 * pitch);   // [24][pieces]: on their way past the registers
#pragma unroll 1
    for (int p = lane + 32 * q; p < pieces; p += 32 * HCC_SPLITS)
#pragma unroll
        for (int r = 0; r < 3; r++) cp_async16(wm + (b + 8 * r) * pieces + p, a.fn + (size_t)(b + 8 * r) * ME + (size_t)(p / per) * E + d0 + (p % per) * 8);
    pdl_wait();                  // the streams and y come from earlier kernels; the mixer rows do not

    double sq = 0.0;
    {
        float cb[MM], po[M];
        if (a.y) {
#pragma unroll
            for (int i = 0; i < MM; i++) cb[i] = __ldcg(a.comb + (size_t)t * MM + i);
#pragma unroll
            for (int i = 0; i < M; i++) po[i] = __ldcg(a.post + (size_t)t * M + i);
        }
#pragma unroll 1
        for (int d = tid; d < W; d += HCC_THREADS) {
            float hv[M];
#pragma unroll
            for (int i = 0; i < M; i++) hv[i] = __ldcg(ht + (size_t)i * E + d);
            if (a.y) {
                // the pending hc_post of the previous site: h'[j][d] = post[j] y[d] + sum_i comb[i][j] h[i][d] (src/core/glm53f_ops.c:612-625)
                const double y = (double)__ldcg(a.y + (size_t)t * E + d0 + d);
                double h[M];
#pragma unroll
                for (int i = 0; i < M; i++) h[i] = (double)hv[i];
#pragma unroll
                for (int j = 0; j < M; j++) {
                    double v = (double)po[j] * y;
#pragma unroll
                    for (int i = 0; i < M; i++) v = fma((double)cb[i * M + j], h[i], v);
                    hv[j] = (float)v;
                    ht[(size_t)j * E + d] = hv[j];
                }
            }
#pragma unroll
            for (int i = 0; i < M; i++) {
                const double h = (double)hv[i];
                at(i, d) = h;
                sq = fma(h, h, sq);
            }
        }
    }
    sq = warp_sum(sq);
    if (lane == 0) red[warp] = sq;
    cp_async_wait();
    __syncthreads();

    // ---- mixer rows
    {
        double acc[3] = {};
        uint32_t special = 0;                            // an infinity or NaN among this lane's mixer elements: no place among the scaled ones
        auto products = [&](auto widen) {
#pragma unroll 1
            for (int p = lane + 32 * q; p < pieces; p += 32 * HCC_SPLITS) {    // (rolled: this code runs from a cold instruction cache)
                const double2 *h = hd + (p / per) * 4 * pitch + p % per;
                uint4 wv[3];
#pragma unroll
                for (int r = 0; r < 3; r++) wv[r] = wm[(b + 8 * r) * pieces + p];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const double2 v = h[e * pitch];
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        const uint32_t u = e == 0 ? wv[r].x : e == 1 ? wv[r].y : e == 2 ? wv[r].z : wv[r].w;
                        special |= bf16_special(u);
                        acc[r] = fma(widen(u << 16), v.x, acc[r]);
                        acc[r] = fma(widen(u), v.y, acc[r]);
                    }
                }
            }
        };
        products([](uint32_t u) { return bf16_bits_f64(u); });
#pragma unroll
        for (int r = 0; r < 3; r++) acc[r] *= BF16_BITS_SCALE;
        if (__any_sync(0xffffffffu, special)) {
            acc[0] = acc[1] = acc[2] = 0.0;
            products([](uint32_t u) { return (double)__uint_as_float(u & 0xffff0000u); });
        }
#pragma unroll
        for (int r = 0; r < 3; r++) {
            acc[r] = warp_sum(acc[r]);
            if (lane == 0) mine[q][b + 8 * r] = acc[r];
        }
        if (tid == 0) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < HCC_WARPS; w++) s += red[w];
            mine[0][MIX] = s;
        }
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();

    // ---- every CTA: the token's sums in CTA order, the norm factor, the gates
    if (tid <= MIX) {
        double part[HCC_CTAS][HCC_SPLITS];
#pragma unroll
        for (uint32_t r = 0; r < HCC_CTAS; r++)
#pragma unroll
            for (int k = 0; k < HCC_SPLITS; k++) part[r][k] = k == 0 || tid < MIX ? ld_cluster_f64(&mine[k][tid], r) : 0.0;
        double s = 0.0;
#pragma unroll
        for (uint32_t r = 0; r < HCC_CTAS; r++) {
            double v = part[r][0];
#pragma unroll
            for (int k = 1; k < HCC_SPLITS; k++) v += part[r][k];
            s += v;
        }
        dots[tid] = s;
    }
    __syncthreads();
    if (tid < MIX) mx[tid] = (float)(dots[tid] * (double)(float)rsqrt_newton(dots[MIX] / (double)ME + (double)a.rms_eps));
    __syncthreads();
    if (warp == 0) {
        cluster_arrive();                                // nothing of this warp goes into sum x^2
        if (rank == 0) {
            // row softmax + eps, then column / row normalisations (src/core/glm53f_ops.c:577-598): a
            // lane per matrix element, the row's / column's members gathered with shuffles
            const int el = lane < MM ? lane : 0, i = el / M, j = el % M;
            const int k = 2 * M + el;
            const double l = (double)mul_add_unfused(mx[k], a.scale[2], a.base[k]);
            double top = -INFINITY;
#pragma unroll
            for (int jj = 0; jj < M; jj++) top = fmax(top, __shfl_sync(0xffffffffu, l, i * M + jj));
            const double ex = exp(l - top);
            double z = 0.0;
#pragma unroll
            for (int jj = 0; jj < M; jj++) z += __shfl_sync(0xffffffffu, ex, i * M + jj);
            const double v = sinkhorn_passes<M>(ex / z + eps, M, i, j, 2 * a.iters - 1, eps);
            if (lane < MM) a.comb[(size_t)t * MM + lane] = (float)v;
            __syncwarp();
        }
        cluster_wait();
    } else {
        // x[d] = sum_i pre[i] * h[i][d] in FP64 (src/core/glm53f_ops.c:603-607) for this CTA's columns
        constexpr int NW = HCC_THREADS - 32;
        const int wt = tid - 32;
        if (wt < M) {
            pre[wt] = (double)sigmoid_host(mul_add_unfused(mx[wt], a.scale[0], a.base[wt])) + eps;
            if (rank == 0) a.post[(size_t)t * M + wt] = __fmul_rn(2.0f, sigmoid_host(mul_add_unfused(mx[M + wt], a.scale[1], a.base[M + wt])));
        }
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(NW) : "memory");     // `pre` comes from threads of these warps
        double s2 = 0.0;
#pragma unroll 1
        for (int d = wt; d < W; d += NW) {
            double v = 0.0;
#pragma unroll
            for (int i = 0; i < M; i++) v += pre[i] * at(i, d);
            const float xv = (float)v;
            xs[d] = xv;
            s2 += (double)xv * (double)xv;
        }
        s2 = warp_sum(s2);
        if (lane == 0) red[warp] = s2;
        asm volatile("bar.sync 1, %0;" ::"n"(NW) : "memory");
        if (wt == 0) {
            double v = 0.0;
#pragma unroll
            for (int w = 1; w < HCC_WARPS; w++) v += red[w];
            mine_s2 = v;
        }
        __syncwarp();
        cluster_arrive();
        const float nw = wt < W ? a.norm_w[d0 + wt] : 0.f;
        cluster_wait();
        // ---- the sub-block's input: RMSNorm(x) * w (glm53f_rmsnorm, src/core/glm53f_ops.c:473-480)
        double part[HCC_CTAS], tot = 0.0;
#pragma unroll
        for (uint32_t r = 0; r < HCC_CTAS; r++) part[r] = ld_cluster_f64(&mine_s2, r);
#pragma unroll
        for (uint32_t r = 0; r < HCC_CTAS; r++) tot += part[r];
        const float f = (float)rsqrt_newton(tot / (double)E + (double)a.rms_eps);
#pragma unroll 1
        for (int d = wt; d < W; d += NW) a.xn[(size_t)t * E + d0 + d] = __fmul_rn(d == wt ? nw : a.norm_w[d0 + d], __fmul_rn(xs[d], f));
    }
    // no CTA leaves while another may still read its shared memory
    cluster_arrive();
    cluster_wait();
}

// ---- the same site for several positions (four streams): a cluster takes eight positions at once.
// A cluster per position multiplies the mixer rows, which every position shares, position by position, with sums like
// FP64's made of ten FP32 instructions per term (acc2.cuh): 45 us for 64 positions, and one CTA per position 442 us for 2048. With
// eight positions the mixer product is a contraction, [24 rows] x [8 positions] over the CTA's columns, and the FP64 matrix
// instruction does it: 64 FMA per clock and SM, while a mixer element becomes a double once per eight products and a
// stream element once per 24. The columns' order in the sum is the lanes' own: lane q of four takes eight consecutive columns, one
// 16-byte piece of a mixer row and two of a stream, for eight steps of the instruction. Everything else is in FP64
// too, with a column's streams converted once. A CTA keeps its columns of the eight positions in shared memory from the first
// load to the last store; gates, Sinkhorn and norms run as in the cluster kernel above, the Sinkhorn chain of position r in
// warp 0 of CTA r. 64 positions: 26 us, 45 with a cluster
// per position; 2048: 222, 442 with a CTA per position (the FP64 products alone 45, HBM 56: a cluster is a chain of phases, and two CTAs
// of 100 KB fit an SM).
constexpr int HCG_POS = 8, HCG_WARPS = 8, HCG_THREADS = HCG_WARPS * 32, HCG_M = 4, HCG_MIX = (2 + HCG_M) * HCG_M;
static_assert(HCG_POS == HCC_CTAS && HCG_POS == HCG_WARPS && HCG_MIX == 24, "a CTA of the cluster and a warp per position; three tiles of rows");
// streams of a position in shared memory: 4 more than a multiple of 32 words, so that two positions' pieces share a wavefront
__host__ __device__ constexpr int hcg_pitch(int W) { return (HCG_M * W + 31) / 32 * 32 + 4; }

__global__ void __cluster_dims__(HCC_CTAS, 1, 1) __launch_bounds__(HCG_THREADS, 2) hc_pre_group_kernel(const HcFused a, int T)
{
    extern __shared__ __align__(16) float hs[];                  // [8][pitch]: this CTA's columns of the positions' streams
    __shared__ double part[HCG_WARPS][HCG_MIX + 1][HCG_POS];     // the warps' parts of the dots, and of sum h^2
    __shared__ double mine[HCG_MIX + 1][HCG_POS], dots[HCG_MIX + 1][HCG_POS], mine_s2[HCG_POS];
    __shared__ double cbs[HCG_POS][HCG_M * HCG_M + HCG_M], pre[HCG_POS][HCG_M];
    __shared__ float mx[HCG_POS][HCG_MIX], factor[HCG_POS];
    constexpr int M = HCG_M, MM = M * M, MIX = HCG_MIX;
    pdl_trigger();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const uint32_t rank = cluster_cta_rank();
    const int E = a.E, ME = M * E, W = E / HCC_CTAS, d0 = (int)rank * W, P = hcg_pitch(W);
    const int t0 = blockIdx.y * HCG_POS, np = T - t0 < HCG_POS ? T - t0 : HCG_POS;
    const double eps = (double)a.hc_eps;

    float *ys = hs + HCG_POS * P;                                // [8][W]: the pending output
    float *norm = ys + HCG_POS * W;                              // [W]
    const int groups = (W + 127) / 128;                          // of 128 columns of a position: at most 8
    // The warp's blocks of 32 columns of a stream; the first two blocks' mixer rows are asked for before anything else.
    const int per = (W + 31) / 32, blocks = M * per;
    uint4 wn[2][3];
    auto load_rows = [&](uint4 (&w)[3], int blk) {
        const int c = (blk % per) * 32 + q * 8;
#pragma unroll
        for (int m = 0; m < 3; m++)
            w[m] = blk < blocks && c < W ? __ldg(reinterpret_cast<const uint4 *>(a.fn + (size_t)(m * 8 + g) * ME + (size_t)(blk / per) * E + d0 + c)) : make_uint4(0u, 0u, 0u, 0u);
    };
    load_rows(wn[0], warp);
    load_rows(wn[1], warp + HCG_WARPS);
    for (int i = tid * 4; i < W; i += HCG_THREADS * 4) cp_async16(norm + i, a.norm_w + d0 + i);
    pdl_wait();

    // ---- the streams, all of them on their way at once: 80 KB per SM and CTA, one round trip
    for (int i = tid; i < HCG_POS * M * (W / 4); i += HCG_THREADS) {
        const int p = i / (M * (W / 4)), r = i % (M * (W / 4)), k = r / (W / 4), c = (r % (W / 4)) * 4;
        float *dst = hs + p * P + k * W + c;
        if (p < np) cp_async16(dst, a.h + (size_t)(t0 + p) * ME + (size_t)k * E + d0 + c);
        else        *reinterpret_cast<float4 *>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (a.y) {
        for (int i = tid; i < np * (W / 4); i += HCG_THREADS) {
            const int p = i / (W / 4), c = (i % (W / 4)) * 4;
            cp_async16(ys + p * W + c, a.y + (size_t)(t0 + p) * E + d0 + c);
        }
        for (int i = tid; i < np * (MM + M); i += HCG_THREADS) {
            const int p = i / (MM + M), k = i % (MM + M);
            cbs[p][k] = (double)(k < MM ? __ldcg(a.comb + (size_t)(t0 + p) * MM + k) : __ldcg(a.post + (size_t)(t0 + p) * M + k - MM));
        }
    }
    cp_async_wait();
    __syncthreads();
    // ---- the pending hc_post of the previous site (src/core/glm53f_ops.c:612-625): warp p has position p
    if (a.y && warp < np) {
        const int p = warp;
        float *hp = hs + p * P, *ht = a.h + (size_t)(t0 + p) * ME + d0;
#pragma unroll 1
        for (int c = lane * 4; c < W; c += 128) {
            double hx[M], hy[M], hz[M], hw[M];
#pragma unroll
            for (int i = 0; i < M; i++) {
                const float4 v = *reinterpret_cast<const float4 *>(hp + i * W + c);
                hx[i] = (double)v.x; hy[i] = (double)v.y; hz[i] = (double)v.z; hw[i] = (double)v.w;
            }
            const float4 yv = *reinterpret_cast<const float4 *>(ys + p * W + c);
            const double yx = (double)yv.x, yy = (double)yv.y, yz = (double)yv.z, yw = (double)yv.w;
#pragma unroll 1
            for (int j = 0; j < M; j++) {                        // rolled: a launch runs this code once or twice, from a cold cache
                const double po = cbs[p][MM + j];
                double sx = po * yx, sy = po * yy, sz = po * yz, sw = po * yw;
#pragma unroll
                for (int i = 0; i < M; i++) {
                    const double cb = cbs[p][i * M + j];
                    sx = fma(cb, hx[i], sx); sy = fma(cb, hy[i], sy); sz = fma(cb, hz[i], sz); sw = fma(cb, hw[i], sw);
                }
                const float4 v = make_float4((float)sx, (float)sy, (float)sz, (float)sw);
                *reinterpret_cast<float4 *>(hp + j * W + c) = v;
                *reinterpret_cast<float4 *>(ht + (size_t)j * E + c) = v;
            }
        }
    }
    __syncthreads();

    // ---- mixer rows, and the sums of squares of the values that the lanes have as doubles then anyway
    {
        double acc[2][3][2] = {}, sq[4] = {};                    // (several sums each: a product waits for the one before it in its sum)
        uint32_t special = 0;                                    // an infinity or NaN among this lane's mixer elements
        auto multiply = [&](const uint4 (&wv)[3], int blk, auto widen) {
            const int c = (blk % per) * 32 + q * 8;
            float hv[8];
            if (c < W) {
                const float *hp = hs + g * P + (blk / per) * W + c;
                const float4 h0 = *reinterpret_cast<const float4 *>(hp), h1 = *reinterpret_cast<const float4 *>(hp + 4);
                hv[0] = h0.x; hv[1] = h0.y; hv[2] = h0.z; hv[3] = h0.w; hv[4] = h1.x; hv[5] = h1.y; hv[6] = h1.z; hv[7] = h1.w;
            } else {
#pragma unroll
                for (int k = 0; k < 8; k++) hv[k] = 0.f;
            }
            // Two steps' factors become doubles while the two before them are multiplied, in registers of their own: written as
            // plain expressions they shared a few registers and every product waited for the one before to have read them.
            double av[2][2][3], bv[2][2];
            auto take = [&](int j) {
#pragma unroll
                for (int k = 0; k < 2; k++) {
#pragma unroll
                    for (int m = 0; m < 3; m++) {
                        const uint32_t u = j == 0 ? wv[m].x : j == 1 ? wv[m].y : j == 2 ? wv[m].z : wv[m].w;
                        widen(av[j & 1][k][m], k ? u : u << 16);
                    }
                    asm volatile("cvt.f64.f32 %0, %1;" : "=d"(bv[j & 1][k]) : "f"(hv[2 * j + k]));
                }
            };
            take(0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j < 3) take(j + 1);
#pragma unroll
                for (int k = 0; k < 2; k++) {
#pragma unroll
                    for (int m = 0; m < 3; m++) mma_f64(acc[k][m], av[j & 1][k][m], bv[j & 1][k]);
                    sq[2 * (j & 1) + k] = fma(bv[j & 1][k], bv[j & 1][k], sq[2 * (j & 1) + k]);
                }
            }
        };
        auto step = [&](uint4 (&wv)[3], int blk) {
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const uint32_t u[4] = {wv[m].x, wv[m].y, wv[m].z, wv[m].w};
#pragma unroll
                for (int k = 0; k < 4; k++) special |= bf16_special(u[k]);
            }
            multiply(wv, blk, [](double &d, uint32_t u) {
                d = bf16_bits_f64(u);
            });
            load_rows(wv, blk + 2 * HCG_WARPS);
        };
#pragma unroll 1
        for (int blk = warp; blk < blocks; blk += 2 * HCG_WARPS) {
            step(wn[0], blk);
            if (blk + HCG_WARPS < blocks) step(wn[1], blk + HCG_WARPS);
        }
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
            for (int i = 0; i < 2; i++) acc[0][m][i] = (acc[0][m][i] + acc[1][m][i]) * BF16_BITS_SCALE;
        if (__any_sync(0xffffffffu, special)) {
            // those have no place among the scaled ones: the warp's products once more, element by element
            sq[0] = sq[1] = sq[2] = sq[3] = 0.0;
#pragma unroll
            for (int m = 0; m < 3; m++) acc[0][m][0] = acc[0][m][1] = acc[1][m][0] = acc[1][m][1] = 0.0;
#pragma unroll 1
            for (int blk = warp; blk < blocks; blk += HCG_WARPS) {
                uint4 wv[3];
                load_rows(wv, blk);
                multiply(wv, blk, [](double &d, uint32_t u) { d = (double)__uint_as_float(u & 0xffff0000u); });
            }
#pragma unroll
            for (int m = 0; m < 3; m++)
#pragma unroll
                for (int i = 0; i < 2; i++) acc[0][m][i] += acc[1][m][i];
        }
        double ss = (sq[0] + sq[1]) + (sq[2] + sq[3]);
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (q == 0) part[warp][MIX][g] = ss;
#pragma unroll
        for (int m = 0; m < 3; m++) { part[warp][m * 8 + g][2 * q] = acc[0][m][0]; part[warp][m * 8 + g][2 * q + 1] = acc[0][m][1]; }
    }
    __syncthreads();
    if (tid < (MIX + 1) * HCG_POS) {
        const int k = tid / HCG_POS, p = tid % HCG_POS;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < HCG_WARPS; w++) s += part[w][k][p];
        mine[k][p] = s;
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();

    // ---- every CTA: the positions' sums in CTA order, the norm factors, the gates
    if (tid < (MIX + 1) * HCG_POS) {
        double s = 0.0;
#pragma unroll
        for (uint32_t r = 0; r < HCC_CTAS; r++) s += ld_cluster_f64(&mine[0][0] + tid, r);
        (&dots[0][0])[tid] = s;
    }
    __syncthreads();
    if (tid < MIX * HCG_POS) {
        const int k = tid / HCG_POS, p = tid % HCG_POS;
        const float inv = (float)rsqrt_newton(dots[MIX][p] / (double)ME + (double)a.rms_eps);
        mx[p][k] = (float)(dots[k][p] * (double)inv);
    }
    __syncthreads();
    if (tid < HCG_POS * M) pre[tid / M][tid % M] = (double)sigmoid_host(mul_add_unfused(mx[tid / M][tid % M], a.scale[0], a.base[tid % M])) + eps;
    __syncthreads();
    if (warp == 0) {
        cluster_arrive();                                        // nothing of this warp goes into the sums of x^2
        if ((int)rank < np) {
            // position `rank`: row softmax + eps, then column / row normalisations (src/core/glm53f_ops.c:577-598)
            const float *m = mx[rank];
            const int t = t0 + (int)rank, el = lane < MM ? lane : 0, i = el / M, j = el % M, k = 2 * M + el;
            const double l = (double)mul_add_unfused(m[k], a.scale[2], a.base[k]);
            double top = -INFINITY;
#pragma unroll
            for (int jj = 0; jj < M; jj++) top = fmax(top, __shfl_sync(0xffffffffu, l, i * M + jj));
            const double ex = exp(l - top);
            double z = 0.0;
#pragma unroll
            for (int jj = 0; jj < M; jj++) z += __shfl_sync(0xffffffffu, ex, i * M + jj);
            const double v = sinkhorn_passes<M>(ex / z + eps, M, i, j, 2 * a.iters - 1, eps);
            if (lane < MM) a.comb[(size_t)t * MM + lane] = (float)v;
            if (lane >= MM && lane < MM + M) {
                const int i2 = lane - MM;
                a.post[(size_t)t * M + i2] = __fmul_rn(2.0f, sigmoid_host(mul_add_unfused(m[M + i2], a.scale[1], a.base[M + i2])));
            }
            __syncwarp();
        }
        cluster_wait();
    } else {
        // x[d] = sum_i pre[i] * h[i][d] in FP64 (src/core/glm53f_ops.c:603-607) for this CTA's columns of the eight positions
        // (a warp takes 128 columns of a position at a time)
        constexpr int NT = HCG_THREADS - 32;
        const int wt = tid - 32;
        for (int i = warp - 1; i < HCG_POS * groups; i += HCG_WARPS - 1) {
            const int p = i / groups, c = i % groups * 128 + lane * 4;
            float *hp = hs + p * P + c;
            double s2 = 0.0;
            if (c < W) {
                double x = 0.0, y = 0.0, z = 0.0, w = 0.0;
#pragma unroll
                for (int k = 0; k < M; k++) {
                    const float4 v = *reinterpret_cast<const float4 *>(hp + k * W);
                    const double pr = pre[p][k];
                    x += pr * (double)v.x; y += pr * (double)v.y; z += pr * (double)v.z; w += pr * (double)v.w;
                }
                const float4 xv = make_float4((float)x, (float)y, (float)z, (float)w);
                *reinterpret_cast<float4 *>(hp) = xv;            // (this thread alone reads these columns)
                x = (double)xv.x; y = (double)xv.y; z = (double)xv.z; w = (double)xv.w;
                s2 = fma(x, x, y * y) + fma(z, z, w * w);
            }
            s2 = warp_sum(s2);
            if (lane == 0) (&part[0][0][0])[i] = s2;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        if (wt < HCG_POS) {
            double s = 0.0;
            for (int i = 0; i < groups; i++) s += (&part[0][0][0])[wt * groups + i];
            mine_s2[wt] = s;
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        // the sub-blocks' inputs: RMSNorm(x) * w (:473-480)
        if (wt < HCG_POS) {
            double tot = 0.0;
#pragma unroll
            for (uint32_t r = 0; r < HCC_CTAS; r++) tot += ld_cluster_f64(&mine_s2[wt], r);
            factor[wt] = (float)rsqrt_newton(tot / (double)E + (double)a.rms_eps);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        for (int i = warp - 1; i < np * groups; i += HCG_WARPS - 1) {
            const int p = i / groups, c = i % groups * 128 + lane * 4;
            if (c < W) {
                const float4 v = *reinterpret_cast<const float4 *>(hs + p * P + c), w = *reinterpret_cast<const float4 *>(norm + c);
                const float f = factor[p];
                *reinterpret_cast<float4 *>(a.xn + (size_t)(t0 + p) * E + d0 + c) =
                    make_float4(__fmul_rn(w.x, __fmul_rn(v.x, f)), __fmul_rn(w.y, __fmul_rn(v.y, f)), __fmul_rn(w.z, __fmul_rn(v.z, f)), __fmul_rn(w.w, __fmul_rn(v.w, f)));
            }
        }
    }
    // no CTA leaves while another may still read its shared memory
    cluster_arrive();
    cluster_wait();
}

// From here on eight positions to a cluster (hc_pre_group_kernel) are as fast as a cluster for each (hc_pre_one_kernel), or faster. Alone, 5 us of launch
// included, a site takes 24.6 us with the former at any of these sizes and with the latter 14.4 up to 15 positions, which all run at once, 24.6 from 16
// on, 32.8 for 32, 51 for 64; with the streams' expansion 26.7 against 18.5 for 15, 26.8 for 16, 28.7 for 18, 39 for 32. A KDA + MoE layer of 12
// sequences 280 us against 260, of 16: 292.4 and 289.8, of 18: 304 both, of 32: 347 and 366.
constexpr int HCG_MIN_T = 17;

static bool hc_pre_cluster_takes(int M, int E)
{
    const int W = E / HCC_CTAS;
    return E % (HCC_CTAS * 8) == 0 && W <= HCC_MAX_W && M * W <= HCC_MAX_HS && M * M <= 32 && M <= G5B_MAX_HC;
}

bool hc_pre_fused_supported(const HcW &w, int M, int E)
{
    if (w.fn.dt != DT_BF16) return false;
    if (hc_pre_cluster_takes(M, E)) return true;
    return E <= HCF_MAX_E && E % (HCF_SLICES * 8) == 0 && M <= G5B_MAX_HC &&
           M * (E / HCF_SLICES) <= HCF_MAX_E * G5B_MAX_HC / HCF_SLICES && E / HCF_SLICES <= HC_THREADS;
}

void hc_pre_fused(cudaStream_t st, float *xn, float *post, float *comb, float *h, const float *y_pending,
                  const HcW &w, const float *norm_w, double *part, int *counters, int T, int M, int E, int iters,
                  float hc_eps, float rms_eps)
{
    HcFused a{xn, post, comb, h, y_pending, static_cast<const uint16_t *>(w.fn.w), w.base, w.scale, norm_w, part,
              counters, M, E, iters, hc_eps, rms_eps};
    if (T >= HCG_MIN_T && M == HCG_M && hc_pre_cluster_takes(M, E)) {
        const size_t smem = ((size_t)HCG_POS * (hcg_pitch(E / HCC_CTAS) + E / HCC_CTAS) + E / HCC_CTAS) * sizeof(float);
        static SmemGrant grant;
        if (dev_opt_in_smem((const void *)hc_pre_group_kernel, smem + (20 << 10), grant)) {
            G5B_LAUNCH(hc_pre_group_kernel, dim3(HCC_CTAS, (T + HCG_POS - 1) / HCG_POS), HCG_THREADS, smem, st, a, T);
            return;
        }
    }
    if (M == HCO_M && hc_pre_cluster_takes(M, E)) {
        const size_t smem = hco_smem(E / HCC_CTAS);
        static SmemGrant grant;
        if (dev_opt_in_smem((const void *)hc_pre_one_kernel, smem + (8 << 10), grant)) {
            G5B_LAUNCH_PDL(hc_pre_one_kernel, dim3(HCC_CTAS, T), dim3(HCC_THREADS), smem, st, a);
            return;
        }
    }
    if (hc_pre_cluster_takes(M, E)) G5B_LAUNCH_PDL(hc_pre_cluster_kernel, dim3(HCC_CTAS, T), dim3(HCC_THREADS), 0, st, a);
    else                            G5B_LAUNCH(hc_pre_fused_kernel, dim3(HCF_SLICES, T), HC_THREADS, 0, st, a);
}

// h'[j][d] = post[j]*y[d] + sum_i comb[i][j]*h[i][d] in FP64, in place: a thread owns column d of
// every stream (src/core/glm53f_ops.c:612-625; note comb is used transposed).
__global__ void hc_post_kernel(float *h, const float *y, const float *post, const float *comb, int M, int E)
{
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.y;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= E) return;
    float *ht = h + (size_t)t * M * E;
    double hv[G5B_MAX_HC];
    for (int i = 0; i < M; i++) hv[i] = (double)ht[(size_t)i * E + d];
    const double yv = (double)y[(size_t)t * E + d];
    const float *cb = comb + (size_t)t * M * M, *po = post + (size_t)t * M;
    for (int j = 0; j < M; j++) {
        double s = (double)po[j] * yv;
        for (int i = 0; i < M; i++) s += (double)cb[i * M + j] * hv[i];
        ht[(size_t)j * E + d] = (float)s;
    }
}

void hc_post(cudaStream_t st, float *h, const float *y, const float *post, const float *comb, int T,
             int M, int E)
{
    G5B_LAUNCH_PDL(hc_post_kernel, dim3((E + 127) / 128, T), dim3(128), 0, st, h, y, post, comb, M, E);
}

}  // namespace g5b
