// kda.cu - the gated delta-rule linear attention step (KDA), everything between the input
// projections and the output projection.
//
// Reference: glm53f_kda_layer and kda_step (src/core/glm53f_ops.c:630-755). Its device form was
// nine launches per layer and token (three k_shortconv, k_kda_prep, k_kda_decay, k_kda_read,
// k_kda_write, k_kda_out, k_onorm_gate; src/gpu/glm53f_gpu_kernels.cu:243-450) that passed over
// the 64 KB per-head state four times. Here it is short convolution + SiLU of q/k/v with the
// carried history, L2 norm of q and k, beta and the per-channel decay, the recurrence, and the
// gated per-head RMSNorm of the output, with the state in registers, read once and written once
// per call however many tokens the call carries:
//   one position of one sequence, head_dim 64 or 128   kda_step_kernel, a cluster of CTAs per head
//   one position of each of several sequences          kda_each_kernel, a CTA per head and sequence
//   several positions                                  kda_prep_kernel, kda_scan_kernel, kda_out_kernel
//   other head sizes                                   kda_core_kernel, a CTA per head, the state in memory
//
// The one-position and the any-size kernel keep the reference's order of FP32 operations (decay row
// i, u_j += S_ij k_i, S_ij += k_i u_j, o_j += S_ij q_i, ascending i, products and sums rounded
// separately) and its exactly rounded exponential. The kernels over many rows do not: products are
// fused, sums taken in parts, o from the decayed state, exponentials within 0.53 units (expf_near).
#include "common.cuh"
#include "kernels.h"

namespace g5b {

struct KdaArgs {
    float *o;
    const float *q, *k, *v, *z, *braw, *gb;
    const float *q_conv, *k_conv, *v_conv, *A_log, *dt_bias, *o_norm;
    float *state;
    int T, H, D, K;
    int head0;                    // the grid covers heads head0 .. head0 + gridDim.x - 1 of the H heads
    float gate_lb, rms_eps;
    size_t seq_stride;            // floats between the states of consecutive sequences (grid.y > 1:
                                  // CTA (h, s) advances sequence s by the T positions at rows s*T ...)
    const uint16_t *f_b, *g_b;    // optional (T == 1): z and gb are computed here from lrf / lrg
    const float *lrf, *lrg;
    float *snap;                  // optional: a second state buffer (same layout) that receives the state as it
    int snap_after;               // is after position snap_after of the call (speculative decode keeps it to fall back on)
};

// conv + SiLU of one channel at one position; `past` holds K-1 previous inputs, oldest first.
__device__ __forceinline__ float conv_step(float cur, const float *w, float *past, int K)
{
    const int hist = K - 1;
    float acc = __fmul_rn(w[hist], cur);
    for (int j = 0; j < hist; j++) acc = mul_add_unfused(w[j], past[j], acc);
    for (int j = 0; j + 1 < hist; j++) past[j] = past[j + 1];
    if (hist > 0) past[hist - 1] = cur;
    return __fmul_rn(acc, sigmoid_host(acc));
}

// Any head_dim up to 512: one CTA per head, a thread per column, the state column re-read from memory.
__global__ void __launch_bounds__(512) kda_core_kernel(const KdaArgs a)
{
    __shared__ float sq[512], sk[512], sal[512];
    __shared__ double red[32];
    const int h = a.head0 + blockIdx.x, d = threadIdx.x;
    const int D = a.D, P = a.H * D, K = a.K, hist = K - 1;
    const bool live = d < D;
    const int ch = h * D + (live ? d : 0);
    float *state = a.state + (size_t)blockIdx.y * a.seq_stride;
    float *S = state + (size_t)h * D * D;
    float *cs = state + (size_t)a.H * D * D;
    const int row0 = blockIdx.y * a.T;                       // first activation row of this sequence

    float pq[16], pk[16], pv[16], wq[17], wk[17], wv[17];
    for (int j = 0; j < hist; j++) {
        pq[j] = cs[(size_t)ch * hist + j];
        pk[j] = cs[(size_t)P * hist + (size_t)ch * hist + j];
        pv[j] = cs[(size_t)2 * P * hist + (size_t)ch * hist + j];
    }
    for (int j = 0; j < K; j++) {
        wq[j] = a.q_conv[(size_t)ch * K + j];
        wk[j] = a.k_conv[(size_t)ch * K + j];
        wv[j] = a.v_conv[(size_t)ch * K + j];
    }
    const float ea = expf_host(a.A_log[h]);
    const float dtb = a.dt_bias[ch], onw = a.o_norm[live ? d : 0];
    const float qscale = 1.0f / sqrtf((float)D);

    for (int t = 0; t < a.T; t++) {
        const size_t off = (size_t)(row0 + t) * P + ch;
        float qv = 0.f, kv = 0.f, vv = 0.f;
        if (live) {
            qv = conv_step(a.q[off], wq, pq, K);
            kv = conv_step(a.k[off], wk, pk, K);
            vv = conv_step(a.v[off], wv, pv, K);
        }
        // l2norm: divide by sqrt(sum of squares + 1e-6), sums in FP64 (glm53f_ops.c:661-667)
        const double qq = block_sum(live ? (double)qv * (double)qv : 0.0, red);
        const double kk = block_sum(live ? (double)kv * (double)kv : 0.0, red);
        const float qinv = (float)(1.0 / sqrt(qq + (double)1e-6f));
        const float kinv = (float)(1.0 / sqrt(kk + (double)1e-6f));
        const float beta = sigmoid_host(a.braw[(size_t)(row0 + t) * a.H + h]);
        __syncthreads();
        if (live) {
            sq[d] = __fmul_rn(__fmul_rn(qv, qinv), qscale);
            sk[d] = __fmul_rn(kv, kinv);
            const float g = __fmul_rn(a.gate_lb, sigmoid_host(__fmul_rn(ea, __fadd_rn(a.z[off], dtb))));
            sal[d] = expf_host(g);
        }
        __syncthreads();

        float ov = 0.f;
        if (live) {
            float u = 0.f;
            for (int i = 0; i < D; i++) {
                const float s = __fmul_rn(S[(size_t)i * D + d], sal[i]);
                S[(size_t)i * D + d] = s;
                u = __fadd_rn(u, __fmul_rn(s, sk[i]));
            }
            u = __fmul_rn(__fsub_rn(vv, u), beta);
            for (int i = 0; i < D; i++) {
                const float s = __fadd_rn(S[(size_t)i * D + d], __fmul_rn(sk[i], u));
                S[(size_t)i * D + d] = s;
                ov = __fadd_rn(ov, __fmul_rn(s, sq[i]));
            }
        }
        // per-head RMSNorm with weight, then the sigmoid output gate (glm53f_ops.c:748-752)
        const double oo = block_sum(live ? (double)ov * (double)ov : 0.0, red);
        if (live) {
            const float inv = (float)(1.0 / sqrt(oo / (double)D + (double)a.rms_eps));
            const float n = __fmul_rn(onw, __fmul_rn(ov, inv));
            a.o[off] = __fmul_rn(n, sigmoid_host(a.gb[off]));
        }
        if (a.snap && t == a.snap_after && live) {
            float *sn = a.snap + (size_t)blockIdx.y * a.seq_stride;
            float *Sn = sn + (size_t)h * D * D, *cn = sn + (size_t)a.H * D * D;
            for (int i = 0; i < D; i++) Sn[(size_t)i * D + d] = S[(size_t)i * D + d];
            for (int j = 0; j < hist; j++) {
                cn[(size_t)ch * hist + j] = pq[j];
                cn[(size_t)P * hist + (size_t)ch * hist + j] = pk[j];
                cn[(size_t)2 * P * hist + (size_t)ch * hist + j] = pv[j];
            }
        }
    }

    if (live) {
        for (int j = 0; j < hist; j++) {
            cs[(size_t)ch * hist + j] = pq[j];
            cs[(size_t)P * hist + (size_t)ch * hist + j] = pk[j];
            cs[(size_t)2 * P * hist + (size_t)ch * hist + j] = pv[j];
        }
    }
}

// Several positions of one sequence (prompts, the two-position pass of speculative decode), or, with a convolution of another
// width than four, one position each of many sequences. What does not depend on the previous position - three convolutions with SiLU, the gate, the
// l2norm sums - runs for all positions at once (kda_prep_kernel); the state update
// alone walks the positions (kda_scan_kernel); the output's norm and gate follow for all positions at once
// (kda_out_kernel).
//
// The scan: the columns of the state are independent of each other, so a head's 128 are dealt to CTAs, and a column's
// rows to PARTS lanes, in registers. Both products of a position are taken with the decayed state, o = q.(aS) + (q.k) u,
// so that one round of shuffles serves them and the next position waits for u alone; the positions' vectors arrive by
// asynchronous copies, 8 positions ahead. Many positions are bound by that chain and by shared-memory wavefronts (vector
// loads and shuffles, 48 % of what there could be): eight lanes to a column, one transposed sum for its two values. 2048 positions of
// 64 heads: 5.2 ms with a thread per column, 1.05 with two columns to a lane of half as many warps, now 1.00. One position of
// many sequences is bound by the state's memory traffic: four lanes to a column read it in whole 32-byte sectors.
// The sums of a column are taken in parts with four accumulators each, products fused.
struct KdaPrep {
    KdaArgs a;
    float *qn, *kn, *vn, *al, *beta;        // [rows][P] normalised q (scaled), normalised k, v, exp(gate); [rows][H][2] beta, q.k
    int heads;                              // of this launch
};

// A CTA takes KDA_TILE positions of one head, in two passes: a thread per channel of q, k, v and the gate walks the positions, four at a
// time and two to an instruction, its weights and the last K - 1 inputs in registers; then a warp per position takes the norms of q and k
// from shared memory. KW: the width of the convolution, 0 for one known at run time only. (q and k are wanted twice, by channel and by
// position; a warp that kept all of a position's vectors took eight positions one after the other, each 17 KB of instructions and a chain
// of seventeen divisions with their branches: 5 us a position however few there were.) Bound by the instructions of the exponentials and
// reciprocals, 16 of them a channel; its memory traffic would take 10 us for 256 positions of 64 heads. With inputs that come from memory:
// 2 positions 15 -> 5 us, 8: 41 -> 6, 50: 41 -> 12, 200: 52 -> 27, 256: 52 -> 31.
constexpr int KDA_TILE = 16;
template <int DS, int KW>
__global__ void __launch_bounds__(4 * DS) kda_prep_kernel(const KdaPrep p)
{
    pdl_trigger();
    const KdaArgs &a = p.a;
    constexpr int D = DS, C = DS / 32, U = 4;               // channels per lane of the second pass; positions of a step of the first
    struct alignas(4 * C) Vec { float v[C]; };
    __shared__ __align__(16) float xs[4][KDA_TILE][D];       // the inputs; q's and k's give way to the convolutions' results
    const int tiles = (a.T + KDA_TILE - 1) / KDA_TILE, seq = blockIdx.y / tiles, t0 = (blockIdx.y - seq * tiles) * KDA_TILE;
    const int h = a.head0 + blockIdx.x, P = a.H * D, K = KW ? KW : a.K, hist = K - 1, nt = a.T - t0 < KDA_TILE ? a.T - t0 : KDA_TILE;
    const int c = threadIdx.x / D, d = threadIdx.x % D, ch = h * D + d;                 // (c: the same for a whole warp)
    const size_t first = ((size_t)seq * a.T + t0) * P + ch;
    const float *x = (c == 0 ? a.q : c == 1 ? a.k : c == 2 ? a.v : a.z) + first;
    const float *wp = (c == 0 ? a.q_conv : c == 1 ? a.k_conv : a.v_conv) + (size_t)ch * K;
    float w[KW ? KW : 1];
    if (KW && c < 3)
#pragma unroll
        for (int j = 0; j < KW; j++) w[j] = wp[j];
    const float dt = c == 3 ? a.dt_bias[ch] : 0.f, ea = c == 3 ? expf_host(a.A_log[h]) : 0.f;
    pdl_wait();
    {
        const float *row = x - d + d % (D / 4) * 4;            // D / 4 threads to a row of 16-byte pieces
#pragma unroll
        for (int t = d / (D / 4); t < KDA_TILE; t += 4)
            if (t < nt) cp_async16(&xs[c][t][d % (D / 4) * 4], row + (size_t)t * P);
    }
    // the input before position tt of the tile: earlier rows of this call, or the carried history (oldest first)
    const float *cs = a.state + (size_t)seq * a.seq_stride + (size_t)a.H * D * D + (size_t)c * P * hist + (size_t)ch * hist;
    auto before = [&](int tt) { return t0 + tt >= 0 ? x[(ptrdiff_t)tt * P] : cs[hist + t0 + tt]; };
    float past[KW ? KW - 1 + U : 1];
    if (c < 3)
#pragma unroll
        for (int j = 0; j + 1 < KW; j++) past[j] = before(j - (KW - 1));
    cp_async_wait();
    __syncthreads();
    if (c == 3) {
#pragma unroll 1
        for (int t = 0; t < nt; t += U) {
            float g[U];
#pragma unroll
            for (int j = 0; j < U; j++) g[j] = __fmul_rn(ea, __fadd_rn(xs[3][t + j][d], dt));
#pragma unroll
            for (int j = 0; j < U; j += 2) {
                sigmoid_near2(g[j], g[j + 1], g[j], g[j + 1]);
                expf_near2(__fmul_rn(a.gate_lb, g[j]), __fmul_rn(a.gate_lb, g[j + 1]), g[j], g[j + 1]);
            }
#pragma unroll
            for (int j = 0; j < U; j++)
                if (t + j < nt) p.al[first + (size_t)(t + j) * P] = g[j];
        }
    } else {
#pragma unroll 1
        for (int t = 0; t < nt; t += U) {
            float y[U];
            if constexpr (KW != 0) {
#pragma unroll
                for (int j = 0; j < U; j++) past[KW - 1 + j] = xs[c][t + j][d];
#pragma unroll
                for (int j = 0; j < U; j++) {
                    y[j] = __fmul_rn(w[KW - 1], past[KW - 1 + j]);
#pragma unroll
                    for (int i = 0; i + 1 < KW; i++) y[j] = mul_add_unfused(w[i], past[j + i], y[j]);
                }
#pragma unroll
                for (int j = 0; j + 1 < KW; j++) past[j] = past[j + U];
            } else {
                for (int j = 0; j < U; j++) {
                    const int tt = t + j < nt ? t + j : nt - 1;
                    float v = __fmul_rn(wp[hist], x[(size_t)tt * P]);
                    for (int i = 0; i < hist; i++) v = mul_add_unfused(wp[i], before(tt - hist + i), v);
                    y[j] = v;
                }
            }
            float s[U];
#pragma unroll
            for (int j = 0; j < U; j += 2) sigmoid_near2(y[j], y[j + 1], s[j], s[j + 1]);
#pragma unroll
            for (int j = 0; j < U; j++)
                if (t + j < nt) {
                    const float v = __fmul_rn(y[j], s[j]);
                    if (c < 2) xs[c][t + j][d] = v;
                    else p.vn[first + (size_t)(t + j) * P] = v;
                }
        }
    }
    __syncthreads();
    // l2norm: divide by sqrt(sum of squares + 1e-6), sums in FP64 (glm53f_ops.c:661-667); one half of the warp sums q's, the other k's
    const int lane = threadIdx.x & 31;
    const bool upper = lane & 16;
    const float qscale = 1.0f / sqrtf((float)D);
    for (int t = threadIdx.x >> 5; t < nt; t += D / 8) {
        const size_t rr = (size_t)seq * a.T + t0 + t;
        const float braw = a.braw[rr * a.H + h];
        const Vec yq = *reinterpret_cast<const Vec *>(&xs[0][t][lane * C]), yk = *reinterpret_cast<const Vec *>(&xs[1][t][lane * C]);
        double qq = 0.0, kk = 0.0, qk = 0.0;
#pragma unroll
        for (int i = 0; i < C; i++) {
            qq = fma((double)yq.v[i], (double)yq.v[i], qq);
            kk = fma((double)yk.v[i], (double)yk.v[i], kk);
        }
        double sum = (upper ? kk : qq) + __shfl_xor_sync(0xffffffffu, upper ? qq : kk, 16);
#pragma unroll
        for (int m = 8; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        const float inv = (float)rsqrt_newton(sum + (double)1e-6f), other = __shfl_xor_sync(0xffffffffu, inv, 16);
        const float qinv = upper ? other : inv, kinv = upper ? inv : other;
        Vec qn, kn;
#pragma unroll
        for (int i = 0; i < C; i++) {
            qn.v[i] = __fmul_rn(__fmul_rn(yq.v[i], qinv), qscale);
            kn.v[i] = __fmul_rn(yk.v[i], kinv);
            qk = fma((double)qn.v[i], (double)kn.v[i], qk);
        }
        qk = warp_sum(qk);
        *reinterpret_cast<Vec *>(p.qn + rr * P + h * D + lane * C) = qn;
        *reinterpret_cast<Vec *>(p.kn + rr * P + h * D + lane * C) = kn;
        const float beta = sigmoid_near(braw);
        if (lane == 0) *reinterpret_cast<float2 *>(p.beta + (rr * a.H + h) * 2) = make_float2(beta, (float)qk);
    }
}

constexpr int KDA_TB = 8;
template <int DS, int PARTS, int CPL, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) kda_scan_kernel(const KdaPrep p)
{
    pdl_trigger();
    constexpr int D = DS, R = DS / PARTS, PART = R + 4, LC = 32 / PARTS;    // rows per lane; their stride in shared memory (other banks); lanes side by side
    constexpr int COLS = LC * CPL * WARPS, NT = 32 * WARPS;                // columns of the CTA
    __shared__ __align__(16) float vec[2][KDA_TB][3][PARTS * PART];        // decay, k, q
    __shared__ __align__(16) float sv[2][KDA_TB][COLS];
    __shared__ float2 sb[2][KDA_TB];
    const KdaArgs &a = p.a;
    const int groups = D / COLS, hl = blockIdx.x / groups, h = a.head0 + hl, col0 = (blockIdx.x % groups) * COLS, seq = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane / LC, cc = warp * LC * CPL + (lane % LC) * CPL, col = col0 + cc;
    const int P = a.H * D, hist = a.K - 1, row0 = seq * a.T;
    float *state = a.state + (size_t)seq * a.seq_stride;
    float *S = state + (size_t)h * D * D + (size_t)part * R * D + col;
    pdl_wait();
    auto fetch = [&](int t0, int buf) {
        const int nt = a.T - t0 < KDA_TB ? a.T - t0 : KDA_TB;
        constexpr int Q = D / 4;                                     // 16-byte pieces of a vector
        for (int i = threadIdx.x; i < nt * 3 * Q; i += NT) {
            const int j = i / (3 * Q), w = (i / Q) % 3, c = i % Q;
            const float *src = (w == 0 ? p.al : w == 1 ? p.kn : p.qn) + (size_t)(row0 + t0 + j) * P + h * D + c * 4;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&vec[buf][j][w][(c * 4 / R) * PART + (c * 4) % R]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        }
        for (int i = threadIdx.x; i < nt * (COLS / 4); i += NT) {
            const int j = i / (COLS / 4), c = i % (COLS / 4);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sv[buf][j][c * 4]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p.vn + (size_t)(row0 + t0 + j) * P + h * D + col0 + c * 4) : "memory");
        }
        if (threadIdx.x < nt) sb[buf][threadIdx.x] = __ldcg(reinterpret_cast<const float2 *>(p.beta) + (size_t)(row0 + t0 + threadIdx.x) * a.H + h);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    F2 s[CPL][R / 2];
#pragma unroll
    for (int c = 0; c < CPL; c++)
#pragma unroll
        for (int i = 0; i < R / 2; i++) s[c][i] = f2(S[(size_t)(2 * i) * D + c], S[(size_t)(2 * i + 1) * D + c]);
    auto put_state = [&](float *dst) {
#pragma unroll
        for (int c = 0; c < CPL; c++)
#pragma unroll
            for (int i = 0; i < R / 2; i++) {
                float x, y;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(s[c][i].v));
                dst[(size_t)(2 * i) * D + c] = x; dst[(size_t)(2 * i + 1) * D + c] = y;
            }
    };
    int buf = 0;
    for (int t0 = 0; t0 < a.T; t0 += KDA_TB, buf ^= 1) {
        const int nt = a.T - t0 < KDA_TB ? a.T - t0 : KDA_TB;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();                                             // this group's vectors are there, the other buffer is free
        if (t0 + KDA_TB < a.T) fetch(t0 + KDA_TB, buf ^ 1);
#pragma unroll 2
        for (int j = 0; j < nt; j++) {
            const float4 *al4 = reinterpret_cast<const float4 *>(&vec[buf][j][0][part * PART]), *k4 = reinterpret_cast<const float4 *>(&vec[buf][j][1][part * PART]),
                         *q4 = reinterpret_cast<const float4 *>(&vec[buf][j][2][part * PART]);
            const F2 zero = f2(0.f, 0.f);
            F2 u0[CPL], u1[CPL], o0[CPL], o1[CPL], k[R / 2];
#pragma unroll
            for (int c = 0; c < CPL; c++) u0[c] = u1[c] = o0[c] = o1[c] = zero;
#pragma unroll
            for (int i = 0; i < R / 4; i++) {
                const float4 al = al4[i], kk = k4[i], q = q4[i];
                k[2 * i] = f2(kk.x, kk.y); k[2 * i + 1] = f2(kk.z, kk.w);
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    s[c][2 * i] = f2_mul(s[c][2 * i], f2(al.x, al.y));
                    s[c][2 * i + 1] = f2_mul(s[c][2 * i + 1], f2(al.z, al.w));
                    u0[c] = f2_fma(s[c][2 * i], k[2 * i], u0[c]);
                    u1[c] = f2_fma(s[c][2 * i + 1], k[2 * i + 1], u1[c]);
                    o0[c] = f2_fma(s[c][2 * i], f2(q.x, q.y), o0[c]);
                    o1[c] = f2_fma(s[c][2 * i + 1], f2(q.z, q.w), o1[c]);
                }
            }
            const float2 b = sb[buf][j];
            float *out = a.o + (size_t)(row0 + t0 + j) * P + h * D + col;
            float u[CPL];
            if constexpr (PARTS == 8) {
                // two sums over the eight lanes of a column: half of them go on with u, half with o
                const float x = __fadd_rn(f2_sum(u0[0]), f2_sum(u1[0])), y = __fadd_rn(f2_sum(o0[0]), f2_sum(o1[0]));
                const bool is_o = lane & 16;
                float v = __fadd_rn(is_o ? y : x, __shfl_xor_sync(0xffffffffu, is_o ? x : y, 16));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
                u[0] = __fmul_rn(__fsub_rn(sv[buf][j][cc], __shfl_sync(0xffffffffu, v, lane & 3)), b.x);
                if ((lane & 28) == 16) *out = __fmaf_rn(b.y, u[0], v);
            } else {
                float o = __fadd_rn(f2_sum(o0[0]), f2_sum(o1[0]));
                u[0] = __fadd_rn(f2_sum(u0[0]), f2_sum(u1[0]));
#pragma unroll
                for (int m = LC; m < 32; m <<= 1) {
                    u[0] = __fadd_rn(u[0], __shfl_xor_sync(0xffffffffu, u[0], m));
                    o = __fadd_rn(o, __shfl_xor_sync(0xffffffffu, o, m));
                }
                u[0] = __fmul_rn(__fsub_rn(sv[buf][j][cc], u[0]), b.x);
                if (part == 0) *out = __fmaf_rn(b.y, u[0], o);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const F2 uu = f2(u[c], u[c]);
#pragma unroll
                for (int i = 0; i < R / 2; i++) s[c][i] = f2_fma(k[i], uu, s[c][i]);
            }
            if (a.snap && t0 + j == a.snap_after) put_state(a.snap + (size_t)h * D * D + (size_t)part * R * D + col);
        }
    }
    put_state(S);
    // the convolution histories of this CTA's channels: the K - 1 inputs before position `upto` (the call's rows, older
    // ones from the old history, which the preparation has read)
    float *cs = state + (size_t)a.H * D * D;
    auto histories = [&](float *dst, int upto) {
        const float *src[3] = {a.q, a.k, a.v};
        for (int i = threadIdx.x; i < 3 * COLS; i += NT) {
            const int w = i / COLS, ch = h * D + col0 + i % COLS;
            float nv[16];
            for (int j = 0; j < hist; j++) {
                const int tt = upto - hist + j;
                nv[j] = tt >= 0 ? src[w][(size_t)(row0 + tt) * P + ch] : cs[(size_t)w * P * hist + (size_t)ch * hist + (hist + tt)];
            }
            for (int j = 0; j < hist; j++) dst[(size_t)w * P * hist + (size_t)ch * hist + j] = nv[j];
        }
    };
    if (a.snap && a.snap_after + 1 <= a.T) histories(a.snap + (size_t)a.H * D * D, a.snap_after + 1);   // before cs changes (each channel by one thread)
    histories(cs, a.T);
}

// Per-head RMSNorm with weight, then the sigmoid output gate (glm53f_ops.c:748-752), in place; a warp per row and head.
template <int DS>
__global__ void __launch_bounds__(256) kda_out_kernel(const KdaArgs a, int heads)
{
    pdl_trigger();
    constexpr int D = DS, C = DS / 32;
    const int lane = threadIdx.x & 31, hl = blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_wait();
    if (hl >= heads) return;
    const int h = a.head0 + hl;
    const size_t off = (size_t)blockIdx.y * a.H * D + h * D + lane * C;
    float o[C];
    double oo = 0.0;
#pragma unroll
    for (int i = 0; i < C; i++) { o[i] = a.o[off + i]; oo += (double)o[i] * (double)o[i]; }
    oo = warp_sum(oo);
    const float inv = (float)rsqrt_newton(oo / (double)D + (double)a.rms_eps);
#pragma unroll
    for (int i = 0; i < C; i++)
        a.o[off + i] = __fmul_rn(__fmul_rn(a.o_norm[lane * C + i], __fmul_rn(o[i], inv)), sigmoid_near(a.gb[off + i]));
}

// One position of each of several sequences, convolutions of width 4: a CTA takes a head of a sequence from its inputs to its gated output.
// Bound by the states' way from HBM and back (64 sequences of 64 heads: 0.54 GB, 82 us). The three kernels above, of which the scan
// read a state in pieces of 32 bytes, took 171 us a layer (27 + 139 + 5); here a thread holds two columns of 32 rows, asked for
// before anything else, so that 128 KB are on their way to an SM while the convolutions, norms and gates of the two CTAs on it are
// computed. Arithmetic as above: products fused, sums in parts of eight rows. 64 sequences:
// 111 us, 7: 17.3 (34 before); a step of 64 sequences over eight layers 6.80 -> 6.39 ms.
template <int DS>
__global__ void __launch_bounds__(256, 2) kda_each_kernel(const KdaArgs a)
{
    pdl_trigger();
    constexpr int D = DS, KW = 4, HIST = KW - 1, CP = D / 2, RG = 256 / CP, R = D / RG, CH = (3 * D + 255) / 256;
    __shared__ __align__(16) float sal[D], sk[D], sq[D], raw[3 * D];
    __shared__ __align__(16) F2 us[RG][CP], os[RG][CP];
    __shared__ double red[8][3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cp = tid % CP, rg = tid / CP, h = a.head0 + blockIdx.x, seq = blockIdx.y, P = a.H * D;
    float *state = a.state + (size_t)seq * a.seq_stride, *cs = state + (size_t)a.H * D * D;
    unsigned long long *S = reinterpret_cast<unsigned long long *>(state + (size_t)h * D * D + (size_t)rg * R * D + 2 * cp);
    F2 s[R];
#pragma unroll
    for (int i = 0; i < R; i++) s[i].v = __ldcs(S + (size_t)i * (D / 2));
    float w[CH][KW], past[CH][HIST];
#pragma unroll
    for (int n = 0; n < CH; n++) {
        const int i = tid + 256 * n, c = i / D, ch = h * D + i % D;
        if (i < 3 * D) {
            const float *wp = (c == 0 ? a.q_conv : c == 1 ? a.k_conv : a.v_conv) + (size_t)ch * KW, *hp = cs + (size_t)c * P * HIST + (size_t)ch * HIST;
#pragma unroll
            for (int j = 0; j < KW; j++) w[n][j] = wp[j];
#pragma unroll
            for (int j = 0; j < HIST; j++) past[n][j] = hp[j];
        }
    }
    const float dt = tid < D ? a.dt_bias[h * D + tid] : 0.f, onw = tid < D ? a.o_norm[tid] : 0.f;
    const float ea = expf_host(a.A_log[h]), qscale = 1.0f / sqrtf((float)D);
    pdl_wait();
    const size_t off = (size_t)seq * P + h * D;
    const float z = tid < D ? a.z[off + tid] : 0.f, gate = tid < D ? a.gb[off + tid] : 0.f, braw = a.braw[(size_t)seq * a.H + h];
#pragma unroll
    for (int n = 0; n < CH; n++) {
        const int i = tid + 256 * n, c = i / D, d = i % D;
        if (i < 3 * D) {
            const float now = (c == 0 ? a.q : c == 1 ? a.k : a.v)[off + d];
            float y = __fmul_rn(w[n][HIST], now);
#pragma unroll
            for (int j = 0; j < HIST; j++) y = mul_add_unfused(w[n][j], past[n][j], y);
            raw[i] = __fmul_rn(y, sigmoid_near(y));
            float *hp = cs + (size_t)c * P * HIST + (size_t)(h * D + d) * HIST;      // (each channel by one thread)
            hp[0] = past[n][1]; hp[1] = past[n][2]; hp[2] = now;
        }
    }
    __syncthreads();
    // l2norm: divide by sqrt(sum of squares + 1e-6), sums in FP64 (glm53f_ops.c:661-667)
    const float yq = tid < D ? raw[tid] : 0.f, yk = tid < D ? raw[D + tid] : 0.f;
    {
        const double qq = warp_sum((double)yq * (double)yq), kk = warp_sum((double)yk * (double)yk);
        if (lane == 0) { red[warp][0] = qq; red[warp][1] = kk; }
    }
    if (tid < D) sal[tid] = expf_near(__fmul_rn(a.gate_lb, sigmoid_near(__fmul_rn(ea, __fadd_rn(z, dt)))));
    __syncthreads();
    double tq = 0.0, tk = 0.0;
#pragma unroll
    for (int i = 0; i < D / 32; i++) { tq += red[i][0]; tk += red[i][1]; }
    const float qinv = (float)rsqrt_newton(tq + (double)1e-6f), kinv = (float)rsqrt_newton(tk + (double)1e-6f);
    if (tid < D) { sq[tid] = __fmul_rn(__fmul_rn(yq, qinv), qscale); sk[tid] = __fmul_rn(yk, kinv); }
    __syncthreads();
    // q.k of the normalised vectors, for o = q.(aS) + (q.k) u
    {
        const double qk = tid < D ? warp_sum((double)sq[tid] * (double)sk[tid]) : 0.0;
        if (tid < D && lane == 0) red[warp][2] = qk;
    }
    const float beta = sigmoid_near(braw);
    F2 u[4], o[4];                                                  // four sums of eight rows each (one of 32: 1.4 times the rounding error, and no faster)
#pragma unroll
    for (int j = 0; j < 4; j++) u[j] = o[j] = f2(0.f, 0.f);
    const float4 *al4 = reinterpret_cast<const float4 *>(sal + rg * R), *k4 = reinterpret_cast<const float4 *>(sk + rg * R), *q4 = reinterpret_cast<const float4 *>(sq + rg * R);
#pragma unroll
    for (int i = 0; i < R / 4; i++) {
        const float4 al = al4[i], k = k4[i], q = q4[i];
        s[4 * i] = f2_mul(s[4 * i], f2(al.x, al.x)); s[4 * i + 1] = f2_mul(s[4 * i + 1], f2(al.y, al.y));
        s[4 * i + 2] = f2_mul(s[4 * i + 2], f2(al.z, al.z)); s[4 * i + 3] = f2_mul(s[4 * i + 3], f2(al.w, al.w));
        u[0] = f2_fma(s[4 * i], f2(k.x, k.x), u[0]); u[1] = f2_fma(s[4 * i + 1], f2(k.y, k.y), u[1]);
        u[2] = f2_fma(s[4 * i + 2], f2(k.z, k.z), u[2]); u[3] = f2_fma(s[4 * i + 3], f2(k.w, k.w), u[3]);
        o[0] = f2_fma(s[4 * i], f2(q.x, q.x), o[0]); o[1] = f2_fma(s[4 * i + 1], f2(q.y, q.y), o[1]);
        o[2] = f2_fma(s[4 * i + 2], f2(q.z, q.z), o[2]); o[3] = f2_fma(s[4 * i + 3], f2(q.w, q.w), o[3]);
    }
    us[rg][cp] = f2_add(f2_add(u[0], u[1]), f2_add(u[2], u[3])); os[rg][cp] = f2_add(f2_add(o[0], o[1]), f2_add(o[2], o[3]));
    __syncthreads();
    float ux = 0.f, uy = 0.f, ox = 0.f, oy = 0.f;
#pragma unroll
    for (int i = 0; i < RG; i++) {
        const float2 p = *reinterpret_cast<const float2 *>(&us[i][cp]), q = *reinterpret_cast<const float2 *>(&os[i][cp]);
        ux = __fadd_rn(ux, p.x); uy = __fadd_rn(uy, p.y); ox = __fadd_rn(ox, q.x); oy = __fadd_rn(oy, q.y);
    }
    double qk = 0.0;
#pragma unroll
    for (int i = 0; i < D / 32; i++) qk += red[i][2];
    ux = __fmul_rn(__fsub_rn(raw[2 * D + 2 * cp], ux), beta); uy = __fmul_rn(__fsub_rn(raw[2 * D + 2 * cp + 1], uy), beta);
    ox = __fmaf_rn((float)qk, ux, ox); oy = __fmaf_rn((float)qk, uy, oy);
    const F2 uu = f2(ux, uy);
#pragma unroll
    for (int i = 0; i < R / 4; i++) {
        const float4 k = k4[i];
        const F2 r0 = f2_fma(f2(k.x, k.x), uu, s[4 * i]), r1 = f2_fma(f2(k.y, k.y), uu, s[4 * i + 1]), r2 = f2_fma(f2(k.z, k.z), uu, s[4 * i + 2]), r3 = f2_fma(f2(k.w, k.w), uu, s[4 * i + 3]);
        __stcs(S + (size_t)(4 * i) * (D / 2), r0.v); __stcs(S + (size_t)(4 * i + 1) * (D / 2), r1.v);
        __stcs(S + (size_t)(4 * i + 2) * (D / 2), r2.v); __stcs(S + (size_t)(4 * i + 3) * (D / 2), r3.v);
    }
    // per-head RMSNorm with weight, then the sigmoid output gate (glm53f_ops.c:748-752)
    if (rg == 0) { sal[2 * cp] = ox; sal[2 * cp + 1] = oy; }          // (the decays have been read: the barrier above)
    __syncthreads();
    const float ov = tid < D ? sal[tid] : 0.f;
    const double oo = warp_sum((double)ov * (double)ov);
    if (lane == 0) red[warp][0] = oo;
    __syncthreads();
    if (tid < D) {
        double tot = 0.0;
#pragma unroll
        for (int i = 0; i < D / 32; i++) tot += red[i][0];
        const float inv = (float)rsqrt_newton(tot / (double)D + (double)a.rms_eps);
        a.o[off + tid] = __fmul_rn(__fmul_rn(onw, __fmul_rn(ov, inv)), sigmoid_near(gate));
    }
}

// One position of one sequence. The chain of a single step is all latency: convolutions, norms, gates, two sums over the
// state, the output's norm. A cluster takes a head, 32 columns of the state to a CTA of 256 threads; what all columns need
// (q, k, the decays with their low-rank up-projection) every CTA computes for itself, and only the sum of squares of the
// output crosses the cluster. Weights and state travel before the wait for the kernel in front. Every value is that of
// the sequential recurrence, bit for bit: i ascending, rounded term by term, 256 dependent additions of one warp with a
// lane per column. (One CTA per head with its 64 KB of state and 255 registers a thread: 17.8 us cold, now 10.6, 8.7 of them behind the products.)
constexpr int KDA_STEP_PITCH(int D) { return 2 * D + 16; }               // bytes: consecutive rows begin on different banks
constexpr int KDA_STEP_SMEM(int D, bool low_rank) { return D * 32 * 4 + (low_rank ? (D + 32) * KDA_STEP_PITCH(D) : 0); }
template <int DS, int KW>
__global__ void __cluster_dims__(DS / 32, 1, 1) __launch_bounds__(256) kda_step_kernel(const KdaArgs a)
{
    pdl_trigger();
    constexpr int D = DS, CL = DS / 32, PITCH = KDA_STEP_PITCH(DS), TASKS = 2 * D + 32;
    extern __shared__ __align__(16) uint8_t smem[];
    float *st = reinterpret_cast<float *>(smem);                         // [D][32]: this CTA's columns of the state
    uint8_t *lrw = smem + D * 32 * 4;                                    // D rows of f_b, then 32 rows of g_b
    __shared__ __align__(16) float vec[3][D];                            // decay, k, q
    __shared__ __align__(16) float lr[2][D];
    __shared__ float raw[TASKS], sgb[32];
    __shared__ double mine;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % CL, h = a.head0 + blockIdx.x / CL, col0 = rank * 32, P = a.H * D, K = KW ? KW : a.K, hist = K - 1;
    float *S = a.state + (size_t)h * D * D + col0, *cs = a.state + (size_t)a.H * D * D;
    for (int i = tid; i < D * 8; i += 256)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(st + i * 4)), "l"(S + (size_t)(i >> 3) * D + (i & 7) * 4) : "memory");
    if (a.f_b) {
        constexpr int PER = D / 8;
        for (int i = tid; i < (D + 32) * PER; i += 256) {
            const int row = i / PER, piece = i % PER;
            const uint16_t *src = (row < D ? a.f_b + ((size_t)h * D + row) * D : a.g_b + ((size_t)h * D + col0 + row - D) * D) + piece * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(lrw + (size_t)row * PITCH + piece * 16)), "l"(src) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // convolution channels: q, then k, of the whole head, then v of this CTA's columns; two per thread at most
    const float *const xs[3] = {a.q, a.k, a.v}, *const ws[3] = {a.q_conv, a.k_conv, a.v_conv};
    int which[2], ch[2];
    bool has[2], own[2];
    float w[2][KW ? KW : 1], past[2][KW ? KW : 1];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int task = tid + n * 256;
        has[n] = task < TASKS;
        which[n] = task < D ? 0 : task < 2 * D ? 1 : 2;
        const int c = which[n] < 2 ? task % D : col0 + task - 2 * D;
        own[n] = has[n] && c >= col0 && c < col0 + 32;
        ch[n] = h * D + c;
        if (has[n]) {
#pragma unroll
            for (int j = 0; j < KW; j++) w[n][j] = ws[which[n]][(size_t)ch[n] * KW + j];
#pragma unroll
            for (int j = 0; j + 1 < KW; j++) past[n][j] = cs[(size_t)which[n] * P * hist + (size_t)ch[n] * hist + j];
        }
    }
    const float ea = expf_host(a.A_log[h]), qscale = 1.0f / sqrtf((float)D);
    const float dtb = a.dt_bias[h * D + tid % D], onw = a.o_norm[col0 + lane];
    // everything above is weights and this layer's own state; from here on the kernel in front is read
    pdl_wait();
    float now[2];
#pragma unroll
    for (int n = 0; n < 2; n++)
        if (has[n]) now[n] = xs[which[n]][ch[n]];
    const float beta_raw = a.braw[h];
    if (a.f_b)
        for (int i = tid; i < 2 * D; i += 256) lr[i / D][i % D] = (i < D ? a.lrf : a.lrg)[i % D];
    // ---- convolutions and SiLU
#pragma unroll
    for (int n = 0; n < 2; n++)
        if (has[n]) {
            float y;
            if (KW) {
                y = __fmul_rn(w[n][KW ? KW - 1 : 0], now[n]);
#pragma unroll
                for (int j = 0; j + 1 < KW; j++) y = mul_add_unfused(w[n][j], past[n][j], y);
            } else {
                const float *wp = ws[which[n]] + (size_t)ch[n] * K, *pp = cs + (size_t)which[n] * P * hist + (size_t)ch[n] * hist;
                y = __fmul_rn(wp[hist], now[n]);
                for (int j = 0; j < hist; j++) y = mul_add_unfused(wp[j], pp[j], y);
            }
            raw[tid + n * 256] = __fmul_rn(y, sigmoid_host(y));
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- decays, this CTA's output gates (z = f_b lrf, gb = g_b lrg: even and odd columns apart, ascending) and the l2norm
    // (divide by sqrt(sum of squares + 1e-6), sums in FP64, glm53f_ops.c:661-667): each to warps of its own
    if (tid < D + 32) {
        const bool gate = tid >= D;
        float z;
        if (a.f_b) {
            const uint8_t *row = lrw + (size_t)tid * PITCH;
            const float *x = lr[gate ? 1 : 0];
            F2 t = f2(0.f, 0.f);
#pragma unroll 4
            for (int c = 0; c < D; c += 8) {
                const uint4 v = *reinterpret_cast<const uint4 *>(row + 2 * c);
                const float4 x0 = *reinterpret_cast<const float4 *>(x + c), x1 = *reinterpret_cast<const float4 *>(x + c + 4);
                float lo, hi;
                bf16x2_to_f32(v.x, lo, hi); t = f2_fma(f2(lo, hi), f2(x0.x, x0.y), t);
                bf16x2_to_f32(v.y, lo, hi); t = f2_fma(f2(lo, hi), f2(x0.z, x0.w), t);
                bf16x2_to_f32(v.z, lo, hi); t = f2_fma(f2(lo, hi), f2(x1.x, x1.y), t);
                bf16x2_to_f32(v.w, lo, hi); t = f2_fma(f2(lo, hi), f2(x1.z, x1.w), t);
            }
            z = f2_sum(t);
        } else z = gate ? a.gb[h * D + col0 + tid - D] : a.z[h * D + tid];
        if (gate) sgb[tid - D] = sigmoid_host(z);
        else      vec[0][tid] = expf_host(__fmul_rn(a.gate_lb, sigmoid_host(__fmul_rn(ea, __fadd_rn(z, dtb)))));
    } else if (warp >= 6) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < D / 32; i++) { const double v = (double)raw[(warp - 6) * D + lane + 32 * i]; t = fma(v, v, t); }
        t = warp_sum(t);
        const float inv = (float)rsqrt_newton(t + (double)1e-6f);
#pragma unroll
        for (int i = 0; i < D / 32; i++) {
            const float v = __fmul_rn(raw[(warp - 6) * D + lane + 32 * i], inv);
            vec[warp == 6 ? 2 : 1][lane + 32 * i] = warp == 6 ? __fmul_rn(v, qscale) : v;
        }
    }
    __syncthreads();
    // ---- the state's columns: decay, u = k.S, S += k (v - u) beta, o = q.S
    float o = 0.f;
    if (warp == 0) {
        float u = 0.f;
        const float4 *al4 = reinterpret_cast<const float4 *>(vec[0]), *k4 = reinterpret_cast<const float4 *>(vec[1]), *q4 = reinterpret_cast<const float4 *>(vec[2]);
        float *sc = st + lane;
        const float beta = sigmoid_host(beta_raw);
#pragma unroll 8
        for (int i = 0; i < D / 4; i++) {
            const float4 al = al4[i], kk = k4[i];
            const float s0 = __fmul_rn(sc[(4 * i) * 32], al.x), s1 = __fmul_rn(sc[(4 * i + 1) * 32], al.y), s2 = __fmul_rn(sc[(4 * i + 2) * 32], al.z),
                        s3 = __fmul_rn(sc[(4 * i + 3) * 32], al.w);
            u = __fadd_rn(u, __fmul_rn(s0, kk.x)); u = __fadd_rn(u, __fmul_rn(s1, kk.y));
            u = __fadd_rn(u, __fmul_rn(s2, kk.z)); u = __fadd_rn(u, __fmul_rn(s3, kk.w));
        }
        u = __fmul_rn(__fsub_rn(raw[2 * D + lane], u), beta);
#pragma unroll 8
        for (int i = 0; i < D / 4; i++) {
            const float4 al = al4[i], kk = k4[i], q = q4[i];
            const float s0 = __fadd_rn(__fmul_rn(sc[(4 * i) * 32], al.x), __fmul_rn(kk.x, u)), s1 = __fadd_rn(__fmul_rn(sc[(4 * i + 1) * 32], al.y), __fmul_rn(kk.y, u)),
                        s2 = __fadd_rn(__fmul_rn(sc[(4 * i + 2) * 32], al.z), __fmul_rn(kk.z, u)), s3 = __fadd_rn(__fmul_rn(sc[(4 * i + 3) * 32], al.w), __fmul_rn(kk.w, u));
            float *Sp = S + (size_t)(4 * i) * D + lane;
            Sp[0] = s0; Sp[D] = s1; Sp[2 * D] = s2; Sp[3 * D] = s3;
            o = __fadd_rn(o, __fmul_rn(s0, q.x)); o = __fadd_rn(o, __fmul_rn(s1, q.y));
            o = __fadd_rn(o, __fmul_rn(s2, q.z)); o = __fadd_rn(o, __fmul_rn(s3, q.w));
        }
        const double oo = warp_sum((double)o * (double)o);
        if (lane == 0) mine = oo;
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    // ---- per-head RMSNorm with weight, then the sigmoid output gate (glm53f_ops.c:748-752)
    if (warp == 0) {
        double tot = 0.0;
#pragma unroll
        for (int r = 0; r < CL; r++) tot += ld_cluster_f64(&mine, r);
        const float inv = (float)rsqrt_newton(tot / (double)D + (double)a.rms_eps);
        a.o[h * D + col0 + lane] = __fmul_rn(__fmul_rn(onw, __fmul_rn(o, inv)), sgb[lane]);
    }
    // the histories move on by one (every CTA of the head has read them: the barrier above); each channel by one thread
#pragma unroll
    for (int n = 0; n < 2; n++)
        if (own[n] && hist > 0) {
            float *hp = cs + (size_t)which[n] * P * hist + (size_t)ch[n] * hist;
            if (KW) {
#pragma unroll
                for (int j = 0; j + 2 < KW; j++) hp[j] = past[n][j + 1];
            } else
                for (int j = 0; j + 1 < hist; j++) hp[j] = hp[j + 1];
            hp[hist - 1] = now[n];
        }
    __syncwarp();
    cluster_arrive();                                    // no CTA leaves while another may still read its sum
    cluster_wait();
}

template <int DS, int KW>
static bool kda_step(cudaStream_t st, const KdaArgs &a, int heads)
{
    static SmemGrant grant;
    const size_t smem = KDA_STEP_SMEM(DS, a.f_b != nullptr);
    // (with the static arrays it is above the 48 KB that need no consent before the dynamic part alone is)
    if (!dev_opt_in_smem((const void *)kda_step_kernel<DS, KW>, smem + (8 << 10), grant)) return false;
    G5B_LAUNCH_PDL((kda_step_kernel<DS, KW>), dim3(heads * (DS / 32)), dim3(256), smem, st, a);
    return true;
}

constexpr int KDA_EARLY_T = 8;        // positions whose scan is shorter than a launch
template <int DS>
static void kda_rows(cudaStream_t st, const KdaArgs &a, const KdaScratch &x, int heads, int n_seq)
{
    KdaPrep p{a, x.qn, x.kn, x.vn, x.al, x.beta, heads};
    const dim3 pg(heads, (a.T + KDA_TILE - 1) / KDA_TILE * n_seq);
    if (a.K == 4) G5B_LAUNCH_PDL((kda_prep_kernel<DS, 4>), pg, dim3(4 * DS), 0, st, p);
    else          G5B_LAUNCH_PDL((kda_prep_kernel<DS, 0>), pg, dim3(4 * DS), 0, st, p);
    // (many positions: launched the ordinary way - launched early, its few long-running CTAs crowd the SMs that the preparation
    // leaves first, seven to an SM, and the others idle)
    if (a.T > KDA_EARLY_T) G5B_LAUNCH((kda_scan_kernel<DS, 8, 1, 4>), dim3(heads * (DS / 16), n_seq), dim3(128), 0, st, p);
    else if (a.T > 1)      G5B_LAUNCH_PDL((kda_scan_kernel<DS, 8, 1, 4>), dim3(heads * (DS / 16), n_seq), dim3(128), 0, st, p);
    else                   G5B_LAUNCH_PDL((kda_scan_kernel<DS, 4, 1, 4>), dim3(heads * (DS / 32), n_seq), dim3(128), 0, st, p);
    G5B_LAUNCH_PDL(kda_out_kernel<DS>, dim3((heads + 7) / 8, a.T * n_seq), dim3(256), 0, st, a, heads);
}

int kda_core(cudaStream_t st, float *o, const float *q, const float *k, const float *v, const float *z,
              const float *braw, const float *gb, const float *q_conv, const float *k_conv,
              const float *v_conv, const float *A_log, const float *dt_bias, const float *o_norm,
              float *state, int T, const KdaShape &s, int n_seq, size_t seq_stride, const KdaLowRank *lr, int head0, int heads,
              float *snap, int snap_after, const KdaScratch *scratch)
{
    const bool fused = lr && T == 1 && n_seq <= 1 && (s.D == 64 || s.D == 128);
    KdaArgs a{o, q, k, v, z, braw, gb, q_conv, k_conv, v_conv, A_log, dt_bias, o_norm, state,
              T, s.H, s.D, s.K, head0, s.gate_lb, s.rms_eps, seq_stride,
              fused ? static_cast<const uint16_t *>(lr->f_b) : nullptr, fused ? static_cast<const uint16_t *>(lr->g_b) : nullptr,
              fused ? lr->lrf : nullptr, fused ? lr->lrg : nullptr, snap, snap_after};
    const dim3 grid(heads > 0 ? heads : s.H, n_seq < 1 ? 1 : n_seq);
    const bool known = s.K >= 1 && s.K <= 17 && (s.D == 128 || s.D == 64);
    if (known && T * grid.y == 1) {
        const bool ok = s.D == 128 ? (s.K == 4 ? kda_step<128, 4>(st, a, (int)grid.x) : kda_step<128, 0>(st, a, (int)grid.x))
                                   : (s.K == 4 ? kda_step<64, 4>(st, a, (int)grid.x) : kda_step<64, 0>(st, a, (int)grid.x));
        if (ok) return 0;
        if (fused) return -1;                // the kernel below does not take the up-projections itself
    } else if (known && T == 1 && s.K == 4) {
        if (s.D == 128) G5B_LAUNCH_PDL(kda_each_kernel<128>, grid, dim3(256), 0, st, a);
        else            G5B_LAUNCH_PDL(kda_each_kernel<64>, grid, dim3(256), 0, st, a);
        return 0;
    } else if (known && scratch) {
        if (s.D == 128) kda_rows<128>(st, a, *scratch, (int)grid.x, (int)grid.y);
        else            kda_rows<64>(st, a, *scratch, (int)grid.x, (int)grid.y);
        return 0;
    }
    G5B_LAUNCH(kda_core_kernel, grid, ((s.D + 31) / 32) * 32, 0, st, a);
    return 0;
}

}  // namespace g5b
