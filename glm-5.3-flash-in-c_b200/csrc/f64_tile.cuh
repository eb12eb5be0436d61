// f64_tile.cuh - out[z][t][n] = sum_k A[z][t][k] B[z](k, n) with FP64 sums, A in FP32 and B in BF16: the router's scores
// and the absorption of W_k into the queries for many positions at once.
//
// The FP64 pipe (16 FMA per clock and SM) bounds both. A float becomes a double at half that rate, so a loop that
// converts its factors for every product, or for four, mostly converts; here a CTA converts a 32 x 32 block of each
// factor once (BF16 by shifting bits, which needs no FP64 instruction) and uses it for 32 products, and a thread holds
// 4 x 4 sums. Two warps to a CTA, eight CTAs to an SM: products of some CTAs beside the conversions of others. Few rows of A:
// tiles of eight, 1 x 4 sums to a thread, since a tile of 32 would multiply padding for most of its time.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace g5b {

// v = hi + mid + lo exactly enough (24 bits), each a BF16
__device__ __forceinline__ void split3_bf16(float v, __nv_bfloat16 &hi, __nv_bfloat16 &mid, __nv_bfloat16 &lo)
{
    hi = __float2bfloat16_rn(v);
    const float e1 = v - __bfloat162float(hi);
    mid = __float2bfloat16_rn(e1);
    lo = __float2bfloat16_rn(e1 - __bfloat162float(mid));
}

// Where an absorbed query goes: doubles [query][head][KL], or, for the tensor-core attention core, the float of v * scale
// as three BF16 terms [query][head][term][KL] (split here once, not by every CTA that multiplies the query).
struct QueryOut {
    double *qa; __nv_bfloat16 *terms; double scale; int H, KL;
    __device__ __forceinline__ void put(int t, int h, int c, double v) const
    {
        if (terms) {
            __nv_bfloat16 *d = terms + ((size_t)t * H + h) * 3 * KL + c;
            split3_bf16((float)(v * scale), d[0], d[KL], d[2 * KL]);
        } else qa[((size_t)t * H + h) * KL + c] = v;
    }
};

struct F64Tile {
    const float *A; const uint16_t *B; double *out;
    size_t lda, ldb, ldo;         // elements between rows
    size_t za, zb, zo;            // elements between the problems of blockIdx.z (heads, or stretches of k)
    int T, N, K;                  // K: a multiple of 32, rows of A and B 16-byte aligned
    QueryOut q;                   // K_ROWS: the results are absorbed queries of head blockIdx.z
};
constexpr int F64_N = 32, F64_K = 32, F64_THREADS = 64, F64_PITCH = 34;

__device__ __forceinline__ double bf16_to_f64(uint32_t h)
{
    const uint32_t m = h & 0x7fffu, e = m & 0x7f80u;
    if (e - 0x80u < 0x7f00u) return __hiloint2double((int)(((h & 0x8000u) << 16) | ((m << 13) + 0x38000000u)), 0);
    return (double)bf16_to_f32((uint16_t)h);                      // zero, subnormal, infinite, NaN
}

// K_ROWS: B's rows run along n (element (k, n) at B[k * ldb + n], N a multiple of 8); otherwise along k (B[n * ldb + k]).
template <bool K_ROWS, int TR>
__global__ void __launch_bounds__(F64_THREADS, 8) f64_tile_kernel(const F64Tile p)
{
    pdl_trigger();
    constexpr int F64_T = 8 * TR;                                 // rows of A in a tile
    __shared__ __align__(16) double sa[F64_K][F64_T + 2], sb[F64_K][F64_PITCH];
    const int tid = threadIdx.x, t0 = blockIdx.y * F64_T, n0 = blockIdx.x * F64_N;
    const float *A = p.A + (size_t)blockIdx.z * p.za;
    const uint16_t *Bm = p.B + (size_t)blockIdx.z * p.zb;
    double *out = K_ROWS ? nullptr : p.out + (size_t)blockIdx.z * p.zo;
    const int row = tid & 31, half = tid >> 5;                    // a thread loads 16 consecutive k of one row of B
    const int arow = tid % F64_T, ak = tid / F64_T * (4 * TR);    // and 4 TR of one of A
    const bool alive = t0 + arow < p.T;
    const int tt = (tid >> 3) * TR, nn = (tid & 7) * 4;
    float4 ra[TR];
    uint4 rb[2];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < TR; i++)
            ra[i] = alive ? *reinterpret_cast<const float4 *>(A + (size_t)(t0 + arow) * p.lda + k0 + ak + i * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            if (K_ROWS) {
                const int k = k0 + (tid >> 2) + 16 * i, n = n0 + (tid & 3) * 8;
                rb[i] = n < p.N ? *reinterpret_cast<const uint4 *>(Bm + (size_t)k * p.ldb + n) : make_uint4(0u, 0u, 0u, 0u);
            } else
                rb[i] = n0 + row < p.N ? *reinterpret_cast<const uint4 *>(Bm + (size_t)(n0 + row) * p.ldb + k0 + half * 16 + i * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    double acc[TR][4];
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
    load(0);
    for (int k0 = 0; k0 < p.K; k0 += F64_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TR; i++) {
            const int k = ak + i * 4;
            sa[k][arow] = (double)ra[i].x; sa[k + 1][arow] = (double)ra[i].y; sa[k + 2][arow] = (double)ra[i].z; sa[k + 3][arow] = (double)ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t u[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const double lo = bf16_to_f64(u[j] & 0xffffu), hi = bf16_to_f64(u[j] >> 16);
                if (K_ROWS) {
                    const int k = (tid >> 2) + 16 * i, n = (tid & 3) * 8 + 2 * j;
                    sb[k][n] = lo; sb[k][n + 1] = hi;
                } else {
                    const int k = half * 16 + i * 8 + 2 * j;
                    sb[k][row] = lo; sb[k + 1][row] = hi;
                }
            }
        }
        __syncthreads();
        if (k0 + F64_K < p.K) load(k0 + F64_K);
#pragma unroll 4
        for (int k = 0; k < F64_K; k++) {
            double av[TR];
            if constexpr (TR == 4) {
                const double2 a0 = *reinterpret_cast<const double2 *>(&sa[k][tt]), a1 = *reinterpret_cast<const double2 *>(&sa[k][tt + 2]);
                av[0] = a0.x; av[1] = a0.y; av[2] = a1.x; av[3] = a1.y;
            } else av[0] = sa[k][tt];
            const double2 b0 = *reinterpret_cast<const double2 *>(&sb[k][nn]), b1 = *reinterpret_cast<const double2 *>(&sb[k][nn + 2]);
            const double bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < TR; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TR; i++)
        if (t0 + tt + i < p.T)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (n0 + nn + j < p.N) {
                    if (K_ROWS) p.q.put(t0 + tt + i, blockIdx.z, n0 + nn + j, acc[i][j]);
                    else        out[(size_t)(t0 + tt + i) * p.ldo + n0 + nn + j] = acc[i][j];
                }
}

inline int f64_tile_rows(int T) { return T > 16 ? 32 : 8; }      // (two tiles of eight are as fast as one of 32)
template <bool K_ROWS>
void f64_tile(cudaStream_t st, const F64Tile &p, int z)
{
    const int rows = f64_tile_rows(p.T);
    const dim3 grid((p.N + F64_N - 1) / F64_N, (p.T + rows - 1) / rows, z);
    // (launched the ordinary way: launched early, the CTAs crowd the SMs that the kernel in front has left, eight to an SM, and
    // the FP64 pipes of the others idle - 486 us became 963)
    if (rows == 32) G5B_LAUNCH((f64_tile_kernel<K_ROWS, 4>), grid, F64_THREADS, 0, st, p);
    else            G5B_LAUNCH((f64_tile_kernel<K_ROWS, 1>), grid, F64_THREADS, 0, st, p);
}

}  // namespace g5b
