// f64_tile.cuh - out[z][t][n] = sum_k A[z][t][k] B[z](k, n) with FP64 sums, A in FP32 and B in BF16: the router's scores,
// the absorption of W_k into the queries and the value projection for several positions at once.
//
// The FP64 pipe bounds both: 64 FMA per clock and SM, as DFMA or as mma.sync.m8n8k4 (measured: 63 and 64), while a float
// becomes a double at 16 per clock and SM. Threads that hold 4 x 4 sums read 64 bytes of shared memory for 16 products and
// shared memory, not the pipe, bounds them (12 FMA per clock and SM); the matrix instruction reads each factor once for
// eight products in every lane, so a warp with 4 x 4 of its tiles reads 2 KB for 4096 products. A CTA converts a block of 32 k of each factor
// once (BF16 by shifting bits, which needs no FP64 instruction). 64 queries of 64 heads, K = 256, N = 512: 49 us, 115 with threads of 4 x 4 sums (the pipe alone: 28).
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
    __device__ __forceinline__ void put2(int t, int h, int c, double v0, double v1) const    // c even
    {
        if (terms) {
            __nv_bfloat162 *d = reinterpret_cast<__nv_bfloat162 *>(terms + ((size_t)t * H + h) * 3 * KL + c), x, y, z;
            split3_bf16((float)(v0 * scale), x.x, y.x, z.x);
            split3_bf16((float)(v1 * scale), x.y, y.y, z.y);
            d[0] = x; d[KL / 2] = y; d[KL] = z;
        } else *reinterpret_cast<double2 *>(qa + ((size_t)t * H + h) * KL + c) = make_double2(v0, v1);
    }
};

struct F64Tile {
    const float *A; const uint16_t *B; double *out;
    size_t lda, ldb, ldo;         // elements between rows
    size_t za, zb, zo;            // elements between the problems of blockIdx.z (heads, or stretches of k)
    int T, N, K;                  // K: a multiple of 32, rows of A and B 16-byte aligned
    QueryOut q;                   // K_ROWS: the results are absorbed queries of head blockIdx.z
    float *rounded;               // otherwise, instead of out if not null: the sums rounded to floats
};
constexpr int F64_N = 64, F64_K = 32, F64_THREADS = 128;
// Rows of the blocks in shared memory, in doubles: 4 more than a multiple of 16, so that the 4 x 4 or 8 x 4 elements that a
// half-warp of the matrix instruction reads lie in different banks, and no more than that.
constexpr int F64_KPITCH = F64_K + 4, F64_NPITCH = F64_N + 4;

// c += a b, 8 x 8 x 4: a = A[lane / 4][lane % 4], b = B[lane % 4][lane / 4], c[i] = C[lane / 4][2 (lane % 4) + i]
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

__device__ __forceinline__ double bf16_to_f64(uint32_t h)
{
    const uint32_t m = h & 0x7fffu, e = m & 0x7f80u;
    if (e - 0x80u < 0x7f00u) return __hiloint2double((int)(((h & 0x8000u) << 16) | ((m << 13) + 0x38000000u)), 0);
    return (double)bf16_to_f32((uint16_t)h);                      // zero, subnormal, infinite, NaN
}

// A BF16's bits (the upper half of u) put where a double has them: its value times 2^-896, zero and subnormal ones too. Two instructions,
// where the exponent's own bias takes eight; a sum of such products is scaled back at the end. Sums lose nothing to underflow
// before 2^-52 of terms whose BF16 factor is above 2^-110. Infinities and NaN have no place among them (bf16_special).
constexpr double BF16_BITS_SCALE = 0x1p896;
__device__ __forceinline__ double bf16_bits_f64(uint32_t u)
{
    double d;
    asm volatile("{\n\t.reg .b32 t;\n\tshr.s32 t, %1, 3;\n\tand.b32 t, t, 0x8fffe000;\n\tmov.b64 %0, {0, t};\n\t}" : "=d"(d) : "r"(u));
    return d;
}
__device__ __forceinline__ uint32_t bf16_special(uint32_t two) { return ((two & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }

// K_ROWS: B's rows run along n (element (k, n) at B[k * ldb + n], N a multiple of 8); otherwise along k (B[n * ldb + k]).
// A CTA of four warps takes 8 TM rows of A and 64 columns: TM = 8: two by two warps of 32 x 32 each, otherwise a warp has 16
// of the columns.
template <bool K_ROWS, int TM>
__global__ void __launch_bounds__(F64_THREADS, 4) f64_tile_kernel(const F64Tile p)
{
    pdl_trigger();
    constexpr int ROWS = 8 * TM, MT = TM == 8 ? 4 : TM, NT = TM == 8 ? 4 : 2;
    constexpr int BR = K_ROWS ? F64_K : F64_N, BP = K_ROWS ? F64_NPITCH : F64_KPITCH;
    __shared__ __align__(16) double sa[ROWS][F64_KPITCH], sb[BR][BP];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int t0 = blockIdx.y * ROWS, n0 = blockIdx.x * F64_N;
    const int wm = TM == 8 ? (warp >> 1) * 32 : 0, wn = TM == 8 ? (warp & 1) * 32 : warp * 16;
    const float *A = p.A + (size_t)blockIdx.z * p.za;
    const uint16_t *Bm = p.B + (size_t)blockIdx.z * p.zb;
    // A: eight lanes take 32 k of a row. B: four lanes take 32 k of a row, or eight lanes 64 n of a k.
    constexpr int AL = (ROWS * 8 + F64_THREADS - 1) / F64_THREADS, BL = 2;
    float4 ra[AL];
    uint4 rb[BL];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < AL; i++) {
            const int r = (tid >> 3) + i * (F64_THREADS / 8);
            ra[i] = r < ROWS && t0 + r < p.T ? *reinterpret_cast<const float4 *>(A + (size_t)(t0 + r) * p.lda + k0 + (tid & 7) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < BL; i++) {
            if (K_ROWS) {
                const int k = k0 + (tid >> 3) + 16 * i, n = n0 + (tid & 7) * 8;
                rb[i] = n < p.N ? *reinterpret_cast<const uint4 *>(Bm + (size_t)k * p.ldb + n) : make_uint4(0u, 0u, 0u, 0u);
            } else {
                const int n = n0 + (tid >> 2) + 32 * i;
                rb[i] = n < p.N ? *reinterpret_cast<const uint4 *>(Bm + (size_t)n * p.ldb + k0 + (tid & 3) * 8) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    double acc[MT][NT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    load(0);
    for (int k0 = 0; k0 < p.K; k0 += F64_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < AL; i++) {
            const int r = (tid >> 3) + i * (F64_THREADS / 8);
            if (ROWS * 8 % F64_THREADS == 0 || r < ROWS) {
                double2 *d = reinterpret_cast<double2 *>(&sa[r][(tid & 7) * 4]);
                d[0] = make_double2((double)ra[i].x, (double)ra[i].y);
                d[1] = make_double2((double)ra[i].z, (double)ra[i].w);
            }
        }
#pragma unroll
        for (int i = 0; i < BL; i++) {
            double2 *d = reinterpret_cast<double2 *>(K_ROWS ? &sb[(tid >> 3) + 16 * i][(tid & 7) * 8] : &sb[(tid >> 2) + 32 * i][(tid & 3) * 8]);
            const uint32_t u[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) d[j] = make_double2(bf16_to_f64(u[j] & 0xffffu), bf16_to_f64(u[j] >> 16));
        }
        __syncthreads();
        if (k0 + F64_K < p.K) load(k0 + F64_K);
#pragma unroll
        for (int k = 0; k < F64_K; k += 4) {
            double av[MT], bv[NT];
#pragma unroll
            for (int i = 0; i < MT; i++) av[i] = sa[wm + i * 8 + g][k + q];
#pragma unroll
            for (int j = 0; j < NT; j++) bv[j] = K_ROWS ? sb[k + q][wn + j * 8 + g] : sb[wn + j * 8 + g][k + q];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < NT; j++) mma_f64(acc[i][j], av[i], bv[j]);
        }
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const int t = t0 + wm + i * 8 + g;
        if (t < p.T)
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const int n = n0 + wn + j * 8 + 2 * q;        // (N is even)
                if (n < p.N) {
                    if (K_ROWS) p.q.put2(t, blockIdx.z, n, acc[i][j][0], acc[i][j][1]);
                    else {
                        const size_t at = (size_t)blockIdx.z * p.zo + (size_t)t * p.ldo + n;
                        if (p.rounded) *reinterpret_cast<float2 *>(p.rounded + at) = make_float2((float)acc[i][j][0], (float)acc[i][j][1]);
                        else           *reinterpret_cast<double2 *>(p.out + at) = make_double2(acc[i][j][0], acc[i][j][1]);
                    }
                }
            }
    }
}

// Rows of A in a CTA's tile: what there are, in steps of 8, 16, 32 (padding costs the pipe as much as rows do), 64 beyond.
inline int f64_tile_rows(int T) { return T <= 8 ? 8 : T <= 16 ? 16 : T <= 32 ? 32 : 64; }
// N even, out and ldo too
template <bool K_ROWS>
void f64_tile(cudaStream_t st, const F64Tile &p, int z)
{
    const int rows = f64_tile_rows(p.T);
    const dim3 grid((p.N + F64_N - 1) / F64_N, (p.T + rows - 1) / rows, z);
    // (launched the ordinary way: launched early, the CTAs crowd the SMs that the kernel in front has left, several to an SM, and
    // the FP64 pipes of the others idle)
    switch (rows) {
    case 8:  G5B_LAUNCH((f64_tile_kernel<K_ROWS, 1>), grid, F64_THREADS, 0, st, p); break;
    case 16: G5B_LAUNCH((f64_tile_kernel<K_ROWS, 2>), grid, F64_THREADS, 0, st, p); break;
    case 32: G5B_LAUNCH((f64_tile_kernel<K_ROWS, 4>), grid, F64_THREADS, 0, st, p); break;
    default: G5B_LAUNCH((f64_tile_kernel<K_ROWS, 8>), grid, F64_THREADS, 0, st, p);
    }
}

}  // namespace g5b
