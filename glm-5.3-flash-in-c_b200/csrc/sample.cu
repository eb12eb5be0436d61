// sample.cu - the next token drawn from the logits on the device: temperature, then nucleus
// (top-p) truncation, then one draw from a counter-based generator.
//
// The reference decodes greedily only (src/cli/glm53f_run.c:492-494 takes the arg-max on the host);
// this is the sampled counterpart, kept on the GPU so that a decode loop never returns to the host
// between steps. The definition, which tests restate in numpy on the same logits:
//   p_i    = (float) exp((double) ((l_i - max l) / temperature))             (float subtract, divide)
//   Z      = sum_i p_i                                                       (FP64)
//   tau    = the largest probability value with  sum_{p_i >= tau} p_i >= top_p * Z
//            (the nucleus is every token at least that probable; top_p >= 1 keeps all of them)
//   u      = (mix64(seed ^ mix64(step + 1)) >> 11) * 2^-53                   (in [0, 1))
//   token  = the first index i, in index order, whose running nucleus mass exceeds u * (nucleus mass)
// FP64 sums are taken in a different association on the two sides, so a draw can differ only when
// a running sum falls within rounding (1e-16 relative) of a threshold.
//
// Four small launches over the whole GPU (as one CTA walking the vocabulary seven times a draw from 154880 logits
// took 1.9 ms, as much as the eight decoder layers before it; now a sampled token takes 41 us more than a greedy
// one with a nucleus of 0.95, 9 us more with top_p = 1):
//   max    each CTA's largest logit
//   prob   p_i, each CTA's mass, and the mass per bin of the upper 12 bits of p (p >= 0: bits order like values)
//   cut    every CTA finds the bin in which the nucleus mass is reached (top_p < 1), adds the mass of its
//          tokens above that bin, and lists its tokens inside it
//   pick   one CTA: tau among the listed tokens (radix over the lower 20 bits), the masses of the CTAs' index
//          ranges completed, then the range and the token that hold the drawn point
// The grid is one CTA per 1024 tokens: 152 CTAs for the released vocabulary, about one per SM.
#include <math.h>

#include "common.cuh"
#include "kernels.h"

namespace g5b {

constexpr int SMP_THREADS = 256, SMP_PICK = 1024;
constexpr int SMP_RANGE = 1024;           // tokens per CTA at least
constexpr int SMP_MAX_PARTS = 1024;
constexpr int SMP_BITS = 20, SMP_BINS = 1 << (32 - SMP_BITS);

__device__ __forceinline__ uint64_t smp_mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

struct SampleArgs {
    const float *logits;   // [V]
    float *prob;           // [V]
    double *bins;          // [SMP_BINS] mass per bin
    double *mass;          // [parts] nucleus mass of each CTA's range
    float *top;            // [parts] largest logit of each range
    double *above;         // [1] mass of the bins above the cut bin
    int *list;             // [V] tokens of the cut bin
    int *count;            // [1] how many, then the cut bin
    int *out;              // [1]
    int V, range, parts;
    float temperature, top_p;
    uint64_t seed, step;
};

// Sums of v over the threads up to and including this one, and over the whole block (total). red: 32 doubles.
__device__ __forceinline__ double block_scan(double v, double *red, double &total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    __syncthreads();
    if (lane == 31) red[wid] = v;
    __syncthreads();
    double before = 0.0;
    total = 0.0;
    for (int w = 0; w < nw; w++) { if (w == wid) before = total; total += red[w]; }
    return before + v;
}

__global__ void __launch_bounds__(SMP_THREADS) sample_max_kernel(const SampleArgs a)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float wmax[SMP_THREADS / 32];
    for (int i = blockIdx.x * SMP_THREADS + threadIdx.x; i < SMP_BINS; i += gridDim.x * SMP_THREADS) a.bins[i] = 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.count[0] = 0;
    const int i1 = min(a.V, ((int)blockIdx.x + 1) * a.range);
    float m = -INFINITY;
    for (int i = blockIdx.x * a.range + threadIdx.x; i < i1; i += SMP_THREADS) m = fmaxf(m, a.logits[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < SMP_THREADS / 32; w++) m = fmaxf(m, wmax[w]);
        a.top[blockIdx.x] = m;
    }
}

__global__ void __launch_bounds__(SMP_THREADS) sample_prob_kernel(const SampleArgs a)
{
    pdl_trigger();
    pdl_wait();
    __shared__ double bin[SMP_BINS];
    __shared__ double red[32];
    __shared__ float wmax[SMP_THREADS / 32];
    const bool cut = a.top_p < 1.0f;
    float m = -INFINITY;
    for (int i = threadIdx.x; i < a.parts; i += SMP_THREADS) m = fmaxf(m, a.top[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    if (cut) for (int i = threadIdx.x; i < SMP_BINS; i += SMP_THREADS) bin[i] = 0.0;
    __syncthreads();
    m = wmax[0];
    for (int w = 1; w < SMP_THREADS / 32; w++) m = fmaxf(m, wmax[w]);
    const int i1 = min(a.V, ((int)blockIdx.x + 1) * a.range);
    double z = 0.0;
    for (int i = blockIdx.x * a.range + threadIdx.x; i < i1; i += SMP_THREADS) {
        const float p = expf_host(__fdiv_rn(__fsub_rn(a.logits[i], m), a.temperature));
        a.prob[i] = p;
        if (cut) atomicAdd(&bin[__float_as_uint(p) >> SMP_BITS], (double)p);
        else     z += (double)p;
    }
    if (!cut) {
        z = block_sum(z, red);
        if (threadIdx.x == 0) a.mass[blockIdx.x] = z;
        return;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < SMP_BINS; i += SMP_THREADS)
        if (bin[i] != 0.0) atomicAdd(a.bins + i, bin[i]);
}

__global__ void __launch_bounds__(SMP_THREADS) sample_cut_kernel(const SampleArgs a)
{
    pdl_trigger();
    pdl_wait();
    constexpr int PER = SMP_BINS / SMP_THREADS;
    __shared__ double red[32];
    __shared__ int s_bin, s_first, s_some;
    // thread t holds bins SMP_BINS - 1 - t PER - k, the largest values first
    double b[PER], own = 0.0, z;
#pragma unroll
    for (int k = 0; k < PER; k++) { b[k] = a.bins[SMP_BINS - 1 - (int)threadIdx.x * PER - k]; own += b[k]; }
    if (threadIdx.x == 0) { s_bin = 0; s_first = SMP_THREADS; s_some = 0; }
    const double upto = block_scan(own, red, z), target = (double)a.top_p * z;
    if (own != 0.0) { atomicMax(&s_some, (int)threadIdx.x); if (upto >= target) atomicMin(&s_first, (int)threadIdx.x); }
    __syncthreads();
    if ((int)threadIdx.x == (s_first < SMP_THREADS ? s_first : s_some)) {      // (rounding: none reaches it, the last one holds it)
        double run = upto - own, at_run = run;
        int at_k = 0;
        for (int k = 0; k < PER; k++) {
            if (b[k] == 0.0) continue;
            at_k = k; at_run = run;
            run += b[k];
            if (run >= target) break;
        }
        s_bin = SMP_BINS - 1 - (int)threadIdx.x * PER - at_k;
        if (blockIdx.x == 0) { *a.above = at_run; a.count[1] = s_bin; }
    }
    __syncthreads();
    const unsigned at = (unsigned)s_bin;
    const int i1 = min(a.V, ((int)blockIdx.x + 1) * a.range);
    double mass = 0.0;
    for (int i = blockIdx.x * a.range + threadIdx.x; i < i1; i += SMP_THREADS) {
        const float p = a.prob[i];
        const unsigned q = __float_as_uint(p) >> SMP_BITS;
        if (q > at) mass += (double)p;
        else if (q == at) {                      // lanes of one warp that have one take their places together
            const unsigned lanes = __activemask(), rank = __popc(lanes & ((1u << (threadIdx.x & 31)) - 1u));
            const int leader = __ffs(lanes) - 1;
            int base = 0;
            if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(a.count, __popc(lanes));
            a.list[__shfl_sync(lanes, base, leader) + (int)rank] = i;
        }
    }
    mass = block_sum(mass, red);
    if (threadIdx.x == 0) a.mass[blockIdx.x] = mass;
}

__global__ void __launch_bounds__(SMP_PICK) sample_pick_kernel(const SampleArgs a)
{
    pdl_trigger();
    pdl_wait();
    __shared__ double red[32], hist[256], range_mass[SMP_MAX_PARTS];
    __shared__ double s_run;
    __shared__ unsigned s_prefix;
    __shared__ int s_owner, s_pick, s_last;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool cut = a.top_p < 1.0f;
    const int n = cut ? *a.count : 0;
    unsigned tau = 0u;                           // bits of the smallest probability kept; 0 keeps everything
    range_mass[tid] = tid < a.parts ? a.mass[tid] : 0.0;
    if (tid == 0) { s_owner = SMP_MAX_PARTS; s_pick = a.V; s_last = -1; s_prefix = cut ? (unsigned)a.count[1] << SMP_BITS : 0u; s_run = cut ? *a.above : 0.0; }
    if (cut) {
        // the target again from the bins, added the way the cut kernel did (the first SMP_THREADS threads' order
        // does not matter here beyond rounding)
        double z = 0.0;
        for (int i = tid; i < SMP_BINS; i += SMP_PICK) z += a.bins[i];
        z = block_sum(z, red);
        const double target = (double)a.top_p * z;
        for (int shift = SMP_BITS - 8; ; shift = shift > 8 ? shift - 8 : 0) {
            const int done = shift == SMP_BITS - 8 ? 12 : shift == SMP_BITS - 16 ? 20 : 28;      // bits already fixed
            const int width = done == 28 ? 4 : 8;
            if (tid < 256) hist[tid] = 0.0;
            __syncthreads();
            const unsigned prefix = s_prefix, mask = ~0u << (32 - done);
            for (int j = tid; j < n; j += SMP_PICK) {
                const float p = a.prob[a.list[j]];
                const unsigned bits = __float_as_uint(p);
                if ((bits & mask) == prefix) atomicAdd(&hist[(bits >> shift) & ((1u << width) - 1u)], (double)p);
            }
            __syncthreads();
            if (tid < 32) {
                // the digit at which the running mass reaches the target: lane l owns digits 255 - 8 l ... 248 - 8 l
                double c[8], own = 0.0;
#pragma unroll
                for (int k = 0; k < 8; k++) { c[k] = hist[255 - 8 * lane - k]; own += c[k]; }
                double incl = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                double run = s_run + (incl - own);
                const bool reach = run + own >= target;
                const unsigned who = __ballot_sync(0xffffffffu, reach && own != 0.0);
                const unsigned some = __ballot_sync(0xffffffffu, own != 0.0);
                // (rounding may leave the target just past the last member: then the lowest digit present)
                const int leader = who ? __ffs(who) - 1 : some ? 31 - __clz(some) : 31;
                __syncwarp();
                if (lane == leader) {
                    int d = 0, low = 0;
                    double low_run = run;
                    bool found = false;
                    for (int k = 0; k < 8 && !found; k++) {
                        if (c[k] == 0.0) continue;
                        low = k; low_run = run;
                        if (run + c[k] >= target) found = true;
                        else run += c[k];
                    }
                    d = 255 - 8 * lane - low;
                    s_run = low_run;
                    s_prefix = prefix | ((unsigned)d << shift);
                }
            }
            __syncthreads();
            if (shift == 0) break;
        }
        tau = s_prefix;
        for (int j = tid; j < n; j += SMP_PICK) {
            const int i = a.list[j];
            const float p = a.prob[i];
            if (__float_as_uint(p) >= tau) atomicAdd(&range_mass[i / a.range], (double)p);
        }
    }
    __syncthreads();
    // ---- the draw: the range that holds the point, then the token
    double total;
    const double own = range_mass[tid], upto = block_scan(own, red, total);
    const double u = (double)(smp_mix64(a.seed ^ smp_mix64(a.step + 1)) >> 11) * (1.0 / 9007199254740992.0);
    const double want = u * total;
    if (own != 0.0) { atomicMax(&s_last, tid); if (upto > want) atomicMin(&s_owner, tid); }
    __syncthreads();
    const int owner = s_owner < a.parts ? s_owner : s_last >= 0 ? s_last : 0;
    if (tid == owner) s_run = upto - own;
    __syncthreads();
    const int i0 = owner * a.range, i1 = min(a.V, i0 + a.range);
    if (tid == 0) s_last = -1;
    double run = s_run;
    for (int base = i0; base < i1; base += SMP_PICK) {
        const int i = base + tid;
        const float p = i < i1 ? a.prob[i] : 0.f;
        const bool keep = i < i1 && __float_as_uint(p) >= tau;
        double sum;
        const double at = run + block_scan(keep ? (double)p : 0.0, red, sum);   // (its barriers order s_last above)
        if (keep) { atomicMax(&s_last, i); if (at > want) atomicMin(&s_pick, i); }
        __syncthreads();
        if (s_pick < a.V) break;
        run += sum;
    }
    __syncthreads();
    if (tid == 0) *a.out = s_pick < a.V ? s_pick : s_last >= 0 ? s_last : 0;     // rounding left the point just past the last member
}

// Scratch: [bins | masses] doubles, [prob] floats, [list] ints, [top] floats, the rest.
static size_t sample_parts(int V, int &range)
{
    range = (V + SMP_MAX_PARTS - 1) / SMP_MAX_PARTS;
    if (range < SMP_RANGE) range = SMP_RANGE;
    return (size_t)((V + range - 1) / range);
}

size_t sample_scratch_bytes(int V)
{
    return (SMP_BINS + SMP_MAX_PARTS + 1) * sizeof(double) + (size_t)V * 8 + SMP_MAX_PARTS * 4 + 8;
}

void sample_token(cudaStream_t st, int *out, const float *logits, void *scratch, int V, float temperature, float top_p,
                  uint64_t seed, uint64_t step)
{
    SampleArgs a;
    a.logits = logits;
    a.bins = static_cast<double *>(scratch);
    a.mass = a.bins + SMP_BINS;
    a.above = a.mass + SMP_MAX_PARTS;
    a.prob = reinterpret_cast<float *>(a.above + 1);
    a.list = reinterpret_cast<int *>(a.prob + V);
    a.top = reinterpret_cast<float *>(a.list + V);
    a.count = reinterpret_cast<int *>(a.top + SMP_MAX_PARTS);
    a.out = out;
    a.V = V; a.temperature = temperature; a.top_p = top_p; a.seed = seed; a.step = step;
    a.parts = (int)sample_parts(V, a.range);
    G5B_LAUNCH_PDL(sample_max_kernel, dim3(a.parts), dim3(SMP_THREADS), 0, st, a);
    G5B_LAUNCH_PDL(sample_prob_kernel, dim3(a.parts), dim3(SMP_THREADS), 0, st, a);
    if (top_p < 1.0f) G5B_LAUNCH_PDL(sample_cut_kernel, dim3(a.parts), dim3(SMP_THREADS), 0, st, a);
    G5B_LAUNCH_PDL(sample_pick_kernel, dim3(1), dim3(SMP_PICK), 0, st, a);
}

}  // namespace g5b
