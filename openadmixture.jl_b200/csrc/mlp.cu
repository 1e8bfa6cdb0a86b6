/*
 * mlp.cu -- the learned warm start: genotype sketch, a small MLP encoder (forward, backward,
 * Adam) and the closed-form P step that turns a predicted Q into a starting P.
 *
 * This part has no counterpart in the reference.  Its hook is run_admixture's init_q / init_p
 * (driver.jl:52-53,161-166,183-188): the predicted Q and the derived P replace the random start
 * and the EM priming.
 *
 * Features of individual i: the dosages of S fixed sketch SNPs (int8; 3 = missing) and R
 * projections of the frequency-standardised dosages onto fixed +-1 directions,
 *   proj_ir = S^-1/2 sum_s (d_is - 2 f_s) / sqrt(2 f_s (1 - f_s)) * sign_rs     (missing -> 0).
 * Network: x = [d - 2f | proj] (S + R) -> ReLU(W1 x + b1) (H) -> ReLU(W2 . + b2) (H) ->
 * softmax(W3 . + b3) (K).  Loss: cross-entropy against soft targets (aligned converged Q).
 * All matrices are row-major FP32 (W1: (S+R) x H, W2: H x H, W3: H x K).
 *
 * Every product of the forward and backward passes is one tensor-core GEMM (k_gemm_tc): a CTA
 * owns a 128 x 64 tile of the output in TMEM; each 32-deep slice of the reduction is loaded by
 * the CTA's threads through an operand functor (dense, transposed, or the network input built
 * on the fly from the dosages), split into BF16 high and low parts, and multiplied as
 * hi*hi + lo*hi + hi*lo by tcgen05 (about 2^-17 relative per product, FP32 accumulation).  The
 * accumulator restarts every 128 of the reduction and the threads add it into FP32 registers,
 * so no FP32 partial sees more than 24 of the tensor core's accumulations.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "../../include/admix.h"
#include "col_words.h"
#include "common.cuh"
#include "synth.h"
#include "tc05.cuh"

namespace cg = cooperative_groups;

namespace {

/* 2-bit code -> dosage: 00 -> 0, 10 -> 1, 11 -> 2, 01 (missing) -> 3 */
__device__ __forceinline__ int8_t dosage_of(int c) { return c == 1 ? (int8_t)3 : (int8_t)(c == 0 ? 0 : c - 1); }

/* Allele frequency of each sketch SNP: one block per SNP.  The dosage sum and the non-missing count are integers by
 * popcount of the code bits (codes 10 and 11 have the high bit, 11 also the low one; 01 is missing), a word at a time
 * where the columns are word-aligned. */
__global__ void __launch_bounds__(128)
k_sketch_freq(const uint8_t *__restrict__ bed, int64_t pitch, int64_t I, const int32_t *__restrict__ snps,
              float *__restrict__ freq)
{
    __shared__ double red[4];
    const uint8_t *col = bed + (size_t)snps[blockIdx.x] * pitch;
    const int64_t Ib = (I + 3) / 4, full = I / 4;    /* bytes; bytes without padding bits */
    long long a = 0, n = 0;
    auto add = [&](uint32_t v, uint32_t mask) {
        const uint32_t lo = v & 0x55555555u & mask, hi = (v >> 1) & 0x55555555u & mask;
        a += __popc(hi) + __popc(hi & lo);
        n += __popc(mask & 0x55555555u) - __popc(lo & ~hi);
    };
    int64_t b0 = 0;
    if ((((uintptr_t)bed | (uintptr_t)pitch) & 3u) == 0) {
        const int64_t nw = full / 4;
        for (int64_t w = threadIdx.x; w < nw; w += blockDim.x) add(__ldg((const uint32_t *)col + w), 0xFFFFFFFFu);
        b0 = 4 * nw;
    }
    for (int64_t b = b0 + threadIdx.x; b < Ib; b += blockDim.x)
        add(col[b], b < full ? 0xFFu : (1u << (2 * (int)(I & 3))) - 1u);
    const double sa = block_sum((double)a, red);
    const double sn = block_sum(2.0 * (double)n, red);
    if (threadIdx.x == 0) freq[blockIdx.x] = sn > 0.0 ? (float)(sa / sn) : 0.5f;
}

/* Dosage sketch (I x S int8) and the R standardised projections (I x R).  A block owns the 4 individuals of one byte of
 * the columns, a thread every 256th sketch SNP: its byte, its hash (the signs) and its standardisation serve
 * four individuals, and the next SNP's byte is in flight while this one's 32 sums are formed.  With one individual
 * a block, the gathers and the hash were repeated for each: 20,000 x 4,096 in 0.90 ms, now 0.45.  Bound: one FMA
 * per cell and direction and the signs' unpacking, at the 8 warps per SM that 128 sums a thread allow. */
constexpr int SK_THREADS = 256;

__global__ void __launch_bounds__(SK_THREADS, 1)
k_sketch(const uint8_t *__restrict__ bed, int64_t pitch, int64_t I, const int32_t *__restrict__ snps,
         int S, const float *__restrict__ freq, int R, uint64_t seed, int8_t *__restrict__ dos,
         float *__restrict__ proj)
{
    __shared__ float sh[4][SK_THREADS / 32][32];      /* the warps' sums */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint8_t *row = bed + blockIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * 4;
    const int ni = (int)min((int64_t)4, I - i0);
    float acc[4][32];
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int r = 0; r < 32; ++r) acc[v][r] = 0.f;
    uint32_t byte = 0u;
    int32_t next = 0;
    float f = 0.f, fn = 0.f;
    if (tid < S) {
        byte = row[(size_t)snps[tid] * pitch];
        f = freq[tid];
    }
    if (tid + SK_THREADS < S) next = snps[tid + SK_THREADS];
    for (int s = tid; s < S; s += SK_THREADS) {
        uint32_t bn = 0u;
        if (s + SK_THREADS < S) {
            bn = row[(size_t)next * pitch];
            fn = freq[s + SK_THREADS];
        }
        if (s + 2 * SK_THREADS < S) next = snps[s + 2 * SK_THREADS];
        const float w = rsqrtf(fmaxf(2.f * f * (1.f - f), 1e-6f));
        const uint32_t h = (uint32_t)syn_hash3(seed, (uint64_t)s, 0);
        float z[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const uint32_t c = (byte >> (2 * v)) & 3u;
            const int8_t d = dosage_of((int)c);
            if (v < ni) dos[(size_t)(i0 + v) * S + s] = d;
            z[v] = c == 1u ? 0.f : ((float)d - 2.f * f) * w;   /* a missing dosage adds 0 to every sum */
        }
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            const float sg = __uint_as_float(0xBF800000u ^ ((h << (31 - r)) & 0x80000000u));   /* bit r: +1, else -1 */
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[v][r] = fmaf(z[v], sg, acc[v][r]);
        }
        byte = bn;
        f = fn;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            float x = acc[v][r];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) sh[v][warp][r] = x;
        }
    __syncthreads();
    const float scale = rsqrtf((float)S);
    const int v = tid >> 5;
    if (v < ni && lane < R) {
        float x = 0.f;
        for (int w = 0; w < SK_THREADS / 32; ++w) x += sh[v][w][lane];
        proj[(size_t)(i0 + v) * R + lane] = x * scale;
    }
}

} // namespace

extern "C" int admix_sketch(const uint8_t *d_bed, int64_t pitch, int64_t I, const int32_t *d_snps, int32_t S,
                            int32_t R, uint64_t seed, float *d_freq, int8_t *d_dos, float *d_proj, void *stream)
{
    if (!d_bed || !d_snps || !d_freq || !d_dos || !d_proj || I < 1 || S < 1 || R < 0 || R > 32 || pitch < (I + 3) / 4)
        return ADMIX_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    k_sketch_freq<<<S, 128, 0, st>>>(d_bed, pitch, I, d_snps, d_freq);
    k_sketch<<<(unsigned)((I + 3) / 4), SK_THREADS, 0, st>>>(d_bed, pitch, I, d_snps, S, d_freq, R, seed, d_dos, d_proj);
    return cudaGetLastError() == cudaSuccess ? ADMIX_OK : ADMIX_ERR_CUDA;
}

namespace {

/* ---- operand loaders: row r of an operand, 8 consecutive elements of the reduction from c0 (a multiple of 8).  load()
 * only reads memory, so that a slice's reads are all in flight together and a slice ahead of their use;
 * values() turns them into numbers, zero past the operand's bounds. ---- */
struct LoadF {                     /* dense FP32: element (r, c) at p[r * sr + c * sc] */
    const float *p; int64_t sr, sc;
    struct Raw { float v[8]; };
    __device__ __forceinline__ void load(Raw &w, int64_t r, int64_t c0, int64_t rows, int64_t cols) const
    {
        const float *q = p + r * sr + c0 * sc;
        if (sc == 1 && (((uintptr_t)p | (uintptr_t)(sr * 4)) & 15u) == 0 && r < rows && c0 + 8 <= cols) {
            const float4 a = *(const float4 *)q, b = *(const float4 *)(q + 4);
            w.v[0] = a.x; w.v[1] = a.y; w.v[2] = a.z; w.v[3] = a.w;
            w.v[4] = b.x; w.v[5] = b.y; w.v[6] = b.z; w.v[7] = b.w;
            return;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) w.v[e] = (r < rows && c0 + e < cols) ? q[e * sc] : 0.f;
    }
    __device__ __forceinline__ void values(float (&v)[8], const Raw &w, int64_t, int64_t, int64_t, int64_t) const
    {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = w.v[e];
    }
};
/* the network input [dosage - 2f (0 if missing) | projections]; a dosage byte or a projection's bits per element */
struct LoadX {                     /* row = individual, reduction = feature */
    const int8_t *dos; const float *center; const float *proj; int S, R;
    struct Raw { uint32_t v[8]; };
    __device__ __forceinline__ void load(Raw &w, int64_t m, int64_t k0, int64_t rows, int64_t cols) const
    {
        if (m < rows && k0 + 8 <= S && (((uintptr_t)dos | (uintptr_t)S) & 7u) == 0) {
            const uint2 x = *(const uint2 *)(dos + m * S + k0);   /* k0 is a multiple of 8 */
#pragma unroll
            for (int e = 0; e < 8; ++e) w.v[e] = ((e < 4 ? x.x : x.y) >> (8 * (e & 3))) & 0xFFu;
            return;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int64_t k = k0 + e;
            w.v[e] = 0u;
            if (m < rows && k < cols) w.v[e] = k < S ? (uint32_t)(uint8_t)dos[m * S + k] : __float_as_uint(proj[m * R + (k - S)]);
        }
    }
    __device__ __forceinline__ void values(float (&v)[8], const Raw &w, int64_t m, int64_t k0, int64_t rows, int64_t cols) const
    {
        if (k0 + 8 <= S) {
            float c[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) c[e] = __ldg(center + k0 + e);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = (m < rows && w.v[e] != 3u) ? (float)(int8_t)w.v[e] - c[e] : 0.f;
            return;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int64_t k = k0 + e;
            if (k < S) v[e] = (m < rows && w.v[e] != 3u) ? (float)(int8_t)w.v[e] - __ldg(center + k) : 0.f;
            else v[e] = __uint_as_float(w.v[e]);
        }
    }
};
struct LoadXT {                    /* row = feature, reduction = individual */
    LoadX x;
    struct Raw { uint32_t v[8]; };
    __device__ __forceinline__ void load(Raw &w, int64_t k, int64_t m0, int64_t rows, int64_t cols) const
    {
        if (k < x.S) {
#pragma unroll
            for (int e = 0; e < 8; ++e) w.v[e] = m0 + e < cols ? (uint32_t)(uint8_t)x.dos[(m0 + e) * x.S + k] : 3u;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) w.v[e] = (k < rows && m0 + e < cols) ? __float_as_uint(x.proj[(m0 + e) * x.R + (k - x.S)]) : 0u;
        }
    }
    __device__ __forceinline__ void values(float (&v)[8], const Raw &w, int64_t k, int64_t, int64_t, int64_t) const
    {
        const float c = k < x.S ? __ldg(x.center + k) : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = k < x.S ? (w.v[e] == 3u ? 0.f : (float)(int8_t)w.v[e] - c) : __uint_as_float(w.v[e]);
    }
};

constexpr int GT_M = 128, GT_N = 64, GT_K = 32;   /* output tile rows x columns, reduction slice */
constexpr int GT_THREADS = 512;
constexpr int GT_D = 4;                             /* slices per fresh accumulation */
constexpr uint32_t GT_WAIT = 1u << 22;              /* polls of a bounded wait */
/* one stage: A hi, A lo (128 x 32 BF16, K-major core matrices), B hi, B lo (64 x 32) */
constexpr uint32_t GT_A = GT_M * GT_K * 2, GT_B = GT_N * GT_K * 2;
constexpr uint32_t GT_STAGE = 2 * GT_A + 2 * GT_B;
constexpr uint32_t GT_SMEM = 2 * GT_STAGE + 1024;
constexpr uint32_t GT_PART = GT_M * GT_N * 4;       /* one block's FP32 sums */
constexpr uint32_t GT_A_LBO = GT_M * 16, GT_B_LBO = GT_N * 16;

/* 8 values as BF16 high parts (rounded to nearest) and the BF16 of the remainders, v = hi + lo, packed in pairs */
__device__ __forceinline__ void split8(const float (&v)[8], uint4 &hi, uint4 &lo)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        h[e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
        l[e] = pack_bf16x2(v[2 * e] - __uint_as_float(h[e] << 16), v[2 * e + 1] - __uint_as_float(h[e] & 0xFFFF0000u));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

/* C[m, n] = alpha * sum_k A(m, k) B(k, n) (+ bias[n]); relu if act; times [mask(m, n) > 0] if mask.
 * 512 threads, one 128 x 64 output tile per CTA: thread t owns output row (TMEM lane) 32 (warp % 4) + lane and the 16
 * columns from 16 (warp / 4), and converts one granule of A (row t % 128) and, for t < 256, one of B.  Two smem
 * stages: the threads convert slice c+1 while the tensor core multiplies slice c, and the global reads of
 * slice c+2 are in flight meanwhile.  B is given by its rows: element (n, k) of loader B is B(k, n).
 * Bound: the operands' conversion on the CUDA cores, at the latency of one slice where the grid is small (hence 12
 * elements a thread).  128 threads that read each of their 48 elements where they converted it put 48 memory
 * latencies in series: the encoder's first layer on 20,000
 * individuals took 2.78 ms, its weight gradient on 4,096 2.27 ms; now 0.75 and 0.20.  Every wait is
 * bounded; a CTA whose wait runs out writes NaN into its tile, and the ReLU keeps NaN, so that the failure shows in the loss.
 *
 * CL > 1: a cluster of CL CTAs shares a tile.  Each takes nb blocks of GT_D slices at a time and leaves every block's
 * sums in its shared memory; then each adds all CTAs' blocks for its 16 / CL of a thread's columns, in the order
 * of the reduction, so the result is bit for bit that of one CTA (a CTA whose wait ran out leaves NaN in its slots).  A
 * 256 x 256 weight gradient over 4,096 individuals (8 tiles) took one CTA per tile 176 us at the latency of its 128
 * slices.  CL = 2 keeps the 64 registers of two CTAs per SM, but its blocks' slots (113 KB) leave room for one. */
template <class LA, class LB, int CL>
__global__ void __launch_bounds__(GT_THREADS, CL == 8 ? 1 : 2)
k_gemm_tc(LA A, LB B, int64_t M, int64_t N, int64_t Kd, float alpha, const float *__restrict__ bias, int act,
          const float *__restrict__ mask, float *__restrict__ C, int64_t ldc, int nb)
{
    constexpr int NE = 16 / CL;          /* columns a thread owns in the end */
    extern __shared__ __align__(1024) uint8_t smraw[];
    uint8_t *sm = (uint8_t *)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t bar[2];          /* MMAs of the slice in stage s done */
    __shared__ uint32_t tmem_holder;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int64_t m0 = (int64_t)blockIdx.y * GT_M, n0 = (int64_t)blockIdx.x * GT_N;
    if (warp == 0) tmem_alloc_warp(&tmem_holder, GT_N);
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_holder;
    const int col0 = 16 * (warp >> 2);
    const uint32_t my_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    bool ok = true;
    auto wait = [&](uint64_t *b, uint32_t parity) {
        if (!ok) return;
        for (uint32_t n = 0; n < GT_WAIT; ++n) {
            if (mbar_try_wait(b, parity)) return;
            if ((n & 255u) == 255u && abort_flag) break;
        }
        ok = false;
        abort_flag = 1;
    };
    float acc[NE];
#pragma unroll
    for (int n = 0; n < NE; ++n) acc[n] = 0.f;
    float *part = (float *)(sm + 2 * GT_STAGE) + tid;     /* element e of block slot b: part[(16 b + e) * GT_THREADS] */
    auto drain = [&](int slot) {   /* the finished accumulation block into the FP32 registers or its slot */
        tc_fence_after_sync();
        float v[16];
        tmem_ld16(my_tmem, v);
        if constexpr (CL == 1) {
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[e] += v[e];
        } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) part[(16 * slot + e) * GT_THREADS] = v[e];
        }
    };
    const int nch = (int)((Kd + GT_K - 1) / GT_K), nblk = (nch + GT_D - 1) / GT_D;
    const int rank = CL == 1 ? 0 : (int)blockIdx.z, rounds = CL == 1 ? 1 : (nblk + CL * nb - 1) / (CL * nb);
    /* this CTA's slices of a round */
    auto first = [&](int round) { return CL == 1 ? 0 : (round * CL + rank) * nb * GT_D; };
    auto count = [&](int round) { return CL == 1 ? nch : max(0, min(nch - first(round), nb * GT_D)); };
    constexpr uint32_t idesc = idesc_bf16_f32(GT_M, GT_N);
    typename LA::Raw ra;
    typename LB::Raw rb;
    const int am = tid & (GT_M - 1), ag = tid >> 7, bn = tid & (GT_N - 1), bg = tid >> 6;
    const bool hasb = tid < GT_N * GT_K / 8;
    static_assert(GT_M * GT_K / 8 == GT_THREADS, "one granule of A a thread");
    auto fetch = [&](int c) {
        const int64_t k0 = (int64_t)c * GT_K;
        A.load(ra, m0 + am, k0 + 8 * ag, M, Kd);
        if (hasb) B.load(rb, n0 + bn, k0 + 8 * bg, N, Kd);
    };
    if (count(0) > 0) fetch(first(0));
    int n = 0;                                            /* slices so far */
    for (int round = 0; round < rounds; ++round) {
        const int c0 = first(round), len = count(round);
        for (int i = 0; i < len; ++i, ++n) {
            const int c = c0 + i, st = n & 1;
            uint8_t *Ah = sm + st * GT_STAGE, *Al = Ah + GT_A, *Bh = Al + GT_A, *Bl = Bh + GT_B;
            if (n >= 2) wait(&bar[st], (uint32_t)(((n - 2) >> 1) & 1));   /* stage st is free again */
            const int64_t k0 = (int64_t)c * GT_K;
            float v[8];
            uint4 h, l;
            A.values(v, ra, m0 + am, k0 + 8 * ag, M, Kd);
            split8(v, h, l);
            *(uint4 *)(Ah + ag * GT_A_LBO + 16 * am) = h;
            *(uint4 *)(Al + ag * GT_A_LBO + 16 * am) = l;
            if (hasb) {
                B.values(v, rb, n0 + bn, k0 + 8 * bg, N, Kd);
                split8(v, h, l);
                *(uint4 *)(Bh + bg * GT_B_LBO + 16 * bn) = h;
                *(uint4 *)(Bl + bg * GT_B_LBO + 16 * bn) = l;
            }
            if (i + 1 < len) fetch(c + 1);
            else if (round + 1 < rounds && count(round + 1) > 0) fetch(first(round + 1));
            fence_async_smem();
            if (i > 0 && i % GT_D == 0) {   /* the block ending at the slice before: its MMAs done */
                wait(&bar[(n - 1) & 1], (uint32_t)(((n - 1) >> 1) & 1));
                if (ok) drain(i / GT_D - 1);
            }
            tc_fence_before_sync();
            __syncthreads();
            tc_fence_after_sync();
            if (tid == 0 && ok) {
                const uint32_t ah = smem_u32(Ah), al = smem_u32(Al), bh = smem_u32(Bh), bl = smem_u32(Bl);
#pragma unroll
                for (int ks = 0; ks < GT_K / 16; ++ks) {
                    const uint32_t ao = ks * 2 * GT_A_LBO, bo = ks * 2 * GT_B_LBO;
                    const uint32_t fresh = (i % GT_D == 0 && ks == 0) ? 0u : 1u;
                    tc_mma_bf16(tmem, umma_desc_kmajor(ah + ao, GT_A_LBO, 128), umma_desc_kmajor(bh + bo, GT_B_LBO, 128),
                                idesc, fresh);
                    tc_mma_bf16(tmem, umma_desc_kmajor(al + ao, GT_A_LBO, 128), umma_desc_kmajor(bh + bo, GT_B_LBO, 128),
                                idesc, 1u);
                    tc_mma_bf16(tmem, umma_desc_kmajor(ah + ao, GT_A_LBO, 128), umma_desc_kmajor(bl + bo, GT_B_LBO, 128),
                                idesc, 1u);
                }
                tc_commit(&bar[st]);
            }
        }
        if (len > 0) {   /* the last block */
            wait(&bar[(n - 1) & 1], (uint32_t)(((n - 1) >> 1) & 1));
            if (ok) drain((len - 1) / GT_D);
        }
        if constexpr (CL > 1) {
            cg::cluster_group cl = cg::this_cluster();
            ok = __syncthreads_and(ok);
            if (!ok)
                for (int e = 0; e < 16 * nb; ++e) part[e * GT_THREADS] = __int_as_float(0x7fc00000);
            cl.sync();
            const int left = nblk - round * CL * nb;              /* blocks from this round on */
            for (int r = 0; r < CL; ++r) {
                const float *src = cl.map_shared_rank(part, r) + (size_t)rank * NE * GT_THREADS;
                for (int slot = 0; slot < min(nb, left - r * nb); ++slot)
#pragma unroll
                    for (int e = 0; e < NE; ++e) acc[e] += src[(16 * slot + e) * GT_THREADS];
            }
            cl.sync();                                            /* the slots are read */
        }
    }
    ok = __syncthreads_and(ok);
    if (!ok && tid == 0) {   /* give MMAs still in flight a bounded moment before the TMEM goes */
        mbar_wait_bounded(&bar[0], 0u, 1024u); mbar_wait_bounded(&bar[0], 1u, 1024u);
        mbar_wait_bounded(&bar[1], 0u, 1024u); mbar_wait_bounded(&bar[1], 1u, 1024u);
    }
    const int64_t m = m0 + 32 * (warp & 3) + (tid & 31);
    if (m < M) {
#pragma unroll
        for (int n = 0; n < NE; ++n) {
            const int64_t col = n0 + col0 + rank * NE + n;
            if (col >= N) break;
            float v = alpha * acc[n] + (bias ? bias[col] : 0.f);
            if (act && v <= 0.f) v = 0.f;                         /* NaN stays */
            if (mask && !(mask[m * ldc + col] > 0.f)) v = 0.f;
            C[m * ldc + col] = ok ? v : __int_as_float(0x7fc00000);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc_warp(tmem, GT_N);
}

/* The dynamic shared memory limit belongs to the device, and callers may change devices and threads between two calls: set
 * before every launch (0.2 us) instead of remembered. */
template <class LA, class LB, int CL>
cudaError_t allow_smem(size_t bytes)
{
    return cudaFuncSetAttribute(k_gemm_tc<LA, LB, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

/* A tile per cluster of CL CTAs, each holding at most NB blocks' sums at a time */
template <int CL, int NB, class LA, class LB>
cudaError_t gemm_split(LA A, LB B, int64_t M, int64_t N, int64_t Kd, float alpha, const float *bias, int act,
                       const float *mask, float *C, int64_t ldc, dim3 grid, int64_t nblk, cudaStream_t st)
{
    const cudaError_t e = allow_smem<LA, LB, CL>(GT_SMEM + NB * GT_PART);
    if (e != cudaSuccess) return e;
    const int64_t rounds = (nblk + CL * NB - 1) / (CL * NB);
    const int nb = (int)((nblk + CL * rounds - 1) / (CL * rounds));
    grid.z = CL;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = CL;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(GT_THREADS);
    cfg.dynamicSmemBytes = GT_SMEM + (size_t)nb * GT_PART;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_gemm_tc<LA, LB, CL>, A, B, M, N, Kd, alpha, bias, act, mask, C, ldc, nb);
}

template <class LA, class LB>
cudaError_t gemm(LA A, LB B, int64_t M, int64_t N, int64_t Kd, float alpha, const float *bias, int act,
                 const float *mask, float *C, int64_t ldc, cudaStream_t st)
{
    dim3 grid((unsigned)((N + GT_N - 1) / GT_N), (unsigned)((M + GT_M - 1) / GT_M));
    const int64_t tiles = (int64_t)grid.x * grid.y, nblk = (Kd + GT_K * GT_D - 1) / (GT_K * GT_D);
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    /* Few tiles leave most SMs idle.  Eight CTAs per tile (one per SM: 177 KB) up to 4/3 of a wave, a sixth of the SMs' number of
     * tiles: encoder forward pass of 300 / 640 / 1,024 individuals (12 / 20 / 32 tiles on 148 SMs, 33 blocks in its first layer)
     * 91 / 133 / 180 us, with one CTA per tile 238 / 227 / 229, with two 172 / 168 / 168.  Two (one per SM as well: 113 KB) up to
     * one wave: 2,048 individuals (64 tiles) 175 us against 230; at 128 tiles 307 against 233.  Two blocks are worth
     * eight CTAs (40 individuals, second layer too: 86 -> 78 us); two CTAs need the blocks to pay for their rounds. */
    if (6 * tiles <= sms && nblk >= 2)
        return gemm_split<8, 4>(A, B, M, N, Kd, alpha, bias, act, mask, C, ldc, grid, nblk, st);
    if (2 * tiles <= sms && nblk >= 8)
        return gemm_split<2, 2>(A, B, M, N, Kd, alpha, bias, act, mask, C, ldc, grid, nblk, st);
    e = allow_smem<LA, LB, 1>(GT_SMEM);
    if (e != cudaSuccess) return e;
    k_gemm_tc<LA, LB, 1><<<grid, GT_THREADS, GT_SMEM, st>>>(A, B, M, N, Kd, alpha, bias, act, mask, C, ldc, 0);
    return cudaGetLastError();
}

/* row softmax of logits (n x K) into probs; with targets: dlogits = (probs - target) / n and the
 * summed cross-entropy added (atomically) into *loss */
__global__ void k_softmax_ce(const float *__restrict__ logits, int64_t n, int K, float *__restrict__ probs,
                             const float *__restrict__ target, float *__restrict__ dlogits, float *__restrict__ loss)
{
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    const float *z = logits + m * K;
    float mx = z[0];
    for (int k = 1; k < K; ++k) mx = fmaxf(mx, z[k]);
    float s = 0.f;
    for (int k = 0; k < K; ++k) s += expf(z[k] - mx);
    const float ls = logf(s);
    float l = 0.f;
    for (int k = 0; k < K; ++k) {
        const float pk = expf(z[k] - mx - ls);
        probs[m * K + k] = pk;
        if (target) {
            dlogits[m * K + k] = (pk - target[m * K + k]) / (float)n;
            l -= target[m * K + k] * (z[k] - mx - ls);
        }
    }
    if (target && loss) atomicAdd(loss, l);
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                       float *__restrict__ m2, int64_t n, float lr, float b1, float b2, float eps, float c1, float c2)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const float gt = g[t];
        const float a = b1 * m1[t] + (1.f - b1) * gt, b = b2 * m2[t] + (1.f - b2) * gt * gt;
        m1[t] = a; m2[t] = b;
        w[t] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
    }
}

} // namespace

namespace {

/* column sums of dY (M x N), a thread per column and row slice, 32 reads in flight: four launches of a backward
 * pass on 4,096 individuals took 12 us more with one at a time */
__global__ void k_colsum_atomic(const float *__restrict__ dY, int64_t M, int64_t N, float *__restrict__ db)
{
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const int64_t rows = (M + gridDim.y - 1) / gridDim.y;
    const int64_t m0 = (int64_t)blockIdx.y * rows, m1 = min(M, m0 + rows);
    float s = 0.f;
#pragma unroll 32
    for (int64_t m = m0; m < m1; ++m) s += __ldg(dY + m * N + n);
    atomicAdd(db + n, s);
}

cudaError_t colsum(const float *dY, int64_t M, int64_t N, float *db, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(db, 0, sizeof(float) * N, st);
    if (e != cudaSuccess) return e;
    const unsigned gy = (unsigned)std::min<int64_t>(64, std::max<int64_t>(1, M / 256));
    k_colsum_atomic<<<dim3((unsigned)((N + 127) / 128), gy), 128, 0, st>>>(dY, M, N, db);
    return cudaGetLastError();
}

struct ColRead {
    __device__ __forceinline__ uint32_t byte(const uint8_t *p) const { return __ldg(p); }
    __device__ __forceinline__ uint32_t word(const uint8_t *p) const { return __ldg((const uint32_t *)p); }
};

/* closed-form P step from Q: p_kj = sum_i nm q_ki g_ij / (2 sum_i nm q_ki), clamped to
 * [1e-5, 1-1e-5] like project_p! (projections.jl:69-74).  A thread owns two SNPs, one in each half of its paired
 * FP32 sums; q is staged through shared memory 64 individuals at a time with each value twice, so a pair of cells
 * takes one paired FMA per cluster and sum and no duplication of the genotype factors, which a table gives per code
 * pair.  A missing cell adds zeros, so no thread branches on the genotype.  Each sum is the same per-k FP32 sequence
 * as a per-cell loop that skips the missing cells.  W = 8: columns aligned to 8 bytes; otherwise
 * aligned words, shifted (col_words.h).
 * Bound: instruction issue at the few warps that J / 2 threads are (the sums of a SNP are serial chains over the
 * individuals).  I=20k, J=100k, K=8: 2.53 ms with one SNP a thread and a byte per load, 1.88 now; two pairs a
 * thread, or the clusters split over two threads, repeat the staging or the decoding and take 2.35 to 2.46.
 * Registers up to K = 8: as many as it takes; left to itself the compiler chose 72 with spills for K = 3 (4,001 x 1,003,
 * unaligned columns: 150 us, 123 so).  Above, its own choice: K = 11 at 20,003 x 100,001 takes 2.66 ms, 3.42 with more. */
template <int K, int W>
__global__ void __launch_bounds__(64, K <= 8 ? 1 : 0)
k_warm_p(const uint8_t *__restrict__ bed, int64_t pitch, int64_t I, int64_t J, const double *__restrict__ q,
         double *__restrict__ p)
{
    constexpr int K2 = (K + 1) / 2;                  /* 16-byte groups of two doubled values per individual */
    __shared__ __align__(16) float4 qs[64 * K2];
    const int64_t ja = ((int64_t)blockIdx.x * 64 + threadIdx.x) * 2, jb = ja + 1;
    const uint8_t *ca = bed + (size_t)(ja < J ? ja : 0) * pitch, *cb = bed + (size_t)(jb < J ? jb : 0) * pitch;
    const int64_t Ib = (I + 3) / 4;
    float2 num[2 * K2], den[2 * K2];                  /* (SNP a, SNP b): sum_i q_ki g_ij and sum_i nm q_ki */
#pragma unroll
    for (int k = 0; k < 2 * K2; ++k) num[k] = den[k] = make_float2(0.f, 0.f);
    /* factors by code pair (code of a | code of b << 2): (g_a, g_b) and (nm_a, nm_b) as BF16 pairs (exact), 16 copies
     * so that a half-warp's 8-byte loads never share a bank */
    __shared__ __align__(16) uint2 tab[16 * 16];
    for (int t = threadIdx.x; t < 256; t += 64) {
        const uint32_t c0 = (uint32_t)(t >> 4) & 3u, c1 = (uint32_t)(t >> 6);
        auto gf = [](uint32_t c) { return c == 3u ? 2.f : (c == 2u ? 1.f : 0.f); };   /* codes 00 -> 0, 10 -> 1, 11 -> 2 */
        auto mf = [](uint32_t c) { return c == 1u ? 0.f : 1.f; };                      /* 01: missing */
        tab[t] = make_uint2(pack_bf16x2(gf(c0), gf(c1)), pack_bf16x2(mf(c0), mf(c1)));
    }
    const uint8_t *tl = (const uint8_t *)tab + 8 * (threadIdx.x & 15);
    /* 8 two-bit codes spread to the low halves of 8 nibbles */
    auto spread = [](uint32_t x) {
        x = (x | (x << 8)) & 0x00FF00FFu;
        x = (x | (x << 4)) & 0x0F0F0F0Fu;
        return (x | (x << 2)) & 0x33333333u;
    };
    /* the 16 bytes of 64 individuals of a column, missing past its end */
    auto codes = [&](const uint8_t *col, int64_t i0, int64_t limit, uint32_t (&w)[4]) {
        const int64_t b0 = i0 >> 2;
#pragma unroll
        for (int v = 0; v < 4; ++v) w[v] = 0x55555555u;
        if (b0 + 16 <= limit) {
            if (W == 8) {
                const uint2 x = __ldg((const uint2 *)(col + b0)), y = __ldg((const uint2 *)(col + b0) + 1);
                w[0] = x.x; w[1] = x.y; w[2] = y.x; w[3] = y.y;
            } else {
                block_words(ColRead{}, col + b0, w);
            }
        } else {
            block_bytes(ColRead{}, col, b0, Ib, w);
        }
    };
    /* this thread's q values of the next 64 individuals; 0 past I, which adds nothing whatever the codes there */
    float qa[K2], qb[K2];
    auto fetch = [&](int64_t i0) {
#pragma unroll
        for (int e = 0; e < K2; ++e) {
            const int t = threadIdx.x + e * 64, ii = t / K2, k = 2 * (t - ii * K2);
            const double *src = q + (size_t)K * (i0 + ii) + k;
            qa[e] = i0 + ii < I ? (float)src[0] : 0.f;
            qb[e] = (i0 + ii < I && k + 1 < K) ? (float)src[1] : 0.f;
        }
    };
    uint32_t wa[4], wb[4];
    const int64_t limit = W == 8 ? Ib : word_limit(blockIdx.x == gridDim.x - 1, Ib);
    const int64_t limit0 = W == 8 ? Ib : first_word_limit(blockIdx.x == 0, bed, limit);
    codes(ca, 0, limit0, wa);
    codes(cb, 0, limit0, wb);
    fetch(0);
    for (int64_t i0 = 0; i0 < I; i0 += 64) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < K2; ++e) qs[threadIdx.x + e * 64] = make_float4(qa[e], qa[e], qb[e], qb[e]);
        __syncthreads();
        uint32_t na[4] = {wa[0], wa[1], wa[2], wa[3]}, nb[4] = {wb[0], wb[1], wb[2], wb[3]};
        if (i0 + 64 < I) {
            fetch(i0 + 64);
            codes(ca, i0 + 64, limit, na);
            codes(cb, i0 + 64, limit, nb);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
#pragma unroll 1
            for (int hw = 0; hw < 2; ++hw) {
                const uint32_t x = spread((wa[v] >> (16 * hw)) & 0xFFFFu) | (spread((wb[v] >> (16 * hw)) & 0xFFFFu) << 2);
                const float4 *qv = qs + (16 * v + 8 * hw) * K2;
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const uint2 f = *(const uint2 *)(tl + ((t < 2 ? x << (7 - 4 * t) : x >> (4 * t - 7)) & 0x780u));
                    const float2 g = make_float2(__uint_as_float(f.x << 16), __uint_as_float(f.x & 0xFFFF0000u));
                    const float2 m = make_float2(__uint_as_float(f.y << 16), __uint_as_float(f.y & 0xFFFF0000u));
#pragma unroll
                    for (int h = 0; h < K2; ++h) {
                        const float4 y = qv[t * K2 + h];
                        const float2 y0 = make_float2(y.x, y.y), y1 = make_float2(y.z, y.w);
                        num[2 * h] = __ffma2_rn(y0, g, num[2 * h]);
                        den[2 * h] = __ffma2_rn(y0, m, den[2 * h]);
                        if (2 * h + 1 < K) {
                            num[2 * h + 1] = __ffma2_rn(y1, g, num[2 * h + 1]);
                            den[2 * h + 1] = __ffma2_rn(y1, m, den[2 * h + 1]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) { wa[v] = na[v]; wb[v] = nb[v]; }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float na = num[k].x, da = 2.f * den[k].x, nb = num[k].y, db = 2.f * den[k].y;
        const double va = da > 0.f ? (double)na / (double)da : 0.5, vb = db > 0.f ? (double)nb / (double)db : 0.5;
        if (ja < J) p[(size_t)K * ja + k] = fmin(fmax(va, 1e-5), 1.0 - 1e-5);
        if (jb < J) p[(size_t)K * jb + k] = fmin(fmax(vb, 1e-5), 1.0 - 1e-5);
    }
}

template <int K>
cudaError_t launch_warm_p(const uint8_t *bed, int64_t pitch, int64_t I, int64_t J, const double *q, double *p, cudaStream_t st)
{
    const unsigned grid = (unsigned)((J + 127) / 128);
    const uintptr_t al = (uintptr_t)bed | (uintptr_t)pitch;
    if ((al & 7u) == 0) k_warm_p<K, 8><<<grid, 64, 0, st>>>(bed, pitch, I, J, q, p);
    else k_warm_p<K, 1><<<grid, 64, 0, st>>>(bed, pitch, I, J, q, p);
    return cudaGetLastError();
}

} // namespace

extern "C" {

int admix_mlp_forward(const admix_mlp *net, int64_t n, const int8_t *dos, const float *center, const float *proj,
                      float *h1, float *h2, float *logits, float *probs, void *stream)
{
    if (!net || n < 1 || !dos || !center || !proj || !h1 || !h2 || !logits || !probs) return ADMIX_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t D = net->S + net->R, H = net->H, K = net->K;
    cudaError_t e = gemm(LoadX{dos, center, proj, net->S, net->R}, LoadF{net->w1, 1, H}, n, H, D, 1.f, net->b1, 1,
                         nullptr, h1, H, st);
    if (e == cudaSuccess) e = gemm(LoadF{h1, H, 1}, LoadF{net->w2, 1, H}, n, H, H, 1.f, net->b2, 1, nullptr, h2, H, st);
    if (e == cudaSuccess) e = gemm(LoadF{h2, H, 1}, LoadF{net->w3, 1, K}, n, K, H, 1.f, net->b3, 0, nullptr, logits, K, st);
    if (e == cudaSuccess) {
        k_softmax_ce<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(logits, n, (int)K, probs, nullptr, nullptr, nullptr);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? ADMIX_OK : ADMIX_ERR_CUDA;
}

int admix_mlp_backward(const admix_mlp *net, const admix_mlp_grads *grad, int64_t n, const int8_t *dos,
                       const float *center, const float *proj, const float *h1, const float *h2, const float *logits,
                       const float *target, float *probs, float *dlogits, float *dh2, float *dh1, float *loss,
                       void *stream)
{
    if (!net || !grad || n < 1 || !target || !dlogits || !dh2 || !dh1) return ADMIX_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t D = net->S + net->R, H = net->H, K = net->K;
    k_softmax_ce<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(logits, n, (int)K, probs, target, dlogits, loss);
    cudaError_t e = cudaGetLastError();
    /* layer 3 */
    if (e == cudaSuccess) e = gemm(LoadF{h2, 1, H}, LoadF{dlogits, 1, K}, H, K, n, 1.f, nullptr, 0, nullptr, grad->w3, K, st);
    if (e == cudaSuccess) e = colsum(dlogits, n, K, grad->b3, st);
    if (e == cudaSuccess) e = gemm(LoadF{dlogits, K, 1}, LoadF{net->w3, K, 1}, n, H, K, 1.f, nullptr, 0, h2, dh2, H, st);
    /* layer 2 */
    if (e == cudaSuccess) e = gemm(LoadF{h1, 1, H}, LoadF{dh2, 1, H}, H, H, n, 1.f, nullptr, 0, nullptr, grad->w2, H, st);
    if (e == cudaSuccess) e = colsum(dh2, n, H, grad->b2, st);
    if (e == cudaSuccess) e = gemm(LoadF{dh2, H, 1}, LoadF{net->w2, H, 1}, n, H, H, 1.f, nullptr, 0, h1, dh1, H, st);
    /* layer 1 */
    if (e == cudaSuccess)
        e = gemm(LoadXT{LoadX{dos, center, proj, net->S, net->R}}, LoadF{dh1, 1, H}, D, H, n, 1.f, nullptr, 0, nullptr,
                 grad->w1, H, st);
    if (e == cudaSuccess) e = colsum(dh1, n, H, grad->b1, st);
    return e == cudaSuccess ? ADMIX_OK : ADMIX_ERR_CUDA;
}

int admix_mlp_adam(float *w, const float *g, float *m, float *v, int64_t n, float lr, float beta1, float beta2,
                   float eps, int32_t t, void *stream)
{
    if (!w || !g || !m || !v || n < 1 || t < 1) return ADMIX_ERR_ARG;
    const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
    const unsigned grid = (unsigned)std::min<int64_t>(4096, (n + 255) / 256);
    k_adam<<<grid, 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? ADMIX_OK : ADMIX_ERR_CUDA;
}

int admix_warm_p(const uint8_t *d_bed, int64_t pitch, int64_t I, int64_t J, int32_t K, const double *d_q,
                 double *d_p, void *stream)
{
    if (!d_bed || !d_q || !d_p || I < 1 || J < 1 || K < 1 || K > ADMIX_MAX_K || pitch < (I + 3) / 4)
        return ADMIX_ERR_ARG;
    cudaError_t e = cudaErrorInvalidValue;
    ADMIX_DISPATCH_K(K, e = launch_warm_p<KK>(d_bed, pitch, I, J, d_q, d_p, (cudaStream_t)stream));
    return e == cudaSuccess ? ADMIX_OK : ADMIX_ERR_CUDA;
}

} /* extern "C" */
