/*
 * sweeps_f64.cu -- the FP64 ("plain") decode-fused sweeps over the packed genotype matrix.
 *
 * Every kernel decodes the 2-bit PLINK codes in place (loops.jl:529-534), recomputes
 * qp = sum_k q_ki p_kj (qp_block!, loops.jl:303-314) and accumulates in FP64.  Unlike the
 * reference's CUDA.jl kernels (cuda/kernels.jl), which add every cell's contribution into
 * global memory with FP64 atomics, each accumulator here has one owner thread; a sweep that
 * needs more parallelism than its owners provide is split into S slices whose partial sums
 * the consumer kernel adds in a fixed order.  Results are deterministic run to run.
 */
#include "common.cuh"
#include "kernels.h"

/* ===================================================================== FP64 tensor-core tiles
 *
 * Every sum of this form is a contraction over cells, so it runs on the FP64 matrix unit
 * (mma.sync ... f64, the only FP64 form of the tensor core: tcgen05 has no FP64 kind): a warp owns
 * 16 rows (individuals or SNPs) and walks the other axis 8 columns at a time.
 *   1. qp of the 16 x 8 cells is one product of the rows' coefficients (in registers) with the
 *      columns' (in shared memory): lane (g, t) = (lane / 4, lane % 4) receives the cells of rows
 *      g, g + 8 and columns 2t, 2t + 1.
 *   2. The lane turns its four cells into weights.  Column pair (2t, 2t + 1) of the result is
 *      the A operand's (t, t + 4) of the next product when that product's B rows are read in the
 *      same order, so the weights never leave their registers.
 *   3. The sums are products of the weights with tables of the columns' factors (pairs x_k x_k2,
 *      then x_k), a 16-byte shared load per 8 x 8 block of B; the accumulators stay in registers.
 * Measured on a B200: m16n8k8 reaches 18.5e12 FMA/s (64 per clock and SM), the same rate as and
 * shared with DFMA, which reaches 14e12 from registers; the gain over one thread per row is that
 * a cell's qp, reciprocal and weights are formed once and that the operands of 1,024 FMAs
 * are one load per lane, where a scalar loop needs a shared load per two FMAs. */

/* Both are collectives of the whole warp: volatile, so that the compiler leaves each where every lane executes it even if
 * only some lanes use the result, and callers reconverge (__syncwarp) after a branch that lanes take apart. */
__device__ __forceinline__ void dmma_k8(double (&d)[4], const double (&a)[4], double b0, double b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
__device__ __forceinline__ void dmma_k4(double (&d)[4], double a0, double a1, double b0)
{
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3]) : "d"(a0), "d"(a1), "d"(b0));
}

constexpr int F_THREADS = 256;               /* 8 warps */
constexpr int F_ROWS = 128;                  /* rows of a CTA: 16 per warp */

/* Columns per chunk: K * chunk <= 256, so each thread stages one coefficient per chunk.  Table rows
 * are 8 doubles longer than a chunk: a row stride of 64 bytes modulo 128 keeps the 16-byte B loads of
 * 8 lanes (2 rows x 4 column pairs) in different banks. */
__host__ __device__ constexpr int f_chunk(int K) { return K <= 8 ? 32 : 16; }

/* CTAs per SM: two where 128 registers a thread hold the accumulators */
__host__ __device__ constexpr int f_resident(int K, int mode) { return (K <= 8 || mode == 1) ? 2 : 1; }

/* rows' coefficients x[row][k] of rows g and g + 8 as A operands: a[s] = x[g][4s + t], x[g + 8][4s + t] */
template <int K>
struct RowA {
    static constexpr int KQ = (K + 3) / 4;
    double a[KQ][2];
    __device__ __forceinline__ void load(const double *__restrict__ x, int64_t r0, int64_t r1, int64_t n, int t)
    {
#pragma unroll
        for (int s = 0; s < KQ; ++s) {
            const int k = 4 * s + t;
            a[s][0] = (k < K) ? (r0 < n ? x[(size_t)K * r0 + k] : 0.5 / K) : 0.0;
            a[s][1] = (k < K) ? (r1 < n ? x[(size_t)K * r1 + k] : 0.5 / K) : 0.0;
        }
    }
    /* qp of the 16 x 8 cells whose column coefficients are c[k * CS + column]; (g, t) of this lane */
    template <int CS>
    __device__ __forceinline__ void dot(double (&qp)[4], const double *c, int g, int t) const
    {
#pragma unroll
        for (int i = 0; i < 4; ++i) qp[i] = 0.0;
#pragma unroll
        for (int s = 0; s < KQ; ++s) dmma_k4(qp, a[s][0], a[s][1], c[(4 * s + t) * CS + g]);
    }
};

/* 1 / x to at most one ulp from the correctly rounded quotient (which 99.7 % of values give) for normal x well inside the
 * exponent range: the hardware's approximation (20 bits) and one third-order Householder step, r (1 + e + e^2) with
 * e = 1 - x r, which leaves e^3 = 2^-60 before its last rounding. */
__device__ __forceinline__ double rcp_fast(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = fma(-x, r, 1.0);
    e = fma(e, e, e);
    return fma(r, e, r);
}

/* 1 / x by division, out of line (one register in, one out) */
__device__ __noinline__ double rcp_div(double x) { return 1.0 / x; }
__device__ __noinline__ double log_call(double x) { return log(x); }

/* The weights of a lane's four cells: qp[e] with code bits (lo, hi) (00, 10, 11: dosage 0, 1, 2; 01: missing, all
 * weights zero).  The dosage's factor 0, 1 or 2 is applied by integer instructions (a selection of zero and one added
 * to the exponent): the FP64 pipe, shared with the products, is the bound. */
struct CellW { double z1[4], z2[4], w1[4], w2[4]; };

template <bool HESS>
__device__ __forceinline__ bool cells_fast(const double (&qp)[4], const uint32_t (&code)[4], CellW &c)
{
    int odd = 0;
    double om[4], r1[4], r2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) om[e] = 1.0 - qp[e];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        odd |= __double2hiint(qp[e]) ^ 0x30000000;
        odd |= __double2hiint(om[e]) ^ 0x30000000;
        r1[e] = rcp_fast(qp[e]);
        r2[e] = rcp_fast(om[e]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool lo = (code[e] & 1u) != 0u, hi = (code[e] & 2u) != 0u;
        const int h1 = __double2hiint(r1[e]) + (lo ? 0x00100000 : 0), h2 = __double2hiint(r2[e]) + (hi ? 0 : 0x00100000);
        c.z1[e] = __hiloint2double(hi ? h1 : 0, hi ? __double2loint(r1[e]) : 0);
        c.z2[e] = __hiloint2double(lo ? 0 : h2, lo ? 0 : __double2loint(r2[e]));
        if (HESS) {
            c.w1[e] = c.z1[e] * r1[e];
            c.w2[e] = c.z2[e] * r2[e];
        }
    }
    return (odd & 0xF0000000) == 0;   /* qp and 1 - qp in [2^-255, 2): the reciprocals and the doubling are safe */
}

/* The same in the mean-imputed form: a missing cell's dosage is gm[e].  Factors of every code, two products a cell more than
 * the exponent trick, and no lane leaves the others: with divisions for a lane's four cells where one was missing, three of four
 * 16 x 8 blocks took them at 1 % missing.  I=10k, J=20k, 1 % missing: EM sums K=3 2.16 -> 0.98 ms, K=8 2.28 -> 1.11
 * (one thread per row 1.41 and 1.99); Q sweep K=3 1.34 -> 0.69, P sweep 1.10 -> 0.52. */
template <bool HESS>
__device__ __forceinline__ bool cells_mean(const double (&qp)[4], const uint32_t (&code)[4], const double (&gm)[4], CellW &c)
{
    int odd = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const double om = 1.0 - qp[e];
        odd |= (__double2hiint(qp[e]) ^ 0x30000000) | (__double2hiint(om) ^ 0x30000000);
        const double r1 = rcp_fast(qp[e]), r2 = rcp_fast(om);
        const bool lo = (code[e] & 1u) != 0u, hi = (code[e] & 2u) != 0u;
        double g = __hiloint2double(hi ? (lo ? 0x40000000 : 0x3FF00000) : 0, 0);
        g = (lo && !hi) ? gm[e] : g;
        c.z1[e] = g * r1;
        c.z2[e] = (2.0 - g) * r2;
        if (HESS) {
            c.w1[e] = c.z1[e] * r1;
            c.w2[e] = c.z2[e] * r2;
        }
    }
    return (odd & 0xF0000000) == 0;
}

/* the general form: dosage g (the SNP's mean gm for a missing cell when imp) and a division each; all weights zero for a
 * cell past the tile's columns (!in), whose placeholder coefficients a row may well take to qp = 0 or 1 */
__device__ __forceinline__ void cell_general(double qp, uint32_t code, bool in, bool imp, double gm, double &z1, double &z2,
                                             double &w1, double &w2)
{
    if (!in) {
        z1 = z2 = w1 = w2 = 0.0;
        return;
    }
    const bool miss = (code & 3u) == 1u, nm = !miss || imp;
    const double g = (miss && imp) ? gm : gval((int)(code & 3u));
    const double r1 = rcp_div(qp), r2 = rcp_div(1.0 - qp);
    z1 = (nm && g != 0.0) ? g * r1 : 0.0;
    z2 = (nm && g != 2.0) ? (2.0 - g) * r2 : 0.0;
    w1 = z1 * r1;
    w2 = z2 * r2;
}

/* A lane's four cells in the general form, out of line: inlined, its calls made the sweeps spill from K = 5 on.  Columns (e >> 1)
 * are past the tile's where !in0, !in1. */
struct CellIn { double qp[4], gm[4]; uint32_t code[4]; };
__device__ __noinline__ void cells_general(const CellIn *x, bool in0, bool in1, bool imp, CellW *o)
{
#pragma unroll
    for (int e = 0; e < 4; ++e)
        cell_general(x->qp[e], x->code[e], (e >> 1) ? in1 : in0, imp, x->gm[e], o->z1[e], o->z2[e], o->w1[e], o->w2[e]);
}

/* ===================================================================== loglik */

/* loglikelihood_kernel (cuda/kernels.jl:2-32) / loglikelihood_loop_skipmissing
 * (loops.jl:517-539); with mu != NULL the non-skipmissing loglikelihood_loop (loops.jl:493-514),
 * whose missing cells count with the SNP's mean dosage mu_j.
 *
 * Rows = SNPs; CTAs take units of (128 SNPs, slice of individuals) in turn, so the number of
 * partial sums is bounded by the grid.  A cell's factor qp^g (1-qp)^(2-g) is folded into a running
 * product (the exponent moved into an integer every 16 cells) and
 * one log is taken per thread.  A lane whose 32-individual chunk has a group of four outside
 * [2^-255, 2) or a negative factor (qp at or beyond 0 or 1, NaN) takes a log per cell in a second pass over the
 * chunk.  Mean-imputed (IMP): a row's missing cells share the dosage mu_j, so the lane keeps the products of their qp and of their
 * 1 - qp in the same way and takes two logs per row and unit.  A log per cell for every chunk of such a handle: K=3,
 * I=10k, J=20k, 1 % missing 1.49 ms (one thread per 4 individuals 1.12), now 0.35, whatever the share of missing cells.
 * Measured on a B200 (I=10k, J=100k): K=5 4.4 -> 1.18 ms, K=12 (I=20k, J=60k) 13.2 -> 1.8 ms against one
 * thread per 4 individuals with an FP64 log per cell; four CTAs per SM beat two by 7 % up to K = 8 (64 registers)
 * and lose 1-2 % above, where the row coefficients take more registers.  What bounds it now: per 16 x 8 cells
 * 32 cycles of the matrix unit per 4 clusters, 24 of FP64 scalars and about 50 integer selections.
 * PADDED: columns at a pitch that is a multiple of 16 bytes, padding coded missing (the handle's layout);
 * otherwise the caller's own columns, read bytewise up to Ib with the tail masked. */
template <int K>
struct LL {
    static constexpr int IC = 32, CS = IC + 4;                /* CS: 32 bytes modulo 128, 4 rows x 4 columns conflict-free */
    static constexpr int KR = RowA<K>::KQ * 4;
    static constexpr int PT = (K * IC + F_THREADS - 1) / F_THREADS;
};

template <bool PADDED>
__device__ __forceinline__ uint2 codes32(const uint8_t *__restrict__ bed, int64_t pitch, int64_t Ib, int64_t I, int64_t j, int64_t J,
                                         int64_t ic)
{
    if (j >= J) return make_uint2(0x55555555u, 0x55555555u);
    const uint8_t *src = bed + (size_t)j * pitch + (size_t)(ic >> 2);
    if (PADDED) return __ldg((const uint2 *)src);
    uint32_t v[2] = {0u, 0u};
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        uint32_t byte = 0x55u;
        const int64_t b = (ic >> 2) + n;
        if (b < Ib) {
            byte = __ldg(src + n);
            const int64_t left = I - 4 * b;               /* individuals of this byte */
            if (left < 4) {
                const uint32_t keep = (1u << (2 * (int)left)) - 1u;
                byte = (byte & keep) | (0x55u & ~keep);
            }
        }
        v[n >> 2] |= byte << (8 * (n & 3));
    }
    return make_uint2(v[0], v[1]);
}

template <int K, bool PADDED, bool IMP>
__global__ void __launch_bounds__(F_THREADS, (K <= 8 && !IMP ? 4 : 2))
k_loglik_f64(const uint8_t *__restrict__ bed, int64_t I, int64_t J, int64_t Ib, int64_t pitch,
             const double *__restrict__ q, const double *__restrict__ p, int64_t nblk, int64_t nunit,
             int64_t islice, double *__restrict__ partial, const double *__restrict__ mu)
{
    using C = LL<K>;
    constexpr int IC = C::IC, CS = C::CS, KR = C::KR, PT = C::PT;
    __shared__ double qs[2][KR * CS];
    __shared__ double red[F_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    for (int e = tid; e < 2 * KR * CS; e += F_THREADS) (&qs[0][0])[e] = 0.0;
    double acc = 0.0, prod = 1.0;
    int64_t ex = 0;
    for (int64_t u = blockIdx.x; u < nunit; u += gridDim.x) {
        const int64_t js = (u % nblk) * F_ROWS + warp * 16, i0 = (u / nblk) * islice, i1 = min(I, i0 + islice);
        const int nch = (int)((i1 - i0 + IC - 1) / IC);
        const int64_t ja = js + g, jb = js + g + 8;
        RowA<K> A;
        A.load(p, ja, jb, J, t);
        /* IMP: the rows' means, and the running products of qp (element 0, 1: rows a, b) and 1 - qp (2, 3) over missing cells */
        const double ga = (IMP && ja < J) ? mu[ja] : 0.0, gb = (IMP && jb < J) ? mu[jb] : 0.0;
        double mp[4] = {1.0, 1.0, 1.0, 1.0};
        int mx[4] = {0, 0, 0, 0};
        double qv[PT];
        auto fetch = [&](int c) {   /* the chunk's q: individuals past I read 0.5 / K (their codes are missing) */
#pragma unroll
            for (int n = 0; n < PT; ++n) {
                const int e = tid + n * F_THREADS;
                const int64_t i = i0 + (int64_t)c * IC + e / K;
                qv[n] = (e < K * IC) ? (i < I ? q[(size_t)K * (i0 + (int64_t)c * IC) + e] : 0.5 / K) : 0.0;
            }
        };
        auto stage = [&](int c) {
#pragma unroll
            for (int n = 0; n < PT; ++n) {
                const int e = tid + n * F_THREADS;
                if (e < K * IC) qs[c & 1][(e % K) * CS + e / K] = qv[n];
            }
        };
        __syncthreads();                                  /* the previous unit is done with qs */
        fetch(0);
        stage(0);
        uint2 wa = codes32<PADDED>(bed, pitch, Ib, I, ja, J, i0), wb = codes32<PADDED>(bed, pitch, Ib, I, jb, J, i0);
        __syncthreads();
        for (int c = 0; c < nch; ++c) {
            uint2 na = wa, nb = wb;
            if (c + 1 < nch) {
                fetch(c + 1);
                na = codes32<PADDED>(bed, pitch, Ib, I, ja, J, i0 + (int64_t)(c + 1) * IC);
                nb = codes32<PADDED>(bed, pitch, Ib, I, jb, J, i0 + (int64_t)(c + 1) * IC);
            }
            const double *qc = qs[c & 1];
            /* the lane's codes of block b: bits 16 b + 4 t .. + 3 of each row's 64 bits */
            const uint32_t xa[2] = {wa.x >> (4 * t), wa.y >> (4 * t)}, xb[2] = {wb.x >> (4 * t), wb.y >> (4 * t)};
            /* the factors of block b's cells (e & 2: row b, e & 1: column 2t + 1), 1 where missing */
            auto factors = [&](int b, double (&qp)[4], double (&f)[4]) {
                A.template dot<CS>(qp, qc + 8 * b, g, t);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t cc = ((e & 2) ? xb[b >> 1] : xa[b >> 1]) >> (16 * (b & 1) + 2 * (e & 1));
                    const bool lo = cc & 1u, hi = cc & 2u;
                    const double om = 1.0 - qp[e];
                    const double x = (hi ? qp[e] : om) * (lo ? qp[e] : om);
                    f[e] = (lo && !hi) ? 1.0 : x;
                }
            };
            const int left = (int)min((int64_t)IC, I - (i0 + (int64_t)c * IC));
            int odd = 0, sgn = 0;
            double m[IC / 8], cm[4] = {1.0, 1.0, 1.0, 1.0};
#pragma unroll
            for (int b = 0; b < IC / 8; ++b) {
                double qp[4], f[4];
                factors(b, qp, f);
                m[b] = (f[0] * f[1]) * (f[2] * f[3]);
                odd |= __double2hiint(m[b]) ^ 0x30000000;
                sgn |= __double2hiint(f[0]) | __double2hiint(f[1]) | __double2hiint(f[2]) | __double2hiint(f[3]);
                if (IMP) {
                    double a[4], o[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint32_t cc = ((e & 2) ? xb[b >> 1] : xa[b >> 1]) >> (16 * (b & 1) + 2 * (e & 1));
                        const bool miss = (cc & 3u) == 1u && 8 * b + 2 * t + (e & 1) < left;
                        a[e] = miss ? qp[e] : 1.0;
                        o[e] = miss ? 1.0 - qp[e] : 1.0;
                        sgn |= __double2hiint(a[e]) | __double2hiint(o[e]);
                    }
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const double x = a[2 * r] * a[2 * r + 1], y = o[2 * r] * o[2 * r + 1];
                        odd |= (__double2hiint(x) ^ 0x30000000) | (__double2hiint(y) ^ 0x30000000);
                        cm[r] *= x;
                        cm[2 + r] *= y;
                    }
                }
            }
            const bool ok = ((odd & 0xF0000000) | (sgn & 0x80000000)) == 0;
            if (ok) prod *= (m[0] * m[1]) * (m[2] * m[3]);   /* four groups in [2^-255, 2): normal */
            if (IMP && ok)
#pragma unroll
                for (int r = 0; r < 4; ++r) {                 /* likewise, the exponent moved into mx */
                    mp[r] *= cm[r];
                    const int h = __double2hiint(mp[r]);
                    mx[r] += ((h >> 20) & 0x7FF) - 1023;
                    mp[r] = __hiloint2double((h & 0x800FFFFF) | 0x3FF00000, __double2loint(mp[r]));
                }
            if (__any_sync(0xffffffffu, !ok)) {              /* again, with a log per cell in the lanes that need it */
#pragma unroll 1
                for (int b = 0; b < IC / 8; ++b) {
                    double qp[4], f[4];
                    factors(b, qp, f);
                    if (!ok) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            acc += log_call(f[e]);
                            const uint32_t cc = (((e & 2) ? xb[b >> 1] : xa[b >> 1]) >> (16 * (b & 1) + 2 * (e & 1))) & 3u;
                            if (IMP && cc == 1u && ((e & 2) ? jb : ja) < J && 8 * b + 2 * t + (e & 1) < left) {
                                const double gm = (e & 2) ? gb : ga;   /* loglikelihood_loop: the missing dosage imputed by mu_j */
                                acc += gm * log_call(qp[e]) + (2.0 - gm) * log_call(1.0 - qp[e]);
                            }
                        }
                    }
                    __syncwarp();                            /* the next block's product is the whole warp's */
                }
            }
            const int64_t bits = __double_as_longlong(prod);
            ex += ((bits >> 52) & 0x7FF) - 1023;
            prod = __longlong_as_double((bits & ~(0x7FFLL << 52)) | (1023LL << 52));
            if (c + 1 < nch) stage(c + 1);
            wa = na;
            wb = nb;
            __syncthreads();
        }
        if (IMP) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const double gm = (r & 1) ? gb : ga, f = (r & 2) ? 2.0 - gm : gm;
                if (((r & 1) ? jb : ja) < J) acc += f * (log_call(mp[r]) + (double)mx[r] * 0.69314718055994530942);
            }
        }
    }
    acc += log_call(prod) + (double)ex * 0.69314718055994530942;
    const double s = block_sum(acc, red);
    if (tid == 0) partial[blockIdx.x] = s;
}

/* Fixed-order sum of n partials into *out (one block of 1024 threads). */
__global__ void __launch_bounds__(1024)
k_sum_partials(const double *__restrict__ partial, int64_t n, double *__restrict__ out)
{
    __shared__ double red[32];
    double v = 0.0;
    for (int64_t t = threadIdx.x; t < n; t += blockDim.x) v += partial[t];
    const double s = block_sum(v, red);
    if (threadIdx.x == 0) *out = s;
}

/* The Q side's EM accumulators, every 256 SNPs into totals of their own and at the last chunk back: z1 p + z2 (1-p) is
 * near 2 in every cell, and a serial chain of thousands of nearly equal terms loses several ulp (q against 64 bits at 5,984 x
 * 16,795, K=6: 7.9e-16 of its norm, 3.0e-16 with the shorter slices of one thread per row, 2.5e-16 so).  The other sums'
 * errors are those of one thread per row without it (median ratio 1.00 over 23 cohorts), and gradients and Hessians
 * would need twice their registers. */
template <int CH, int N>
__device__ __forceinline__ void em_fold(int c, int nch, double (&acc)[N][4], double (&tot)[N][4])
{
    constexpr int PER = 256 / CH;
    if (nch <= PER || ((c + 1) % PER != 0 && c != nch - 1)) return;
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            tot[n][e] += acc[n][e];
            acc[n][e] = c == nch - 1 ? tot[n][e] : 0.0;
        }
}

/* ===================================================================== Q side */

/* With mu != NULL every kernel below runs the reference's non-skipmissing twin (update_q_loop!,
 * em_q_loop!, update_p_loop!, em_p_loop!, loops.jl:589-608,679-698,840-865,896-921): a missing
 * cell counts with g = mu_j, the SNP's mean dosage, and weight 1.
 *
 * Per-individual accumulators over SNPs j.  MODE 0 (update_q_loop_skipmissing!,
 * loops.jl:867-894; update_q_kernel!, cuda/kernels.jl:102-137): entries e < T are the
 * packed upper triangle of XtX_q (T = K(K+1)/2), entries T..T+K-1 are Xtz_q.
 * MODE 1 (em_q_loop_skipmissing!, loops.jl:610-632): E = K entries sum_j (z1 p_k + z2 (1-p_k)),
 * finalised into q_next by k_emq_finalize.
 *   z1 = nm g / qp, z2 = nm (2-g) / (1-qp), w1 = z1 / qp, w2 = z2 / (1-qp)
 *   XtX[k,k2] += w1 p_k p_k2 + w2 (1-p_k)(1-p_k2),   Xtz[k] += z1 p_k + z2 (1-p_k)
 * A CTA owns 128 individuals and a slice of SNPs.  Per chunk of SNPs the columns' coefficients p_k
 * and 1 - p_k (three buffers) and the pair tables p_k p_k2 and (1-p_k)(1-p_k2) (two buffers) are in
 * shared memory, so one barrier per chunk suffices: while chunk c is summed, chunk c+1's pair
 * tables are built and chunk c+2's coefficients and genotypes are in flight.
 * Bound: the FP64 pipe.  Per 16 x 8 cells and warp 64 cycles a product (2 per 8 columns of pairs and of
 * coefficients, half of one per 4 clusters for qp) and 9 scalar FP64 instructions a cell.  Measured on a B200
 * against one thread per individual: K=5 (I=10k, J=100k) 11.9 -> 4.7 ms, 67 % of the pipe's rate; K=12 (I=20k,
 * J=60k) 74 -> 17.7 ms, 78 %. */
template <int K, int MODE>
struct QSide {
    static constexpr int T = K * (K + 1) / 2;
    static constexpr int E = MODE == 0 ? T + K : K;
    static constexpr int NH = MODE == 0 ? (T + 7) / 8 : 0;     /* 8-column tiles of pairs */
    static constexpr int NG = (K + 7) / 8;                     /* ... and of coefficients */
    static constexpr int JC = f_chunk(K), CS = JC + 8;
    static constexpr int CO = 2 * 8 * NG * CS;                 /* doubles of one coefficient buffer: p rows, 1-p rows */
    static constexpr int TB = 2 * 8 * NH * CS;                 /* doubles of one pair-table buffer */
    static constexpr int GW = JC * 8;                          /* genotype words of one chunk (32 bytes per SNP) */
    static constexpr size_t smem = sizeof(double) * (size_t)(3 * CO + 2 * TB) + 4 * (size_t)(3 * GW) + 2 * (size_t)(8 * NH) + 8 * (size_t)(3 * JC);
};

template <int K, int MODE, bool IMP>
__global__ void __launch_bounds__(F_THREADS, f_resident(K, MODE))
k_sweep_q_f64(const uint8_t *__restrict__ bed, int64_t I, int64_t J, int64_t pitch,
              const double *__restrict__ q, const double *__restrict__ p,
              int64_t jslice, double *__restrict__ out, const double *__restrict__ mu)
{
    using C = QSide<K, MODE>;
    constexpr int T = C::T, E = C::E, NH = C::NH, NG = C::NG, JC = C::JC, CS = C::CS;
    extern __shared__ __align__(16) double sm[];
    double *co = sm, *tb = sm + 3 * C::CO;
    uint32_t *gw = (uint32_t *)(tb + 2 * C::TB);
    uint8_t *lut = (uint8_t *)(gw + 3 * C::GW);                /* (k, k2) of pair n at lut[2n], lut[2n + 1] */
    double *ms = (double *)(lut + 2 * 8 * NH);                 /* IMP: the chunks' SNP means, three buffers */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int64_t i0 = (int64_t)blockIdx.x * F_ROWS;
    const int64_t ia = i0 + warp * 16 + g, ib = ia + 8;
    const int64_t j0 = (int64_t)blockIdx.y * jslice, j1 = min(J, j0 + jslice);
    const int nch = (int)((j1 - j0 + JC - 1) / JC);

    RowA<K> A;
    A.load(q, ia, ib, I, t);
    for (int e = tid; e < 3 * C::CO + 2 * C::TB; e += F_THREADS) sm[e] = 0.0;   /* rows past K and T stay zero */
    if (MODE == 0)
        for (int n = tid; n < T; n += F_THREADS) {
            int k, k2;
            tri_pair(n, k, k2);
            lut[2 * n] = (uint8_t)k;
            lut[2 * n + 1] = (uint8_t)k2;
        }
    double pv = 0.5, mv = 0.0;
    uint32_t gv = 0x55555555u;
    /* chunk c's coefficient (SNP tid / K, k = tid % K; 0.5 past the slice) and genotype word (SNP
     * tid / 8, 16 individuals tid % 8; missing past the slice and past the column) of this thread */
    auto fetch = [&](int c) {
        const int64_t jc = j0 + (int64_t)c * JC;
        if (tid < K * JC) pv = (jc + tid / K < j1) ? p[(size_t)K * jc + tid] : 0.5;
        if (IMP && tid < JC) mv = (jc + tid < j1) ? mu[jc + tid] : 0.0;
        if (tid < 8 * JC) {
            const int64_t j = jc + (tid >> 3), byte = (i0 >> 2) + 4 * (tid & 7);
            gv = (j < j1 && byte < pitch) ? __ldg((const uint32_t *)(bed + (size_t)j * pitch + byte)) : 0x55555555u;
        }
    };
    auto stage = [&](int c) {
        const int s = c % 3;
        if (tid < K * JC) {
            double *o = co + s * C::CO + (tid % K) * CS + tid / K;
            o[0] = pv;
            o[8 * NG * CS] = 1.0 - pv;
        }
        if (tid < 8 * JC) gw[s * C::GW + tid] = gv;
        if (IMP && tid < JC) ms[s * JC + tid] = mv;
    };
    auto pairs = [&](int c) {
        if (MODE != 0) return;
        const double *ps = co + (c % 3) * C::CO, *os = ps + 8 * NG * CS;
        double *ta = tb + (c & 1) * C::TB, *tc = ta + 8 * NH * CS;
#pragma unroll 2
        for (int e = tid; e < T * JC; e += F_THREADS) {
            const int n = e / JC, jj = e % JC, k = lut[2 * n] * CS + jj, k2 = lut[2 * n + 1] * CS + jj;
            ta[n * CS + jj] = ps[k] * ps[k2];
            tc[n * CS + jj] = os[k] * os[k2];
        }
    };
    double acc[NH + NG][4], tot[MODE == 1 ? NG : 1][4];
#pragma unroll
    for (int n = 0; n < NH + NG; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = tot[MODE == 1 ? n : 0][e] = 0.0;

    __syncthreads();
    if (nch > 0) { fetch(0); stage(0); }
    if (nch > 1) { fetch(1); stage(1); }
    __syncthreads();
    if (nch > 0) pairs(0);
    __syncthreads();
    for (int c = 0; c < nch; ++c) {
        if (c + 2 < nch) fetch(c + 2);
        if (c + 1 < nch) pairs(c + 1);
        const double *ps = co + (c % 3) * C::CO, *os = ps + 8 * NG * CS;
        const double *ta = tb + (c & 1) * C::TB, *tc = ta + 8 * NH * CS;
        const uint32_t *gc = gw + (c % 3) * C::GW + warp;
        auto weights = [&](int b, CellW &w) {   /* element e = row (e & 1), SNP 2t + (e >> 1): result element 2 (e & 1) + (e >> 1) */
            double d[4], qp[4];
            A.template dot<CS>(d, ps + 8 * b, g, t);
            const uint32_t c0 = gc[8 * (8 * b + 2 * t)] >> (2 * g), c1 = gc[8 * (8 * b + 2 * t + 1)] >> (2 * g);
            const uint32_t code[4] = {c0, c0 >> 16, c1, c1 >> 16};
#pragma unroll
            for (int e = 0; e < 4; ++e) qp[e] = d[2 * (e & 1) + (e >> 1)];
            double gm[4] = {0.0, 0.0, 0.0, 0.0};
            if (IMP) {
                const double2 m = *(const double2 *)(ms + (c % 3) * JC + 8 * b + 2 * t);
                gm[0] = gm[1] = m.x;
                gm[2] = gm[3] = m.y;
            }
            const bool fast = IMP ? cells_mean<MODE == 0>(qp, code, gm, w) : cells_fast<MODE == 0>(qp, code, w);
            const auto in = [&](int e) { return j0 + (int64_t)c * JC + 8 * b + 2 * t + (e >> 1) < j1; };
            if (!fast) {
                CellIn x;
                CellW y;
#pragma unroll
                for (int e = 0; e < 4; ++e) { x.qp[e] = qp[e]; x.gm[e] = gm[e]; x.code[e] = code[e]; }
                cells_general(&x, in(0), in(2), IMP, &y);
                w = y;
            } else if (IMP && c == nch - 1) {   /* the placeholders' codes are missing */
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!in(e)) w.z1[e] = w.z2[e] = w.w1[e] = w.w2[e] = 0.0;
            }
            __syncwarp();                                      /* the sums are the whole warp's products */
        };
        auto sums = [&](int b, const CellW &w) {
            const int bo = g * CS + 8 * b + 2 * t;
#pragma unroll
            for (int n = 0; n < NH + NG; ++n) {
                const double2 x = *(const double2 *)((n < NH ? ta + n * 8 * CS : ps + (n - NH) * 8 * CS) + bo);
                dmma_k8(acc[n], n < NH ? w.w1 : w.z1, x.x, x.y);
            }
#pragma unroll
            for (int n = 0; n < NH + NG; ++n) {
                const double2 x = *(const double2 *)((n < NH ? tc + n * 8 * CS : os + (n - NH) * 8 * CS) + bo);
                dmma_k8(acc[n], n < NH ? w.w2 : w.z2, x.x, x.y);
            }
        };
#pragma unroll 2
        for (int b = 0; b < JC / 8; ++b) {
            CellW w;
            weights(b, w);
            sums(b, w);
        }
        if (c + 2 < nch) stage(c + 2);
        if constexpr (MODE == 1) em_fold<JC>(c, nch, acc, tot);
        __syncthreads();
    }
#pragma unroll
    for (int n = 0; n < NH + NG; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int col = (n < NH ? 8 * n : 8 * (n - NH)) + 2 * t + (e & 1);
            const int64_t i = (e & 2) ? ib : ia;
            if (i < I && col < (n < NH ? T : K)) out[((size_t)blockIdx.y * I + i) * E + (n < NH ? 0 : E - K) + col] = acc[n][e];
        }
}

/* em_q! finalisation (algorithms_inner.jl:89): q_next[k,i] = q[k,i] * sum_s acc / (2J). */
/* q_next[k,i] = q[k,i] sum_j (z1 p_k + z2 (1-p_k)) / 2J from S slices of per-individual rows of E
 * entries whose sums start at entry off (E = K, off = 0 for the EM sweep; E = T + K, off = T for
 * the gradient entries of a gradient / Hessian sweep, which are the same sums) */
__global__ void k_emq_finalize(int64_t I, int K, int64_t J, int S, int E, int off, const double *__restrict__ parts,
                               const double *__restrict__ q, double *__restrict__ q_next)
{
    const int64_t n = (int64_t)K * I;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / K, k = t - i * K;
        double s = 0.0;
        for (int sl = 0; sl < S; ++sl) s += parts[((size_t)sl * I + i) * E + off + k];
        q_next[t] = q[t] * s / (double)(2 * J);
    }
}

/* ===================================================================== P side */

/* Per-SNP accumulators over individuals i.  MODE 0 (update_p_loop_skipmissing!,
 * loops.jl:923-950; update_p_kernel!, cuda/kernels.jl:139-174): e < T packed XtX_p,
 * T..T+K-1 Xtz_p, with
 *   XtX[k,k2] += nm (g/qp^2 + (2-g)/(1-qp)^2) q_k q_k2,  Xtz[k] += nm (g/qp - (2-g)/(1-qp)) q_k.
 * MODE 1 (em_p_loop_skipmissing!, loops.jl:700-721): E = 2K entries sum_i z1 q_k and
 * sum_i z2 q_k, finalised by k_emp_finalize.  The Q side with the axes swapped: a CTA owns 128 SNPs
 * and a slice of individuals (slices start on multiples of 32), whose q_k and q_k q_k2 tables are in
 * shared memory; a lane reads the codes of its two SNPs straight from their columns, a chunk ahead.
 * Measured as above: K=5 5.0 -> 3.3 ms, K=12 43 -> 11.0 ms. */
template <int K, int MODE>
struct PSide {
    static constexpr int T = K * (K + 1) / 2;
    static constexpr int E = MODE == 0 ? T + K : 2 * K;
    static constexpr int NH = MODE == 0 ? (T + 7) / 8 : 0;
    static constexpr int NG = (K + 7) / 8;
    static constexpr int NA = MODE == 0 ? NH + NG : 2 * NG;    /* accumulator tiles */
    static constexpr int IC = f_chunk(K), CS = IC + 8;
    static constexpr int CO = 8 * NG * CS, TB = 8 * NH * CS;
    static constexpr size_t smem = sizeof(double) * (size_t)(3 * CO + 2 * TB) + 2 * (size_t)(8 * NH);
};

template <int K, int MODE, bool IMP>
__global__ void __launch_bounds__(F_THREADS, f_resident(K, MODE))
k_sweep_p_f64(const uint8_t *__restrict__ bed, int64_t I, int64_t J, int64_t pitch,
              const double *__restrict__ q, const double *__restrict__ p,
              int64_t islice, double *__restrict__ out, const double *__restrict__ mu)
{
    using C = PSide<K, MODE>;
    constexpr int T = C::T, E = C::E, NH = C::NH, NG = C::NG, NA = C::NA, IC = C::IC, CS = C::CS;
    extern __shared__ __align__(16) double sm[];
    double *co = sm, *tb = sm + 3 * C::CO;
    uint8_t *lut = (uint8_t *)(tb + 2 * C::TB);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int64_t ja = (int64_t)blockIdx.x * F_ROWS + warp * 16 + g, jb = ja + 8;
    const int64_t i0 = (int64_t)blockIdx.y * islice, i1 = min(I, i0 + islice);
    const int nch = (int)((i1 - i0 + IC - 1) / IC);

    RowA<K> A;
    A.load(p, ja, jb, J, t);
    const double ga = (IMP && ja < J) ? mu[ja] : 0.0, gb = (IMP && jb < J) ? mu[jb] : 0.0;
    for (int e = tid; e < 3 * C::CO + 2 * C::TB; e += F_THREADS) sm[e] = 0.0;
    if (MODE == 0)
        for (int n = tid; n < T; n += F_THREADS) {
            int k, k2;
            tri_pair(n, k, k2);
            lut[2 * n] = (uint8_t)k;
            lut[2 * n + 1] = (uint8_t)k2;
        }
    double qv = 0.0;
    auto fetch = [&](int c) {   /* individuals past I: 0.5 / K, their codes are missing */
        const int64_t ic = i0 + (int64_t)c * IC;
        if (tid < K * IC) qv = (ic + tid / K < I) ? q[(size_t)K * ic + tid] : 0.5 / K;
    };
    auto stage = [&](int c) {
        if (tid < K * IC) co[(c % 3) * C::CO + (tid % K) * CS + tid / K] = qv;
    };
    auto pairs = [&](int c) {
        if (MODE != 0) return;
        const double *qs = co + (c % 3) * C::CO;
        double *ta = tb + (c & 1) * C::TB;
#pragma unroll 2
        for (int e = tid; e < T * IC; e += F_THREADS) {
            const int n = e / IC, ii = e % IC;
            ta[n * CS + ii] = qs[lut[2 * n] * CS + ii] * qs[lut[2 * n + 1] * CS + ii];
        }
    };
    /* the chunk's codes of SNP j (IC / 4 bytes of its column) */
    auto codes = [&](int64_t j, int c) -> uint2 {
        if (j >= J) return make_uint2(0x55555555u, 0x55555555u);
        const uint8_t *src = bed + (size_t)j * pitch + (size_t)((i0 + (int64_t)c * IC) >> 2);
        if (IC == 32) return __ldg((const uint2 *)src);
        return make_uint2(__ldg((const uint32_t *)src), 0u);
    };
    double acc[NA][4];
#pragma unroll
    for (int n = 0; n < NA; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0;

    __syncthreads();
    uint2 wa = make_uint2(0u, 0u), wb = wa;
    if (nch > 0) { fetch(0); stage(0); wa = codes(ja, 0); wb = codes(jb, 0); }
    if (nch > 1) { fetch(1); stage(1); }
    __syncthreads();
    if (nch > 0) pairs(0);
    __syncthreads();
    for (int c = 0; c < nch; ++c) {
        uint2 na = wa, nb = wb;
        if (c + 1 < nch) { na = codes(ja, c + 1); nb = codes(jb, c + 1); }
        if (c + 2 < nch) fetch(c + 2);
        if (c + 1 < nch) pairs(c + 1);
        const double *qs = co + (c % 3) * C::CO, *ta = tb + (c & 1) * C::TB;
        auto weights = [&](int b, CellW &w) {
            double d[4], qp[4];
            A.template dot<CS>(d, qs + 8 * b, g, t);
            const int sh = 16 * (b & 1) + 4 * t;
            const uint32_t ca = ((b & 2) ? wa.y : wa.x) >> sh, cb = ((b & 2) ? wb.y : wb.x) >> sh;
            const uint32_t code[4] = {ca, cb, ca >> 2, cb >> 2};
#pragma unroll
            for (int e = 0; e < 4; ++e) qp[e] = d[2 * (e & 1) + (e >> 1)];
            const double gm[4] = {ga, gb, ga, gb};
            const bool fast = IMP ? cells_mean<MODE == 0>(qp, code, gm, w) : cells_fast<MODE == 0>(qp, code, w);
            const auto in = [&](int e) { return i0 + (int64_t)c * IC + 8 * b + 2 * t + (e >> 1) < i1; };
            if (!fast) {
                CellIn x;
                CellW y;
#pragma unroll
                for (int e = 0; e < 4; ++e) { x.qp[e] = qp[e]; x.gm[e] = gm[e]; x.code[e] = code[e]; }
                cells_general(&x, in(0), in(2), IMP, &y);
                w = y;
            } else if (IMP && c == nch - 1) {   /* the placeholders' codes are missing */
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (!in(e)) w.z1[e] = w.z2[e] = w.w1[e] = w.w2[e] = 0.0;
            }
            __syncwarp();
            if (MODE == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    w.w1[e] += w.w2[e];                        /* nm (g/qp^2 + (2-g)/(1-qp)^2) */
                    w.z1[e] -= w.z2[e];                        /* nm (g/qp - (2-g)/(1-qp)) */
                }
            }
        };
        auto sums = [&](int b, const CellW &w) {
            const int bo = g * CS + 8 * b + 2 * t;
#pragma unroll
            for (int n = 0; n < (MODE == 0 ? NA : NG); ++n) {
                const double2 x = *(const double2 *)((n < NH ? ta + n * 8 * CS : qs + (n - NH) * 8 * CS) + bo);
                dmma_k8(acc[n], n < NH ? w.w1 : w.z1, x.x, x.y);
                if (MODE == 1) dmma_k8(acc[NG + n], w.z2, x.x, x.y);
            }
        };
#pragma unroll 2
        for (int b = 0; b < IC / 8; ++b) {
            CellW w;
            weights(b, w);
            sums(b, w);
        }
        if (c + 2 < nch) stage(c + 2);
        wa = na;
        wb = nb;
        __syncthreads();
    }
#pragma unroll
    for (int n = 0; n < NA; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool hess = n < NH;
            const int col = 8 * (hess ? n : (n - NH) % NG) + 2 * t + (e & 1);
            const int off = hess ? 0 : (MODE == 0 ? T : (n / NG) * K);
            const int64_t j = (e & 2) ? jb : ja;
            if (j < J && col < (hess ? T : K)) out[((size_t)blockIdx.y * J + j) * E + off + col] = acc[n][e];
        }
}

/* em_p! finalisation (algorithms_inner.jl:133-137): A = p sum z1 q, B = (1-p) sum z2 q,
 * p_next = A / (A + B). */
__global__ void k_emp_finalize(int64_t J, int K, int S, const double *__restrict__ parts,
                               const double *__restrict__ p, double *__restrict__ p_next)
{
    const int64_t n = (int64_t)K * J;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / K;
        const int k = (int)(t - j * K);
        double a = 0.0, b = 0.0;
        for (int sl = 0; sl < S; ++sl) {
            const double *o = parts + ((size_t)sl * J + j) * (2 * K);
            a += o[k];
            b += o[K + k];
        }
        const double pk = p[t];
        const double A = pk * a, B = (1.0 - pk) * b;
        p_next[t] = A / (A + B);
    }
}

/* Sum S slices of packed accumulators (E = T + K per problem) and expand to the
 * reference's K x K x n / K x n layout (for host dumps). */
__global__ void k_expand_hess(int64_t nprob, int K, int S, const double *__restrict__ parts,
                              double *__restrict__ XtX, double *__restrict__ Xtz)
{
    const int T = K * (K + 1) / 2, E = T + K;
    const int64_t n = nprob * (int64_t)E;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t pr = t / E;
        const int e = (int)(t - pr * E);
        double s = 0.0;
        for (int sl = 0; sl < S; ++sl) s += parts[(size_t)sl * n + t];
        if (e < T) {
            int k, k2;
            tri_pair(e, k, k2);
            XtX[(size_t)K * K * pr + k2 + (size_t)K * k] = s;
            XtX[(size_t)K * K * pr + k + (size_t)K * k2] = s;
        } else {
            Xtz[(size_t)K * pr + (e - T)] = s;
        }
    }
}

/* ===================================================================== decode counts */

/* Missing-code counts, bit-exact: code 01 <=> low bit 1, high bit 0.  Thread = one byte
 * column position b over a slice of SNPs; padding bits of the last byte are masked. */
__global__ void __launch_bounds__(256)
k_decode_counts(const uint8_t *__restrict__ bed, int64_t I, int64_t J, int64_t Ib, int64_t pitch, int64_t jslice,
                unsigned long long *__restrict__ miss_snp, unsigned long long *__restrict__ miss_ind)
{
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t j0 = (int64_t)blockIdx.y * jslice, j1 = min(J, j0 + jslice);
    const bool valid = b < Ib;
    unsigned mask = 0x55u;
    if (valid && b == Ib - 1 && (I & 3)) mask = 0x55u >> (2 * (4 - (I & 3)));
    unsigned c[4] = {0, 0, 0, 0};
    for (int64_t j = j0; j < j1; ++j) {
        unsigned m = 0;
        if (valid) {
            const unsigned byte = __ldg(bed + (size_t)j * pitch + b);
            m = byte & ~(byte >> 1) & mask;
            c[0] += m & 1u; c[1] += (m >> 2) & 1u; c[2] += (m >> 4) & 1u; c[3] += (m >> 6) & 1u;
        }
        unsigned cnt = __popc(m);
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(miss_snp + j, (unsigned long long)cnt);
    }
    if (valid)
        for (int s = 0; s < 4; ++s) {
            const int64_t i = 4 * b + s;
            if (i < I && c[s]) atomicAdd(miss_ind + i, (unsigned long long)c[s]);
        }
}

/* ===================================================================== SNP means */

/* g.mu of the SnpLinAlg (additive model): per SNP the mean dosage over its non-missing
 * individuals, NaN when all are missing.  One block per SNP over its padded column (padding is
 * coded missing, so it never counts).  Per byte: codes 10 and 11 have the high bit, 11 also the
 * low bit, so sum g = popc(hi) + popc(hi & lo) and the missing count is popc(lo & ~hi). */
__global__ void __launch_bounds__(256)
k_snp_means(const uint8_t *__restrict__ bed, int64_t J, int64_t pitch, double *__restrict__ mu)
{
    __shared__ double red[8];
    const int64_t j = blockIdx.x;
    if (j >= J) return;
    const uint8_t *col = bed + (size_t)j * pitch;
    long long gs = 0, nn = 0;
    for (int64_t b = threadIdx.x; b < pitch; b += blockDim.x) {
        const unsigned v = col[b];
        const unsigned lo = v & 0x55u, hi = (v >> 1) & 0x55u;
        gs += __popc(hi) + __popc(hi & lo);
        nn += 4 - __popc(lo & ~hi);
    }
    const double sg = block_sum((double)gs, red);
    const double sn = block_sum((double)nn, red);
    if (threadIdx.x == 0) mu[j] = sn > 0.0 ? sg / sn : __longlong_as_double(0x7ff8000000000000LL);
}

cudaError_t launch_snp_means(const uint8_t *bed, int64_t J, int64_t pitch, double *mu, cudaStream_t st)
{
    k_snp_means<<<(unsigned)J, 256, 0, st>>>(bed, J, pitch, mu);
    return cudaGetLastError();
}

/* ===================================================================== launchers */

template <int K>
static cudaError_t launch_loglik_t(const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                                   const double *p, const LoglikPlan &pl, bool padded, double *partial, double *out,
                                   cudaStream_t st, const double *mu)
{
    const int64_t Ib = (I + 3) / 4;
    if (mu)   /* handles only: padded */
        k_loglik_f64<K, true, true><<<(unsigned)pl.gx, F_THREADS, 0, st>>>(bed, I, J, Ib, pitch, q, p, pl.nblk, pl.nunit, pl.islice, partial, mu);
    else if (padded)
        k_loglik_f64<K, true, false><<<(unsigned)pl.gx, F_THREADS, 0, st>>>(bed, I, J, Ib, pitch, q, p, pl.nblk, pl.nunit, pl.islice, partial, mu);
    else
        k_loglik_f64<K, false, false><<<(unsigned)pl.gx, F_THREADS, 0, st>>>(bed, I, J, Ib, pitch, q, p, pl.nblk, pl.nunit, pl.islice, partial, mu);
    k_sum_partials<<<1, 1024, 0, st>>>(partial, pl.gx, out);
    return cudaGetLastError();
}

/* Units of 128 SNPs x a slice of individuals, taken in turn by at most four CTAs per SM: about
 * eight units per CTA where the cohort has that many (the last round is then at most an eighth
 * empty), slices of at least 256 individuals (below that a unit's setup shows), at most one
 * partial sum per CTA whatever the cohort's size. */
LoglikPlan plan_loglik(int64_t I, int64_t J, int sms)
{
    LoglikPlan pl;
    const int64_t cap = std::max<int64_t>(1, 4 * (int64_t)sms);
    pl.nblk = std::max<int64_t>(1, (J + F_ROWS - 1) / F_ROWS);
    const int64_t want = (8 * cap + pl.nblk - 1) / pl.nblk;                 /* slices for eight units per CTA */
    const int64_t full = (cap + pl.nblk - 1) / pl.nblk;                     /* ... for one */
    int64_t ns = std::min(want, std::max<int64_t>(1, I / 256));
    ns = std::max(ns, std::min(full, std::max<int64_t>(1, I / 64)));
    pl.islice = std::max<int64_t>(32, ((I + ns - 1) / ns + 31) / 32 * 32);
    pl.nunit = pl.nblk * std::max<int64_t>(1, (I + pl.islice - 1) / pl.islice);
    pl.gx = (int)std::min(pl.nunit, cap);
    return pl;
}

cudaError_t launch_loglik_f64(int K, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                              const double *p, const LoglikPlan &pl, bool padded, double *partial, double *out,
                              cudaStream_t st, const double *mu)
{
    cudaError_t e = cudaErrorInvalidValue;
    ADMIX_DISPATCH_K(K, e = launch_loglik_t<KK>(bed, I, J, pitch, q, p, pl, padded, partial, out, st, mu));
    return e;
}

/* CTAs of 128 rows; slices are multiples of 32 columns and at least 64 long. */
static SweepPlan plan_f64(int K, int64_t rows, int64_t cols, int sms, int64_t smax)
{
    return plan_rows(rows, cols, sms, f_resident(K, 0), 32, 2, smax);
}

SweepPlan plan_sweep_q(int K, int64_t I, int64_t J, int sms, int64_t smax) { return plan_f64(K, I, J, sms, smax); }
SweepPlan plan_sweep_p(int K, int64_t I, int64_t J, int sms, int64_t smax) { return plan_f64(K, J, I, sms, smax); }

template <int K, int MODE>
static cudaError_t launch_sweep_q_t(const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                                    const double *p, const SweepPlan &pl, double *out, cudaStream_t st,
                                    const double *mu)
{
    using C = QSide<K, MODE>;
    dim3 grid((unsigned)pl.gx, (unsigned)pl.S);
    if (mu) k_sweep_q_f64<K, MODE, true><<<grid, F_THREADS, C::smem, st>>>(bed, I, J, pitch, q, p, pl.slice, out, mu);
    else k_sweep_q_f64<K, MODE, false><<<grid, F_THREADS, C::smem, st>>>(bed, I, J, pitch, q, p, pl.slice, out, mu);
    return cudaGetLastError();
}

cudaError_t launch_sweep_q_f64(int K, int mode, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                               const double *q, const double *p, const SweepPlan &pl, double *out,
                               cudaStream_t st, const double *mu)
{
    cudaError_t e = cudaErrorInvalidValue;
    if (mode == 0) { ADMIX_DISPATCH_K(K, (e = launch_sweep_q_t<KK, 0>(bed, I, J, pitch, q, p, pl, out, st, mu))); }
    else { ADMIX_DISPATCH_K(K, (e = launch_sweep_q_t<KK, 1>(bed, I, J, pitch, q, p, pl, out, st, mu))); }
    return e;
}

template <int K, int MODE>
static cudaError_t launch_sweep_p_t(const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                                    const double *p, const SweepPlan &pl, double *out, cudaStream_t st,
                                    const double *mu)
{
    using C = PSide<K, MODE>;
    dim3 grid((unsigned)pl.gx, (unsigned)pl.S);
    if (mu) k_sweep_p_f64<K, MODE, true><<<grid, F_THREADS, C::smem, st>>>(bed, I, J, pitch, q, p, pl.slice, out, mu);
    else k_sweep_p_f64<K, MODE, false><<<grid, F_THREADS, C::smem, st>>>(bed, I, J, pitch, q, p, pl.slice, out, mu);
    return cudaGetLastError();
}

cudaError_t launch_sweep_p_f64(int K, int mode, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                               const double *q, const double *p, const SweepPlan &pl, double *out,
                               cudaStream_t st, const double *mu)
{
    cudaError_t e = cudaErrorInvalidValue;
    if (mode == 0) { ADMIX_DISPATCH_K(K, (e = launch_sweep_p_t<KK, 0>(bed, I, J, pitch, q, p, pl, out, st, mu))); }
    else { ADMIX_DISPATCH_K(K, (e = launch_sweep_p_t<KK, 1>(bed, I, J, pitch, q, p, pl, out, st, mu))); }
    return e;
}

static int grid_for(int64_t n, int sms)
{
    int64_t b = (n + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)sms * 16));
}

cudaError_t launch_emq_finalize(int64_t I, int K, int64_t J, int S, const double *parts,
                                const double *q, double *q_next, int sms, cudaStream_t st, int E, int off)
{
    k_emq_finalize<<<grid_for((int64_t)K * I, sms), 256, 0, st>>>(I, K, J, S, E > 0 ? E : K, off, parts, q, q_next);
    return cudaGetLastError();
}

cudaError_t launch_emp_finalize(int64_t J, int K, int S, const double *parts, const double *p,
                                double *p_next, int sms, cudaStream_t st)
{
    k_emp_finalize<<<grid_for((int64_t)K * J, sms), 256, 0, st>>>(J, K, S, parts, p, p_next);
    return cudaGetLastError();
}

cudaError_t launch_expand_hess(int64_t nprob, int K, int S, const double *parts, double *XtX,
                               double *Xtz, int sms, cudaStream_t st)
{
    const int E = K * (K + 1) / 2 + K;
    k_expand_hess<<<grid_for(nprob * E, sms), 256, 0, st>>>(nprob, K, S, parts, XtX, Xtz);
    return cudaGetLastError();
}

cudaError_t launch_sum_doubles(const double *src, int64_t n, double *dst, cudaStream_t st)
{
    k_sum_partials<<<1, 1024, 0, st>>>(src, n, dst);
    return cudaGetLastError();
}

cudaError_t launch_decode_counts(const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                                 unsigned long long *miss_snp, unsigned long long *miss_ind,
                                 int sms, cudaStream_t st)
{
    const int64_t Ib = (I + 3) / 4;
    const int gx = (int)((Ib + 255) / 256);
    int64_t gy = std::max<int64_t>(1, std::min<int64_t>(((int64_t)sms * 8 + gx - 1) / gx, J));
    const int64_t jslice = (J + gy - 1) / gy;
    gy = (J + jslice - 1) / jslice;
    k_decode_counts<<<dim3(gx, (unsigned)gy), 256, 0, st>>>(bed, I, J, Ib, pitch, jslice, miss_snp, miss_ind);
    return cudaGetLastError();
}

template <int K, int MODE, bool IMP>
static cudaError_t prepare_mode_t()
{
    cudaError_t e = cudaFuncSetAttribute(k_sweep_q_f64<K, MODE, IMP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)QSide<K, MODE>::smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sweep_p_f64<K, MODE, IMP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PSide<K, MODE>::smem);
    return e;
}

template <int K>
static cudaError_t prepare_sweeps_t()
{
    cudaError_t e = prepare_mode_t<K, 0, false>();
    if (e == cudaSuccess) e = prepare_mode_t<K, 1, false>();
    if (e == cudaSuccess) e = prepare_mode_t<K, 0, true>();
    if (e == cudaSuccess) e = prepare_mode_t<K, 1, true>();
    return e;
}

/* Dynamic shared-memory limits of the sweep kernels for this K; called once per handle
 * before any launch (and so before any stream capture). */
cudaError_t prepare_sweeps(int K)
{
    cudaError_t e = cudaErrorInvalidValue;
    ADMIX_DISPATCH_K(K, e = prepare_sweeps_t<KK>());
    return e;
}

/* Padding of the last genotype byte of every column (individuals >= I) set to the missing code
 * 01, so kernels that read whole 16-byte groups need no per-individual bound checks.  The
 * reference never reads those bits (its loops stop at I), so this changes no result. */
__global__ void k_mask_tail(uint8_t *__restrict__ bed, int64_t I, int64_t J, int64_t pitch)
{
    const int64_t Ib = (I + 3) / 4;
    const int r = (int)(I & 3);
    const unsigned keep = (1u << (2 * r)) - 1u;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < J; j += (int64_t)gridDim.x * blockDim.x) {
        uint8_t *b = bed + (size_t)j * pitch + (Ib - 1);
        *b = (uint8_t)((*b & keep) | (0x55u & ~keep));
    }
}

cudaError_t launch_mask_tail(uint8_t *bed, int64_t I, int64_t J, int64_t pitch, int sms, cudaStream_t st)
{
    if ((I & 3) == 0) return cudaSuccess;
    k_mask_tail<<<grid_for(J, sms), 256, 0, st>>>(bed, I, J, pitch);
    return cudaGetLastError();
}
