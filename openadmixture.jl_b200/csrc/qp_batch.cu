/*
 * qp_batch.cu -- batched per-individual simplex QPs and per-SNP box QPs of the block SQP
 * updates (update_q! / update_p!, algorithms_inner.jl:199-228 and 275-306), fused with the
 * x + delta step and the projection (projections.jl).
 *
 * A group of 4 to 32 lanes solves one problem, lane r holding row r of the (K+2)^2 or (K+1)^2 tableau in
 * registers; a sweep broadcasts the pivot column by shuffles.  The solver is the Jennrich-Sampson sweep /
 * active-set method of qp.jl:171-317, step for step: every entry sees the same operations in the
 * same order as in a serial solve.  Products feeding a sum are rounded separately (__dmul_rn /
 * __dadd_rn), as in the reference's plain Julia loops, so the tableau arithmetic is the same IEEE
 * sequence as the oracle's; only the accumulated XtX / Xtz inputs differ in their last bits.
 *
 * A problem is one serial chain of about 2 K sweeps, so one thread per problem (its tableau in shared
 * memory) ran at the latency of K^2-long chains with 11 warps per SM.
 * Measured on a B200, Q / P block: K=3, 203 / 517 problems 13 / 11 -> 6.8 / 7.0 us; K=6, 20k / 50k problems
 * 143 / 216 -> 28 / 32 us; K=12, 20k / 60k 368 / 843 -> 134 / 238 us.
 */
#include "common.cuh"
#include "kernels.h"

namespace {

constexpr int QB = 128;   /* threads per block */
constexpr uint32_t FULL = 0xffffffffu;

/* rows of the tableau, lanes of a group */
template <int K, bool SIMPLEX>
struct QP {
    static constexpr int C = SIMPLEX ? 1 : 0;
    static constexpr int N = K + C + 1;
    static constexpr int G = N <= 4 ? 4 : (N <= 8 ? 8 : (N <= 16 ? 16 : 32));
    static constexpr int T = K * (K + 1) / 2, E = T + K;
    static constexpr int PER = QB / G;                /* problems per block */
};

__device__ __forceinline__ double pick(bool p, double a, double b) { return p ? a : b; }

/* element k of this lane's row */
template <int N>
__device__ __forceinline__ double row_at(const double (&A)[N], int k)
{
    double v = A[0];
#pragma unroll
    for (int c = 1; c < N; ++c) v = pick(c == k, A[c], v);
    return v;
}

/* sweep! (qp.jl:297-317) of row and column k in the groups where on; every lane of the warp calls it */
template <int N, int G>
__device__ __forceinline__ void sweep(double (&A)[N], int r, int k, bool inverse, bool on)
{
    double tmp = row_at<N>(A, k);                     /* A(r, k) */
    const double piv = 1.0 / __shfl_sync(FULL, tmp, k, G);
    if (r == k) tmp = inverse ? 1.0 : -1.0;
    const double own = __dmul_rn(piv, tmp);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const double pv = __shfl_sync(FULL, own, i, G);
        const double a = (i == k || r == k) ? 0.0 : A[i];
        const double v = __dsub_rn(a, __dmul_rn(pv, tmp));
        A[i] = pick(on, v, A[i]);
    }
}

/* quadratic_program! (qp.jl:171-292) with pmin = 0, pmax = 1, on every group of the warp (those with !live
 * do nothing).  Returns the iteration count or 0 on failure; lane r's delta is left as the reference
 * leaves it. */
template <int K, bool SIMPLEX>
__device__ __forceinline__ int quadratic_program(double (&A)[QP<K, SIMPLEX>::N], int r, double par, bool live, double &delta)
{
    using P = QP<K, SIMPLEX>;
    constexpr int N = P::N, G = P::G, E = N - 1;
    const double small = 1e-5, tol = 1e-8;
    const int shift = (threadIdx.x & 31) & ~(G - 1);
    const uint32_t gmask = G == 32 ? FULL : ((1u << (G & 31)) - 1u);
    delta = 0.0;
    bool run = live;
    const double d = row_at<N>(A, r);
#pragma unroll 1
    for (int i = 0; i < K; ++i) {
        const double di = __shfl_sync(FULL, d, i, G), ai = __shfl_sync(FULL, row_at<N>(A, i), i, G);
        run = run && !(di <= 0.0 || ai < __dmul_rn(di, tol));
        sweep<N, G>(A, r, i, false, run);
    }
    if (SIMPLEX) {
        const double ai = __shfl_sync(FULL, A[K], K, G);
        run = run && !(ai >= 0.0);
        sweep<N, G>(A, r, K, false, run);
    }
    bool swept = r < K;
    int st = 0;
#pragma unroll 1
    for (int iteration = 1; iteration <= 1000; ++iteration) {
        if (!__any_sync(FULL, run)) break;
        /* the longest step to the box that the swept coordinates allow */
        const double ui = A[E];
        double a = 1.0;
        if (swept) {
            const double ai = (ui > 0.0) ? (1.0 - par - delta) : (0.0 - par - delta);
            if (fabs(ui) > 1e-10) a = fmin(a, ai / ui);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) a = fmin(a, __shfl_xor_sync(FULL, a, o, G));
        if (swept && run) {
            delta = __dadd_rn(delta, __dmul_rn(a, ui));
            A[E] = __dmul_rn(1.0 - a, ui);
        }
        const uint32_t sw = __ballot_sync(FULL, swept) >> shift;
#pragma unroll
        for (int i = 0; i < K; ++i) {                 /* A(E, i) = A(i, E) */
            const double v = __shfl_sync(FULL, A[E], i, G);
            A[i] = pick(run && r == E && ((sw >> i) & 1u), v, A[i]);
        }
        const double xi = par + delta, uj = A[E];
        const bool crit = swept && fabs(row_at<N>(A, r)) > 1e-10 && ((0.0 >= xi - small) || (1.0 <= xi + small));
        const bool viol = !swept && r < K && ((uj > 0.0 && 0.0 >= xi - small) || (uj < 0.0 && 1.0 <= xi + small));
        const uint32_t bc = (__ballot_sync(FULL, crit) >> shift) & gmask, bv = (__ballot_sync(FULL, viol) >> shift) & gmask;
        const bool out = bc != 0u;                    /* a critical coordinate leaves, else a violating one enters */
        const int p = __ffs((int)(out ? bc : bv)) - 1;
        if (run && p < 0) {
            st = iteration;
            run = false;
        }
        sweep<N, G>(A, r, p < 0 ? 0 : p, out, run);
        if (run && r == p) swept = !out;
    }
    return st;
}

/* project_q! (projections.jl:27-59) of the K values held one per lane (lanes < K); s: K doubles of shared
 * memory of this group */
template <int K, int G>
__device__ __forceinline__ double project_simplex(double b, int r, double *s)
{
    const double pc = 1e-5;
    const double tau = 1.0 - __dmul_rn((double)K, pc);
    b -= pc;
    int rank = 0;                                     /* place in descending order */
    bool nan = r < K && b != b;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const double v = __shfl_sync(FULL, b, i, G);
        rank += (v > b || (v == b && i < r)) ? 1 : 0;
        nan = nan || v != v;
    }
    __syncwarp();
    if (r < K) s[nan ? r : rank] = b;
    __syncwarp();
    if (nan && r == 0)                                /* unordered values: the serial insertion sort's order */
        for (int i = 0; i < K; ++i) {
            const double v = s[i];
            int k = i;
            while (k > 0 && s[k - 1] < v) { s[k] = s[k - 1]; --k; }
            s[k] = v;
        }
    __syncwarp();
    double tsum = 0.0, tmax = 0.0;
    bool bget = false;
#pragma unroll 1
    for (int i = 0; i < K - 1; ++i) {
        tsum += s[i];
        tmax = (tsum - tau) / (double)(i + 1);
        if (tmax >= s[i + 1]) { bget = true; break; }
    }
    if (!bget) tmax = (tsum + s[K - 1] - tau) / (double)K;
    return fmax(b - tmax, 0.0) + pc;
}

/* damp_retry (the mixed-precision form only): a problem whose QP fails is solved once more with
 * the Hessian's diagonal scaled by 1 + K/512.  A BF16 Hessian rounds every pair product p_k p_k'
 * on its own, so a problem whose exact Hessian is nearly singular can come out slightly
 * indefinite and fail the reference's pivot tests; the scaling covers that rounding (K * 2^-9
 * per row, Gershgorin) and only shortens the Newton step -- the fixed point is set by the
 * gradient.  The FP64 form never retries: a failed QP leaves the reference's zero step. */
template <int K, bool SIMPLEX>
__global__ void __launch_bounds__(QB)
k_qp(int64_t nprob, const double *__restrict__ parts, int S, const double *__restrict__ x,
     double *__restrict__ x_next, int32_t *__restrict__ status, int32_t *__restrict__ fail_count,
     const double *__restrict__ vt, int mu_mode, int damp_retry)
{
    using P = QP<K, SIMPLEX>;
    constexpr int N = P::N, G = P::G, T = P::T, E = P::E;
    __shared__ double sm[P::PER * E];
    const int r = threadIdx.x & (G - 1);              /* row of the tableau */
    const int64_t pr = (int64_t)blockIdx.x * P::PER + threadIdx.x / G;
    const bool live = pr < nprob;
    double *sums = sm + (threadIdx.x / G) * E;
    const double par = (live && r < K) ? x[(size_t)K * pr + r] : 0.0;

    /* the slices' partial sums, added in slice order */
    const int64_t stride = nprob * (int64_t)E;
    for (int e = r; e < E; e += G) {
        double s = 0.0;
        if (live) {
            const double *src = parts + (size_t)pr * E + e;
#pragma unroll 8
            for (int sl = 0; sl < S; ++sl) s += src[(size_t)sl * stride];
        }
        sums[e] = s;
    }
    __syncwarp();

    int st = 0;
    double delta = 0.0;
#pragma unroll 1
    for (int attempt = 0; attempt < (damp_retry ? 2 : 1); ++attempt) {
        const bool todo = live && st == 0;
        if (!__any_sync(FULL, todo)) break;
        const double dscale = attempt ? 1.0 + (double)K / 512.0 : 1.0;
        /* create_tableau! (qp.jl:8-76): H, border -r = Xtz (r = -Xtz, algorithms_inner.jl:201) */
        double A[N];
#pragma unroll
        for (int c = 0; c < N; ++c) A[c] = 0.0;
        if (r < K) {
#pragma unroll
            for (int c = 0; c < K; ++c) {
                A[c] = sums[c <= r ? tri_index(c, r) : tri_index(r, c)];
                if (c == r) A[c] *= dscale;
            }
            A[N - 1] = sums[T + r];
        } else if (r == N - 1) {
#pragma unroll
            for (int c = 0; c < K; ++c) A[c] = sums[T + c];
        }
        if (SIMPLEX) {
            double mu = 0.0;
            if (mu_mode == 1) {
                /* tmp_k = H v[:,1]; tmp_k = V' tmp_k; mu = 2 (|tmp_k|_1 - 2 tmp_k[1]) / K */
                double t1 = 0.0, t2 = 0.0, n1 = 0.0, first = 0.0;
#pragma unroll
                for (int j = 0; j < K; ++j) t1 = __dadd_rn(t1, __dmul_rn(A[j], vt[j]));
#pragma unroll
                for (int j = 0; j < K; ++j)
                    t2 = __dadd_rn(t2, __dmul_rn(vt[(r < K ? r : 0) + K * j], __shfl_sync(FULL, t1, j, G)));
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    const double s = __shfl_sync(FULL, t2, i, G);
                    n1 += fabs(s);
                    if (i == 0) first = s;
                }
                mu = (n1 - __dmul_rn(2.0, first)) / (double)K;
                mu = __dmul_rn(2.0, mu);
            }
            double sx = 0.0;
#pragma unroll
            for (int i = 0; i < K; ++i) sx += __shfl_sync(FULL, par, i, G);
            if (r < K) {
#pragma unroll
                for (int c = 0; c < K; ++c) A[c] += mu;
                A[K] = 1.0;
            } else if (r == K) {
#pragma unroll
                for (int c = 0; c < K; ++c) A[c] = 1.0;
                A[N - 1] = 1.0 - sx;
            } else if (r == N - 1) {
                A[K] = 1.0 - sx;
            }
        }
        double dl;
        const int s1 = quadratic_program<K, SIMPLEX>(A, r, par, todo, dl);
        if (todo) {
            st = s1;
            delta = dl;
        }
    }
    if (live && r == 0) {
        if (status) status[pr] = st;
        if (st == 0 && fail_count) atomicAdd(fail_count, 1);
    }
    double b = par + delta;
    if (SIMPLEX) b = project_simplex<K, G>(b, r, sums);
    else b = fmin(fmax(b, 1e-5), 1.0 - 1e-5);         /* project_p! */
    if (live && r < K) x_next[(size_t)K * pr + r] = b;
}

template <int K, bool SIMPLEX>
cudaError_t launch_qp_t(int64_t nprob, const double *parts, int S, const double *x, double *x_next,
                        int32_t *status, int32_t *fail_count, const double *vt, int mu_mode, int damp_retry,
                        cudaStream_t st)
{
    if (nprob <= 0) return cudaSuccess;
    constexpr int per = QP<K, SIMPLEX>::PER;
    const unsigned grid = (unsigned)((nprob + per - 1) / per);
    k_qp<K, SIMPLEX><<<grid, QB, 0, st>>>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_qp(int K, bool simplex, int64_t nprob, const double *parts, int S,
                      const double *x, double *x_next, int32_t *status, int32_t *fail_count,
                      const double *vt, int mu_mode, int damp_retry, cudaStream_t st)
{
    cudaError_t e = cudaErrorInvalidValue;
    if (simplex) { ADMIX_DISPATCH_K(K, (e = launch_qp_t<KK, true>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry, st))); }
    else { ADMIX_DISPATCH_K(K, (e = launch_qp_t<KK, false>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry, st))); }
    return e;
}
