/*
 * qp_batch.cu -- batched per-individual simplex QPs and per-SNP box QPs of the block SQP
 * updates (update_q! / update_p!, algorithms_inner.jl:199-228 and 275-306), fused with the
 * x + delta step and the projection (projections.jl).
 *
 * A group of 4 to 32 lanes solves one problem (one thread where there are very many small ones, below), lane r holding row r of
 * the (K+2)^2 or (K+1)^2 tableau in registers; a sweep broadcasts the pivot column by shuffles.  The solver is the Jennrich-Sampson sweep /
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

/* ---- one thread per problem, for small tableaus in large numbers ----
 *
 * The tableau lives in shared memory in an [element][thread] layout, so a warp's accesses to the same element are
 * consecutive.  A problem is a serial chain, but where there are more problems than lanes on the GPU the chains overlap
 * anyway, and a group of 4 or 8 lanes for 2 to 6 rows repeats each pivot's division and selections in every lane.
 * 500k problems, one thread / lanes: K=1 13 / 33 us, K=2 29 / 48, K=4 113 / 158 (box), K=3 78 / 143 (simplex); from K = 5 on
 * the lanes are equal within 6 % or better (K=5 217 / 225, K=6 399 / 299).  Every entry sees the same operations in the same order as in
 * the lanes' solve: the same bits. */
constexpr int SB = 32;   /* problems (threads) per block */
constexpr int SERIAL_K = 4;

template <int N>
struct Tab {
    double *base;
    int tid;
    __device__ __forceinline__ double &operator()(int r, int c) const { return base[((r) * N + (c)) * SB + tid]; }
};

/* sweep! (qp.jl:297-317) */
template <int N>
__device__ __noinline__ void sweep_serial(const Tab<N> &A, double *tmp, int k, bool inverse)
{
    const double piv = 1.0 / A(k, k);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        tmp[i * SB] = A(i, k);
        A(i, k) = 0.0;
        A(k, i) = 0.0;
    }
    tmp[k * SB] = inverse ? 1.0 : -1.0;
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
        const double pv = __dmul_rn(piv, tmp[i * SB]);
#pragma unroll
        for (int j = 0; j < N; ++j) A(j, i) = __dsub_rn(A(j, i), __dmul_rn(pv, tmp[j * SB]));
    }
}

/* quadratic_program! (qp.jl:171-292) with pmin = 0, pmax = 1.  Returns the iteration count
 * or 0 on failure; delta is left as the reference leaves it. */
template <int K, int C>
__device__ int quadratic_program_serial(const Tab<K + C + 1> &A, double *tmp, double *d,
                                 const double (&par)[K], double (&delta)[K])
{
    constexpr int N = K + C + 1, E = N - 1;
    const double small = 1e-5, tol = 1e-8;
#pragma unroll
    for (int i = 0; i < K; ++i) delta[i] = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) d[i * SB] = A(i, i);
#pragma unroll 1
    for (int i = 0; i < K; ++i) {
        const double di = d[i * SB];
        if (di <= 0.0 || A(i, i) < __dmul_rn(di, tol)) return 0;
        sweep_serial<N>(A, tmp, i, false);
    }
    uint32_t swept = (K >= 32) ? 0xffffffffu : ((1u << K) - 1u);
#pragma unroll 1
    for (int i = K; i < K + C; ++i) {
        if (A(i, i) >= 0.0) return 0;
        sweep_serial<N>(A, tmp, i, false);
    }
    for (int iteration = 1; iteration <= 1000; ++iteration) {
        double a = 1.0;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (swept & (1u << i)) {
                const double ui = A(i, E);
                const double ai = (ui > 0.0) ? (1.0 - par[i] - delta[i]) : (0.0 - par[i] - delta[i]);
                if (fabs(ui) > 1e-10) a = fmin(a, ai / ui);
            }
        }
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (swept & (1u << i)) {
                const double ui = A(i, E);
                delta[i] = __dadd_rn(delta[i], __dmul_rn(a, ui));
                A(i, E) = __dmul_rn(1.0 - a, ui);
                A(E, i) = A(i, E);
            }
        }
        int pick = -1;
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (pick < 0) {
                const double xi = par[i] + delta[i];
                const bool critical = (0.0 >= xi - small) || (1.0 <= xi + small);
                if ((swept & (1u << i)) && fabs(A(i, i)) > 1e-10 && critical) pick = i;
            }
        }
        if (pick >= 0) {
            sweep_serial<N>(A, tmp, pick, true);
            swept &= ~(1u << pick);
            continue;
        }
#pragma unroll
        for (int i = 0; i < K; ++i) {
            if (pick < 0) {
                const double ui = A(i, E);
                const double xi = par[i] + delta[i];
                bool violation = ui > 0.0 && 0.0 >= xi - small;
                violation = violation || (ui < 0.0 && 1.0 <= xi + small);
                if (!(swept & (1u << i)) && violation) pick = i;
            }
        }
        if (pick >= 0) {
            sweep_serial<N>(A, tmp, pick, false);
            swept |= (1u << pick);
            continue;
        }
        return iteration;
    }
    return 0;
}

/* project_q! (projections.jl:27-59) on K values held in registers; s is scratch. */
template <int K>
__device__ __forceinline__ void project_simplex_serial(double (&b)[K], double *s)
{
    const double pc = 1e-5;
    const double tau = 1.0 - __dmul_rn((double)K, pc);
#pragma unroll
    for (int i = 0; i < K; ++i) b[i] -= pc;
    /* descending insertion sort of the values (order of equal values is immaterial) */
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const double v = b[i];
        int k = i;
        while (k > 0 && s[(k - 1) * SB] < v) { s[k * SB] = s[(k - 1) * SB]; --k; }
        s[k * SB] = v;
    }
    double tsum = 0.0, tmax = 0.0;
    bool bget = false;
    for (int i = 0; i < K - 1; ++i) {
        tsum += s[i * SB];
        tmax = (tsum - tau) / (double)(i + 1);
        if (tmax >= s[(i + 1) * SB]) { bget = true; break; }
    }
    if (!bget) tmax = (tsum + s[(K - 1) * SB] - tau) / (double)K;
#pragma unroll
    for (int i = 0; i < K; ++i) b[i] = fmax(b[i] - tmax, 0.0) + pc;
}

template <int K, bool SIMPLEX>
__global__ void __launch_bounds__(SB)
k_qp_serial(int64_t nprob, const double *__restrict__ parts, int S, const double *__restrict__ x,
     double *__restrict__ x_next, int32_t *__restrict__ status, int32_t *__restrict__ fail_count,
     const double *__restrict__ vt, int mu_mode, int damp_retry)
{
    constexpr int C = SIMPLEX ? 1 : 0;
    constexpr int N = K + C + 1;
    constexpr int T = K * (K + 1) / 2, E = T + K;
    extern __shared__ double sm[];
    const int tid = threadIdx.x;
    const int64_t pr = (int64_t)blockIdx.x * SB + tid;
    if (pr >= nprob) return;           /* no block-level synchronisation below */
    Tab<N> A{sm, tid};
    double *tmp = sm + N * N * SB + tid;
    double *d = tmp + N * SB;

    double par[K], delta[K];
#pragma unroll
    for (int k = 0; k < K; ++k) par[k] = x[(size_t)K * pr + k];

    /* create_tableau! (qp.jl:8-76): H, border -r = Xtz (r = -Xtz, algorithms_inner.jl:201) */
    const int64_t stride = nprob * (int64_t)E;
    const double *src = parts + (size_t)pr * E;
    int st = 0;
    for (int attempt = 0; attempt < (damp_retry ? 2 : 1) && st == 0; ++attempt) {
    const double dscale = attempt ? 1.0 + (double)K / 512.0 : 1.0;
#pragma unroll 1
    for (int k2 = 0; k2 < K; ++k2) {
#pragma unroll 1
        for (int k = 0; k <= k2; ++k) {
            const int e = tri_index(k, k2);
            double s = 0.0;
            for (int sl = 0; sl < S; ++sl) s += src[(size_t)sl * stride + e];
            if (k == k2) s *= dscale;
            A(k, k2) = s;
            A(k2, k) = s;
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
        for (int sl = 0; sl < S; ++sl) s += src[(size_t)sl * stride + T + k];
        A(N - 1, k) = s;
        A(k, N - 1) = s;
    }
    A(N - 1, N - 1) = 0.0;
    if (SIMPLEX) {
        double mu = 0.0;
        if (mu_mode == 1) {
            /* tmp_k = H v[:,1]; tmp_k = V' tmp_k; mu = 2 (|tmp_k|_1 - 2 tmp_k[1]) / K */
            /* t1 is staged in the d column (free until quadratic_program fills it) */
#pragma unroll 1
            for (int i = 0; i < K; ++i) {
                double s = 0.0;
#pragma unroll 1
                for (int j = 0; j < K; ++j) s = __dadd_rn(s, __dmul_rn(A(i, j), vt[j]));
                d[i * SB] = s;
            }
            double n1 = 0.0, first = 0.0;
#pragma unroll 1
            for (int i = 0; i < K; ++i) {
                double s = 0.0;
#pragma unroll 1
                for (int j = 0; j < K; ++j) s = __dadd_rn(s, __dmul_rn(vt[i + K * j], d[j * SB]));
                n1 += fabs(s);
                if (i == 0) first = s;
            }
            mu = (n1 - __dmul_rn(2.0, first)) / (double)K;
            mu = __dmul_rn(2.0, mu);
        }
#pragma unroll
        for (int j = 0; j < K; ++j)
#pragma unroll
            for (int i = 0; i < K; ++i) A(i, j) += mu;
#pragma unroll
        for (int i = 0; i < K; ++i) { A(K, i) = 1.0; A(i, K) = 1.0; }
        A(K, K) = 0.0;
        double sx = 0.0;
#pragma unroll
        for (int i = 0; i < K; ++i) sx += par[i];
        A(K + 1, K) = 1.0 - sx;
        A(K, K + 1) = 1.0 - sx;
        A(K + 1, K + 1) = 0.0;
    }

    st = quadratic_program_serial<K, C>(A, tmp, d, par, delta);
    }   /* attempts */
    if (status) status[pr] = st;
    if (st == 0 && fail_count) atomicAdd(fail_count, 1);

    double b[K];
#pragma unroll
    for (int k = 0; k < K; ++k) b[k] = par[k] + delta[k];
    if (SIMPLEX) {
        project_simplex_serial<K>(b, tmp);
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) b[k] = fmin(fmax(b[k], 1e-5), 1.0 - 1e-5);   /* project_p! */
    }
#pragma unroll
    for (int k = 0; k < K; ++k) x_next[(size_t)K * pr + k] = b[k];
}

template <int K, bool SIMPLEX>
constexpr size_t qp_serial_smem()
{
    constexpr int N = K + (SIMPLEX ? 1 : 0) + 1;
    return sizeof(double) * (size_t)SB * (N * N + 2 * N);
}

template <int K, bool SIMPLEX>
cudaError_t launch_qp_t(int64_t nprob, const double *parts, int S, const double *x, double *x_next,
                        int32_t *status, int32_t *fail_count, const double *vt, int mu_mode, int damp_retry,
                        int sms, cudaStream_t st)
{
    if (nprob <= 0) return cudaSuccess;
    /* One thread per problem where the lanes of all groups are more than the GPU holds (half of it up to K = 2).  One thread /
     * lanes in us either side of the line (box, 152k and 303k lanes of 148 SMs): K=2 20k problems 9 / 7, 50k 9 / 9, 100k 11 / 13;
     * K=3 50k 15 / 13, 100k 17 / 18, 200k 30 / 29; K=4 20k 19 / 13, 50k 23 / 22, 100k 33 / 37; simplex K=3 20k 13 / 11,
     * 50k 15 / 19, 100k 21 / 33. */
    if constexpr (K <= SERIAL_K) {
        if (nprob * QP<K, SIMPLEX>::G * (K <= 2 ? 2 : 1) > (int64_t)sms * 2048) {
            k_qp_serial<K, SIMPLEX><<<(unsigned)((nprob + SB - 1) / SB), SB, qp_serial_smem<K, SIMPLEX>(), st>>>(
                nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry);
            return cudaGetLastError();
        }
    }
    constexpr int per = QP<K, SIMPLEX>::PER;
    const unsigned grid = (unsigned)((nprob + per - 1) / per);
    k_qp<K, SIMPLEX><<<grid, QB, 0, st>>>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_qp(int K, bool simplex, int64_t nprob, const double *parts, int S,
                      const double *x, double *x_next, int32_t *status, int32_t *fail_count,
                      const double *vt, int mu_mode, int damp_retry, int sms, cudaStream_t st)
{
    cudaError_t e = cudaErrorInvalidValue;
    if (simplex) { ADMIX_DISPATCH_K(K, (e = launch_qp_t<KK, true>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry, sms, st))); }
    else { ADMIX_DISPATCH_K(K, (e = launch_qp_t<KK, false>(nprob, parts, S, x, x_next, status, fail_count, vt, mu_mode, damp_retry, sms, st))); }
    return e;
}
