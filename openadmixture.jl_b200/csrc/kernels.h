/*
 * kernels.h -- host-side launchers of libadmix's device kernels (internal).
 */
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <vector>
#include "common.cuh"

/* gx CTAs (= partial sums) over nunit units: nblk blocks of 128 SNPs x slices of islice individuals */
struct LoglikPlan { int gx = 1; int64_t nblk = 1, nunit = 1, islice = 32; };
/* Device buffers listed first, then carved from one allocation (256-byte aligned): on a B200 host an
 * allocation takes 0.35 to 0.45 ms and its free 0.3 to 0.5, so 17 of them cost more than a small solve (and a pinned
 * block, which single handles no longer have, 1.1 to 2.9 ms). */
struct Carver {
    struct Item { void **p; size_t bytes; };
    std::vector<Item> items;
    size_t total = 0;
    template <typename T>
    void add(T **p, size_t count)
    {
        const size_t b = (sizeof(T) * (count ? count : 1) + 255) / 256 * 256;
        items.push_back({(void **)p, b});
        total += b;
    }
    cudaError_t carve(void **arena)
    {
        const cudaError_t e = cudaMalloc(arena, total ? total : 256);
        if (e != cudaSuccess) {
            *arena = nullptr;
            cudaGetLastError();
            return e;
        }
        uint8_t *at = (uint8_t *)*arena;
        for (const Item &i : items) {
            *i.p = (void *)at;
            at += i.bytes;
        }
        return cudaSuccess;
    }
};

struct SweepPlan  { int gx = 1, S = 1; int64_t slice = 1; int rows = 128; };   /* rows of a CTA */

LoglikPlan plan_loglik(int64_t I, int64_t J, int sms);
/* Slices of the second axis for CTAs of 128 rows, per_sm of which are resident per SM: whole waves, slices
 * a multiple of unit columns and at least min_units of them long, at most smax slices. */
SweepPlan plan_rows(int64_t rows, int64_t cols, int sms, int per_sm, int64_t unit, int64_t min_units, int64_t smax);
/* at most smax slices (a handle's partial-sum buffers are sized for its first plans) */
SweepPlan plan_sweep_q(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);
SweepPlan plan_sweep_p(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);

/* FP64 sweeps (sweeps_f64.cu) */
cudaError_t prepare_sweeps(int K);
/* mu (J doubles, the SNP means) != nullptr selects the reference's non-skipmissing loops.  padded: the
 * handle's column layout (16-byte pitch, padding coded missing). */
cudaError_t launch_loglik_f64(int K, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                              const double *p, const LoglikPlan &pl, bool padded, double *partial, double *out,
                              cudaStream_t st, const double *mu = nullptr);
cudaError_t launch_sweep_q_f64(int K, int mode, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                               const double *q, const double *p, const SweepPlan &pl, double *out,
                               cudaStream_t st, const double *mu = nullptr);
cudaError_t launch_sweep_p_f64(int K, int mode, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                               const double *q, const double *p, const SweepPlan &pl, double *out,
                               cudaStream_t st, const double *mu = nullptr);
/* g.mu of the SnpLinAlg: mean non-missing dosage per SNP of the padded device genotypes */
cudaError_t launch_snp_means(const uint8_t *bed, int64_t J, int64_t pitch, double *mu, cudaStream_t st);
/* SKFR AIM pre-selection (csrc/skfr.cu) on padded device genotypes; clusters_out: I, aims_out:
 * up to aims_capacity sorted SNP indices (n_aims: how many there are) */
cudaError_t skfr_run(const uint8_t *bed, int64_t pitch, int64_t I, int64_t J, int K, int64_t sparsity, int local,
                     int max_iter, int tries, uint64_t seed, cudaStream_t st, int32_t *clusters_out, int32_t *aims_out,
                     int64_t aims_capacity, int64_t *n_aims, double *objective_out, int32_t *iters_out);
/* fixed-order FP64 sum of n doubles into *dst (one block) */
cudaError_t launch_sum_doubles(const double *src, int64_t n, double *dst, cudaStream_t st);
cudaError_t launch_emq_finalize(int64_t I, int K, int64_t J, int S, const double *parts,
                                const double *q, double *q_next, int sms, cudaStream_t st, int E = 0, int off = 0);
cudaError_t launch_emp_finalize(int64_t J, int K, int S, const double *parts, const double *p,
                                double *p_next, int sms, cudaStream_t st);
cudaError_t launch_expand_hess(int64_t nprob, int K, int S, const double *parts, double *XtX,
                               double *Xtz, int sms, cudaStream_t st);
cudaError_t launch_decode_counts(const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                                 unsigned long long *miss_snp, unsigned long long *miss_ind,
                                 int sms, cudaStream_t st);

/* mixed-precision sweeps on tensor cores (sweeps_mixed.cu) */
cudaError_t prepare_mixed(int K);
/* The mixed-form plans pick their slice count for whole waves of resident CTAs, at most smax
 * slices (the partial-sum buffers of a handle are sized for its first plans). */
SweepPlan plan_sweep_q_mixed(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);
/* The mixed Q sweep first builds its per-chunk P packages in pkg (sweep_q_mixed_pkg_bytes). */
cudaError_t launch_sweep_q_mixed(int K, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                                 const double *p, const SweepPlan &pl, double *out, int *err, uint8_t *pkg,
                                 cudaStream_t st);
size_t sweep_q_mixed_pkg_bytes(int K, int64_t J);

SweepPlan plan_sweep_p_mixed(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);
SweepPlan plan_em_p_mixed(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);
/* The mixed P sweep first builds its per-chunk Q packages in pkg (sweep_p_mixed_pkg_bytes); pl: of plan_sweep_p_mixed
 * (mode 0) or plan_em_p_mixed (mode 1).
 * mode 0: gradient / Hessian rows (T + K); mode 1: the EM P-step's two sums (2K, k_emp_finalize). */
cudaError_t launch_sweep_p_mixed(int K, int mode, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch,
                                 const double *q, const double *p, const SweepPlan &pl, double *out, int *err,
                                 uint8_t *pkg, cudaStream_t st);
size_t sweep_p_mixed_pkg_bytes(int K, int64_t I);
/* The mixed log-likelihood first builds its per-chunk Q limb packages in pkg (this many bytes). */
size_t loglik_mixed_pkg_bytes(int K, int64_t I);
/* one CTA whose bounded wait on an mbarrier nothing completes runs out and sets *err */
cudaError_t launch_wait_probe(int *err, uint32_t polls, cudaStream_t st);
SweepPlan plan_loglik_mixed(int K, int64_t I, int64_t J, int sms, int64_t smax = INT64_MAX);
/* err and pkg are accepted for symmetry with the sweeps; the log-likelihood stays on the CUDA cores. */
cudaError_t launch_loglik_mixed(int K, const uint8_t *bed, int64_t I, int64_t J, int64_t pitch, const double *q,
                                const double *p, const SweepPlan &pl, double *partial, double *out, int *err,
                                uint8_t *pkg, cudaStream_t st);

cudaError_t launch_mask_tail(uint8_t *bed, int64_t I, int64_t J, int64_t pitch, int sms, cudaStream_t st);

/* batched QP + projection (qp_batch.cu) */
cudaError_t launch_qp(int K, bool simplex, int64_t nprob, const double *parts, int S,
                      const double *x, double *x_next, int32_t *status, int32_t *fail_count,
                      const double *vt, int mu_mode, int damp_retry, int sms, cudaStream_t st);

/* quasi-Newton (qn.cu) */
struct QNPlan { int blocks = 1; };
QNPlan plan_qn(int64_t n, int sms);
cudaError_t launch_qn(int Q, int64_t I, int64_t J, int K, const double *x0, const double *x1,
                      const double *x2, double *U, double *V, double *x_tmp, double *partial,
                      const QNPlan &pl, DevScalars *sc, int sms, cudaStream_t st);
cudaError_t launch_lbqn(int Q, int64_t I, int64_t J, int K, const double *x0, const double *x1,
                        const double *x2, double *U, double *V, double *x_tmp, double *partial,
                        const QNPlan &pl, DevScalars *sc, int sms, cudaStream_t st);
cudaError_t launch_iter_begin(DevScalars *sc, cudaStream_t st);
cudaError_t launch_accept(int64_t n, const double *x_tmp, const double *x_next2, double *x,
                          DevScalars *sc, int sms, cudaStream_t st);
cudaError_t launch_copy(int64_t n, const double *src, double *dst, int sms, cudaStream_t st);
