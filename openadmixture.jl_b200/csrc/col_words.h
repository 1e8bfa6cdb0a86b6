/*
 * col_words.h -- 16 bytes (64 individuals) of a packed genotype column at any alignment, for kernels that take the
 * caller's own columns.  Host code too: the reads are the caller's functor, so that a program can watch them.
 */
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define COL_FN __host__ __device__ __forceinline__
#else
#define COL_FN inline
#endif

/* A column's 16-byte block b0 may be read as aligned words where b0 + 16 <= the limit of its group of columns.  A fifth word can
 * pass the end of the caller's genotypes by up to three bytes in the last column's last whole block, and block 0's
 * first word can begin that far before them in the first column of an unaligned base.  The group (a CTA's columns) that
 * holds the last or the first column gives up that block: one test for all its threads, and no register more than a plain end. */
COL_FN int64_t word_limit(bool has_last, int64_t Ib) { return has_last ? Ib / 16 * 16 - 1 : Ib; }
COL_FN int64_t first_word_limit(bool has_first, const uint8_t *genotypes, int64_t limit)
{
    return has_first && ((uintptr_t)genotypes & 3u) ? 0 : limit;
}

/* The 16 bytes at p, from the four or five aligned words that hold them */
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Read>
COL_FN void block_words(const Read &read, const uint8_t *p, uint32_t (&w)[4])
{
    const uint32_t mis = (uint32_t)((uintptr_t)p & 3u);
    const uint8_t *al = p - mis;
    uint32_t x[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) x[v] = (v < 4 || mis) ? read.word(al + 4 * v) : 0u;
#pragma unroll
#ifdef __CUDA_ARCH__
    for (int v = 0; v < 4; ++v) w[v] = __funnelshift_r(x[v], x[v + 1], 8 * mis);
#else
    for (int v = 0; v < 4; ++v) w[v] = (uint32_t)((((uint64_t)x[v + 1] << 32) | x[v]) >> (8 * mis));
#endif
}

/* Bytes [b0, b0 + 16) of the column at col up to its Ib, one at a time; w holds 0x55 (missing) for the others */
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Read>
COL_FN void block_bytes(const Read &read, const uint8_t *col, int64_t b0, int64_t Ib, uint32_t (&w)[4])
{
#pragma unroll
    for (int n = 0; n < 16; ++n)
        if (b0 + n < Ib) w[n >> 2] = (w[n >> 2] & ~(0xFFu << (8 * (n & 3)))) | ((uint32_t)read.byte(col + b0 + n) << (8 * (n & 3)));
}
