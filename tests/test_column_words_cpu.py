"""Reads of 16 column bytes at any alignment (csrc/col_words.h, the code that the learned start's P step runs): for every
small geometry, and every 16-byte block of every column, all reads stay inside the caller's genotypes and the
words hold the column's bytes, missing past its end.  The header is compiled for the host with readers that check."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "openadmixture.jl_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "col_words.h"
static const uint8_t *first, *end;
static long outside = 0, wrong = 0, words = 0;
struct Read {
    uint8_t byte(const uint8_t *p) const { if (p < first || p >= end) { ++outside; return 0; } return *p; }
    uint32_t word(const uint8_t *p) const
    {
        ++words;
        if ((uintptr_t)p & 3u) ++wrong;
        uint32_t v = 0;
        for (int n = 0; n < 4; ++n) v |= (uint32_t)byte(p + n) << (8 * n);
        return v;
    }
};
int main()
{
    std::vector<uint8_t> store(16384);
    for (size_t n = 0; n < store.size(); ++n) store[n] = (uint8_t)(n * 37 + 11);
    const uint8_t *base = store.data() + (16 - ((uintptr_t)store.data() & 15u)) % 16 + 64;
    for (int off = 0; off < 8; ++off)
        for (int64_t Ib = 1; Ib <= 70; ++Ib)
            for (int64_t pitch = Ib; pitch <= Ib + 4; ++pitch)
                for (int64_t J : {1, 2, 3, 5, 130}) {      /* groups of 128 columns */
                    first = base + off;
                    end = first + (J - 1) * pitch + Ib;   /* the last column need not be padded to the pitch */
                    for (int64_t j = 0; j < J; ++j) {
                        const uint8_t *col = first + j * pitch;
                        const int64_t limit = word_limit(j / 128 == (J - 1) / 128, Ib), limit0 = first_word_limit(j < 128, first, limit);
                        for (int64_t b0 = 0; b0 < Ib; b0 += 16) {
                            uint32_t w[4] = {0x55555555u, 0x55555555u, 0x55555555u, 0x55555555u};
                            if (b0 + 16 <= (b0 == 0 ? limit0 : limit)) block_words(Read{}, col + b0, w);
                            else block_bytes(Read{}, col, b0, Ib, w);
                            for (int n = 0; n < 16; ++n) {
                                const uint8_t want = b0 + n < Ib ? col[b0 + n] : 0x55;
                                if ((uint8_t)(w[n >> 2] >> (8 * (n & 3))) != want) ++wrong;
                            }
                        }
                    }
                }
    std::printf("outside %ld wrong %ld words %d\n", outside, wrong, words > 0);
    return 0;
}
"""


def test_reads_stay_inside_the_callers_genotypes(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["outside", "0", "wrong", "0", "words", "1"], out
