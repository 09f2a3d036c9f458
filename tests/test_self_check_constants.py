"""The host self-check of the 30-bit engine's constants and CRT table notices a wrong one: every constant
that the kernels read, changed by a little in turn (a program built from the library's host sources)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "engel-cuda-negacyclic-multiply_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include <cstdio>
#include <string>
#include <vector>
#include "hostmath.h"
using namespace nc;

static int bad = 0;
static void expect(bool found, const char* what, int bits) {
    if (!found) { std::printf("not noticed: %s at %d bits\n", what, bits); ++bad; }
}

int main() {
    for (int bits : {9, 31, 32, 40, 41, 434, 868, 947}) {
        const int L = (bits + 31) / 32;
        std::vector<uint32_t> q(size_t(L), 0x9e3779b9u);
        q[0] |= 1u;
        const int top = bits - 32 * (L - 1);
        q[size_t(L) - 1] = (top == 32 ? ~0u : (1u << top) - 1u) & (0xb7e15162u | (1u << (top - 1)) | (L == 1 ? 1u : 0u));
        QConst32 c{};
        const std::string err = build_qconst32(q.data(), L, 10, &c);
        if (!err.empty()) { std::printf("%s\n", err.c_str()); return 1; }
        const std::vector<uint8_t> table = crt32_table(c);
        const std::string ok = check_qconst32(c), ok2 = check_crt32_table(c, table);
        if (!ok.empty() || !ok2.empty()) { std::printf("%d bits: %s%s\n", bits, ok.c_str(), ok2.c_str()); return 1; }
#define CHANGED(field, by)                          \
    {                                               \
        QConst32 w = c;                             \
        w.field += by;                              \
        expect(!check_qconst32(w).empty(), #field, bits); \
    }
        CHANGED(top_byte, 1)
        CHANGED(top_shift, 1)
        CHANGED(top_shift, -1)
        CHANGED(top_neg_m, 1)
        CHANGED(top_neg_m, (1ull << 40))
        CHANGED(mu1, 1)
        CHANGED(mu1, -1)
        CHANGED(neg_q[0], 1)
        CHANGED(neg_q[c.LW], 1)
        CHANGED(neg_m[0], 1)
        CHANGED(q[L - 1], 1)
        CHANGED(y[c.k - 1], 1)
        CHANGED(mq[(c.k - 1) * (kMaxL + 2)], 1)
        // the table: a weight's lowest and highest byte, a quotient byte, a byte that has to be zero
        auto at = [&](int K, int col) { return size_t(col / 8) * 2048 + size_t(K / 16) * 128 + size_t(col % 8) * 16 + size_t(K % 16); };
        const int LW = int(c.LW), last = 4 * int(c.k) - 1;
        for (int K : {0, last})
            for (int col : {0, 4 * L - 1, 4 * LW, 4 * LW + 3}) {
                std::vector<uint8_t> w = table;
                w[at(K, col)] ^= 1;
                expect(!check_crt32_table(c, w).empty(), "table byte", bits);
            }
        if (last < 255) {
            std::vector<uint8_t> w = table;
            w[at(255, 0)] = 1;
            expect(!check_crt32_table(c, w).empty(), "padding byte of a row", bits);
        }
        std::vector<uint8_t> w = table;
        w.pop_back();
        expect(!check_crt32_table(c, w).empty(), "table size", bits);
    }
    for (const PrimeConst32& p : prime_set32())
        expect(p.p > (7u << 27), "prime above 7/8 of 2^30", 30);
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not CUDA_INCLUDE.exists(), reason="needs g++ and the CUDA headers")
def test_changed_constants_are_noticed(tmp_path):
    src = tmp_path / "check.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", f"-I{CUDA_INCLUDE}", str(src), str(CSRC / "hostmath.cpp"), "-o",
                    str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
