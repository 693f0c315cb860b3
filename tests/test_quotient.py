"""The division by a shared reciprocal (quotient in vct_device.cuh) rounds as
an IEEE division does, for all normal operands whose quotient and remainder
neither overflow nor underflow.

Only the significands matter: a = A, b = B with 2^23 <= A, B < 2^24.  The
first quotient q is within 1.5 units in its last place (y is off by half a
unit, its product with a by half of one), so the remainder, a whole multiple
of the product of both units and at most 1.5 x 2^24 of them, is off by one of
them or exact, and q + r y is within (1.5 x 2^-24 + 2^-23) units of a / b.  It
rounds as a / b does unless a midpoint of two neighbouring floats lies that
near.  The distance of a / b to the midpoint (2k + 1) / 2 units is
|c| / 2B units, where c = 2^25 A - (2k + 1) B (2^24 A where A >= B) is a whole
number other than 0: at most 7 in magnitude in question.  So for every B and
every such c all A are found from the congruence, and the two divisions
compared."""

from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHECK = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#define __device__
#define __forceinline__ inline
QUOTIENT
int main() {
    long long pairs = 0, wrong = 0;
    for (int below = 0; below < 2; ++below) {  // quotients in [1/2, 1), or [1, 2)
        const int bits = below ? 25 : 24;
        for (uint64_t B = 1u << 23; B < (1u << 24); ++B) {
            const int s = __builtin_ctzll(B);
            const uint64_t odd = B >> s;
            uint64_t inv = odd;  // its inverse modulo 2^64
            for (int i = 0; i < 5; ++i) inv *= 2 - odd * inv;
            const float b = (float)B, y = 1.0f / b;
            for (int c = -7; c <= 7; ++c) {
                if (c == 0 || (c & ((1 << s) - 1)) || s > 2 || !((c >> s) & 1)) continue;
                const uint64_t m = 1ull << (bits - s);
                for (uint64_t k = (uint64_t)(int64_t)(-(c >> s)) * inv & (m - 1); k < (1ull << bits); k += m) {
                    if (k < (1ull << (bits - 1))) continue;  // the quotient's leading bit
                    const int64_t n = (int64_t)(k * B) + c;
                    const uint64_t A = (uint64_t)n >> bits;
                    if ((A << bits) != (uint64_t)n || A < (1u << 23) || A >= (1u << 24) || (A < B) != (below == 1)) continue;
                    ++pairs;
                    const float a = (float)A;
                    if (quotient(a, b, y) != a / b) ++wrong;
                }
            }
        }
    }
    std::printf("%lld %lld\n", pairs, wrong);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_quotient_is_the_ieee_division(tmp_path):
    with open(os.path.join(ROOT, "vct_gb300", "csrc", "vct_device.cuh")) as f:
        body = re.search(r"__device__ __forceinline__ float quotient\(.*?\n}\n", f.read(), re.S).group(0)
    src, exe = tmp_path / "quotient.cpp", str(tmp_path / "quotient")
    src.write_text(_CHECK.replace("QUOTIENT", body.replace("fmaf(", "std::fma(")))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(src), "-o", exe], check=True)
    pairs, wrong = map(int, subprocess.run([exe], capture_output=True, text=True, check=True, timeout=600).stdout.split())
    assert pairs > 10_000_000 and wrong == 0
