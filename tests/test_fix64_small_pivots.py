"""CPU: columns of small pivots in the fixed-point factorisation (csrc/fix64.cuh) against
long double. Their entries are small as well (an entry of an SPD matrix is at most the
root of its pivot and diagonal entry), and scaling them by a large reciprocal root must
keep what they hold: the result is good to a unit of 2^-60 at every pivot.

Bound: half a unit of rounding, three truncations of a quarter unit each, and the
reciprocal root's relative 2^-59.
"""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpu-bundle-adjustment_gb300" / "csrc"

PROGRAM = r"""
#include "fix64.cuh"
#include <cmath>
#include <cstdio>
#include <random>
using namespace gba::fx;
int main() {
    std::mt19937_64 r(3);
    long double sum = 0;
    int n = 0;
    for (int i = 0; i < 1000000; ++i) {
        const long long d = static_cast<long long>(r() >> (5 + r() % 59));
        if (d <= 0) continue;
        // |c| up to 0.7 2^30 sqrt(d): any column entry whose row holds it
        const long double top = 0.7L * 0x1p30L * sqrtl(static_cast<long double>(d));
        const long long c = static_cast<long long>(top * (static_cast<long double>(r() >> 11) / 0x1p53L * 2 - 1));
        bool bad = false;
        const long long x = scale(c, rsqrt_fixed(d), &bad);
        const long double want = ldexpl(static_cast<long double>(c) / sqrtl(static_cast<long double>(d)), 30);
        const long double err = (x - want) * (c < 0 ? -1 : 1);
        if (bad || fabsl(err) > 1.25L + fabsl(want) * 0x1p-59L) {
            std::printf("d %lld c %lld: %lld, want %.3Lf\n", d, c, x, want);
            return 1;
        }
        sum += err;
        ++n;
    }
    std::printf("mean error towards zero %.3Lf units\n", -sum / n);
    return fabsl(sum / n) > 0.5L;  // truncations alone, not rounding, may lean towards zero
}
"""


def test_scaled_entries_of_small_pivots(tmp_path):
    cxx = shutil.which("g++") or pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", f"-I{CSRC}", str(src), "-o",
                    str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
