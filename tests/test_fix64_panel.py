"""CPU: the products within a panel of the fixed-point factorisation (csrc/fix64.cuh)
against 128-bit integers.

Bounds, in units of 2^-60: the low halves' product, left out, is below 2^56 2^-60, and
a value is rounded to nearest (passed on, to a quarter unit; with the low halves to
2^-15 of that more). A panel's 63 squares together lose
at most 63/16 and on average 63/48; the same sums split at 2^30 lose four times that.
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
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
    std::mt19937_64 r(5);
    for (int i = 0; i < 300000; ++i) {
        const long long v = ((static_cast<long long>(r() >> 3) - (1ll << 60)) >> (r() % 61)) / 4 * 3;
        const long long w = ((static_cast<long long>(r() >> 3) - (1ll << 60)) >> (r() % 61)) / 4 * 3;
        const Limbs29 a = split29(v), b = split29(w);
        CHECK((static_cast<__int128>(a.hi) << 29) + a.lo == v && a.lo >= -(1 << 28) && a.lo < (1 << 28));
        const Acc29 half{v / 2 * 4, 0};
        CHECK(value(half) == v / 2 && quarters(half) == v / 2 * 4);
        Acc29 acc{0, 0};
        fms(acc, a, b);
        const long double want = -ldexpl(static_cast<long double>(static_cast<__int128>(v) * w), -60);
        CHECK(fabsl(value(acc) - want) <= 0.5L + 0.125L + 0.0625L);
        CHECK(fabsl(quarters(acc) / 4.0L - want) <= 0.125L + 0.0625L);
        Acc29 full{0, 0};
        fms_full(full, a, b);
        CHECK(fabsl(quarters(full) / 4.0L - want) <= 0.126L);
        // the matrix itself, in quarter units
        const int e = static_cast<int>(r() % 2000) - 1000;
        bool bad = false;
        const double d = ldexp(static_cast<double>(v), e - 60);
        const long long f = to_fixed<kFracC>(d, e, &bad);
        if (bad) CHECK(std::abs(v) > 3ll << 58);
        else CHECK(f == ldexpl(static_cast<long double>(d), 62 - e) && std::abs(v) <= 3ll << 58);
    }
    // a diagonal entry: 63 squares, random and with the low halves at their largest
    long double sum = 0;
    for (int i = 0; i < 20000; ++i) {
        const long long d = (1ll << 59) - 1;
        Acc29 acc{4 * d, 0};
        __int128 exact = static_cast<__int128>(d) << 60;
        for (int k = 0; k < 63; ++k) {
            long long v = static_cast<long long>(r() >> 5) / 7;  // squares add up to less than 1/2
            if (i < 2) v = (v >> 29 << 29) + (i ? (1ll << 28) - 1 : 1ll << 28);
            fms(acc, split29(v), split29(v));
            exact -= static_cast<__int128>(v) * v;
        }
        const long double err = value(acc) - ldexpl(static_cast<long double>(exact), -60);
        CHECK(exact > 0 && err >= -0.625L && err <= 63 / 16.0L + 0.625L);
        if (i >= 2) sum += err;
    }
    std::printf("mean %.3Lf units\n", sum / 19998);
    CHECK(fabsl(sum / 19998 - 63 / 48.0L) < 0.05L);
    std::printf("ok\n");
    return 0;
}
"""


def test_products_within_a_panel(tmp_path):
    cxx = shutil.which("g++") or pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", f"-I{CSRC}", str(src), "-o",
                    str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
