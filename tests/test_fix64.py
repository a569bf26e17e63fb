"""CPU: the scaled 64-bit fixed-point arithmetic of the Cholesky factorisation
(csrc/fix64.cuh, the same functions as on the device) against long double.

Bounds: conversions round to nearest; a reciprocal square root is good to 2^-59
(its series' next term is below 2^-63, its operands 2^-61); an entry scaled by it
to one unit of 2^-60 times the pivot's 2^s; a product of limbs to 1.5 units, with the
low halves to half a unit and the 2^-15 that their dropped bits can weigh twice.
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
    std::mt19937_64 r(1);
    for (int i = 0; i < 300000; ++i) {
        const long long d = static_cast<long long>(r() >> (4 + r() % 58));
        if (d <= 0) continue;
        const Rsqrt y = rsqrt_fixed(d);
        const long double want = 1.0L / sqrtl(ldexpl(static_cast<long double>(d), -60));
        const long double got = ldexpl(y.y0, -24 + y.s) / sqrtl(1 - ldexpl(static_cast<long double>(y.e), -64));
        CHECK(fabsl(got / want - 1) < 0x1p-59L);
        bool bad = false;
        const long long c = (static_cast<long long>(r() >> 3) - (1ll << 60)) >> (r() % 45);
        const long double xe = ldexpl(static_cast<long double>(c) / sqrtl(static_cast<long double>(d)), 30);
        const long long x = scale(c, y, &bad);
        if (bad) CHECK(fabsl(xe) > 0.74L * 0x1p60L);
        else CHECK(fabsl(x - xe) <= 1 + ldexpl(1, y.s));
    }
    for (int i = 0; i < 300000; ++i) {
        long long v = (static_cast<long long>(r() >> 3) - (1ll << 60)) >> (r() % 61);
        v = v / 4 * 3;
        long long w = (static_cast<long long>(r() >> 3) - (1ll << 60)) >> (r() % 61);
        w = w / 4 * 3;
        int q[kSlices];
        digits(v, q);
        __int128 s = 0;
        for (int k = 0; k < kSlices; ++k) {
            s += static_cast<__int128>(q[k]) << (54 - 9 * k);
            CHECK(std::abs(q[k]) <= 256);
        }
        CHECK(s == static_cast<__int128>(v) * 4 && std::abs(q[0]) <= 193);
        const Limbs a = split(v), b = split(w);
        CHECK((static_cast<__int128>(a.hi) << 30) + a.lo == v && a.lo >= -(1 << 29) && a.lo < (1 << 29));
        Acc acc{0, 0};
        fms(acc, a, b);
        CHECK(fabsl(static_cast<long double>(value(acc)) + ldexpl(static_cast<long double>(v) * w, -60)) <= 1.5L);
        Acc full{0, 0};
        fms_full(full, a, b);
        const __int128 diff = (static_cast<__int128>(value(full)) << 60) + static_cast<__int128>(v) * w;
        CHECK(fabsl(ldexpl(static_cast<long double>(diff), -60)) <= 0.502L);
        const int e = static_cast<int>(r() % 2100) - 1075;
        CHECK(to_double(v, e) == static_cast<double>(ldexpl(static_cast<long double>(v), e - 60)));
    }
    for (int i = 0; i < 300000; ++i) {
        const double d = bits_double(static_cast<int64_t>(r() & 0x7fffffffffffffffull));
        if (!finite_positive(d)) continue;
        const int e = row_exponent(d);
        const long double s = ldexpl(static_cast<long double>(d), -2 * e);
        CHECK(s >= 0.125L && s < 0.5L);
        bool bad = false;
        const long long f = to_fixed(d, 2 * e, &bad);
        CHECK(!bad && fabsl(f - ldexpl(s, 60)) <= 0.5L && to_fixed(-d, 2 * e, &bad) == -f);
    }
    bool bad = false;
    CHECK(to_fixed(0.0, 0, &bad) == 0 && to_fixed(-0.0, 0, &bad) == 0 && !bad);
    for (double d : {5e-324, 1e-310, 2.3e-308}) CHECK(ldexpl(d, -2 * row_exponent(d)) >= 0.125L);
    for (double d : {HUGE_VAL, -HUGE_VAL, static_cast<double>(NAN), 0.76, 1e300}) {
        bad = false;
        CHECK(to_fixed(d, 0, &bad) == 0 && bad);
    }
    std::printf("ok\n");
    return 0;
}
"""


def test_fixed_point_arithmetic(tmp_path):
    cxx = shutil.which("g++") or pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", f"-I{CSRC}", str(src), "-o",
                    str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
