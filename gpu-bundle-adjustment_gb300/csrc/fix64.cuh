#pragma once
// Scaled 64-bit fixed-point arithmetic of the dense Cholesky factorisation
// (chol.cu). GB300 issues one FP64 FMA per warp and SM sub-partition every 64
// cycles; three 32 x 32 + 64 integer multiply-adds take 12, and the tensor
// cores multiply small integers exactly, so the factorisation runs on integers.
//
// An SPD matrix is scaled symmetrically by powers of two, A_ij 2^-(e_i + e_j),
// so that its diagonal lies in [1/8, 1/2). Every entry of every Schur complement
// then stays below 1/2 and every entry of the scaled factor below 0.71: they are
// held as 64-bit integers, the factor's in units of 2^-60, the others, which are
// rounded once per panel, of 2^-62. The absolute rounding relative to
// sqrt(A_ii A_jj) is hundreds of times finer than that of an FP64 entry of that size.
// An entry far below its diagonal keeps that absolute precision, not FP64's relative
// one: of a coupling of 2^-k some 60 - k bits.
//
// Host and device: the same functions run on the CPU in tests/test_fix64.py.

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define GBA_FX __host__ __device__ __forceinline__
#else
#define GBA_FX inline
#endif

namespace gba {
namespace fx {

constexpr int kFrac = 60;                      // fraction bits
constexpr long long kBig = 3ll << (kFrac - 2);  // 0.75: larger entries do not occur in an SPD matrix

GBA_FX int clz_u64(uint64_t a) {  // a != 0
#ifdef __CUDA_ARCH__
    return __clzll(static_cast<long long>(a));
#else
    return __builtin_clzll(a);
#endif
}
GBA_FX int64_t double_bits(double d) {
    int64_t b;
#ifdef __CUDA_ARCH__
    b = __double_as_longlong(d);
#else
    std::memcpy(&b, &d, 8);
#endif
    return b;
}
GBA_FX double bits_double(int64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}

// Binary exponent (floor of log2) and 53-bit significand of a finite non-zero
// |d|: |d| = m 2^(x - 52), m in [2^52, 2^53).
GBA_FX void decompose(double d, int* x, uint64_t* m) {
    const uint64_t b = static_cast<uint64_t>(double_bits(d)) & 0x7fffffffffffffffull;
    int e = static_cast<int>(b >> 52);
    uint64_t f = b & 0xfffffffffffffull;
    if (e == 0) {  // subnormal
        const int s = clz_u64(f) - 11;
        f <<= s;
        e = 1 - s;
    } else {
        f |= 1ull << 52;
    }
    *x = e - 1023;
    *m = f;
}

GBA_FX bool finite_positive(double d) { return d > 0.0 && d <= 1.7976931348623157e308; }

// Row exponent e of a diagonal entry: d 2^(-2e) in [1/8, 1/2).
GBA_FX int row_exponent(double d) {
    int x;
    uint64_t m;
    decompose(d, &x, &m);
    return (x + 3) >> 1;
}

// d 2^(-e) in fixed point with kF fraction bits (up to 62), rounded to nearest; *bad is
// set where it is not finite or too large for an entry of a scaled SPD matrix (0 is
// returned).
template <int kF = kFrac>
GBA_FX long long to_fixed(double d, int e, bool* bad) {
    const int64_t b = double_bits(d);
    if ((b & 0x7fffffffffffffffll) == 0) return 0;
    if (((b >> 52) & 0x7ff) == 0x7ff) {
        *bad = true;
        return 0;
    }
    int x;
    uint64_t m;
    decompose(d, &x, &m);
    const int s = x - 52 - e + kF;  // |d| 2^-e 2^kF = m 2^s
    uint64_t v;
    if (s >= kF - 52) {
        *bad = true;
        return 0;
    } else if (s >= 0) {
        v = m << s;
    } else if (s > -55) {
        v = (m + (1ull << (-s - 1))) >> -s;
    } else {
        v = 0;
    }
    if (v > static_cast<uint64_t>(kBig) << (kF - kFrac)) {
        *bad = true;
        return 0;
    }
    return b < 0 ? -static_cast<long long>(v) : static_cast<long long>(v);
}

// v 2^-60 2^e as a double, rounded to nearest (ties to even).
GBA_FX double to_double(long long v, int e) {
    if (v == 0) return 0.0;
    const uint64_t a = v < 0 ? 0ull - static_cast<uint64_t>(v) : static_cast<uint64_t>(v);
    const int z = clz_u64(a);
    const uint64_t n = a << z;  // top bit set
    const uint64_t m = n >> 11, r = n & 0x7ff;
    const int x = 1023 + 63 - z - kFrac + e;  // biased exponent
    const uint64_t up = (r > 0x400 || (r == 0x400 && (m & 1))) ? 1 : 0;
    const uint64_t sign = v < 0 ? 1ull << 63 : 0;
    if (x >= 1 && x < 2046) {
        // (m - 2^52) + up may carry into the exponent field, as it should
        return bits_double(static_cast<int64_t>(sign | ((static_cast<uint64_t>(x) << 52) + (m - (1ull << 52)) + up)));
    }
    if (x >= 2046) {  // overflow, or the last binade
        if (x > 2046 || (m + up) >> 53) return bits_double(static_cast<int64_t>(sign | (0x7ffull << 52)));
        return bits_double(static_cast<int64_t>(sign | ((static_cast<uint64_t>(x) << 52) + (m - (1ull << 52)) + up)));
    }
    const int s = 12 - x;  // subnormal: shift the 64-bit significand right past the implicit bit
    if (s > 63) return bits_double(static_cast<int64_t>(sign | (s == 64 && n > (1ull << 63) ? 1 : 0)));
    const uint64_t q = n >> s, rr = n & ((1ull << s) - 1), half = 1ull << (s - 1);
    return bits_double(static_cast<int64_t>(sign | (q + ((rr > half || (rr == half && (q & 1))) ? 1 : 0))));
}

// Products: v = hi 2^30 + lo, lo in [-2^29, 2^29). The product of two entries,
// in units of 2^-60, is hi hi' + (hi lo' + lo hi' + lo lo' 2^-30) 2^-30: sums keep the
// two parts in two 64-bit accumulators. lo lo' is below a quarter unit: fms leaves it
// out, fms_full takes it from the upper halves of the factors.
struct Limbs {
    int hi, lo;
};
GBA_FX Limbs split(long long v) {
    Limbs l;
    l.lo = static_cast<int>(static_cast<uint32_t>(static_cast<uint64_t>(v)) << 2) >> 2;
    l.hi = static_cast<int>((v - l.lo) >> 30);
    return l;
}
struct Acc {
    long long c, m;  // c + m 2^-30
};
GBA_FX void fms(Acc& a, Limbs x, Limbs y) {  // a -= x y
    const int nh = -x.hi, nl = -x.lo;
    a.c += static_cast<long long>(nh) * y.hi;
    a.m += static_cast<long long>(nh) * y.lo;
    a.m += static_cast<long long>(nl) * y.hi;
}
GBA_FX void fms_full(Acc& a, Limbs x, Limbs y) {
    fms(a, x, y);
    a.m += static_cast<long long>(-x.lo >> 15) * (y.lo >> 15);
}
GBA_FX long long value(const Acc& a) { return a.c + ((a.m + (1ll << 29)) >> 30); }

// As the kernels take them: split at 2^29, so that within a panel, whose rounds wait for
// one another, lo lo' can be left out (fms): it is below a 16th of a unit (of the 63
// squares subtracted from a diagonal entry it is 1.3 units together; split at 2^30 5.3,
// and the solution's error at condition 4e3 three times as large). 4,096 unknowns 4.76
// -> 4.84 ms; 5.03 with all products whole. The update of few tiles takes them whole
// (fms_full). The sums are kept, and passed on, in quarter units, as the matrix is:
// entries below 2^61, their products' sums as well; of m, at most 2^62.5
// (Cauchy-Schwarz over 64 columns).
struct Limbs29 {
    int hi, lo;  // v = hi 2^29 + lo, lo in [-2^28, 2^28)
};
GBA_FX Limbs29 split29(long long v) {
    Limbs29 l;
    l.lo = static_cast<int>(static_cast<uint32_t>(static_cast<uint64_t>(v)) << 3) >> 3;
    l.hi = static_cast<int>((v - l.lo) >> 29);
    return l;
}
struct Acc29 {
    long long c, m;  // (c + m 2^-29) / 4
};
constexpr int kFracC = kFrac + 2;  // fraction bits of the matrix: quarter units
GBA_FX void fms(Acc29& a, Limbs29 x, Limbs29 y) {  // a -= x y
    const int nh = -x.hi, nl = -x.lo;
    a.c += static_cast<long long>(nh) * y.hi;
    a.m += static_cast<long long>(nh) * y.lo;
    a.m += static_cast<long long>(nl) * y.hi;
}
GBA_FX void fms_full(Acc29& a, Limbs29 x, Limbs29 y) {
    fms(a, x, y);
    a.m += static_cast<long long>(-x.lo >> 14) * (y.lo >> 15);
}
GBA_FX long long quarters(const Acc29& a) { return a.c + ((a.m + (1ll << 28)) >> 29); }
GBA_FX long long value(const Acc29& a) { return (a.c + ((a.m + (1ll << 30)) >> 29)) >> 2; }  // to nearest

// 1 / sqrt(d 2^-60) = y0 2^-24 (1 - e)^(-1/2) 2^s for d in (0, 2^60): an FP32
// reciprocal square root, the 24-bit y0 in [2^23, 2^24) and s in [1, 31], and
// the deviation e = 1 - d 2^-60 (y0 2^-24 2^s)^2 (|e| < 2^-21). The series
// 1 + e/2 + 3 e^2/8 is taken where it is applied (its next term is below
// 2^-63): its product with the entry then waits for e alone.
struct Rsqrt {
    uint32_t y0;
    int s;
    long long e;   // 2^-64
    uint32_t e2;   // e^2, 2^-64
};
GBA_FX Rsqrt rsqrt_fixed(long long d) {
    Rsqrt o;
    uint32_t yb;
#ifdef __CUDA_ARCH__
    // d as FP32 from its two halves: the 64-bit conversion takes longer
    const float fd = fmaf(static_cast<float>(static_cast<int>(d >> 32)), 4294967296.f,
                          __uint2float_rn(static_cast<uint32_t>(d)));
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(fd));
    yb = __float_as_uint(f);
#else
    const float yf = static_cast<float>(1.0 / __builtin_sqrt(static_cast<double>(static_cast<float>(d))));
    std::memcpy(&yb, &yf, 4);
#endif
    o.y0 = (yb & 0x7fffffu) | 0x800000u;  // 1 / sqrt(d) = y0 2^(E - 150)
    o.s = static_cast<int>(yb >> 23) - 96;
    const uint64_t dn = static_cast<uint64_t>(d) << ((2 * o.s) & 63);
    const uint64_t q = static_cast<uint64_t>(o.y0) * o.y0;
    // d y0^2 2^(2 s) 2^-44 mod 2^64 from 32-bit limbs of the 110-bit product
    const uint32_t a0 = static_cast<uint32_t>(dn), a1 = static_cast<uint32_t>(dn >> 32);
    const uint32_t b0 = static_cast<uint32_t>(q), b1 = static_cast<uint32_t>(q >> 32);
    uint64_t r = (static_cast<uint64_t>(a0) * b0) >> 32;
    r += static_cast<uint64_t>(a0) * b1;
    r += static_cast<uint64_t>(a1) * b0;
    o.e = -static_cast<long long>((r >> 12) + ((static_cast<uint64_t>(a1) * b1) << 20));
    const int e12 = static_cast<int>(o.e >> 12);
    o.e2 = static_cast<uint32_t>((static_cast<long long>(e12) * e12) >> 40);
    return o;
}

GBA_FX long long mulhi_s64(long long a, long long b) {
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return static_cast<long long>((static_cast<__int128>(a) * b) >> 64);
#endif
}

// |c| / sqrt(d) for |c| < 2^61 given rsqrt_fixed(d), to one unit; *bad where the
// result is larger than an entry of a scaled factor can be (0 is returned). The
// entry is shifted by s first: of a small pivot's column, whose entries are small,
// the product then keeps all bits.
GBA_FX long long scale_abs(long long c, const Rsqrt& r, bool* bad) {
    const int s = r.s & 31;
    uint64_t a = c < 0 ? 0ull - static_cast<uint64_t>(c) : static_cast<uint64_t>(c);
    if (a >> (61 - s)) {
        *bad = true;
        return 0;
    }
    a <<= s;
    const uint64_t u = ((static_cast<uint64_t>(static_cast<uint32_t>(a >> 32)) * r.y0) << 10) +
                       ((static_cast<uint64_t>(static_cast<uint32_t>(a)) * r.y0) >> 22);  // units of 2^-62
    const long long k = mulhi_s64(static_cast<long long>(u), r.e);
    const uint64_t k2 = (static_cast<uint64_t>(static_cast<uint32_t>(u >> 31)) * r.e2) >> 33;  // u e^2
    const uint64_t t = u + ((3 * k2) >> 3) + static_cast<uint64_t>(k >> 1);
    if (t > static_cast<uint64_t>(kBig) << 2) {
        *bad = true;
        return 0;
    }
    return static_cast<long long>((t + 3) >> 2);  // the truncations above lean by a quarter unit
}
GBA_FX long long scale(long long c, const Rsqrt& r, bool* bad) {
    const long long x = scale_abs(c, r, bad);
    return c < 0 ? -x : x;
}

// The seven balanced base-512 digits of an entry of the factor (|v| < 0.75),
// most significant first: v = sum_s q_s 2^(52 - 9 s), |q_0| <= 193, else
// |q_s| <= 2^8 (exact in FP16). The last digit holds two bits below the entry's unit,
// so that the digit products left out of an update (s + t > 6) stay
// below one unit.
constexpr int kSlices = 7;
GBA_FX void digits(long long v, int (&q)[kSlices]) {
    v = static_cast<long long>(static_cast<uint64_t>(v) << 2);
#pragma unroll
    for (int s = kSlices - 1; s > 0; --s) {
        const int d = ((static_cast<int>(v) + 256) & 511) - 256;
        q[s] = d;
        v = (v - d) >> 9;
    }
    q[0] = static_cast<int>(v);
}

}  // namespace fx
}  // namespace gba
