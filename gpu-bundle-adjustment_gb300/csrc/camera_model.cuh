#pragma once
// Snavely camera model: residual and analytic Jacobian of one observation,
// shared by the host (FP64 finite-difference entry point) and by the device
// edge kernels (FP64 plain form, FP32 mixed form).
//
// Model (BAL; reference src/lm.cu:58-82 and 93-191 evaluate the same function):
//   X_c = R(a) X + t,  u = -X_c.x / X_c.z,  v = -X_c.y / X_c.z,
//   d   = 1 + k1 r2 + k2 r2^2  (r2 = u^2 + v^2),  pred = f d (u, v),
//   residual = pred - obs.
// Rotation branch: the Rodrigues formula when |a|^2 > 1e-24 (FP64 threshold of
// the reference edge kernel, src/lm.cu:62-63), else the first-order model
// R(a) X = X + a x X with dR X/da = -[X]x and R = I (src/lm.cu:72-76,141-149).
//
// Jacobian derivation used here (own derivation, mathematically equal to the
// reference's): for a rotation vector a, R(a + da) X = R(a) X - [R X]x J_l(a) da,
// with the left Jacobian of SO(3)
//   J_l(a) = (s/th) I + ((1-c)/th) [w]x + (1 - s/th) w w^T,  w = a/th,
// so dX_c/da = -[R X]x J_l(a). With t = th^2 and the entire functions
//   A = s/th = 1 - t C,  B = (1 - c)/t,  C = (1 - A)/t,  c = 1 - t B,
// R = c I + A [a]x + B a a^T and J_l = A I + B [a]x + C a a^T: no root, no
// division, and for t <= 10 (|a| up to 3.16, any rotation) two short power series
// instead of sine and cosine. The camera records (camera_constants) form 1 - c as
// 2 sin^2(th/2), which avoids cancellation at small th.
//   d(u,v)/dX_c = [[-1/z, 0, x/z^2], [0, -1/z, y/z^2]]
//   d pred/d(u,v) = f (d I + 2 L (u,v)^T (u,v)),  L = k1 + 2 k2 r2.

#ifdef __CUDACC__
#define GBA_HD __host__ __device__ __forceinline__
#else
#define GBA_HD inline
#endif

#include <cmath>

namespace gba {
namespace model {

template <typename T>
GBA_HD T msqrt(T x) { return sqrt(x); }
template <>
GBA_HD float msqrt<float>(float x) { return sqrtf(x); }
template <typename T>
GBA_HD void msincos(T x, T* s, T* c) { *s = sin(x); *c = cos(x); }
template <>
GBA_HD void msincos<float>(float x, float* s, float* c) { *s = sinf(x); *c = cosf(x); }
template <typename T>
GBA_HD T msin(T x) { return sin(x); }
template <>
GBA_HD float msin<float>(float x) { return sinf(x); }

template <int N>
struct Factorial { static constexpr double value = N * Factorial<N - 1>::value; };
template <>
struct Factorial<0> { static constexpr double value = 1.0; };

// sum over k = K .. Last of (-t)^(k - K) / (2 k + Off)!
template <int K, int Last, int Off>
struct Series {
    static GBA_HD double at(double t) {
        constexpr double c = 1.0 / Factorial<2 * K + Off>::value;
        if constexpr (K == Last)
            return c;
        else
            return c - t * Series<K + 1, Last, Off>::at(t);
    }
};

// A, B, C and c of t = |a|^2 > 0. The series end where t = 10 leaves less than
// half a unit in the last place of B and C. Their terms alternate and the largest is
// 1/2 (1/6), so they lose no digits. 28 FP64 instructions against about 95 for the
// root, the division, the sine and cosine of th and the sine of th/2: an FP64 edge
// kernel is bound by them.
GBA_HD void rotation_terms(double t, double& A, double& B, double& C, double& c) {
    constexpr int kLast = 13;
    if (t <= 10.0) {
        B = Series<0, kLast, 2>::at(t);
        C = Series<0, kLast, 3>::at(t);
        A = 1.0 - t * C;
        c = 1.0 - t * B;
    } else {  // also a NaN
        const double th = sqrt(t);
        const double sh = sin(0.5 * th);
        c = cos(th);
        A = sin(th) / th;
        B = 2.0 * sh * sh / t;
        C = (1.0 - A) / t;
    }
}

// Residual only.
GBA_HD void residual(const double* cam, const double* X, const double* obs, double* r) {
    double P[3];
    const double* a = cam;
    const double t = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    const double x0 = a[1] * X[2] - a[2] * X[1], x1 = a[2] * X[0] - a[0] * X[2], x2 = a[0] * X[1] - a[1] * X[0];
    if (t > 1e-24) {
        double A, B, C, c;
        rotation_terms(t, A, B, C, c);
        const double q = B * (a[0] * X[0] + a[1] * X[1] + a[2] * X[2]);
        P[0] = c * X[0] + (A * x0 + (q * a[0] + cam[3]));
        P[1] = c * X[1] + (A * x1 + (q * a[1] + cam[4]));
        P[2] = c * X[2] + (A * x2 + (q * a[2] + cam[5]));
    } else {
        P[0] = X[0] + x0 + cam[3];
        P[1] = X[1] + x1 + cam[4];
        P[2] = X[2] + x2 + cam[5];
    }
    const double iz = 1.0 / P[2];
    const double u = -P[0] * iz, v = -P[1] * iz;
    const double r2 = u * u + v * v;
    const double fd = cam[6] * (1.0 + r2 * (cam[7] + cam[8] * r2));
    r[0] = fd * u - obs[0];
    r[1] = fd * v - obs[1];
}

// Residual and Jacobian rows from the rotation R, its left Jacobian J_l, R X and
// tf = (t, f, k1, k2).
GBA_HD void jacobian_rows(const double* R, const double* Jl, const double* RX, bool first_order, const double* tf,
                          const double* X, const double* obs, double* r, double* Jc, double* Jp) {
    const double iz = 1.0 / (RX[2] + tf[2]);
    const double u = -(RX[0] + tf[0]) * iz, v = -(RX[1] + tf[1]) * iz;
    const double r2 = u * u + v * v;
    const double f = tf[3], k1 = tf[4], k2r2 = tf[5] * r2;
    const double d = 1.0 + r2 * (k1 + k2r2);
    const double fd = f * d;
    r[0] = fd * u - obs[0];
    r[1] = fd * v - obs[1];

    // D = f (d I + 2 L [u v]^T [u v]), L = k1 + 2 k2 r2, and
    // M = d(u,v)/dX_c = [[-iz, 0, -u iz], [0, -iz, -v iz]]; g = rows of D M
    const double fL2 = 2.0 * f * (k1 + 2.0 * k2r2);
    const double fu = fL2 * u;
    double g[6];
    g[0] = -(fd + fu * u) * iz;
    g[1] = g[3] = -(fu * v) * iz;
    g[4] = -(fd + fL2 * v * v) * iz;
    g[2] = g[0] * u + g[1] * v;
    g[5] = g[3] * u + g[4] * v;

    // rotation columns: g (-[y]x) J_l, y = R X (main branch) or X (first-order
    // branch); (-[y]x) = [[0,y2,-y1],[-y2,0,y0],[y1,-y0,0]]
    const double y0 = first_order ? X[0] : RX[0];
    const double y1 = first_order ? X[1] : RX[1];
    const double y2 = first_order ? X[2] : RX[2];
    const double fr2 = f * r2;
    for (int row = 0; row < 2; ++row) {
        const double g0 = g[3 * row], g1 = g[3 * row + 1], g2 = g[3 * row + 2];
        const double b0 = g2 * y1 - g1 * y2, b1 = g0 * y2 - g2 * y0, b2 = g1 * y0 - g0 * y1;
        const double p = row == 0 ? u : v;
        for (int j = 0; j < 3; ++j) {
            Jc[row * 9 + j] = b0 * Jl[j] + b1 * Jl[3 + j] + b2 * Jl[6 + j];
            Jc[row * 9 + 3 + j] = g[3 * row + j];
            Jp[row * 3 + j] = first_order ? g[3 * row + j] : g0 * R[j] + g1 * R[3 + j] + g2 * R[6 + j];
        }
        Jc[row * 9 + 6] = d * p;
        Jc[row * 9 + 7] = fr2 * p;
        Jc[row * 9 + 8] = fr2 * r2 * p;
    }
}

// Residual + analytic Jacobian. Jc: 2x9 row-major (a[3], t[3], f, k1, k2);
// Jp: 2x3 row-major.
GBA_HD void residual_jacobian(const double* cam, const double* X, const double* obs, double* r, double* Jc, double* Jp) {
    const double* a = cam;
    const double t = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    const bool first_order = !(t > 1e-24);
    // the branch's R = I + [a]x for the point, J_l = I, dX_c/dX = I and dRX/da = -[X]x
    double A = 1.0, B = 0.0, C = 0.0, c = 1.0;
    if (!first_order) rotation_terms(t, A, B, C, c);
    const double A0 = A * a[0], A1 = A * a[1], A2 = A * a[2];
    const double B0 = B * a[0], B1 = B * a[1], B2 = B * a[2];
    const double C0 = C * a[0], C1 = C * a[1], C2 = C * a[2];
    const double R[9] = {c + B0 * a[0],  B0 * a[1] - A2, B0 * a[2] + A1,
                    B1 * a[0] + A2, c + B1 * a[1],  B1 * a[2] - A0,
                    B2 * a[0] - A1, B2 * a[1] + A0, c + B2 * a[2]};
    const double Jl[9] = {A + C0 * a[0],  C0 * a[1] - B2, C0 * a[2] + B1,
                     C1 * a[0] + B2, A + C1 * a[1],  C1 * a[2] - B0,
                     C2 * a[0] - B1, C2 * a[1] + B0, A + C2 * a[2]};
    double RX[3];
    for (int i = 0; i < 3; ++i) RX[i] = R[3 * i] * X[0] + R[3 * i + 1] * X[1] + R[3 * i + 2] * X[2];
    jacobian_rows(R, Jl, RX, first_order, cam + 3, X, obs, r, Jc, Jp);
}

// Rotated point R(a) X (without translation) and the pieces the Jacobian needs.
template <typename T>
struct Rotation {
    T RX[3];
    T R[9];    // row-major rotation matrix (dRX/dX)
    T Jl[9];   // row-major left Jacobian J_l(a); identity on the first-order branch
    bool first_order;
};

template <typename T>
GBA_HD void rotate(const T* a, const T* X, Rotation<T>& o) {
    const T th2 = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    if (th2 > T(1e-24)) {
        const T th = msqrt(th2);
        const T inv = T(1) / th;
        const T w0 = a[0] * inv, w1 = a[1] * inv, w2 = a[2] * inv;
        T s, c;
        msincos(th, &s, &c);
        const T sh = msin(T(0.5) * th);
        const T omc = T(2) * sh * sh;  // 1 - cos th
        const T wX = w0 * X[0] + w1 * X[1] + w2 * X[2];
        const T cx0 = w1 * X[2] - w2 * X[1];
        const T cx1 = w2 * X[0] - w0 * X[2];
        const T cx2 = w0 * X[1] - w1 * X[0];
        o.RX[0] = c * X[0] + s * cx0 + omc * wX * w0;
        o.RX[1] = c * X[1] + s * cx1 + omc * wX * w1;
        o.RX[2] = c * X[2] + s * cx2 + omc * wX * w2;
        // R = c I + s [w]x + (1-c) w w^T
        o.R[0] = c + omc * w0 * w0;  o.R[1] = -s * w2 + omc * w0 * w1;  o.R[2] = s * w1 + omc * w0 * w2;
        o.R[3] = s * w2 + omc * w1 * w0;  o.R[4] = c + omc * w1 * w1;  o.R[5] = -s * w0 + omc * w1 * w2;
        o.R[6] = -s * w1 + omc * w2 * w0;  o.R[7] = s * w0 + omc * w2 * w1;  o.R[8] = c + omc * w2 * w2;
        // J_l = (s/th) I + ((1-c)/th) [w]x + (1 - s/th) w w^T
        const T p = s * inv, q = omc * inv, g = T(1) - p;
        o.Jl[0] = p + g * w0 * w0;  o.Jl[1] = -q * w2 + g * w0 * w1;  o.Jl[2] = q * w1 + g * w0 * w2;
        o.Jl[3] = q * w2 + g * w1 * w0;  o.Jl[4] = p + g * w1 * w1;  o.Jl[5] = -q * w0 + g * w1 * w2;
        o.Jl[6] = -q * w1 + g * w2 * w0;  o.Jl[7] = q * w0 + g * w2 * w1;  o.Jl[8] = p + g * w2 * w2;
        o.first_order = false;
    } else {
        o.RX[0] = X[0] + (a[1] * X[2] - a[2] * X[1]);
        o.RX[1] = X[1] + (a[2] * X[0] - a[0] * X[2]);
        o.RX[2] = X[2] + (a[0] * X[1] - a[1] * X[0]);
        for (int i = 0; i < 9; ++i) o.R[i] = (i % 4 == 0) ? T(1) : T(0);
        for (int i = 0; i < 9; ++i) o.Jl[i] = (i % 4 == 0) ? T(1) : T(0);
        o.first_order = true;
    }
}

// The same in FP32, with the rotation's sine and cosine (fast there: FP32 callers are
// bound by memory).
GBA_HD void residual_jacobian(const float* cam, const float* X, const float* obs, float* r, float* Jc, float* Jp) {
    using T = float;
    Rotation<T> rot;
    rotate(cam, X, rot);
    const T P0 = rot.RX[0] + cam[3], P1 = rot.RX[1] + cam[4], P2 = rot.RX[2] + cam[5];
    const T iz = T(1) / P2;
    const T u = -P0 * iz, v = -P1 * iz;
    const T r2 = u * u + v * v;
    const T f = cam[6], k1 = cam[7], k2 = cam[8];
    const T d = T(1) + r2 * (k1 + k2 * r2);
    const T L = k1 + T(2) * k2 * r2;
    r[0] = f * d * u - obs[0];
    r[1] = f * d * v - obs[1];

    // D = f (d I + 2 L [u v]^T [u v]), symmetric 2x2
    const T D00 = f * (d + T(2) * L * u * u);
    const T D01 = f * (T(2) * L * u * v);
    const T D11 = f * (d + T(2) * L * v * v);
    // M = d(u,v)/dX_c = [[-iz, 0, -u iz], [0, -iz, -v iz]]
    const T m02 = -u * iz, m12 = -v * iz;
    // DM = D M (2x3) = derivative of pred w.r.t. X_c
    T DM[6];
    DM[0] = -D00 * iz;  DM[1] = -D01 * iz;  DM[2] = D00 * m02 + D01 * m12;
    DM[3] = -D01 * iz;  DM[4] = -D11 * iz;  DM[5] = D01 * m02 + D11 * m12;

    // B = DM * (-[y]x) (2x3), y = R X (main branch) or X (first-order branch,
    // where dRX/da = -[X]x); [y]x = [[0,-y2,y1],[y2,0,-y0],[-y1,y0,0]].
    const T y0 = rot.first_order ? X[0] : rot.RX[0];
    const T y1 = rot.first_order ? X[1] : rot.RX[1];
    const T y2 = rot.first_order ? X[2] : rot.RX[2];
    T B[6];
    for (int row = 0; row < 2; ++row) {
        const T g0 = DM[row * 3 + 0], g1 = DM[row * 3 + 1], g2 = DM[row * 3 + 2];
        // (-[y]x) = [[0,y2,-y1],[-y2,0,y0],[y1,-y0,0]]
        B[row * 3 + 0] = -g1 * y2 + g2 * y1;
        B[row * 3 + 1] = g0 * y2 - g2 * y0;
        B[row * 3 + 2] = -g0 * y1 + g1 * y0;
    }
    for (int row = 0; row < 2; ++row) {
        // rotation columns: B * J_l
        for (int j = 0; j < 3; ++j)
            Jc[row * 9 + j] = B[row * 3 + 0] * rot.Jl[0 * 3 + j] + B[row * 3 + 1] * rot.Jl[1 * 3 + j] +
                              B[row * 3 + 2] * rot.Jl[2 * 3 + j];
        for (int j = 0; j < 3; ++j) Jc[row * 9 + 3 + j] = DM[row * 3 + j];
        const T p = row == 0 ? u : v;
        Jc[row * 9 + 6] = d * p;
        Jc[row * 9 + 7] = f * r2 * p;
        Jc[row * 9 + 8] = f * r2 * r2 * p;
        for (int j = 0; j < 3; ++j)
            Jp[row * 3 + j] = DM[row * 3 + 0] * rot.R[0 * 3 + j] + DM[row * 3 + 1] * rot.R[1 * 3 + j] +
                              DM[row * 3 + 2] * rot.R[2 * 3 + j];
    }
}

// Residual + Jacobian from per-camera constants precomputed once per camera
// (in FP64, stored in T): pre = [R (9, row-major), J_l (9), t (3), f, k1, k2,
// first_order (0 / 1)]. On the first-order branch R = I + [a]x (so R X is the
// branch's X + a x X), J_l = I, and the branch's dRX/da = -[X]x and dX_c/dX = I
// are applied here; otherwise the same formulas as residual_jacobian.
template <typename T>
GBA_HD void residual_jacobian_pre(const T* pre, const T* X, const T* obs, T* r, T* Jc, T* Jp) {
    const T* R = pre;
    const T* Jl = pre + 9;
    const bool first_order = pre[24] != T(0);
    T RX[3];
    for (int i = 0; i < 3; ++i) RX[i] = R[3 * i] * X[0] + R[3 * i + 1] * X[1] + R[3 * i + 2] * X[2];
    const T P0 = RX[0] + pre[18], P1 = RX[1] + pre[19], P2 = RX[2] + pre[20];
    const T iz = T(1) / P2;
    const T u = -P0 * iz, v = -P1 * iz;
    const T r2 = u * u + v * v;
    const T f = pre[21], k1 = pre[22], k2 = pre[23];
    const T d = T(1) + r2 * (k1 + k2 * r2);
    const T L = k1 + T(2) * k2 * r2;
    r[0] = f * d * u - obs[0];
    r[1] = f * d * v - obs[1];
    const T D00 = f * (d + T(2) * L * u * u);
    const T D01 = f * (T(2) * L * u * v);
    const T D11 = f * (d + T(2) * L * v * v);
    const T m02 = -u * iz, m12 = -v * iz;
    T DM[6];
    DM[0] = -D00 * iz;  DM[1] = -D01 * iz;  DM[2] = D00 * m02 + D01 * m12;
    DM[3] = -D01 * iz;  DM[4] = -D11 * iz;  DM[5] = D01 * m02 + D11 * m12;
    const T y0 = first_order ? X[0] : RX[0];
    const T y1 = first_order ? X[1] : RX[1];
    const T y2 = first_order ? X[2] : RX[2];
    for (int row = 0; row < 2; ++row) {
        const T g0 = DM[row * 3 + 0], g1 = DM[row * 3 + 1], g2 = DM[row * 3 + 2];
        const T b0 = -g1 * y2 + g2 * y1, b1 = g0 * y2 - g2 * y0, b2 = -g0 * y1 + g1 * y0;
        for (int j = 0; j < 3; ++j) Jc[row * 9 + j] = b0 * Jl[j] + b1 * Jl[3 + j] + b2 * Jl[6 + j];
        for (int j = 0; j < 3; ++j) Jc[row * 9 + 3 + j] = DM[row * 3 + j];
        const T p = row == 0 ? u : v;
        Jc[row * 9 + 6] = d * p;
        Jc[row * 9 + 7] = f * r2 * p;
        Jc[row * 9 + 8] = f * r2 * r2 * p;
        for (int j = 0; j < 3; ++j)
            Jp[row * 3 + j] = first_order ? DM[row * 3 + j]
                                          : g0 * R[j] + g1 * R[3 + j] + g2 * R[6 + j];
    }
}

// The same in FP64 with the common factors taken once: the FP64 kernels are bound by these instructions.
GBA_HD void residual_jacobian_pre(const double* pre, const double* X, const double* obs, double* r, double* Jc,
                                  double* Jp) {
    const double* R = pre;
    const double* Jl = pre + 9;
    const bool first_order = pre[24] != 0.0;
    double RX[3];
    for (int i = 0; i < 3; ++i) RX[i] = R[3 * i] * X[0] + R[3 * i + 1] * X[1] + R[3 * i + 2] * X[2];
    jacobian_rows(R, Jl, RX, first_order, pre + 18, X, obs, r, Jc, Jp);
}

// The per-camera constants of residual_jacobian_pre, in FP64 (28 slots; the
// last three are padding).
GBA_HD void camera_constants(const double* a, double* o) {
    const double th2 = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    if (th2 > 1e-24) {
        const double th = sqrt(th2);
        const double inv = 1.0 / th;
        const double w0 = a[0] * inv, w1 = a[1] * inv, w2 = a[2] * inv;
        const double s = sin(th), c = cos(th), sh = sin(0.5 * th);
        const double omc = 2.0 * sh * sh;
        o[0] = c + omc * w0 * w0;  o[1] = -s * w2 + omc * w0 * w1;  o[2] = s * w1 + omc * w0 * w2;
        o[3] = s * w2 + omc * w1 * w0;  o[4] = c + omc * w1 * w1;  o[5] = -s * w0 + omc * w1 * w2;
        o[6] = -s * w1 + omc * w2 * w0;  o[7] = s * w0 + omc * w2 * w1;  o[8] = c + omc * w2 * w2;
        const double p = s * inv, q = omc * inv, g = 1.0 - p;
        o[9] = p + g * w0 * w0;  o[10] = -q * w2 + g * w0 * w1;  o[11] = q * w1 + g * w0 * w2;
        o[12] = q * w2 + g * w1 * w0;  o[13] = p + g * w1 * w1;  o[14] = -q * w0 + g * w1 * w2;
        o[15] = -q * w1 + g * w2 * w0;  o[16] = q * w0 + g * w2 * w1;  o[17] = p + g * w2 * w2;
        o[24] = 0.0;
    } else {
        o[0] = 1.0;   o[1] = -a[2]; o[2] = a[1];
        o[3] = a[2];  o[4] = 1.0;   o[5] = -a[0];
        o[6] = -a[1]; o[7] = a[0];  o[8] = 1.0;
        for (int i = 0; i < 9; ++i) o[9 + i] = (i % 4 == 0) ? 1.0 : 0.0;
        o[24] = 1.0;
    }
    for (int i = 0; i < 6; ++i) o[18 + i] = a[3 + i];
    o[25] = o[26] = o[27] = 0.0;
}

}  // namespace model
}  // namespace gba
