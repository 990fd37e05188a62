// TTM3-F energies and gradients of four geometries per warp.  Same model and constants
// as the reference (ttm3f.cpp:92-321, 325-720; Partridge-Schwenke monomer and
// dipole-moment surface ps.cpp:470-836; smeared interactions
// ttm3f-bits-smear.cpp:17-287).
//
// Lane l works for water l / 4 of geometry l % 4 (nw <= 8; above, two geometries) and keeps what it sums for
// that water in registers: it reads the other waters from shared memory in turn and
// forms its own side of every pair, so nothing is accumulated in shared memory (the
// energy alone needs H/H once per pair and M/H once per direction; a gradient forms
// both sides).  The monomer polynomials are Horner forms over compile-time loops whose
// coefficients are constant-bank operands; the incomplete gamma function costs one
// exponential and a short polynomial (see smear_tail).  The induced dipoles iterate as the reference's
// (ttm3f.cpp:268-307), all four geometries at once, each stopping on its own residual,
// the dipole tensors in registers.
// What bounds it: instruction issue at the 8 to 16 warps per SM the registers allow.
// Per-sample kernel: hexamer FP32 energies 372 us per 2^16 samples (1864 before), trimer
// FP64 gradients 268 us per 2^14 (1113 before), when a warp took one geometry, its
// monomers on nw lanes, and added every pair term to shared memory by FP64 atomics.
//
// The induced field is zero before the first sweep (the reference's fill at
// ttm3f.cpp:108-109 starts at Efq and leaves Efd to whatever the heap held).  Every
// loop is bounded; the dipole iteration at 500 sweeps (ttm3f.cpp:31), after which the
// sweep count reads 501 and the caller counts the sample as not converged (the
// reference only asserts, and not under NDEBUG, ttm3f.cpp:309).
#pragma once
#include <cstring>
#include <vector>

#include "common.cuh"

namespace scp3 {
namespace ttm {

// Monomer polynomials by powers (I, J) of the two stretches: the energy's 25 groups
// I >= J, I + J <= 8 with 15 - I - J powers of the bend each (ps.cpp idx1..3), the
// charges' 28 groups I + J <= 6 with 7 - I - J (idxD0..2), both in ascending I, J.
constexpr int kEI = 9, kES = 8, kEK = 15, kDI = 7, kDK = 7;
constexpr int kETerms = 245, kDTerms = 84;
__host__ __device__ constexpr int e_offset(int I, int J)
{
    int o = 0;
    for (int i = 0; i < kEI; i++)
        for (int j = 0; j <= i && i + j <= kES; j++) {
            if (i == I && j == J) return o;
            o += kEK - i - j;
        }
    return o;
}
__host__ __device__ constexpr int d_offset(int I, int J)
{
    int o = 0;
    for (int i = 0; i < kDI; i++)
        for (int j = 0; i + j < kDI; j++) {
            if (i == I && j == J) return o;
            o += kDK - i - j;
        }
    return o;
}

struct Consts {
    double iAA_HH, iAA_HM, iAA_MM;   // 1 / pow(polfac*polfac, 1/6), ttm3f.cpp:25-27
    double aXX13;                    // pow(0.175, 1/3), ttm3f-bits-smear.cpp:201
    double c5z0, coefD0;             // the constant terms, outside the damped sums
    double phh1;                     // f5z*phh1A*exp(phh2), ps.cpp:514
    double e[kETerms], d[kDTerms];   // by group (e_offset, d_offset), powers of the bend ascending
    double s[36];                    // 1 / (2/3)_(n+1)
    float ef[kETerms], df[kDTerms], sf[36];
};

// Defined here: only sampling.cu includes this header (whole-program compilation).
__constant__ Consts kC;

constexpr double kPolarM = 1.444;
constexpr double kDebye = 4.8033324;
constexpr double kChargeCon = 18.22234397655801030455;
constexpr double kGammaM = 0.46, kGamma1 = 1.0 - kGammaM, kGamma2 = kGammaM / 2;  // ttm3f-bits.h:21-23
constexpr double kVdwC = -0.72298855E+03, kVdwD = 0.10211829E+06, kVdwE = 0.37170376E+01;
constexpr double kAXX = 0.175;
constexpr double kGamma23 = 1.3541179394264004169;  // Gamma(2/3)

// scratch per warp beside crd and ms: the charges, [4][3nw] in T, and the dipoles in FP64,
// [4][6nw]: every water's a second time nw places on, so water i's partners i + r lie in
// a row
template <typename T>
__host__ __device__ inline size_t scratch_bytes(int nw)
{
    return (sizeof(T) + 2 * sizeof(double)) * 12 * (size_t)nw;
}

template <typename T>
__device__ __forceinline__ T ce(int k)
{
    if constexpr (sizeof(T) == 8) return kC.e[k];
    else return kC.ef[k];
}
template <typename T>
__device__ __forceinline__ T cd(int k)
{
    if constexpr (sizeof(T) == 8) return kC.d[k];
    else return kC.df[k];
}

// v of the smeared charge-charge term (1 - v) / r: with x = a (r/A)^3, e1 = exp(-x) and
// x13 = a^(1/3) r/A, the reference's 1 - e1 + x13 Gamma(2/3, x) (ttm3f-bits-smear.cpp:
// 17-80, 213-231).  Gamma(2/3, x) = x^(2/3) e1 h(x), h the continued fraction 1/(x +
// 1/3 - 1 (1/3)/(x + 7/3 - 2 (4/3)/(x + 13/3 - ...))), so v = e1 (1 - x h), x13 x^(2/3)
// being x.  1 - x h is smooth: a polynomial of degree 16 (7 in FP32) on each of ten
// intervals, two per octave of x from 1.5 to 48, interpolated at Chebyshev points from
// the fraction (tail_tables; 1e-17 of it, 1e-8), takes 17 fused steps where the
// fraction's recurrence takes 100 and more near its start.  Past x = 37 (17) v is below
// rounding; below 1.5 Gamma(2/3) minus the series of the lower function, v = e1 (1 + x
// S) - x13 Gamma(2/3), S = sum x^n / (2/3)_(n+1) (there the reference's own split, at 5/3;
// further out the two terms would cancel).
constexpr int kTailSpans = 10, kTailN = 17, kTailNf = 8;
struct TailTable {
    double scale[kTailSpans], shift[kTailSpans], c[kTailN][kTailSpans];       // t = x scale - shift in [-1, 1]
    float scalef[kTailSpans], shiftf[kTailSpans], cf[kTailNf][kTailSpans];
};
__device__ TailTable kTail;

template <typename T>
__host__ __device__ __forceinline__ constexpr T tail_end() { return T(sizeof(T) == 4 ? 17.0 : 37.0); }

// Interval of x, 0 .. kTailSpans - 1, for 1.5 <= x <= tail_end(): two per octave, exponent
// and first bit of the fraction, from 1.5 on.
template <typename T>
__host__ __device__ __forceinline__ int tail_interval(T x)
{
    constexpr bool F = sizeof(T) == 4;
#ifdef __CUDA_ARCH__
    if constexpr (F) return (__float_as_int(x) >> 22) - 255;
    else return (__double2hiint(x) >> 19) - 2047;
#else
    // the same bits by way of memory
    if constexpr (F) {
        int32_t b;
        std::memcpy(&b, &x, sizeof(b));
        return (b >> 22) - 255;
    } else {
        int64_t b;
        std::memcpy(&b, &x, sizeof(b));
        return (int)(b >> 51) - 2047;
    }
#endif
}

// Which form smear_tail takes: the interval, -1 the series below 1.5, -2 none.  Only -2 can
// be a NaN (coincident sites, coordinates that are not finite).
template <typename T>
__host__ __device__ __forceinline__ int tail_span(T x)
{
    if (!(x <= tail_end<T>())) return -2;
    return x < T(1.5) ? -1 : tail_interval(x);
}

template <typename T>
__device__ __forceinline__ T smear_tail(T x, T e1, T x13)
{
    constexpr bool F = sizeof(T) == 4;
    const int i = tail_span(x);
    if (i == -2) return x > T(1.5) ? T(0) : x;     // past the table; a NaN stays one
    if (i == -1) {
        T s = T(0);
#pragma unroll
        for (int n = F ? 14 : 22; n >= 0; n--) {
            if constexpr (F) s = s * x + kC.sf[n];
            else s = s * x + kC.s[n];
        }
        return e1 * (T(1) + x * s) - x13 * T(kGamma23);
    }
    T s;
    if constexpr (F) {
        const T t = x * __ldg(kTail.scalef + i) - __ldg(kTail.shiftf + i);
        s = __ldg(&kTail.cf[kTailNf - 1][i]);
#pragma unroll
        for (int k = kTailNf - 2; k >= 0; k--) s = s * t + __ldg(&kTail.cf[k][i]);
    } else {
        const T t = x * __ldg(kTail.scale + i) - __ldg(kTail.shift + i);
        s = __ldg(&kTail.c[kTailN - 1][i]);
#pragma unroll
        for (int k = kTailN - 2; k >= 0; k--) s = s * t + __ldg(&kTail.c[k][i]);
    }
    return e1 * s;
}

// The table, in extended precision: Chebyshev interpolation of 1 - x h(x), as powers of t.
inline void tail_tables(TailTable& o)
{
    auto w = [](long double x) {
        const long double a = 2.0L / 3.0L;
        long double b = x + 1.0L - a, A0 = 0.0L, A1 = 1.0L, B0 = 1.0L, B1 = b;
        for (int k = 1; k <= 200; k++) {
            const long double an = -k * (k - a);
            b += 2.0L;
            const long double A2 = b * A1 + an * A0, B2 = b * B1 + an * B0;
            A0 = A1 / B2, A1 = A2 / B2, B0 = B1 / B2, B1 = 1.0L;
        }
        return 1.0L - x * A1 / B1;
    };
    const long double pi = 3.14159265358979323846264338327950288L;
    for (int i = 0; i < kTailSpans; i++) {
        const long double lo = ldexpl((i & 1) ? 1.0L : 1.5L, (i + 1) / 2), hi = lo + ldexpl(0.5L, (i + 1) / 2);
        o.scale[i] = (double)(2.0L / (hi - lo)), o.shift[i] = (double)((hi + lo) / (hi - lo));
        o.scalef[i] = (float)o.scale[i], o.shiftf[i] = (float)o.shift[i];
        for (int n : {kTailN, kTailNf}) {
            std::vector<long double> f(n), c(n, 0.0L), p(n, 0.0L), t0(n, 0.0L), t1(n, 0.0L);
            for (int k = 0; k < n; k++) f[k] = w(0.5L * (lo + hi) + 0.5L * (hi - lo) * cosl(pi * (k + 0.5L) / n));
            for (int j = 0; j < n; j++) {
                for (int k = 0; k < n; k++) c[j] += f[k] * cosl(pi * j * (k + 0.5L) / n);
                c[j] *= (j ? 2.0L : 1.0L) / n;
            }
            t0[0] = 1.0L, t1[1] = 1.0L;                    // T_0, T_1 as powers of t
            for (int k = 0; k < n; k++) p[k] = c[0] * t0[k] + c[1] * t1[k];
            for (int j = 2; j < n; j++) {
                std::vector<long double> t2(n, 0.0L);
                for (int k = 0; k < n; k++) t2[k] = (k ? 2.0L * t1[k - 1] : 0.0L) - t0[k];
                for (int k = 0; k < n; k++) p[k] += c[j] * t2[k];
                t0 = t1, t1 = t2;
            }
            for (int k = 0; k < n; k++)
                if (n == kTailN) o.c[k][i] = (double)p[k];
                else o.cf[k][i] = (float)p[k];
        }
    }
}

// Smeared interactions of two sites R apart (ttm3f-bits-smear.cpp:97-287); the members
// a caller does not read are not formed.
template <typename T>
struct Smear {
    T ri, x, e1, x13;
    __device__ __forceinline__ Smear(T r2, T iAA)
    {
        ri = inv_sqrt(r2);
        x13 = T(kC.aXX13) * (r2 * ri * iAA);
        x = x13 * x13 * x13;
        e1 = exp(-x);
    }
    __device__ __forceinline__ T ts0() const { return (T(1) - smear_tail(x, e1, x13)) * ri; }
    __device__ __forceinline__ T ts1() const { return (T(1) - e1) * ri * (ri * ri); }
    __device__ __forceinline__ T ts2(T ts1, T iAA) const { return (ts1 - e1 * (T(kAXX) * iAA * iAA * iAA)) * (ri * ri); }
    __device__ __forceinline__ T ts3(T ts2, T iAA) const
    {
        const T c = T(kAXX) * iAA * iAA * iAA;
        return (ts2 - T(0.6) * e1 * (c * c) / ri) * (ri * ri);
    }
};

// A water's own terms: energy (kcal/mol) and the charges of H1 and H2 (elementary
// charges); with G the energy's gradient on H1 and H2 and the charges' derivatives.
template <typename T, bool G>
struct Monomer {
    T e, q1, q2;
    T h1[3], h2[3];                               // kcal/mol/A on H1, H2 (O: minus their sum)
    T f11, f12, f21, f22, g11, g12, g21, g22;     // d q1 / d H1 = f11 roh1 + f12 roh2, d q1 / d H2 = f21 roh1 + f22 roh2; g: q2
};

// pot_nasa and dms_nasa with ttm3 = true (ps.cpp:470-836) for the water at w[9].
template <typename T, bool G>
__device__ __forceinline__ void monomer(const T* w, Monomer<T, G>& o)
{
    constexpr double reoh = 0.958649, b1 = 2.0, roh = 0.9519607159623009, alphaoh = 2.587949757553683;
    constexpr double deohA = 42290.92019288289, phh2 = 12.66426998162947, f5z = 0.999677885;
    constexpr double costhe = -.24780227221366464506, tocal = 0.00285914375100642899, xx = 0.529177249;
    constexpr double ath0 = 1.82400520401572996557, dms1 = 0.5, dms2 = 0.9578, dms3 = 0.012;
    T roh1[3], roh2[3], rhh[3], d1 = 0, d2 = 0, dhh = 0, dot = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        roh1[i] = w[3 + i] - w[i];
        roh2[i] = w[6 + i] - w[i];
        rhh[i] = w[3 + i] - w[6 + i];
        d1 += roh1[i] * roh1[i];
        d2 += roh2[i] * roh2[i];
        dhh += rhh[i] * rhh[i];
        dot += roh1[i] * roh2[i];
    }
    d1 = sqrt(d1);
    d2 = sqrt(d2);
    dhh = sqrt(dhh);
    const T costh = dot / (d1 * d2);
    const T dr1 = d1 - T(reoh), dr2 = d2 - T(reoh), x3 = costh - T(costhe);
    T p[kEI], q[kEI];                              // powers of the two stretches
    p[0] = q[0] = T(1);
    p[1] = dr1 / T(reoh), q[1] = dr2 / T(reoh);
#pragma unroll
    for (int k = 2; k < kEI; k++) p[k] = p[k - 1] * p[1], q[k] = q[k - 1] * q[1];
    const T g2 = dr1 * dr1 + dr2 * dr2;
    // --- pot_nasa (ps.cpp:486-603)
    {
        const T deoh = T(f5z * deohA);
        const T e1x = exp(-T(alphaoh) * (d1 - T(roh))), e2x = exp(-T(alphaoh) * (d2 - T(roh)));
        const T va = deoh * (e1x * (e1x - T(2)) + e2x * (e2x - T(2)));
        const T vb = T(kC.phh1) * exp(-T(phh2) * dhh);
        const T efac = exp(-T(b1) * g2);
        T s0 = 0, s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
        for (int I = 0; I < kEI; I++)
#pragma unroll
            for (int J = 0; J < kEI; J++) {
                if (J > I || I + J > kES) continue;
                const int off = e_offset(I, J), n = kEK - I - J;
                T a = ce<T>(off + n - 1), da = T(0);
#pragma unroll
                for (int k = kEK - 2; k >= 0; k--) {
                    if (k > n - 2) continue;
                    if (G) da = da * x3 + a;
                    a = a * x3 + ce<T>(off + k);
                }
                const T sym = I == J ? T(2) * p[I] * q[I] : p[I] * q[J] + p[J] * q[I];
                s0 += a * sym;
                if (G) {
                    T t1 = T(0), t2 = T(0);
                    if (I) t1 += T(I) * p[I - 1] * q[J], t2 += T(I) * p[J] * q[I - 1];
                    if (J) t1 += T(J) * p[J - 1] * q[I], t2 += T(J) * p[I] * q[J - 1];
                    s1 += a * t1, s2 += a * t2, s3 += da * sym;
                }
            }
        o.e = (va + vb + (T(2) * T(kC.c5z0) + efac * s0) + T(0.44739574026257)) * T(tocal);
        if (G) {
            const T dva1 = T(2.0 * alphaoh) * deoh * e1x * (T(1) - e1x) / d1;
            const T dva2 = T(2.0 * alphaoh) * deoh * e2x * (T(1) - e2x) / d2;
            const T dvb = -T(phh2) * vb / dhh;
            const T dvc1 = (-T(2 * b1) * efac * dr1 * s0 + efac * s1 / T(reoh)) / d1;
            const T dvc2 = (-T(2 * b1) * efac * dr2 * s0 + efac * s2 / T(reoh)) / d2;
            const T dvcc = efac * s3;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                o.h1[i] = T(tocal) * (dva1 * roh1[i] + dvb * rhh[i] + dvc1 * roh1[i] +
                                      dvcc * (roh2[i] / (d1 * d2) - costh * roh1[i] / (d1 * d1)));
                o.h2[i] = T(tocal) * (dva2 * roh2[i] - dvb * rhh[i] + dvc2 * roh2[i] +
                                      dvcc * (roh1[i] / (d1 * d2) - costh * roh2[i] / (d2 * d2)));
            }
        }
    }
    // --- dms_nasa (ps.cpp:605-836)
    const T efacD = exp(-g2);   // b1D = 1
    T p1 = 0, p2 = 0, dp1r1 = 0, dp1r2 = 0, dp1c = 0, dp2r1 = 0, dp2r2 = 0, dp2c = 0;
#pragma unroll
    for (int I = 0; I < kDI; I++)
#pragma unroll
        for (int J = 0; J < kDI; J++) {
            if (I + J >= kDI) continue;
            const int off = d_offset(I, J), n = kDK - I - J;
            T a = cd<T>(off + n - 1), da = T(0);
#pragma unroll
            for (int k = kDK - 2; k >= 0; k--) {
                if (k > n - 2) continue;
                if (G) da = da * x3 + a;
                a = a * x3 + cd<T>(off + k);
            }
            p1 += a * (p[I] * q[J]);
            p2 += a * (p[J] * q[I]);
            if (G) {
                if (I) dp1r1 += a * (T(I) * p[I - 1] * q[J]), dp2r2 += a * (T(I) * p[J] * q[I - 1]);
                if (J) dp1r2 += a * (T(J) * p[I] * q[J - 1]), dp2r1 += a * (T(J) * p[J - 1] * q[I]);
                dp1c += da * (p[I] * q[J]);
                dp2c += da * (p[J] * q[I]);
            }
        }
    constexpr double pa = 0.2999, pb = -0.6932, pc0c = 1.0099, pc1 = -0.1801, pc2 = 0.0892;
    const T pl2 = T(0.5) * (T(3) * costh * costh - T(1));
    const T ang_f = T(pc0c) + costh * T(pc1) + pl2 * T(pc2);
    const T w1 = exp(T(pb) * log(d1)), w2 = exp(T(pb) * log(d2));
    const T pc0 = T(pa) * (w1 + w2) * ang_f;
    const T axb[3] = {roh1[1] * roh2[2] - roh1[2] * roh2[1], -roh1[0] * roh2[2] + roh1[2] * roh2[0],
                      roh1[0] * roh2[1] - roh1[1] * roh2[0]};
    const T sinth = sqrt(axb[0] * axb[0] + axb[1] * axb[1] + axb[2] * axb[2]) / (d1 * d2);
    const T ang = T(dms3) * (atan2(sinth, costh) - T(ath0));
    o.q1 = T(kC.coefD0) + p1 * efacD + pc0 * T(xx) + T(dms1) * (d1 - T(dms2)) + ang;
    o.q2 = T(kC.coefD0) + p2 * efacD + pc0 * T(xx) + T(dms1) * (d2 - T(dms2)) + ang;
    if (G) {
        // derivatives by d1, d2 and cos; those of p by a stretch carry 1 / reoh
        const T dw1 = T(pa * pb * xx) * w1 / d1 * ang_f, dw2 = T(pa * pb * xx) * w2 / d2 * ang_f;
        const T dwc = T(pa * xx) * (w1 + w2) * (T(pc1) + T(3.0 * pc2) * costh);
        const T ef1 = -T(2) * dr1 * efacD, ef2 = -T(2) * dr2 * efacD;
        const T a11 = dp1r1 * efacD / T(reoh) + p1 * ef1 + dw1 + T(dms1);
        const T a12 = dp1r2 * efacD / T(reoh) + p1 * ef2 + dw2;
        const T a1c = dp1c * efacD + dwc - T(dms3) / sinth;
        const T a21 = dp2r1 * efacD / T(reoh) + p2 * ef1 + dw1;
        const T a22 = dp2r2 * efacD / T(reoh) + p2 * ef2 + dw2 + T(dms1);
        const T a2c = dp2c * efacD + dwc - T(dms3) / sinth;
        const T i12 = T(1) / (d1 * d2);
        o.f11 = (a11 - a1c * costh / d1) / d1, o.f12 = a1c * i12;
        o.f22 = (a12 - a1c * costh / d2) / d2, o.f21 = a1c * i12;
        o.g11 = (a21 - a2c * costh / d1) / d1, o.g12 = a2c * i12;
        o.g22 = (a22 - a2c * costh / d2) / d2, o.g21 = a2c * i12;
    }
}

template <typename T>
__device__ __forceinline__ void load3(const T* a, T* r)
{
    r[0] = a[0], r[1] = a[1], r[2] = a[2];
}
template <typename T>
__device__ __forceinline__ T dot3(const T* a, const T* b)
{
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
template <int NG>
__device__ __forceinline__ double sum_geometry(double x)      // over the lanes of a geometry
{
#pragma unroll
    for (int o = NG; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Energies (kcal/mol) of ng <= 4 geometries crd + j * stride (shared memory, T), and with
// G their gradients g + j * 9 nw (shared, kcal/mol/A, complete after the call); ms
// [4][3nw] and sc (scratch_bytes) shared scratch.  Lane l returns the energy of geometry
// l % 4, *iters its Jacobi sweeps (kTtmMaxIter + 1 if capped).  NG = 2: two geometries
// of up to 16 waters instead, lane l on water l / 2 of geometry l % 2.  kMaxNw: most
// waters the instance's registers hold dipole tensors for.
template <typename T, bool G, int NG = 4, int kMaxNw = 32 / NG>
__device__ double energy_warp4(const T* crd, int stride, T* ms, char* sc, double* g, int nw, int ng, int lane, int* iters)
{
    const int j = lane % NG, i = lane / NG, n3 = 3 * nw;
    const bool on = j < ng && i < nw;
    const T* cj = crd + j * stride;
    T* mj = ms + j * n3;
    double* dip = reinterpret_cast<double*>(sc) + j * 2 * n3;
    T* chg = reinterpret_cast<T*>(sc + sizeof(double) * 8 * n3) + j * n3;
    T xO[3], xH[2][3], xM[3], qM = 0, qH[2] = {0, 0};
    double part = 0;
    Monomer<T, G> mo;
    if (on) {
        const T* w = cj + 9 * i;
        load3(w, xO), load3(w + 3, xH[0]), load3(w + 6, xH[1]);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xM[k] = T(kGamma1) * xO[k] + T(kGamma2) * (xH[0][k] + xH[1][k]);
            mj[3 * i + k] = xM[k];
        }
        T w9[9];
#pragma unroll
        for (int k = 0; k < 9; k++) w9[k] = w[k];
        monomer<T, G>(w9, mo);
        part = (double)mo.e;
        const T t = T(kGamma2 / kGamma1), s = mo.q1 + mo.q2;
        qM = -T(kChargeCon) * s / T(kGamma1);
        qH[0] = T(kChargeCon) * (mo.q1 + t * s);
        qH[1] = T(kChargeCon) * (mo.q2 + t * s);
        chg[3 * i] = qM, chg[3 * i + 1] = qH[0], chg[3 * i + 2] = qH[1];
    }
    __syncwarp();
    const T iHH = T(kC.iAA_HH), iHM = T(kC.iAA_HM), iMM = T(kC.iAA_MM);
    T phi[3] = {0, 0, 0}, gO[3] = {0, 0, 0}, gH[2][3] = {{0, 0, 0}, {0, 0, 0}};   // potentials at M, H1, H2
    double efq[3] = {0, 0, 0}, el = 0.0, vdw = 0.0;
    // pair terms, the water's own side (ttm3f.cpp:144-257, 403-520)
    if (on)
#pragma unroll 1
        for (int r = 1; r < nw; r++) {
            const int b = i + r < nw ? i + r : i + r - nw;
            const T* w = cj + 9 * b;
            T yO[3], yH[2][3], yM[3], R[3];
            load3(w, yO), load3(w + 3, yH[0]), load3(w + 6, yH[1]), load3(mj + 3 * b, yM);
            const T pM = chg[3 * b], pH[2] = {chg[3 * b + 1], chg[3 * b + 2]};
#pragma unroll
            for (int l = 0; l < 2; l++) {       // own M, other H
#pragma unroll
                for (int k = 0; k < 3; k++) R[k] = xM[k] - yH[l][k];
                const Smear<T> s(dot3(R, R), iHM);
                const T t0 = s.ts0(), t1 = pH[l] * s.ts1();
                if (G) phi[0] += t0 * pH[l];
                else el += (double)(t0 * pH[l] * qM);
#pragma unroll
                for (int k = 0; k < 3; k++) efq[k] += (double)(t1 * R[k]);
            }
            if (G) {
#pragma unroll
                for (int l = 0; l < 2; l++) {   // own H, other M
#pragma unroll
                    for (int k = 0; k < 3; k++) R[k] = yM[k] - xH[l][k];
                    const Smear<T> s(dot3(R, R), iHM);
                    phi[1 + l] += s.ts0() * pM;
                    const T f = pM * qH[l] * s.ts1();
#pragma unroll
                    for (int k = 0; k < 3; k++) gH[l][k] += f * R[k];
                }
            }
            // H/H: both sides of a gradient; the energy takes the waters i and i + r, r up
            // to nw / 2 (that one from both ends, at half weight)
            if (G || 2 * r <= nw) {
                const T half = 2 * r == nw ? T(0.5) : T(1);
#pragma unroll
                for (int l = 0; l < 2; l++)
#pragma unroll
                    for (int m = 0; m < 2; m++) {
#pragma unroll
                        for (int k = 0; k < 3; k++) R[k] = xH[l][k] - yH[m][k];
                        const Smear<T> s(dot3(R, R), iHH);
                        const T t0 = s.ts0();
                        if (G) {
                            phi[1 + l] += t0 * pH[m];
                            const T f = -pH[m] * qH[l] * s.ts1();
#pragma unroll
                            for (int k = 0; k < 3; k++) gH[l][k] += f * R[k];
                        } else {
                            el += (double)(half * t0 * pH[m] * qH[l]);
                        }
                    }
            }
            {                                   // O/O van der Waals, half of it this water's
#pragma unroll
                for (int k = 0; k < 3; k++) R[k] = xO[k] - yO[k];
                const T r2 = dot3(R, R), rr = sqrt(r2), c6 = T(kVdwC) / (r2 * r2 * r2), ex = T(kVdwD) * exp(-T(kVdwE) * rr);
                vdw += (double)(c6 + ex);
                if (G) {
                    const T f = -(T(6) * c6) / r2 - T(kVdwE) * ex / rr;
#pragma unroll
                    for (int k = 0; k < 3; k++) gO[k] += f * R[k];
                }
            }
            {                                   // M/M
#pragma unroll
                for (int k = 0; k < 3; k++) R[k] = xM[k] - yM[k];
                const Smear<T> s(dot3(R, R), iMM);
                const T t0 = s.ts0(), t1 = pM * s.ts1();
                if (G) phi[0] += t0 * pM;
                else el += 0.5 * (double)(t0 * pM * qM);
#pragma unroll
                for (int k = 0; k < 3; k++) efq[k] += (double)(t1 * R[k]);
            }
        }
    // induced dipoles (ttm3f.cpp:239-307); the iterate is carried in FP64 so the FP32
    // form can still reach its residual target
    double tens[kMaxNw - 1][6];                 // 3 ts2 R R^T - ts1 towards water i + r
#pragma unroll
    for (int r = 1; r < kMaxNw; r++)
        if (on && r < nw) {
            const int b = i + r < nw ? i + r : i + r - nw;
            T R[3];
#pragma unroll
            for (int k = 0; k < 3; k++) R[k] = xM[k] - mj[3 * b + k];
            const Smear<T> s(dot3(R, R), iMM);
            const T t1 = s.ts1(), t2 = T(3) * s.ts2(t1, iMM);
            tens[r - 1][0] = (double)(t2 * R[0] * R[0] - t1);
            tens[r - 1][1] = (double)(t2 * R[0] * R[1]);
            tens[r - 1][2] = (double)(t2 * R[0] * R[2]);
            tens[r - 1][3] = (double)(t2 * R[1] * R[1] - t1);
            tens[r - 1][4] = (double)(t2 * R[1] * R[2]);
            tens[r - 1][5] = (double)(t2 * R[2] * R[2] - t1);
        }
    const double tol = sizeof(T) == 8 ? 1.0e-15 : 1.0e-8;
    const double stath = kDebye / kChargeCon / sqrt((double)nw);
    double cur[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        cur[k] = kPolarM * efq[k];
        if (on) dip[3 * i + k] = dip[n3 + 3 * i + k] = cur[k];
    }
    bool busy = j < ng;
    int it = 0;
    for (int sweep = 0; sweep < kTtmMaxIter; sweep++) {
        __syncwarp();
        double ef[3] = {0, 0, 0}, del2 = 0.0;
        if (on && busy) {
#pragma unroll
            for (int r = 1; r < kMaxNw; r++)
                if (r < nw) {
                    const double* d = dip + 3 * (i + r);
                    const double* t = tens[r - 1];
                    const double dx = d[0], dy = d[1], dz = d[2];
                    ef[0] += t[0] * dx + t[1] * dy + t[2] * dz;
                    ef[1] += t[1] * dx + t[3] * dy + t[4] * dz;
                    ef[2] += t[2] * dx + t[4] * dy + t[5] * dz;
                }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double prev = cur[k];
                double d = kPolarM * (efq[k] + ef[k]);
                d = 0.7 * d + (1.0 - 0.7) * prev;
                cur[k] = d;
                del2 += (d - prev) * (d - prev);
            }
        }
        del2 = sum_geometry<NG>(del2);
        __syncwarp();
        if (busy) {
            if (on)
#pragma unroll
                for (int k = 0; k < 3; k++) dip[3 * i + k] = dip[n3 + 3 * i + k] = cur[k];
            it++;
            if (sqrt(del2) * stath < tol) busy = false;
        }
        if (!__any_sync(0xffffffffu, busy)) break;
    }
    *iters = busy ? kTtmMaxIter + 1 : it;
    __syncwarp();
    if (G) el = 0.5 * ((double)phi[0] * (double)qM + (double)phi[1] * (double)qH[0] + (double)phi[2] * (double)qH[1]);
    const double ind = -(cur[0] * efq[0] + cur[1] * efq[1] + cur[2] * efq[2]);
    const double tot = sum_geometry<NG>(on ? part + el + 0.5 * vdw + 0.5 * ind : 0.0);
    if constexpr (G) {
        // charge-dipole and dipole-dipole forces (ttm3f.cpp:594-676), the water's own side
        if (on) {
            T d[3], dM[3] = {0, 0, 0};
#pragma unroll
            for (int k = 0; k < 3; k++) d[k] = (T)cur[k];
#pragma unroll 1
            for (int r = 1; r < nw; r++) {
                const int b = i + r < nw ? i + r : i + r - nw;
                const T* w = cj + 9 * b;
                T yM[3], R[3], db[3];
                load3(mj + 3 * b, yM);
#pragma unroll
                for (int k = 0; k < 3; k++) db[k] = (T)dip[3 * b + k];
                const T pM = chg[3 * b];
#pragma unroll
                for (int l = 0; l < 2; l++) {   // own dipole, other H
#pragma unroll
                    for (int k = 0; k < 3; k++) R[k] = xM[k] - w[3 + 3 * l + k];
                    const Smear<T> s(dot3(R, R), iHM);
                    const T t1 = s.ts1(), t2 = s.ts2(t1, iHM), p = chg[3 * b + 1 + l], c = T(3) * t2 * dot3(d, R);
#pragma unroll
                    for (int k = 0; k < 3; k++) dM[k] += p * (c * R[k] - t1 * d[k]);
                }
#pragma unroll
                for (int l = 0; l < 2; l++) {   // own H, other dipole
#pragma unroll
                    for (int k = 0; k < 3; k++) R[k] = yM[k] - xH[l][k];
                    const Smear<T> s(dot3(R, R), iHM);
                    const T t1 = s.ts1(), t2 = s.ts2(t1, iHM), dR = dot3(db, R), c = T(3) * t2 * dR;
#pragma unroll
                    for (int k = 0; k < 3; k++) gH[l][k] -= qH[l] * (c * R[k] - t1 * db[k]);
                    phi[1 + l] -= t1 * dR;
                }
#pragma unroll
                for (int k = 0; k < 3; k++) R[k] = xM[k] - yM[k];
                const Smear<T> s(dot3(R, R), iMM);
                const T t1 = s.ts1(), t2 = s.ts2(t1, iMM), t3 = s.ts3(t2, iMM);
                const T diR = dot3(d, R), djR = dot3(db, R), dd = dot3(d, db);
#pragma unroll
                for (int k = 0; k < 3; k++)
                    dM[k] += pM * (T(3) * t2 * diR * R[k] - t1 * d[k]) - qM * (T(3) * t2 * djR * R[k] - t1 * db[k]) -
                             T(3) * t2 * (dd * R[k] + djR * d[k] + diR * db[k]) + T(15) * t3 * diR * djR * R[k];
                phi[0] += t1 * djR;
            }
            // the M site's force onto O, H, H, and the charges' geometry dependence
            // (ttm3f.cpp:680-716, GRDQ of 371-393)
            const T t = T(kGamma2 / kGamma1), P0 = (T(1) + T(2) * t) * phi[0];
            const T A1 = T(kChargeCon) * ((T(1) + t) * phi[1] + t * phi[2] - P0);
            const T A2 = T(kChargeCon) * ((T(1) + t) * phi[2] + t * phi[1] - P0);
            const T u1 = A1 * mo.f11 + A2 * mo.g11, u2 = A1 * mo.f12 + A2 * mo.g12;
            const T v1 = A1 * mo.f21 + A2 * mo.g21, v2 = A1 * mo.f22 + A2 * mo.g22;
            double* gw = g + j * 9 * nw + 9 * i;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const T r1 = xH[0][k] - xO[k], r2 = xH[1][k] - xO[k];
                const T c1 = u1 * r1 + u2 * r2 + mo.h1[k], c2 = v1 * r1 + v2 * r2 + mo.h2[k];
                const T f = dM[k] - qM * (T)efq[k];
                gw[k] = gO[k] + T(kGamma1) * f - (c1 + c2);
                gw[3 + k] = gH[0][k] + T(kGamma2) * f + c1;
                gw[6 + k] = gH[1][k] + T(kGamma2) * f + c2;
            }
        }
        __syncwarp();
    }
    return tot;
}

}  // namespace ttm
}  // namespace scp3
