// qTIP4P/f energies and gradients of four geometries per warp, the geometries and M
// sites staged in the warp's shared memory.  Same terms and constants as the reference
// (qtip4pf.cpp:57-145 monomer, 190-286 pair terms); kcal/mol, Angstrom.
#pragma once
#include "common.cuh"

namespace scp3 {
namespace qt {

constexpr double kChargeCon = 18.22234397655801030455;  // qtip4pf.cpp:61
constexpr double kQM = -1.1128 * kChargeCon;
constexpr double kQH = -kQM / 2;
constexpr double kROHeq = 0.9419;
constexpr double kAHOHeqRad = 107.4 * 3.14159265358979323846 / 180.0;  // aHOHeq*M_PI/180.0
constexpr double kEpsilon = 0.1852;
constexpr double kSigma = 3.1589;
constexpr double kAlphaR = 2.287;
constexpr double kDR = 116.09;
constexpr double kKTheta = 87.85;
constexpr double kGammaM = 0.73612;
constexpr double kGamma1 = (1.0 - kGammaM) / 2;

template <typename T>
__device__ __forceinline__ T monomer(const T* w)
{
    T d1[3], d2[3], r1 = 0, r2 = 0, c = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        d1[k] = w[3 + k] - w[k];
        d2[k] = w[6 + k] - w[k];
        r1 += d1[k] * d1[k];
        r2 += d2[k] * d2[k];
        c += d1[k] * d2[k];
    }
    r1 = sqrt(r1);
    r2 = sqrt(r2);
    const T x1 = T(kAlphaR) * (r1 - T(kROHeq)), x2 = T(kAlphaR) * (r2 - T(kROHeq));
    const T v1 = x1 * x1 * (T(1) - x1 * (T(1) - T(7.0 / 12.0) * x1)) * T(kDR);
    const T v2 = x2 * x2 * (T(1) - x2 * (T(1) - T(7.0 / 12.0) * x2)) * T(kDR);
    const T th = acos(c * (T(1) / r1 / r2));
    const T dth = th - T(kAHOHeqRad);
    return v1 + v2 + T(0.5) * T(kKTheta) * dth * dth;
}

// Water pair p of the row-major upper triangle of nw waters: a < b.
__host__ __device__ __forceinline__ void water_pair_of(int p, int nw, int& a, int& b)
{
    a = 0;
    while (p >= nw - 1 - a) {
        p -= nw - 1 - a;
        a++;
    }
    b = a + 1 + p;
}

// The ten site pairs of waters a < b that the reference's pair loops visit
// (qtip4pf.cpp:213-283): the M site of each water against the two H of the
// other, the four H/H pairs, O/O (Lennard-Jones) and M/M.  The eight sites are
// read once; each term is formed in T and summed in FP64.
template <typename T>
__device__ __forceinline__ double water_pair(int a, int b, const T* crd, const T* ms)
{
    T s[2][4][3];   // [water][O, H1, H2, M][x, y, z]
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int l = 0; l < 3; l++) s[0][l][k] = crd[9 * a + 3 * l + k], s[1][l][k] = crd[9 * b + 3 * l + k];
        s[0][3][k] = ms[3 * a + k];
        s[1][3][k] = ms[3 * b + k];
    }
    // a site of one water with the other's three charges, which add up to zero: the sums
    // stay small
    double e = 0.0;
#pragma unroll
    for (int l = 1; l < 4; l++) {
        const double ql = l == 3 ? kQM : kQH;
        double t = (double)(T(ql * kQM) * inv_sqrt(dist2(s[0][l], s[1][3])));
#pragma unroll
        for (int m = 1; m < 3; m++) t += (double)(T(ql * kQH) * inv_sqrt(dist2(s[0][l], s[1][m])));
        e += t;
    }
    const T s2 = T(kSigma * kSigma) / dist2(s[0][0], s[1][0]);
    const T s6 = s2 * s2 * s2;
    e += (double)(T(4 * kEpsilon) * s6 * (s6 - T(1)));
    return e;
}

// Energies of ng <= 4 geometries crd + j * stride (shared memory, T) at once,
// ms a [4][3nw] shared scratch: lane l works for geometry l % 4 only (M sites and
// monomers as items (water, geometry), pair terms as items (water pair,
// geometry)), so a warp keeps its lanes busy on the per-water and per-pair
// terms; lane l returns the sum of geometry l % 4.
template <typename T>
__device__ double energy_warp4(const T* crd, int stride, T* ms, int nw, int ng, int lane)
{
    const int j = lane & 3;
    const bool on = j < ng;
    const T* cj = crd + j * stride;
    T* mj = ms + j * 3 * nw;
    if (on)
        for (int i = lane >> 2; i < nw; i += 8) {
            const T* w = cj + 9 * i;
#pragma unroll
            for (int k = 0; k < 3; k++) mj[3 * i + k] = T(kGammaM) * w[k] + T(kGamma1) * (w[3 + k] + w[6 + k]);
        }
    __syncwarp();
    double part = 0;    // terms in T, their sums in FP64
    if (on) {
        for (int i = lane >> 2; i < nw; i += 8) part += (double)monomer(cj + 9 * i);
        const int np = nw * (nw - 1) / 2;
        for (int p = lane >> 2; p < np; p += 8) {
            int a, b;
            water_pair_of(p, nw, a, b);
            part += water_pair<T>(a, b, cj, mj);
        }
    }
    part += __shfl_xor_sync(0xffffffffu, part, 4);
    part += __shfl_xor_sync(0xffffffffu, part, 8);
    part += __shfl_xor_sync(0xffffffffu, part, 16);
    return part;
}

// ---------------------------------------------------------------- energy + gradient
// qtip4pf.cpp:252-397 (the E+g operator of the gradient path): the same terms,
// their derivatives in kcal/mol/A.  The M site is gammaM O + gamma1 (H1 + H2), so
// the force on it is spread over the three atoms with those weights.  In the
// precision T (FP64 for the parity form; FP32 for the split form's products),
// each term's energy returned in FP64 and summed in FP64.

template <typename T>
__device__ __forceinline__ T monomer_grad(const T* w, T* gh1, T* gh2)
{
    T d1[3], d2[3], r1 = 0, r2 = 0, c = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        d1[k] = w[3 + k] - w[k];
        d2[k] = w[6 + k] - w[k];
        r1 += d1[k] * d1[k];
        r2 += d2[k] * d2[k];
        c += d1[k] * d2[k];
    }
    r1 = sqrt(r1);
    r2 = sqrt(r2);
    const T x1 = T(kAlphaR) * (r1 - T(kROHeq)), x2 = T(kAlphaR) * (r2 - T(kROHeq));
    const T v1 = x1 * x1 * (T(1.0) - x1 * (T(1.0) - T(7.0 / 12.0) * x1)) * T(kDR);
    const T v2 = x2 * x2 * (T(1.0) - x2 * (T(1.0) - T(7.0 / 12.0) * x2)) * T(kDR);
    const T dv1 = T(kDR) * T(kAlphaR) * x1 * (T(2.0) - x1 * (T(3.0) - T(7.0 / 3.0) * x1));   // dv/dr
    const T dv2 = T(kDR) * T(kAlphaR) * x2 * (T(2.0) - x2 * (T(3.0) - T(7.0 / 3.0) * x2));
    const T cs = c / (r1 * r2);
    const T dth = acos(cs) - T(kAHOHeqRad);
    const T de_dc = -T(kKTheta) * dth / sqrt(T(1.0) - cs * cs);                           // dE/dcos(theta)
    const T i1 = T(1.0) / r1, i2 = T(1.0) / r2;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const T u1 = d1[k] * i1, u2 = d2[k] * i2;
        gh1[k] = dv1 * u1 + de_dc * (u2 - cs * u1) * i1;
        gh2[k] = dv2 * u2 + de_dc * (u1 - cs * u2) * i2;
    }
    return v1 + v2 + T(0.5) * T(kKTheta) * dth * dth;
}

// Energies and gradients of ng <= 4 geometries crd + j * stride at once: lane l works
// for geometry l % 4 and for waters l / 4, l / 4 + 8, ..., whose forces it gathers in
// registers over all other waters.  Every pair is formed from both ends, and nothing is
// added in shared memory: FP64 and FP32 atomics there are compare-and-swap loops, which
// bound this kernel before (hexamer, FP64 gradient path's per-sample kernel 382 us per
// 2^15 samples before, 113 now; FP32 200 and 171 us per 2^16).  ms
// [4][3nw] and g [4][9nw] (FP64) are shared, g complete after the call; lane l returns the
// energy of geometry l % 4.
template <typename T>
__device__ double energy_grad_warp4(const T* crd, int stride, T* ms, double* g, int nw, int ng, int lane)
{
    const int j = lane & 3;
    const bool on = j < ng;
    const T* cj = crd + j * stride;
    T* mj = ms + j * 3 * nw;
    if (on)
        for (int i = lane >> 2; i < nw; i += 8) {
            const T* w = cj + 9 * i;
#pragma unroll
            for (int k = 0; k < 3; k++) mj[3 * i + k] = T(kGammaM) * w[k] + T(kGamma1) * (w[3 + k] + w[6 + k]);
        }
    __syncwarp();
    double part = 0;
    if (on)
        for (int i = lane >> 2; i < nw; i += 8) {
            T s[4][3], f[4][3];                 // O, H1, H2, M: positions, gradients
#pragma unroll
            for (int k = 0; k < 3; k++) {
#pragma unroll
                for (int l = 0; l < 3; l++) s[l][k] = cj[9 * i + 3 * l + k];
                s[3][k] = mj[3 * i + k];
                f[0][k] = f[1][k] = f[2][k] = f[3][k] = T(0);
            }
            double e = 0.0;                     // pair terms, each counted from both ends
#pragma unroll 1
            for (int b = 0; b < nw; b++) {
                if (b == i) continue;
                T o[4][3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
#pragma unroll
                    for (int l = 0; l < 3; l++) o[l][k] = cj[9 * b + 3 * l + k];
                    o[3][k] = mj[3 * b + k];
                }
                auto coulomb = [&](T qq, int x, int y) -> double {
                    const T d0 = s[x][0] - o[y][0], d1 = s[x][1] - o[y][1], d2 = s[x][2] - o[y][2];
                    const T ir = inv_sqrt(d0 * d0 + d1 * d1 + d2 * d2), eu = qq * ir, fu = -eu * (ir * ir);
                    f[x][0] += fu * d0, f[x][1] += fu * d1, f[x][2] += fu * d2;
                    return (double)eu;
                };
#pragma unroll
                for (int l = 1; l < 4; l++) {       // neutral groups, as in water_pair
                    const double ql = l == 3 ? kQM : kQH;
                    double t = coulomb(T(ql * kQM), l, 3);
                    t += coulomb(T(ql * kQH), l, 1);
                    t += coulomb(T(ql * kQH), l, 2);
                    e += t;
                }
                const T d0 = s[0][0] - o[0][0], d1 = s[0][1] - o[0][1], d2 = s[0][2] - o[0][2];
                const T ir2 = T(1.0) / (d0 * d0 + d1 * d1 + d2 * d2);
                const T s2 = T(kSigma * kSigma) * ir2, s6 = s2 * s2 * s2;
                const T fo = T(2.0 * 4 * kEpsilon) * (T(3.0) * s6 - T(6.0) * s6 * s6) * ir2;   // 2 dE/d(r^2)
                f[0][0] += fo * d0, f[0][1] += fo * d1, f[0][2] += fo * d2;
                e += (double)(T(4 * kEpsilon) * s6 * (s6 - T(1.0)));
            }
            T w[9], gh1[3], gh2[3];
#pragma unroll
            for (int k = 0; k < 9; k++) w[k] = s[k / 3][k % 3];
            part += (double)monomer_grad(w, gh1, gh2) + 0.5 * e;
            double* gw = g + j * 9 * nw + 9 * i;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                gw[k] = f[0][k] + T(kGammaM) * f[3][k] - (gh1[k] + gh2[k]);
                gw[3 + k] = f[1][k] + T(kGamma1) * f[3][k] + gh1[k];
                gw[6 + k] = f[2][k] + T(kGamma1) * f[3][k] + gh2[k];
            }
        }
    __syncwarp();
    part += __shfl_xor_sync(0xffffffffu, part, 4);
    part += __shfl_xor_sync(0xffffffffu, part, 8);
    part += __shfl_xor_sync(0xffffffffu, part, 16);
    return part;
}

}  // namespace qt
}  // namespace scp3
