// Oscillator functions and the weights of the gradient estimator, FP64.
#pragma once
#include "internal.h"

namespace scp3 {

// (mode, level) list of a basis descriptor (kind | m << 3 | n << 11 | p << 19)
__host__ __device__ __forceinline__ int decode(uint32_t d, int* m, int* l)
{
    const int kind = (int)(d & 7u), a = (int)((d >> 3) & 255u), b = (int)((d >> 11) & 255u), c = (int)(d >> 19);
    switch (kind) {
        case kGround: return 0;
        case kHo1: m[0] = a, l[0] = 1; return 1;
        case kHo2: m[0] = a, l[0] = 2; return 1;
        case kHo1Ho1: m[0] = a, l[0] = 1, m[1] = b, l[1] = 1; return 2;
        case kHo3: m[0] = a, l[0] = 3; return 1;
        case kHo2Ho1: m[0] = a, l[0] = 2, m[1] = b, l[1] = 1; return 2;
        case kHo1Ho2: m[0] = a, l[0] = 1, m[1] = b, l[1] = 2; return 2;
        default: m[0] = a, l[0] = 1, m[1] = b, l[1] = 1, m[2] = c, l[2] = 1; return 3;
    }
}

// h_l(q) (HarmonicOscillatorBasis.cpp: 1, sqrt2 q, (2q^2 - 1)/sqrt2, (2q^3 - 3q)/sqrt3)
__device__ __forceinline__ double ho(int l, double q)
{
    switch (l) {
        case 0: return 1.0;
        case 1: return 1.4142135623730951 * q;
        case 2: return (2.0 * q * q - 1.0) * 0.70710678118654752;
        default: return (2.0 * q * q - 3.0) * q * 0.57735026918962576;
    }
}

// h_a(q), h_a(0), h_a'(q), d_a(q), d_a'(q) for the oscillator functions h_0..h_3
__device__ __forceinline__ void ho_parts(int a, double q, double& h, double& h0, double& dh, double& d, double& dd)
{
    constexpr double s2 = 1.4142135623730951, is2 = 0.70710678118654752, is3 = 0.57735026918962576;
    switch (a) {
        case 0: h = 1, h0 = 1, dh = 0, d = 0, dd = 0; break;
        case 1: h = s2 * q, h0 = 0, dh = s2, d = s2, dd = 0; break;
        case 2: h = (2 * q * q - 1) * is2, h0 = -is2, dh = 2 * s2 * q, d = s2 * q, dd = s2; break;
        default: h = (2 * q * q - 3) * q * is3, h0 = 0, dh = (6 * q * q - 3) * is3, d = (2 * q * q - 3) * is3,
                 dd = 4 * q * is3; break;
    }
}

// K_ab = u V + w dV/dq_m for mode m at q_m = x, levels (a, b)
__device__ __forceinline__ double stein_weight(int a, int b, double x, double V, double Vm)
{
    double ha, ha0, dha, da, dda, hb, hb0, dhb, db, ddb;
    ho_parts(a, x, ha, ha0, dha, da, dda);
    ho_parts(b, x, hb, hb0, dhb, db, ddb);
    const double r = da * hb + ha0 * db;
    const double dr = dda * hb + da * dhb + ha0 * ddb;
    double u = ha0 * hb0 + 0.5 * dr;
    const double w = 0.5 * r;
    if (a == 3 && b == 3) u = (2 * x * x - 3) * (x * x - 3) * (1.0 / 6.0);   // TripleExcitations.h:763-773
    return u * V + w * Vm;
}

}  // namespace scp3
