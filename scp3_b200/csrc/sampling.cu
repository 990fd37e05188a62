// Per-sample kernels: Sobol point (optionally scrambled) -> BSM -> q = y/sqrt(2)
// -> Cartesian back-transform -> water potential -> anharmonic residual.
// A warp takes four samples at a time; their q and geometries live in the warp's slice
// of shared memory, lanes split the dimensions, the coordinates and the waters.  The FP64 form follows SCP3.cpp:196-223 operation for operation
// where that is cheap (division by sqrt(2), x0 + MUa q then times bohr).
#include "common.cuh"
#include "internal.h"
#include "pes_qtip4pf.cuh"
#include "pes_ttm3f.cuh"
#include "ps_coeffs.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace scp3 {

namespace {

constexpr int kWarpsPerBlock = 8;
constexpr int kRun = 16;          // samples per warp of a batch launch (Gray-code walk)
constexpr int kMinRun = 8;        // fewest samples per warp of a single launch

// Samples a warp carries through the back-transform together, so that every
// shared-memory read of MUa serves this many samples (the back-transform is
// bound by shared-memory bandwidth, MUa being re-read for every sample).
constexpr int kGroup = 4;

template <typename T>
struct WarpSlot {
    T* q;           // [group][qs] normal coordinates (the form's precision)
    T* crd;         // [group][9nw] geometries
    T* ms;          // [group][3nw] M sites
    double* g;      // [group][9nw] gradients (gradient path)
    char* sc;       // TTM3-F scratch, after g
    uint64_t* xs;   // [group][nm0] Sobol states of the group; with tl from crd on (slot_bytes), dead
    uint16_t* tl;   // once the normals are formed: [group * nm0] items of the inverse CDF's tail
    int qs;         // q stride: nm0 rounded up to even (16-byte aligned rows)
};

constexpr size_t round16(size_t b) { return (b + 15) & ~(size_t)15; }

// A group's Sobol states share the bytes of its geometries and of what follows: staged beside
// them they took large clusters a block per SM and L1 (16 waters, 2^16 samples: FP64 1264 us and
// 1933, FP32 with its states behind the geometries 1045 and, over them, 884).  `apart`: behind
// the sites all the same, for the batch's FP32 qTIP4P/f kernel, which spills with the
// overlap (4096 samples of two clusters 72.5 us and 74.5).
template <typename T>
__host__ __device__ inline size_t slot_bytes(int pes, int nm0, int nw, bool grad = false, bool apart = false)
{
    const size_t q = round16(sizeof(T) * kGroup * ((nm0 + 1) & ~1));
    const size_t normals = round16((size_t)kGroup * nm0 * (sizeof(uint64_t) + sizeof(uint16_t)));
    const size_t geometry = round16(sizeof(T) * kGroup * 12 * (size_t)nw);
    const size_t force = (grad ? round16(sizeof(double) * kGroup * 9 * (size_t)nw) : 0) +
                         (pes == SCP3GPU_PES_TTM3F ? round16(ttm::scratch_bytes<T>(nw)) : 0);
    if (apart) return q + geometry + (normals > force ? normals : force);
    return q + (normals > geometry + force ? normals : geometry + force);
}

// kChain: the pointers are formed one from the other, else from the base; the registers of
// the TTM3-F instances decide (2^16 samples, hexamer: gradients FP64 1621 us one from the
// other, 1706 from the base, FP32 1274 and 1360; energies FP64 890 and 916, FP32 424 and 397;
// dimer, FP64 energies 389 and 370).
template <typename T, bool kChain, bool kApart = false>
__device__ inline WarpSlot<T> warp_slot(char* base, int nm0, int nw, bool grad)
{
    WarpSlot<T> s;
    s.qs = (nm0 + 1) & ~1;
    s.q = reinterpret_cast<T*>(base);
    s.crd = s.q + (size_t)kGroup * s.qs;         // whole multiples of 16 bytes each, as the next
    s.ms = s.crd + 9 * nw * kGroup;
    if (kChain) {
        s.g = reinterpret_cast<double*>(s.ms + 3 * nw * kGroup);
        s.sc = reinterpret_cast<char*>(s.g + (grad ? 9 * nw * kGroup : 0));
    } else {
        s.g = nullptr;                           // no gradients there
        s.sc = base + round16(sizeof(T) * kGroup * (s.qs + (size_t)(12 * nw)));
    }
    s.xs = kApart ? reinterpret_cast<uint64_t*>(s.sc) : reinterpret_cast<uint64_t*>(s.crd);
    s.tl = reinterpret_cast<uint16_t*>(s.xs + (size_t)kGroup * nm0);
    return s;
}

// Energies (and with G gradients) of a group's gn geometries in one warp pass: lane l
// returns the energy of geometry l % 4.
template <int PES, typename T, bool G, int NG = kGroup, int NW = 32 / NG>
__device__ __forceinline__ double potential4(const WarpSlot<T>& w, int nw, int gn, int lane, int* iters)
{
    if constexpr (PES == SCP3GPU_PES_QTIP4PF) {
        *iters = 0;
        if constexpr (G) return qt::energy_grad_warp4<T>(w.crd, 9 * nw, w.ms, w.g, nw, gn, lane);
        else return qt::energy_warp4<T>(w.crd, 9 * nw, w.ms, nw, gn, lane);
    } else {
        return ttm::energy_warp4<T, G, NG, NW>(w.crd, 9 * nw, w.ms, w.sc, w.g, nw, gn, lane, iters);
    }
}

constexpr int kDimsPerLane = 4;           // dimensions up to 128 keep their Sobol state in registers

// Standard normals of samples s0 .. s0 + gn - 1 of a warp's range (first sample s_first,
// Sobol index index0 + s): put(j, d, y) for sample s0 + j and dimension d.
// (a) the group's Sobol states, lane-owned by dimension, staged as [sample][dimension]
// (padding samples, s >= nvalid, get u = 0.5, so y = 0); (b) the central branch over all
// gn * dims items, the warp's lanes strided over them, the tail items listed; (c) the
// tail branch (16 % of the items, two logarithms) over the list.
template <typename T, typename Put>
__device__ __forceinline__ void group_normals(const int64_t* __restrict__ vdir, const uint64_t* __restrict__ shift,
                                              int dims, int64_t index0, int64_t s0, int64_t s_first, int64_t nvalid,
                                              int gn, uint64_t* st, uint64_t* xs, uint16_t* tl, int lane, Put put)
{
    for (int j = 0; j < gn; j++) {
        const int64_t s = s0 + j;
        const uint64_t idx = (uint64_t)(index0 + s);
        uint64_t* xj = xs + j * dims;
        if (s >= nvalid) {
            for (int d = lane; d < dims; d += 32) xj[d] = 1ull << 61;
            continue;
        }
#pragma unroll
        for (int jd = 0; jd < kDimsPerLane; jd++) {
            const int d = lane + 32 * jd;
            if (d >= dims) break;
            if (s == s_first) st[jd] = sobol_state(vdir, dims, d, idx);
            else st[jd] ^= (uint64_t)__ldg(vdir + (size_t)(__ffsll((long long)idx) - 1) * dims + d);
            xj[d] = shift ? st[jd] ^ __ldg(shift + d) : st[jd];
        }
        for (int d = lane + 32 * kDimsPerLane; d < dims; d += 32)
            xj[d] = (shift ? __ldg(shift + d) : 0ull) ^ sobol_state(vdir, dims, d, idx);
    }
    __syncwarp();
    const int items = gn * dims;
    const float inv = 1.0f / (float)dims;      // item i is (i / dims, i % dims); exact for i < 2^16
    // two items per lane and round (i, i + 32): two independent chains; every item runs
    // the central formula, the tail items' values are dropped (their denominator may
    // vanish; nothing reads the quotient)
    int ntail = 0;
    const unsigned below = (1u << lane) - 1u;
    for (int i0 = 0; i0 < items; i0 += 64) {
        const int ia = i0 + lane, ib = ia + 32;
        const T ya = ia < items ? bsm_centred<T>(xs[ia]) : T(0);
        const T yb = ib < items ? bsm_centred<T>(xs[ib]) : T(0);
        const T va = bsm_central<T>(ya), vb = bsm_central<T>(yb);
        const bool ta = ia < items && !(fabs(ya) < T(0.42));
        const bool tb = ib < items && !(fabs(yb) < T(0.42));
        if (ia < items && !ta) {
            const int j = (int)(((float)ia + 0.5f) * inv);
            put(j, ia - j * dims, va);
        }
        if (ib < items && !tb) {
            const int j = (int)(((float)ib + 0.5f) * inv);
            put(j, ib - j * dims, vb);
        }
        const unsigned ma = __ballot_sync(0xffffffffu, ta);
        if (ta) tl[ntail + __popc(ma & below)] = (uint16_t)ia;
        ntail += __popc(ma);
        const unsigned mb = __ballot_sync(0xffffffffu, tb);
        if (tb) tl[ntail + __popc(mb & below)] = (uint16_t)ib;
        ntail += __popc(mb);
    }
    __syncwarp();
    for (int t = lane; t < ntail; t += 32) {
        const int i = tl[t];
        const int j = (int)(((float)i + 0.5f) * inv);
        put(j, i - j * dims, bsm_tail<T>(xs[i]));
    }
}

// MUa is staged in shared memory, in the form's precision, when it fits this
// many bytes, as coordinate pairs: for mode k and coordinate group g (64
// coordinates), lane l reads {MUa[k][64g + l], MUa[k][64g + 32 + l]} as one
// word (zero past the last coordinate).
constexpr size_t kMuaSmemMax = 64 * 1024;

__host__ __device__ inline int mua_groups(int nw) { return (9 * nw + 63) / 64; }

// On the gradient path MUa of the selected modes is also staged transposed,
// [coordinate][selected mode] in FP64, when it fits this many bytes: the lane of
// mode m then reads row c at m (consecutive lanes, consecutive words) where a
// read of MUa[k][c] from global memory touched one cache line per lane.
constexpr size_t kMuaTSmemMax = 48 * 1024;
__host__ __device__ inline size_t muat_smem_bytes(int nw, int nm)
{
    return (sizeof(double) * 9 * (size_t)nw * nm + 15) / 16 * 16;   // the warp slots follow, 16-byte aligned
}
template <typename T>
__host__ __device__ inline size_t mua_smem_bytes(int nw, int nm0)
{
    return sizeof(T) * 64 * (size_t)mua_groups(nw) * nm0;
}

template <typename T>
struct Pair;
template <>
struct Pair<double> {
    using type = double2;
};
template <>
struct Pair<float> {
    using type = float2;
};

// G: the gradient path (dV/dq) is compiled in; the energy-only instances keep
// their registers for the energy path.
template <int PES, typename T, bool G = false, int NW = 8, bool kApart = false>
__device__ __forceinline__ void samples_body(const SampleArgs& a, char* smem);

// Blocks per SM the registers must allow: qTIP4P/f, 4 for the FP32 energies (64
// registers), 3 for the FP32 gradients (85), 2 for FP64; TTM3-F keeps its dipole tensors
// in registers: 2 for the energies, 1 for the gradients, 2 for those of clusters of up to
// NW = 4 waters (three tensors per lane instead of seven; trimer gradients, 2^14
// samples: 268 us at one block).
template <int PES, typename T, bool G, int NW = 8>
constexpr int sample_blocks()
{
    if (PES == SCP3GPU_PES_TTM3F) return G && NW > 4 ? 1 : 2;
    return sizeof(T) == 4 ? (G ? 3 : 4) : 2;
}

template <int PES, typename T, bool G, int NW = 8>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, sample_blocks<PES, T, G, NW>())
    samples_kernel(SampleArgs a)
{
    extern __shared__ __align__(16) char smem[];
    samples_body<PES, T, G, NW>(a, smem);
}

template <int PES, typename T>
constexpr bool kBatchApart = PES == SCP3GPU_PES_QTIP4PF && sizeof(T) == 4;

// Several clusters of a batch: cluster blockIdx.y takes args[blockIdx.y].
template <int PES, typename T>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, sample_blocks<PES, T, false>())
    samples_batch_kernel(const SampleArgs* __restrict__ args)
{
    extern __shared__ __align__(16) char smem[];
    // the cluster's arguments in shared memory, read where used (a register copy
    // of the whole block costs occupancy)
    __shared__ SampleArgs a;
    if (threadIdx.x == 0) a = args[blockIdx.y];
    __syncthreads();
    samples_body<PES, T, false, 8, kBatchApart<PES, T>>(a, smem);
}

template <int PES, typename T, bool G, int NW, bool kApart>
__device__ __forceinline__ void samples_body(const SampleArgs& a, char* smem)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nw = a.nw, nm0 = a.nm0, N3 = 9 * nw;
    using T2 = typename Pair<T>::type;
    const size_t mua_b = mua_smem_bytes<T>(nw, nm0);
    const bool mua_in_smem = mua_b <= kMuaSmemMax;
    const int ng = mua_groups(nw);
    const double* MUa = a.MUa;
    T2* mua2 = reinterpret_cast<T2*>(smem);      // [nm0][ng][32] coordinate pairs
    if (mua_in_smem) {
        for (int e = threadIdx.x; e < nm0 * ng * 32; e += blockDim.x) {
            const int l = e & 31, g = (e >> 5) % ng, k = (e >> 5) / ng, c = 64 * g + l;
            T2 m;
            m.x = (T)(c < N3 ? a.MUa[(size_t)k * N3 + c] : 0.0);
            m.y = (T)(c + 32 < N3 ? a.MUa[(size_t)k * N3 + c + 32] : 0.0);
            mua2[e] = m;
        }
        __syncthreads();
    }
    const bool grad = G && a.vq != nullptr;
    const bool muat_in_smem = grad && muat_smem_bytes(nw, a.nm) <= kMuaTSmemMax;
    double* muat = reinterpret_cast<double*>(smem + (mua_in_smem ? mua_b : 0));   // [N3][nm]
    if (muat_in_smem) {
        for (int e = threadIdx.x; e < N3 * a.nm; e += blockDim.x) {
            const int c = e / a.nm, m = e - c * a.nm;
            muat[e] = a.MUa[(size_t)__ldg(a.modes + m) * N3 + c];
        }
        __syncthreads();
    }
    char* slots = smem + (mua_in_smem ? mua_b : 0) + (muat_in_smem ? muat_smem_bytes(nw, a.nm) : 0);
    WarpSlot<T> w = warp_slot<T, G || (sizeof(T) == 8 && NW == 8), kApart>(slots + wib * slot_bytes<T>(PES, nm0, nw, grad, kApart), nm0, nw, grad);
    // Each warp takes one contiguous range of samples, the ranges balanced to
    // within one sample (the grid is sized to the SMs, so there is no tail wave):
    // the Sobol state of the first is formed from the Gray code of its index, the
    // next ones by one XOR per dimension (index k differs from k-1 in direction
    // number ctz(k)).  The range goes in groups of kGroup samples: normals for
    // the group, one back-transform pass and one potential pass for the group, then
    // V, q and dV/dq.
    const int64_t nwarps = (int64_t)gridDim.x * kWarpsPerBlock;
    const int64_t gw = (int64_t)blockIdx.x * kWarpsPerBlock + wib;
    uint64_t st[kDimsPerLane];
    const int64_t s_first = a.n * gw / nwarps, s_end = a.n * (gw + 1) / nwarps;
    const bool sobol = a.normals == nullptr && a.normals32 == nullptr;
    for (int64_t s0 = s_first; s0 < s_end; s0 += kGroup) {
        const int gn = (int)(s_end - s0 < kGroup ? s_end - s0 : kGroup);
        // 1. standard normals -> q   (SCP3.cpp:196-201)
        if (sobol) {
            group_normals<T>(a.vdir, a.shift, nm0, a.index0, s0, s_first, a.nvalid, gn, st, w.xs, w.tl, lane,
                             [&](int j, int d, T y) {
                                 w.q[j * w.qs + d] = sizeof(T) == 4 ? y * T(0.70710678f) : y / T(1.4142135623730951);
                             });
        } else {
            for (int j = 0; j < gn; j++) {
                const int64_t s = s0 + j;
                T* q = w.q + j * w.qs;
                for (int d = lane; d < nm0; d += 32) {
                    double y = 0.0;             // padding sample (the range's tail): contributes nothing
                    if (s < a.nvalid) y = a.normals ? a.normals[s * nm0 + d] : (double)a.normals32[s * nm0 + d];
                    q[d] = (T)(y / 1.4142135623730951);   // by /= sqrt(2.0)
                }
            }
        }
        __syncwarp();
        // 2. r = bohr * (x0 + MUa q)   (SCP3.cpp:208), in the form's precision (FP64
        // for the plain form); a lane's two coordinates (c, c + 32) of every sample
        // of the group in one pass, each summed over k in order (samples past gn
        // compute stale values that are not used)
        if (mua_in_smem) {
            for (int g = 0; g < ng; g++) {
                const int c = 64 * g + lane;
                const T2* mg = mua2 + g * 32 + lane;
                const int kstride = ng * 32;
                T acc0[kGroup], acc1[kGroup];
#pragma unroll
                for (int j = 0; j < kGroup; j++) acc0[j] = acc1[j] = T(0);
                int k = 0;
                for (; k + 1 < nm0; k += 2) {
                    const T2 m0 = mg[k * kstride], m1 = mg[(k + 1) * kstride];
#pragma unroll
                    for (int j = 0; j < kGroup; j++) {
                        const T2 qq = reinterpret_cast<const T2*>(w.q + j * w.qs)[k >> 1];
                        acc0[j] += m0.x * qq.x;
                        acc1[j] += m0.y * qq.x;
                        acc0[j] += m1.x * qq.y;
                        acc1[j] += m1.y * qq.y;
                    }
                }
                if (k < nm0) {
                    const T2 m0 = mg[k * kstride];
#pragma unroll
                    for (int j = 0; j < kGroup; j++) {
                        const T qk = w.q[j * w.qs + k];
                        acc0[j] += m0.x * qk;
                        acc1[j] += m0.y * qk;
                    }
                }
                const T x0a = (T)(c < N3 ? __ldg(a.x0 + c) : 0.0), x0b = (T)(c + 32 < N3 ? __ldg(a.x0 + c + 32) : 0.0);
#pragma unroll
                for (int j = 0; j < kGroup; j++) {
                    if (j >= gn) break;
                    T* crd = w.crd + j * N3;
                    if (c < N3) crd[c] = (T)kBohr * (x0a + acc0[j]);
                    if (c + 32 < N3) crd[c + 32] = (T)kBohr * (x0b + acc1[j]);
                }
            }
        } else {
            for (int j = 0; j < gn; j++) {
                const T* q = w.q + j * w.qs;
                T* crd = w.crd + j * N3;
                for (int c = lane; c < N3; c += 64) {
                    const bool two = c + 32 < N3;
                    double acc0 = 0.0, acc1 = 0.0;
#pragma unroll 4
                    for (int k = 0; k < nm0; k++) {
                        const double qk = (double)q[k];
                        acc0 += MUa[(size_t)k * N3 + c] * qk;
                        if (two) acc1 += MUa[(size_t)k * N3 + c + 32] * qk;
                    }
                    crd[c] = (T)(kBohr * (__ldg(a.x0 + c) + acc0));
                    if (two) crd[c + 32] = (T)(kBohr * (__ldg(a.x0 + c + 32) + acc1));
                }
            }
        }
        __syncwarp();
        // 3. V and, on the gradient path (SCP3.cpp:209-216), dV/dr of the whole group in
        // one warp pass, then dV_anh/dq = MUa^T (bohr dV/dr / autokcal) - omega % q of the
        // group's (sample, selected mode) items over the lanes, summed in FP64
        double e4 = 0.0;
        int iters4 = 0;
        if (!a.skip_pes) {
            if (grad) {
                if constexpr (G) e4 = potential4<PES, T, true, kGroup, NW>(w, nw, gn, lane, &iters4);
            } else {
                e4 = potential4<PES, T, false, kGroup, NW>(w, nw, gn, lane, &iters4);
            }
        }
        if constexpr (G) {
            if (grad) {
                for (int it = lane; it < gn * a.nm; it += 32) {
                    const int j = it / a.nm, m = it - j * a.nm;
                    const int64_t s = s0 + j;
                    const int k = __ldg(a.modes + m);
                    const double* gj = w.g + j * N3;
                    double acc = 0.0;
                    if (muat_in_smem)
                        for (int c = 0; c < N3; c++) acc += muat[(size_t)c * a.nm + m] * gj[c];
                    else
                        for (int c = 0; c < N3; c++) acc += MUa[(size_t)k * N3 + c] * gj[c];
                    a.vq[s * a.nm + m] = s < a.nvalid ? acc * (kBohr / kAuToKcalPerMol) -
                                                            __ldg(a.omega + k) * (double)w.q[j * w.qs + k]
                                                      : 0.0;
                }
                __syncwarp();
            }
        }
        for (int j = 0; j < gn; j++) {
            const int64_t s = s0 + j;
            const T* q = w.q + j * w.qs;
            const double e = __shfl_sync(0xffffffffu, e4, j);
            const int iters = PES == SCP3GPU_PES_TTM3F ? __shfl_sync(0xffffffffu, iters4, j) : 0;
            if (s >= a.nvalid) {
                if (lane == 0) a.v[s] = 0.0;
                for (int m = lane; m < a.nm; m += 32) {
                    if (a.q64) a.q64[s * a.nm + m] = 0.0;
                    if (a.q32) a.q32[s * a.nm + m] = 0.0f;
                }
                continue;
            }
            // V in hartree, anharmonic residual   (SCP3.cpp:219-223)
            double V = 0.0;
            if (!a.skip_pes) {
                double h = 0.0;
                for (int d = lane; d < nm0; d += 32) h += (double)q[d] * (__ldg(a.omega + d) * (double)q[d]);
                h = warp_sum(h);
                V = e / kAuToKcalPerMol - 0.5 * h;
            }
            if (lane == 0) {
                a.v[s] = V;
                if (!isfinite(V)) atomicAdd(a.counters + 0, 1ull);
                if (iters > kTtmMaxIter) atomicAdd(a.counters + 1, 1ull);
            }
            // 4. selected modes, coalesced per sample
            for (int m = lane; m < a.nm; m += 32) {
                const T qm = q[__ldg(a.modes + m)];
                if (a.q64) a.q64[s * a.nm + m] = (double)qm;
                if (a.q32) a.q32[s * a.nm + m] = (float)qm;
            }
        }
        __syncwarp();               // the next group's normals go over its geometries
    }
}

// Energies (and with G gradients) of n geometries, FP64, NG per warp (four; two for TTM3-F
// with more than eight waters); one warp per CTA, so that a few geometries (a Hessian's
// 2N) spread over the SMs.
template <int PES, bool G, int NG = kGroup>
__global__ void __launch_bounds__(32) pes_kernel(int nw, int64_t n, const double* __restrict__ crd,
                                                 double* __restrict__ E, double* __restrict__ grad,
                                                 int* __restrict__ iters_out)
{
    extern __shared__ __align__(16) char smem[];
    const int lane = threadIdx.x, N3 = 9 * nw;
    const WarpSlot<double> w = warp_slot<double, G>(smem, 0, nw, G);
    for (int64_t g0 = (int64_t)blockIdx.x * NG; g0 < n; g0 += (int64_t)gridDim.x * NG) {
        const int gn = (int)(n - g0 < NG ? n - g0 : NG);
        for (int c = lane; c < gn * N3; c += 32) w.crd[c] = crd[g0 * N3 + c];
        __syncwarp();
        int iters = 0;
        const double e = potential4<PES, double, G, NG>(w, nw, gn, lane, &iters);
        if (lane < gn) {
            E[g0 + lane] = e;
            if (iters_out) iters_out[g0 + lane] = iters;
        }
        if (G)
            for (int c = lane; c < gn * N3; c += 32) grad[g0 * N3 + c] = w.g[c];
        __syncwarp();
    }
}

// SCP1 per-sample stage (SCP1.cpp:52-63): contiguous balanced sample ranges per warp with
// the Gray-code Sobol walk, in groups of four samples as the builds' per-sample kernel;
// isqrtM_U staged in shared memory.
constexpr int kS1Warps = 8;

__host__ __device__ inline size_t scp1_slot(int pes, int nw, int dim)
{
    return slot_bytes<double>(pes, dim, nw, true) + sizeof(double) * kGroup * (size_t)dim;
}

template <int PES>
__global__ void __launch_bounds__(kS1Warps * 32, PES == SCP3GPU_PES_TTM3F ? 1 : 2) scp1_samples_kernel(Scp1Args a)
{
    extern __shared__ __align__(16) double s1[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nw = a.nw, dim = a.dim;
    double* U = s1;
    for (int e = threadIdx.x; e < dim * dim; e += blockDim.x) U[e] = a.U[e];
    char* slot = reinterpret_cast<char*>(s1) + round16(sizeof(double) * dim * dim) + (size_t)wib * scp1_slot(PES, nw, dim);
    const WarpSlot<double> w = warp_slot<double, true>(slot, dim, nw, true);      // w.q: y = std_normal % sqrt(d)
    double* dq = reinterpret_cast<double*>(slot + slot_bytes<double>(PES, dim, nw, true));   // [group][dim]
    __syncthreads();
    const int64_t nwarps = (int64_t)gridDim.x * kS1Warps;
    const int64_t gw = (int64_t)blockIdx.x * kS1Warps + wib;
    const int64_t s_first = a.n * gw / nwarps, s_end = a.n * (gw + 1) / nwarps;
    uint64_t st[kDimsPerLane];
    for (int64_t s0 = s_first; s0 < s_end; s0 += kGroup) {
        const int gn = (int)(s_end - s0 < kGroup ? s_end - s0 : kGroup);
        // y = std_normal % sqrt(d)   (SCP1.cpp:54-58)
        group_normals<double>(a.vdir, nullptr, dim, a.index0, s0, s_first, a.n, gn, st, w.xs, w.tl, lane,
                              [&](int j, int d, double y) { w.q[j * w.qs + d] = y * __ldg(a.sqd + d); });
        __syncwarp();
        // dq = isqrtM_U y, r = bohr (q + dq)   (SCP1.cpp:60-61), k in order
        for (int c = lane; c < dim; c += 32) {
            double acc[kGroup] = {};
            for (int k = 0; k < dim; k++) {
                const double u = U[(size_t)k * dim + c];
#pragma unroll
                for (int j = 0; j < kGroup; j++) acc[j] += u * w.q[j * w.qs + k];   // past gn: stale, not used
            }
            const double q0 = __ldg(a.q + c);
#pragma unroll
            for (int j = 0; j < kGroup; j++) {
                if (j >= gn) break;
                dq[j * dim + c] = acc[j];
                w.crd[j * dim + c] = kBohr * (q0 + acc[j]);
            }
        }
        __syncwarp();
        int it = 0;
        const double e = potential4<PES, double, true>(w, nw, gn, lane, &it);
        if (lane < gn) {
            a.V[s0 + lane] = e / kAuToKcalPerMol;
            if (it > kTtmMaxIter) atomicAdd(a.not_converged, 1ull);
        }
        for (int c = lane; c < gn * dim; c += 32) {
            a.G[s0 * dim + c] = w.g[c] * (kBohr / kAuToKcalPerMol);    // UX_ *= bohr/autokcalpmol
            a.D[s0 * dim + c] = dq[c];
        }
        __syncwarp();
    }
}

__global__ void std_normal_kernel(int dims, int64_t index0, int64_t n, const int64_t* __restrict__ vdir,
                                  const uint64_t* __restrict__ shift, double* __restrict__ out)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * dims) return;
    const int64_t s = t / dims;
    const int d = (int)(t - s * dims);
    uint64_t x = sobol_state(vdir, dims, d, (uint64_t)(index0 + s));
    if (shift) x ^= shift[d];
    out[t] = bsm(sobol_uniform(x));
}

// Blocks of the per-sample kernel: one warp per kMinRun samples at least, and
// no more blocks than the SMs hold at once.
template <typename K>
int sample_grid(K kern, size_t smem, int64_t n)
{
    int dev = 0, sms = 148, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kWarpsPerBlock * 32, smem) != cudaSuccess || per < 1)
        per = 1;
    const int64_t want = (n + (int64_t)kMinRun * kWarpsPerBlock - 1) / ((int64_t)kMinRun * kWarpsPerBlock);
    const int64_t cap = (int64_t)per * sms;
    return (int)std::max<int64_t>(1, std::min(want, cap));
}

int grid_for(int64_t nwarps_needed)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t blocks = (nwarps_needed + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t cap = (int64_t)sms * 8;
    return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

template <int PES, typename T>
int launch_samples_t(const SampleArgs& a, cudaStream_t s)
{
    const size_t mua_b = mua_smem_bytes<T>(a.nw, a.nm0);
    const size_t muat_b = muat_smem_bytes(a.nw, a.nm);
    const size_t sm = kWarpsPerBlock * slot_bytes<T>(PES, a.nm0, a.nw, a.vq != nullptr) +
                      (mua_b <= kMuaSmemMax ? mua_b : 0) + (a.vq && muat_b <= kMuaTSmemMax ? muat_b : 0);
    // the FP32 gradient is qTIP4P/f's only (launch_samples)
    constexpr bool kGrad = PES == SCP3GPU_PES_QTIP4PF || sizeof(T) == 8;
    auto kern = a.vq ? samples_kernel<PES, T, kGrad> : samples_kernel<PES, T, false>;
    if constexpr (PES == SCP3GPU_PES_TTM3F)
        if (a.nw <= 4) kern = a.vq ? samples_kernel<PES, T, kGrad, 4> : samples_kernel<PES, T, false, 4>;
    if (int rc = allow_smem(kern)) return rc;
    kern<<<sample_grid(kern, sm, a.n), kWarpsPerBlock * 32, sm, s>>>(a);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

template <int PES, typename T>
int launch_samples_batch_t(const SampleArgs* args_host, const SampleArgs* args_dev, int ncl, int64_t n, cudaStream_t s)
{
    // Shared memory for the largest cluster: warp slots of the largest (nm0, nw)
    // plus the largest MUa that a cluster stages (each cluster decides as the
    // single-cluster kernel does, so its layout fits).
    int nm0 = 0, nw = 0;
    size_t mua = 0;
    for (int c = 0; c < ncl; c++) {
        nm0 = std::max(nm0, args_host[c].nm0);
        nw = std::max(nw, args_host[c].nw);
        const size_t b = mua_smem_bytes<T>(args_host[c].nw, args_host[c].nm0);
        if (b <= kMuaSmemMax) mua = std::max(mua, b);
    }
    const size_t sm = kWarpsPerBlock * slot_bytes<T>(PES, nm0, nw, false, kBatchApart<PES, T>) + mua;
    if (int rc = allow_smem(samples_batch_kernel<PES, T>)) return rc;
    const int per = grid_for((n + kRun - 1) / kRun);   // per cluster; the clusters share the SMs
    samples_batch_kernel<PES, T><<<dim3((unsigned)per, (unsigned)ncl), kWarpsPerBlock * 32, sm, s>>>(args_dev);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

}  // namespace

int launch_samples_batch(int pes, bool fp32, const SampleArgs* args_host, const SampleArgs* args_dev, int ncl,
                         int64_t n, cudaStream_t s)
{
    if (n <= 0 || ncl <= 0) return SCP3GPU_OK;
    if (pes == SCP3GPU_PES_QTIP4PF)
        return fp32 ? launch_samples_batch_t<SCP3GPU_PES_QTIP4PF, float>(args_host, args_dev, ncl, n, s)
                    : launch_samples_batch_t<SCP3GPU_PES_QTIP4PF, double>(args_host, args_dev, ncl, n, s);
    if (pes == SCP3GPU_PES_TTM3F)
        return fp32 ? launch_samples_batch_t<SCP3GPU_PES_TTM3F, float>(args_host, args_dev, ncl, n, s)
                    : launch_samples_batch_t<SCP3GPU_PES_TTM3F, double>(args_host, args_dev, ncl, n, s);
    return fail(SCP3GPU_ERR_ARG, "unknown potential id");
}

int ttm_init_device()
{
    static std::mutex mu;
    static bool done[128] = {false};
    int dev = 0;
    SCP3_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 128) return fail(SCP3GPU_ERR_ARG, "device ordinal out of range");
    if (done[dev]) return SCP3GPU_OK;
    ttm::Consts c;
    c.iAA_HH = 1.0 / std::pow(0.496 * 0.496, 1.0 / 6.0);
    c.iAA_HM = 1.0 / std::pow(0.496 * 0.837, 1.0 / 6.0);
    c.iAA_MM = 1.0 / std::pow(0.837 * 0.837, 1.0 / 6.0);
    c.aXX13 = std::pow(0.175, 1.0 / 3.0);
    c.phh1 = 0.999677885 * 16.94879431193463 * std::exp(12.66426998162947);
    for (int i = 0; i < ttm::kETerms; i++) {   // ps.cpp:508-511: f5z, fbasis, fcore, frest
        const double c5z = 0.999677885 * scp3_ps_c5zA[i] + 0.15860145369897 * scp3_ps_cbasis[i] +
                           -1.6351695982132 * scp3_ps_ccore[i] + 1.0 * scp3_ps_crest[i];
        const int I = scp3_ps_idx1[i] - 1, J = scp3_ps_idx2[i] - 1, K = scp3_ps_idx3[i] - 1;
        if (i == 0) c.c5z0 = c5z;
        c.e[ttm::e_offset(I, J) + K] = i ? c5z : 0.0;
    }
    for (int i = 0; i < ttm::kDTerms; i++) {
        const int I = scp3_ps_idxD0[i] - 1, J = scp3_ps_idxD1[i] - 1, K = scp3_ps_idxD2[i] - 1;
        if (i == 0) c.coefD0 = scp3_ps_coefD[i];
        c.d[ttm::d_offset(I, J) + K] = i ? scp3_ps_coefD[i] : 0.0;
    }
    double ser = 1.0;
    for (int n = 0; n < 36; n++) c.s[n] = ser /= 2.0 / 3.0 + n;
    for (int i = 0; i < ttm::kETerms; i++) c.ef[i] = (float)c.e[i];
    for (int i = 0; i < ttm::kDTerms; i++) c.df[i] = (float)c.d[i];
    for (int n = 0; n < 36; n++) c.sf[n] = (float)c.s[n];
    ttm::TailTable tail;
    ttm::tail_tables(tail);
    SCP3_CUDA(cudaMemcpyToSymbol(ttm::kTail, &tail, sizeof(tail)));
    SCP3_CUDA(cudaMemcpyToSymbol(ttm::kC, &c, sizeof(c)));
    done[dev] = true;
    return SCP3GPU_OK;
}

int launch_samples(int pes, bool fp32, const SampleArgs& a, cudaStream_t s)
{
    if (a.n <= 0) return SCP3GPU_OK;
    if (a.vq && fp32 && pes != SCP3GPU_PES_QTIP4PF)
        return fail(SCP3GPU_ERR_UNSUPPORTED, "gradient path: FP32 potential for qTIP4P/f only");
    if (pes == SCP3GPU_PES_QTIP4PF)
        return fp32 ? launch_samples_t<SCP3GPU_PES_QTIP4PF, float>(a, s)
                    : launch_samples_t<SCP3GPU_PES_QTIP4PF, double>(a, s);
    if (pes == SCP3GPU_PES_TTM3F)
        return fp32 ? launch_samples_t<SCP3GPU_PES_TTM3F, float>(a, s)
                    : launch_samples_t<SCP3GPU_PES_TTM3F, double>(a, s);
    return fail(SCP3GPU_ERR_ARG, "unknown potential id");
}

int launch_pes(int pes, int nw, int64_t n, const double* crd, double* E, double* G, int* iters, cudaStream_t s)
{
    if (n <= 0) return SCP3GPU_OK;
    if (pes != SCP3GPU_PES_QTIP4PF && pes != SCP3GPU_PES_TTM3F) return fail(SCP3GPU_ERR_ARG, "unknown potential id");
    const size_t sm = slot_bytes<double>(pes, 0, nw, G != nullptr);      // under 32 KB at 16 waters
    auto kern = pes == SCP3GPU_PES_TTM3F
                    ? (G ? pes_kernel<SCP3GPU_PES_TTM3F, true> : pes_kernel<SCP3GPU_PES_TTM3F, false>)
                    : (G ? pes_kernel<SCP3GPU_PES_QTIP4PF, true> : pes_kernel<SCP3GPU_PES_QTIP4PF, false>);
    int ng = kGroup;
    if (pes == SCP3GPU_PES_TTM3F && nw > 8) {
        if (G) return fail(SCP3GPU_ERR_ARG, "TTM3-F gradients: at most 8 waters");
        kern = pes_kernel<SCP3GPU_PES_TTM3F, false, 2>;
        ng = 2;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned grid = (unsigned)std::min<int64_t>((n + ng - 1) / ng, (int64_t)sms * 32);
    kern<<<grid, 32, sm, s>>>(nw, n, crd, E, G, iters);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

int launch_scp1_samples(int pes, const Scp1Args& a, cudaStream_t s)
{
    if (a.n <= 0) return SCP3GPU_OK;
    if (pes != SCP3GPU_PES_QTIP4PF && pes != SCP3GPU_PES_TTM3F) return fail(SCP3GPU_ERR_ARG, "unknown potential id");
    const size_t sm = round16(sizeof(double) * a.dim * a.dim) + kS1Warps * scp1_slot(pes, a.nw, a.dim);
    auto kern = pes == SCP3GPU_PES_QTIP4PF ? scp1_samples_kernel<SCP3GPU_PES_QTIP4PF>
                                            : scp1_samples_kernel<SCP3GPU_PES_TTM3F>;
    if (int rc = allow_smem(kern)) return rc;
    int dev = 0, sms = 148, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kS1Warps * 32, sm) != cudaSuccess || per < 1) per = 1;
    const int64_t want = (a.n + 4 * kS1Warps - 1) / (4 * kS1Warps);     // >= 4 samples per warp
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)per * sms));
    kern<<<grid, kS1Warps * 32, sm, s>>>(a);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

int launch_std_normal(int dims, int64_t index0, int64_t n, const int64_t* vdir, const uint64_t* shift, double* out,
                      cudaStream_t s)
{
    const int64_t total = n * dims;
    if (total <= 0) return SCP3GPU_OK;
    std_normal_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(dims, index0, n, vdir, shift, out);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

}  // namespace scp3

// Host-only view of TTM3-F's smearing table, for tests: the interval (0..9) x is looked
// up in, -1 where the table is not read.
extern "C" int scp3gpu_internal_tail_span(double x, int fp32)
{
    return std::max(-1, fp32 ? scp3::ttm::tail_span((float)x) : scp3::ttm::tail_span(x));
}

// Host-only view of the water-pair items of the four-sample qTIP4P/f kernels, for
// tests: ab[2 p], ab[2 p + 1] = the waters a < b of pair p, p < nw (nw - 1) / 2.
extern "C" int scp3gpu_internal_water_pairs(int nw, int* ab)
{
    if (nw < 1 || nw > 64 || !ab) return SCP3GPU_ERR_ARG;
    const int np = nw * (nw - 1) / 2;
    for (int p = 0; p < np; p++) scp3::qt::water_pair_of(p, nw, ab[2 * p], ab[2 * p + 1]);
    return SCP3GPU_OK;
}
