// Sums over samples of products of FP64 values, as exact integer products on the
// tensor cores: sum_s A_i(s) B_j(s) for the plain FP64 form of both estimators
// (ScaledMatrixElements.cpp:951-971 and :102-725).
//
// Why.  The FP64 pipe does 64 FMA per clock and SM, the tensor cores 65536 8-bit
// ones: a product of two 56-bit fixed-point numbers in 34 products of 8-bit digits
// is worth 4 FP64 pipes or so (the clock is lower under this load).  The DFMA kernel this replaces ran at 0.72 of that pipe:
// 8.9 ms per 2^17 samples of the hexamer doubles basis.
//
// Digits.  Within a pass every operand row has one power-of-two scale, 2^e just above
// its largest |value|; a value is rounded to the integer x 2^(55 - e) (|.| < 0.9961 2^55)
// and written as seven balanced base-256 digits, each -128..127, most significant first.
// The product of two rows is sum over digit pairs (i, j) of 2^(8 (14 - i - j)) D_ij;
// the 34 pairs with i + j <= 9 are formed.  Against extended-precision sums of the
// same values, 2^13 samples, norm-wise, and of an FP64 product in brackets: 3.3e-16
// (4.4e-16) for a dimer, 3.0e-16 (5.1e-16) a trimer with TTM3-F, 5.6e-16 (1.1e-15) the
// hexamer; with i + j <= 8 only (28 pairs) about ten times as much.  D_ij is accumulated in
// 32-bit integers, exactly: a run is at most 18432 samples, so a group of equal i + j (up to
// 7 pairs of 2^14) stays below 2^31.
//
// Range.  A value 2^-k of its row's largest keeps 55 - k bits, so a sample that dwarfs the
// others would cost them their bits, above all in the elements where its own term is
// small.  Samples whose |V|, |q_m| or |dV/dq_m| is more than 2^9, 2^4 and 2^9 times that
// quantity's geometric mean over 128 samples of the pass, or not finite, are therefore left
// out of the digits (zero) and of the scales, and their products added in FP64 at the end
// of contract_i8_kernel (add_heavy).  2^4 times the mean of 128 coordinates (0.28 to 0.34)
// is 4.5 or more, which one in 10^9 passes, 2^9 above the largest |V| of 2^17 points of the
// clusters looked at (8 to 490 times the mean), so ordinary builds have such samples rarely
// or not at all: the limits cost a launch of 4 us in place of a memset.  One V of 2^14 at 1, 10^2, 10^3, 10^6 and
// 10^12 times the others' rms, elements in which it vanishes, largest error over the sum
// of |terms|: 2.8e-17, 8.7e-17, 2.8e-17, 2.8e-17, 2.8e-17 (an FP64 product 5.7e-17 in each;
// without the limits 4.9e-17, 2.1e-16, 2.2e-15, 1.5e-12, 1.9e-6).  Hexamer, 2^16 samples,
// 2.0 ms: 0.1 % of them heavy add 2 % to the pass, 1 % a tenth, 10 % as much again and 60 %
// (V spread evenly over 24 decades) 3.3 times as much, 1.6 times an FP64 kernel's time.
// Elements are NaN or infinite where the FP64 products would be; a finite row whose
// products overflow reads NaN.
//
// The splitting into exact partial products is the published one for matrix products on
// narrow units (Ozaki, Ogita, Oishi and Rump); the order of the digits below is this file's.
//
// Operand layout: [row block of 128][k-block of 64 samples][digit][128 rows x 64 B],
// each 8 KB box in the 64-byte-swizzled order the MMA descriptors read (16-byte chunk
// c of row r at c ^ ((r >> 1) & 3)).
//
// contract_i8_kernel: a work unit is (sample range, 128 x 256 tile); four sweeps
// over the unit's k-blocks, for the digit sums 9 and 8, 7 and 6, 5 and 4, 3 and 2; a
// sweep's two sums own the two 256-column TMEM accumulators.  In one k-block of a sweep
// the digits come in a chain (1, 7, 2, 6, 3, 5, 4 for the sums 9 and 8; n, 1, n-1, 2,
// ... with n = 6, 4, 2 for the others) whose neighbours add up to the one and the other
// sum in turn, and whose last pairs with itself, so every digit (A box and two B boxes,
// 24 KB) is loaded once and is free again two steps later: 53 bytes loaded per clock
// and SM, 8 or 9 steps in flight in a ring of 9.  After a sweep eight warps add the two
// accumulators, joined in 64 bits, into the unit's own FP64 partial, by reductions
// that need no read (a read-modify-write took 10 us a drain).
// What bounds it: the tensor pipe under the power limit (one M = 128, N = 256, K = 32
// product takes 128 clocks alone on an SM, like a K = 16 product of kind::f16).
// Bounded waits as in contract_tc.cu.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "contract_i8.h"
#include "hermite.cuh"

namespace scp3 {
namespace i8 {

namespace {

constexpr unsigned long long kWaitNs = 4000000000ull;
#include "tc_ptx.cuh"

constexpr int kDigits = 7, kSweeps = 4, kTile = 128, kN = 256;
constexpr int kBox = kTile * kKB;                  // 8 KB: one digit of 128 rows x 64 samples
constexpr int kSlot = 3 * kBox, kRing = 9;         // A box, two B boxes
constexpr int kRunKB = 288;                        // k-blocks per run: 7 * 2^14 * 18432 < 2^31
constexpr int kThreads = 320, kEpiWarps = 8;
constexpr int kSmem = kRing * kSlot + 1024 + 256 + kEpiWarps * kTile * (int)sizeof(double);
// kind::i8: D S32, A and B signed 8-bit, K-major
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) |
                            ((uint32_t)(kTile >> 4) << 24);
constexpr uint32_t kIdescHalf = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) |
                                ((uint32_t)(kTile >> 4) << 24);      // N = 128: tiles of one B panel

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// 16 columns of each of two accumulators
__device__ __forceinline__ void tmem_ld16x2(uint32_t ta, uint32_t tb, int* a, int* b)
{
    uint32_t r[32];
#define SCP3_LD16(k, t)                                                                                               \
    asm volatile(                                                                                                     \
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"      \
        : "=r"(r[k]), "=r"(r[k + 1]), "=r"(r[k + 2]), "=r"(r[k + 3]), "=r"(r[k + 4]), "=r"(r[k + 5]), "=r"(r[k + 6]), \
          "=r"(r[k + 7]), "=r"(r[k + 8]), "=r"(r[k + 9]), "=r"(r[k + 10]), "=r"(r[k + 11]), "=r"(r[k + 12]),          \
          "=r"(r[k + 13]), "=r"(r[k + 14]), "=r"(r[k + 15])                                                           \
        : "r"(t))
    SCP3_LD16(0, ta);
    SCP3_LD16(16, tb);
#undef SCP3_LD16
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; j++) a[j] = (int)r[j], b[j] = (int)r[16 + j];
}

// One thread owns an element of the partials, so its reductions keep their order
__device__ __forceinline__ void add_f64(double* p, double x)
{
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}

// Sweeps t = 0..3 take digits 1..sweep_digits(t); digit (1 = most significant) of step e
// of sweep t's chain.  Steps e - 1 and e add up to the sweep's larger sum, 9 - 2t, where
// in_large, else to the smaller, 8 - 2t, as the last digit and itself do.
__host__ __device__ __forceinline__ int sweep_digits(int t) { return t ? 8 - 2 * t : 7; }
__host__ __device__ __forceinline__ int chain_digit(int t, int e)
{
    if (t == 0) return (e & 1) ? 7 - (e >> 1) : 1 + (e >> 1);
    return (e & 1) ? (e + 1) >> 1 : 8 - 2 * t - (e >> 1);
}
__host__ __device__ __forceinline__ bool in_large(int t, int e) { return ((e & 1) != 0) == (t != 0); }

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Exponent e with every |value| of the row below 0.996 2^e, from the high word of the
// largest: seven balanced digits hold integers up to 0x7f7f7f7f7f7f7f = 0.9961 2^55
__device__ __forceinline__ int row_exp(int hi) { return max(((hi + 0x2100) >> 20) - 1022, -960); }
__device__ __forceinline__ double row_unit(int hi)     // value of one unit of the row's integers
{
    return hi >= 0x7ff00000 ? __longlong_as_double(0x7ff8000000000000ll) : pow2(row_exp(hi) - 55);
}

__device__ __forceinline__ double zero_unit(int hi) { return hi ? row_unit(hi) : 0.0; }

// ---------------------------------------------------------------- heavy samples
// The high word of a pass's limit of |x|: kLimitV or kLimitQ octaves above the geometric
// mean of kLimitSamples of its values.
constexpr int kLimitV = 9, kLimitQ = 4, kLimitSamples = 128, kLimitValues = 8;
constexpr int kLimitThreads = kLimitSamples * kLimitValues;

__device__ __forceinline__ int high_word(double x) { return __double2hiint(x) & 0x7fffffff; }

// Sample j of the ns that the limits are taken from: one at a scattered place in each of
// ns parts of a pass of k.  Not every (k / ns)-th: Sobol points a power of two apart agree in
// their first digits, so that a coordinate of all of them may lie next to zero (hexamer, 2^17
// samples from some first points on: 9.1 ms instead of 4.1, most samples being over the limit).
__host__ __device__ __forceinline__ long long limit_sample(int j, int ns, long long k)
{
    const long long lo = k * j / ns, hi = k * (j + 1) / ns;
    uint32_t h = (uint32_t)(j + 1) * 2654435769u;
    h = (h ^ (h >> 15)) * 2246822519u;
    return lo + (long long)((h ^ (h >> 13)) % (uint32_t)(hi - lo));
}

// Limits of V, q and dV/dq, kLimitValues of these per block, from limit_sample()s; zeros (padding samples among them) and values that are not finite do not count,
// and with nothing left any value but zero is over the limit.  The high word is the
// logarithm's piecewise linear form, so the sums are integers.  The blocks from lblocks on
// clear rowmax.
__global__ void __launch_bounds__(kLimitThreads) limits_kernel(const double* __restrict__ q, const double* __restrict__ v,
                                                               const double* __restrict__ vq, int nm, long long k,
                                                               int* __restrict__ limits, uint32_t* __restrict__ any,
                                                               int lblocks, int* __restrict__ rowmax, int rows)
{
    const int t = threadIdx.x;
    if ((int)blockIdx.x >= lblocks) {
        const int r = ((int)blockIdx.x - lblocks) * kLimitThreads + t;
        if (r < rows) rowmax[r] = 0;
        return;
    }
    __shared__ int sum[kLimitValues], count[kLimitValues];
    if (t < kLimitValues) sum[t] = count[t] = 0;
    if (blockIdx.x == 0 && t == 0) *any = 0;
    __syncthreads();
    const int ns = (int)min((long long)kLimitSamples, k), nq = 1 + nm + (vq ? nm : 0);
    const int j = t / kLimitValues, i = (int)blockIdx.x * kLimitValues + t % kLimitValues;
    int h = 0;
    if (j < ns && i < nq) {
        const long long s = limit_sample(j, ns, k);
        h = high_word(i == 0 ? v[s] : i <= nm ? q[s * nm + i - 1] : vq[s * nm + i - 1 - nm]);
    }
    if (h > 0 && h < 0x7ff00000) {
        atomicAdd(sum + t % kLimitValues, h >> 10);      // below 2^21 each
        atomicAdd(count + t % kLimitValues, 1);
    }
    __syncthreads();
    if (t < kLimitValues && i < nq) {
        const int octaves = i == 0 || i > nm ? kLimitV : kLimitQ;
        limits[i] = count[t] ? (int)min(((long long)(sum[t] / count[t]) << 10) + ((long long)octaves << 20), 0x7fefffffll) : 0;
    }
}

// Value of a table entry (kind | a << 4 | b << 6 | mode << 8) at the sample with
// coordinates q, potential V and derivatives vq
__device__ __forceinline__ double entry_value(uint32_t sp, const double* q, double V, const double* vq)
{
    const int kind = sp & 15, a = (sp >> 4) & 3, b = (sp >> 6) & 3, m = sp >> 8;
    if (kind == kOne) return 1.0;
    if (kind == kV) return V;
    return kind == kHo ? ho(a, q[m]) : stein_weight(a, kind == kKab ? b : 0, q[m], V, vq[m]);
}

struct HeavyArgs {
    const uint32_t *heavy, *any, *tspec, *xdesc;
    int dual, nm;
    const double *q, *v, *vq;
};

constexpr int kHeavy = 32;                         // samples added at a time

// Adds the heavy samples of a unit's blocks of 32, [w0, w1), to its partial P: the products
// of their row values in FP64, in the order of the samples, kHeavy at a time (8 x 4 elements
// of a 128 x 64 block per thread and round).  All threads of the CTA; buf: kHeavyBytes.
constexpr int kHeavyBytes = kHeavy * (kTile + kN) * (int)sizeof(double) + kHeavy * (int)sizeof(int);
__device__ __forceinline__ void add_heavy(const HeavyArgs& a, int4 ti, int w0, int w1, double* P, uint8_t* buf)
{
    double *sa = reinterpret_cast<double*>(buf), *sb = sa + kHeavy * kTile;     // [sample][row], [sample][column]
    int* list = reinterpret_cast<int*>(sb + kHeavy * kN);
    const int t = threadIdx.x, lane = t & 31, tx = t & 15, ty = t >> 4;
    int nh = 0;
    for (int wb = w0;; wb += 32) {
        const bool end = wb >= w1;
        const uint32_t word = wb + lane < w1 ? a.heavy[wb + lane] : 0u;
        uint32_t words = __ballot_sync(0xffffffffu, word != 0), bits = 0;
        int base = 0;
        for (;;) {                                 // every warp takes the same steps
            while (nh < kHeavy && (bits | words)) {
                if (!bits) {
                    const int l = __ffs((int)words) - 1;
                    words &= words - 1;
                    bits = __shfl_sync(0xffffffffu, word, l);
                    base = (wb + l) * 32;
                }
                if (t == 0) list[nh] = base + __ffs((int)bits) - 1;
                bits &= bits - 1;
                nh++;
            }
            if (nh < kHeavy && !(end && nh)) break;
            __syncthreads();
            for (int e = t; e < nh * (kTile + kN); e += kThreads) {
                const int h = e / (kTile + kN), c = e - h * (kTile + kN);
                if (c >= 2 * kTile && ti.z) continue;
                const int64_t s = list[h];
                int row = c < kTile ? ti.x + c : c < 2 * kTile ? ti.y + c - kTile : ti.w + c - 2 * kTile;
                const bool timesV = a.dual && row >= a.dual;
                if (timesV) row -= a.dual;
                const uint32_t d = a.xdesc[row];
                const double V = a.v[s], *q = a.q + s * a.nm, *vq = a.vq + s * a.nm;
                double val = 0.0;
                if (d != kZeroRow) {
                    val = entry_value(a.tspec[d & 1023u], q, V, vq);
                    if ((d >> 10) & 1023u) val *= entry_value(a.tspec[(d >> 10) & 1023u], q, V, vq);
                    if (d >> 20) val *= entry_value(a.tspec[d >> 20], q, V, vq);
                    if (timesV) val *= V;
                }
                if (c < kTile) sa[h * kTile + c] = val;
                else sb[h * kN + c - kTile] = val;
            }
            __syncthreads();
            if (t < 256)
#pragma unroll 1
                for (int c0 = 0; c0 < (ti.z ? kTile : kN); c0 += 64) {
                    double acc[8][4] = {};
#pragma unroll 1
                    for (int h = 0; h < nh; h++) {
                        double x[8], y[4];
#pragma unroll
                        for (int i = 0; i < 8; i++) x[i] = sa[h * kTile + tx + 16 * i];
#pragma unroll
                        for (int j = 0; j < 4; j++) y[j] = sb[h * kN + c0 + ty + 16 * j];
#pragma unroll
                        for (int i = 0; i < 8; i++)
#pragma unroll
                            for (int j = 0; j < 4; j++) acc[i][j] = fma(x[i], y[j], acc[i][j]);
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            add_f64(P + (size_t)(c0 + ty + 16 * j) * kTile + tx + 16 * i, acc[i][j]);
                }
            __syncthreads();
            nh = 0;
        }
        if (end) return;
    }
}

// Passes of few samples, in FP64 throughout.  CTA b < ntiles ranges: the unit of tile
// b % ntiles and sample range b / ntiles of `ranges`; `batch` samples at a time (few_batch),
// the table's entries, the rows' values and their products, 8 x 4 elements of a 128 x 128
// block per thread.  The other CTAs: the summed rows (from row ndesc of xdesc on), one per
// warp.
constexpr int kFewThreads = 512;

__global__ void __launch_bounds__(kFewThreads, 1)
    few_samples_kernel(const int4* __restrict__ tiles, int ntiles, int ranges, int k, int trows, int batch, int ndesc,
                       int nsum, double* __restrict__ sums, double* __restrict__ partial, int* __restrict__ filled,
                       HeavyArgs a)
{
    extern __shared__ __align__(16) double few[];  // [batch][rows], [batch][columns], [batch][table]
    const int u = blockIdx.x, t = threadIdx.x;
    if (u >= ntiles * ranges) {
        const int i = (u - ntiles * ranges) * (kFewThreads / 32) + (t >> 5);
        if (i >= nsum) return;
        const uint32_t d = a.xdesc[ndesc + i];
        const uint32_t sp[3] = {a.tspec[d & 1023u], a.tspec[(d >> 10) & 1023u], a.tspec[d >> 20]};
        double x = 0.0;
        for (int s = t & 31; s < k; s += 32) {
            const double V = a.v[s], *q = a.q + (int64_t)s * a.nm, *vq = a.vq + (int64_t)s * a.nm;
            x += entry_value(sp[0], q, V, vq) * entry_value(sp[1], q, V, vq) * entry_value(sp[2], q, V, vq);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((t & 31) == 0) sums[i] += x;
        return;
    }
    double *sa = few, *sb = sa + batch * kTile, *tab = sb + batch * kN;
    const int split = u / ntiles, lo = (int)((long long)k * split / ranges), hi = (int)((long long)k * (split + 1) / ranges);
    const int4 ti = tiles[u % ntiles];
    double* P = partial + (size_t)u * (size_t)(kTile * kN);
    bool store = filled[u] == 0;                   // the partial holds nothing yet
    // thread t forms row t of the tile's 128 + 256 (entry 0 is the constant 1)
    const int row = t < kTile ? ti.x + t : t < 2 * kTile ? ti.y + t - kTile : ti.w + t - 2 * kTile;
    const bool on = t < (ti.z ? 2 * kTile : kTile + kN), timesV = a.dual && row >= a.dual;
    const uint32_t d = on ? a.xdesc[timesV ? row - a.dual : row] : kZeroRow;
    double* out = t < kTile ? sa + t : sb + t - kTile;
    const int stride = t < kTile ? kTile : kN;
    const int tx = t & 15, ty = (t >> 4) & 15, c0 = t >> 8 << 6;
    for (int s = lo; s < hi; s += batch, store = false) {
        const int nh = min(batch, hi - s);
        for (int e = t; e < nh * trows; e += kFewThreads) {
            const int h = e / trows, i = e - h * trows;
            const int64_t o = (int64_t)(s + h) * a.nm;
            tab[e] = entry_value(a.tspec[i], a.q + o, a.v[s + h], a.vq + o);
        }
        __syncthreads();
        if (on)
#pragma unroll 4
            for (int h = 0; h < nh; h++) {
                const double* th = tab + h * trows;
                double val = 0.0;
                if (d != kZeroRow) {
                    val = th[d & 1023u] * th[(d >> 10) & 1023u] * th[d >> 20];
                    if (timesV) val *= a.v[s + h];
                }
                out[h * stride] = val;
            }
        __syncthreads();
#pragma unroll 1
        for (int c = c0; c < (ti.z ? kTile : kN); c += 128) {
            double acc[8][4] = {};
#pragma unroll 2
            for (int h = 0; h < nh; h++) {
                double x[8], y[4];
#pragma unroll
                for (int i = 0; i < 8; i++) x[i] = sa[h * kTile + tx + 16 * i];
#pragma unroll
                for (int j = 0; j < 4; j++) y[j] = sb[h * kN + c + ty + 16 * j];
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = fma(x[i], y[j], acc[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    double* p = P + (size_t)(c + ty + 16 * j) * kTile + tx + 16 * i;
                    if (store) *p = acc[i][j];
                    else add_f64(p, acc[i][j]);
                }
        }
        __syncthreads();
    }
    if (t == 0 && lo < hi) filled[u] = 1;          // read by all before the barriers above
}

__global__ void __launch_bounds__(kThreads, 1)
    contract_i8_kernel(const uint8_t* __restrict__ x, long long nkb_alloc, const int* __restrict__ rowmax,
                       const int4* __restrict__ tiles, int ntiles, int nsplit, int nkb_pass, int units,
                       double* __restrict__ partial, int* __restrict__ filled, int* __restrict__ err_flag, HeavyArgs ha)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kRing * kSlot);
    uint64_t* empty = full + kRing;
    uint64_t* acc_full = empty + kRing;
    uint64_t* acc_empty = acc_full + 1;
    uint64_t* drain = acc_empty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    double* cunit = reinterpret_cast<double*>(smem + kRing * kSlot + 256);    // [8 warps][128] units of a warp's columns

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto krange = [&](int u, int& lo, int& hi) {
        const int split = u / ntiles;
        lo = (int)((long long)split * nkb_pass / nsplit);
        hi = (int)((long long)(split + 1) * nkb_pass / nsplit);
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kEpiWarps);
        mbar_init(drain, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int slot = 0;
            uint32_t phase = 0, issued = 0, issued_phase = 0;   // bit per slot
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                int lo, hi;
                krange(u, lo, hi);
                const int4 ti = tiles[u % ntiles];
                const size_t rb = (size_t)nkb_alloc * (kDigits * kBox);
                const uint8_t* pa = x + (ti.x / kTile) * rb;
                const uint8_t* pb0 = x + (ti.y / kTile) * rb;
                const uint8_t* pb1 = x + (ti.w / kTile) * rb;
                for (int r0 = lo; r0 < hi && ok; r0 += kRunKB)
                    for (int t = 0; t < kSweeps && ok; t++)
                        for (int kb = r0; kb < min(hi, r0 + kRunKB) && ok; kb++)
                            for (int e = 0; e < sweep_digits(t); e++) {
                                if (!mbar_wait(empty + slot, phase ^ 1, abort)) {
                                    ok = false;
                                    break;
                                }
                                uint8_t* st = smem + slot * kSlot;
                                mbar_expect_tx(full + slot, ti.z ? 2 * kBox : kSlot);
                                const size_t o = ((size_t)kb * kDigits + chain_digit(t, e) - 1) * kBox;
                                bulk_load(st, pa + o, kBox, full + slot);
                                bulk_load(st + kBox, pb0 + o, kBox, full + slot);
                                if (!ti.z) bulk_load(st + 2 * kBox, pb1 + o, kBox, full + slot);
                                issued |= 1u << slot;
                                issued_phase = (issued_phase & ~(1u << slot)) | phase << slot;
                                if (++slot == kRing) {
                                    slot = 0;
                                    phase ^= 1;
                                }
                            }
            }
            if (*abort) {
                for (int s = 0; s < kRing; s++)
                    if ((issued >> s) & 1) {
                        volatile int never = 0;
                        mbar_wait(full + s, (issued_phase >> s) & 1, &never);
                    }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int slot = 0, use = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
                int lo, hi;
                krange(u, lo, hi);
                const uint32_t idesc = tiles[u % ntiles].z ? kIdescHalf : kIdesc;
                for (int r0 = lo; r0 < hi && ok; r0 += kRunKB)
                    for (int t = 0; t < kSweeps && ok; t++, use++) {
                        const int n = sweep_digits(t);
                        if (!mbar_wait(acc_empty, (use & 1) ^ 1, abort)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        for (int kb = r0; kb < min(hi, r0 + kRunKB) && ok; kb++) {
                            uint64_t pa = 0, pb = 0;
                            int prev = 0;
                            for (int e = 0; e < n; e++) {
                                if (!mbar_wait(full + slot, phase, abort)) {
                                    ok = false;
                                    break;
                                }
                                tc_fence_after();
                                uint8_t* st = smem + slot * kSlot;
                                const uint64_t ca = smem_desc64(st), cb = smem_desc64(st + kBox);
                                if (e) {
                                    const uint32_t d = tmem + (in_large(t, e) ? 0u : (uint32_t)kN);
                                    const uint32_t acc = kb != r0 || e > 2;
                                    mma_i8(d, pa, cb, idesc, acc);
                                    mma_i8(d, pa + 2, cb + 2, idesc, 1);
                                    mma_i8(d, ca, pb, idesc, 1);
                                    mma_i8(d, ca + 2, pb + 2, idesc, 1);
                                    mma_commit(empty + prev);
                                }
                                if (e == n - 1) {      // in sweep 3 the smaller sum's first
                                    mma_i8(tmem + kN, ca, cb, idesc, kb != r0 || n > 2);
                                    mma_i8(tmem + kN, ca + 2, cb + 2, idesc, 1);
                                    mma_commit(empty + slot);
                                }
                                pa = ca, pb = cb, prev = slot;
                                if (++slot == kRing) {
                                    slot = 0;
                                    phase ^= 1;
                                }
                            }
                        }
                        if (ok) mma_commit(acc_full);
                    }
            }
            mma_commit(drain);
            volatile int never = 0;
            mbar_wait(drain, 0, &never);
        }
    } else {
        // warp w reads TMEM lane quadrant w % 4 and column half (w - 2) / 4
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int row = quad * 32 + lane;
        int use = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            int lo, hi;
            krange(u, lo, hi);
            const int4 ti = tiles[u % ntiles];
            const double ra = zero_unit(rowmax[ti.x + row]);
            const bool empty = filled[u] == 0;     // the partial holds nothing yet
            // the warp's `span` columns of the tile from cb: a half, or of one panel a
            // quarter (dimer, 2^14 samples: with four warps at a panel's 128 columns 158.5 us
            // a pass on one card and 163.9 on another, with eight 156.2 and 153.3)
            const int span = ti.z ? kTile / 2 : kTile, cb = half * span;
            // their units; each warp its own copy: warps that met at a barrier here could wait
            // for one whose bounded wait has expired and that has left the loop
            double* cu = cunit + (warp - 2) * kTile;
            __syncwarp();
            for (int c = lane; c < span; c += 32)
                cu[c] = zero_unit(rowmax[(cb + c < kTile ? ti.y : ti.w) + ((cb + c) & (kTile - 1))]);
            __syncwarp();
            double* P = partial + (size_t)u * (size_t)(kTile * kN) + (size_t)cb * kTile + row;
            for (int r0 = lo; r0 < hi && ok; r0 += kRunKB)
                for (int t = 0; t < kSweeps; t++, use++) {
                    // warp-uniform: the TMEM loads below are warp-collective
                    if (!__all_sync(0xffffffffu, mbar_wait(acc_full, use & 1, abort))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const bool store = empty && r0 == lo && t == 0;
                    const double w = ra * pow2(8 * (5 + 2 * t));     // the larger digit sum: 2^(8 (14 - (9 - 2t)))
                    const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)cb;
                    // rows that are zero throughout (padding among them; unit 0) add
                    // nothing, unless to values that are not finite (unit NaN)
#pragma unroll 1
                    for (int c0 = 0; c0 < span; c0 += 16) {
                        double un[16];
                        bool any = false;
#pragma unroll
                        for (int j = 0; j < 16; j++) any |= (un[j] = cu[c0 + j]) != 0.0;
                        if (!any && !store) continue;
                        int a0[16], a1[16];
                        tmem_ld16x2(base + c0, base + kN + c0, a0, a1);
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            // |.| < 2^40: exact through the bits of 1.5 * 2^52
                            const long long d = ((long long)a1[j] << 8) + a0[j] + 0x4338000000000000ll;
                            const bool add = (w != 0.0 && un[j] != 0.0) || w != w || un[j] != un[j];
                            const double val = (__longlong_as_double(d) - 6755399441055744.0) * w * un[j];
                            double* e = P + (size_t)(c0 + j) * kTile;
                            if (store) *e = add ? val : 0.0;
                            else if (add) add_f64(e, val);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty);
                }
            // the others have read it: the last sweep's sums came after their arrivals for the
            // sweep before
            if (threadIdx.x == 64 && lo < hi) filled[u] = 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort) atomicExch(err_flag, 1);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
    if (*ha.any == 0 || *abort) return;
    // the ring is free: every copy has been consumed
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        int lo, hi;
        krange(u, lo, hi);
        add_heavy(ha, tiles[u % ntiles], 2 * lo, 2 * hi, partial + (size_t)u * (size_t)(kTile * kN), smem);
    }
}

// ---------------------------------------------------------------- the operand
// A CTA tabulates the entries the rows use for 32 samples in FP64, one (mode, sample)
// per thread at a time; thread (g, r) then takes 16 of the samples (half g; the scan 8)
// of rows 4r .. 4r+3 and on in steps of the CTA: consecutive rows mostly share their
// first factor, read once.  Table entry i, 16-byte chunk c (0..7) of half g lies at chunk
// 8 g + (c ^ (i / 4 & 7)), and half 1 reads its chunks in the order c ^ 4: the eight
// lanes of a 16-byte phase hold rows four apart, whose entries mostly are four apart too,
// and so meet no bank conflict (with the key i & 7 they did: 2^15 samples of the hexamer
// gradient's digits 381 us, now 308).
constexpr int kS = 32, kScanThreads = 512, kDigitThreads = 256;
constexpr int kModeKinds = 12;     // h1 h2 h3 K10 K20 K30 K11 K12 K13 K22 K23 K33

__device__ __forceinline__ void put_entry(double* tab, int r, int l, double val)
{
    if (r >= 0) tab[r * kS + ((((l >> 4) << 3) + (((l >> 1) & 7) ^ ((r >> 2) & 7))) << 1) + (l & 1)] = val;
}

// entries[m][kind]: table entry or -1; v_entry: V's, or -1.  kFlag: the samples over a
// limit are marked in *heavy (shared, cleared).
template <int kThreadsPerCta, bool kFlag>
__device__ __forceinline__ void build_table(const int16_t* __restrict__ entries, int v_entry, int nm,
                                            const double* __restrict__ q, const double* __restrict__ v,
                                            const double* __restrict__ vq, int64_t s0, double* tab,
                                            const int* __restrict__ limits = nullptr, uint32_t* heavy = nullptr)
{
    const int l = threadIdx.x & 31;
    const int64_t s = s0 + l;
    const double V = v[s];
    bool over = kFlag && high_word(V) > __ldg(limits);
    if (threadIdx.x < kS) put_entry(tab, 0, l, 1.0);
    else if (threadIdx.x < 2 * kS) put_entry(tab, v_entry, l, V);
    for (int m = threadIdx.x >> 5; m < nm; m += kThreadsPerCta / 32) {
        const double x = __ldg(q + s * nm + m);
        if (kFlag) over |= high_word(x) > __ldg(limits + 1 + m);
        const int16_t* e = entries + m * kModeKinds;
#pragma unroll
        for (int a = 1; a <= 3; a++) put_entry(tab, e[a - 1], l, ho(a, x));
        if (!vq) continue;
        const double Vm = __ldg(vq + s * nm + m);
        if (kFlag) over |= high_word(Vm) > __ldg(limits + 1 + nm + m);
#pragma unroll
        for (int a = 1; a <= 3; a++) {
            put_entry(tab, e[2 + a], l, stein_weight(a, 0, x, V, Vm));
#pragma unroll
            for (int b = a; b <= 3; b++) {
                const int k = a == 1 ? 5 + b : a == 2 ? 7 + b : 11;      // K1b at 6.., K2b at 9.., K33 at 11
                if (e[k] >= 0) put_entry(tab, e[k], l, stein_weight(a, b, x, V, Vm));
            }
        }
    }
    if (kFlag) {
        const uint32_t bits = __ballot_sync(0xffffffffu, over);
        if (bits && l == 0) atomicOr(heavy, bits);
    }
}

// the 16 values of half g of entry i; register pair k holds samples 2 (k ^ 4 g), + 1
__device__ __forceinline__ void read16(const double* tab, uint32_t i, int g, double* o)
{
    const double2* t = reinterpret_cast<const double2*>(tab + (size_t)i * kS) + 8 * g;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const double2 d = t[(k ^ (g << 2)) ^ ((i >> 2) & 7)];
        o[2 * k] = d.x, o[2 * k + 1] = d.y;
    }
}

__device__ __forceinline__ void mul16(const double* tab, uint32_t i, int g, double* o)
{
    const double2* t = reinterpret_cast<const double2*>(tab + (size_t)i * kS) + 8 * g;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const double2 d = t[(k ^ (g << 2)) ^ ((i >> 2) & 7)];
        o[2 * k] *= d.x, o[2 * k + 1] *= d.y;
    }
}

// the scan's share: the 8 samples of quarter g (half g / 2); the second half reads its
// chunks in another order, so that two rows' four quarters meet no bank conflict
template <bool kMul>
__device__ __forceinline__ void read8(const double* tab, uint32_t i, int g, double* o)
{
    const double2* t = reinterpret_cast<const double2*>(tab + (size_t)i * kS) + 8 * (g >> 1);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 d = t[(4 * (g & 1) + (k ^ (g & 2))) ^ ((i >> 2) & 7)];
        if (kMul) o[2 * k] *= d.x, o[2 * k + 1] *= d.y;
        else o[2 * k] = d.x, o[2 * k + 1] = d.y;
    }
}

// zero in every table entry at the marked samples
__device__ __forceinline__ void drop_samples(double* tab, int trows, uint32_t marked)
{
#pragma unroll 1
    for (int e = threadIdx.x; e < trows * kS; e += blockDim.x)
        if ((marked >> (e & 31)) & 1) put_entry(tab, e >> 5, e & 31, 0.0);
}

// Row values of `d` (entry indices); `fa` caches the first factor of entry `pia`.
__device__ __forceinline__ void row16(const double* tab, uint32_t d, int g, uint32_t& pia, double* fa, double* o)
{
    const uint32_t ia = d & 1023u, ib = (d >> 10) & 1023u, ic = d >> 20;
    if (ia != pia) {
        read16(tab, ia, g, fa);
        pia = ia;
    }
#pragma unroll
    for (int k = 0; k < 16; k++) o[k] = fa[k];
    if (ib) mul16(tab, ib, g, o);
    if (ic) mul16(tab, ic, g, o);
}

__device__ __forceinline__ int max_hi8(const double* o)
{
    int m = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) m = max(m, __double2hiint(o[k]) & 0x7fffffff);
    return m;
}

// Largest |value| of every row over the pass's samples within the limits (its high word;
// the others are marked in heavy), and the sums of the summed rows over all of them.  CTA (x, y): sample blocks x, x + gridDim.x, ..., rows of chunk y.
// dual: row dual + r is V times row r; the summed rows follow the described ones, and
// xdesc ends on a multiple of four rows.
__global__ void __launch_bounds__(kScanThreads, 1)
    scan_kernel(const int16_t* __restrict__ entries, int v_entry, int trows, const uint32_t* __restrict__ xdesc,
                int ndesc, int dual, int nsum, int per, int nm, const double* __restrict__ q,
                const double* __restrict__ v, const double* __restrict__ vq, int nblk, int* __restrict__ rowmax,
                double* __restrict__ spart, const int* __restrict__ limits, uint32_t* __restrict__ heavy,
                uint32_t* __restrict__ any)
{
    extern __shared__ __align__(16) double tab[];      // [trows][32], then [per] doubles and two words
    double* keep = tab + (size_t)trows * kS;           // (max, max of V times the row) or the sum
    int2* mx = reinterpret_cast<int2*>(keep);
    uint32_t* marks = reinterpret_cast<uint32_t*>(keep + per);     // of this block and of the next
    if (threadIdx.x < 2) marks[threadIdx.x] = 0;
    const int r0 = blockIdx.y * per, r1 = min(ndesc + nsum, r0 + per);
    for (int r = threadIdx.x; r < r1 - r0; r += kScanThreads) keep[r] = 0.0;
    const int g = threadIdx.x & 3, rl = threadIdx.x >> 2, w0 = 4 * (rl & 7);     // w0: rows below in the warp
    for (int b = blockIdx.x, odd = 0; b < nblk; b += gridDim.x, odd ^= 1) {
        __syncthreads();
        build_table<kScanThreads, true>(entries, v_entry, nm, q, v, vq, (int64_t)b * kS, tab, limits, marks + odd);
        __syncthreads();
        const uint32_t hw = marks[odd];
        if (threadIdx.x == 0) {
            marks[odd ^ 1] = 0;                        // read by all before the barrier above
            if (blockIdx.y == 0) heavy[b] = hw;
            if (hw) *any = 1;
        }
        // one round over the rows; with marked samples first the summed rows, then, these
        // samples dropped, the others
#pragma unroll 1
        for (int part = 0; part < (hw ? 2 : 1); part++) {
            const int ra = hw && part == 0 ? max(r0, ndesc) : r0, re = part ? min(r1, ndesc) : r1;
            if (part) {
                __syncthreads();
                drop_samples(tab, trows, hw);
                __syncthreads();
            }
            double vv[8], fa[8];
            if (dual) read8<false>(tab, v_entry, g, vv);
            // whole warps take the same number of rounds: the quarters meet in shuffles
            for (int rb = ra + 4 * rl; rb - w0 < re; rb += kScanThreads) {
                uint32_t pia = kZeroRow;
                uint32_t d4[4] = {kZeroRow, kZeroRow, kZeroRow, kZeroRow};
                if (rb < re) *reinterpret_cast<uint4*>(d4) = __ldg(reinterpret_cast<const uint4*>(xdesc + rb));
                const bool sum = rb - w0 + 32 > ndesc;     // the warp holds summed rows
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int row = rb + u;
                    const uint32_t d = d4[u];
                    double o[8];
                    int m = 0, mv = 0;
                    double t = 0.0;
                    if (d != kZeroRow) {
                        const uint32_t ia = d & 1023u, ib = (d >> 10) & 1023u, ic = d >> 20;
                        if (ia != pia) {
                            read8<false>(tab, ia, g, fa);
                            pia = ia;
                        }
#pragma unroll
                        for (int k = 0; k < 8; k++) o[k] = fa[k];
                        if (ib) read8<true>(tab, ib, g, o);
                        if (ic) read8<true>(tab, ic, g, o);
                        if (row < ndesc) {
                            m = max_hi8(o);
                            if (dual) {
#pragma unroll
                                for (int k = 0; k < 8; k++) o[k] *= vv[k];
                                mv = max_hi8(o);
                            }
                        } else {
                            t = ((o[0] + o[1]) + (o[2] + o[3])) + ((o[4] + o[5]) + (o[6] + o[7]));
                        }
                    }
                    if (sum) {
                        t += __shfl_xor_sync(0xffffffffu, t, 1);
                        t += __shfl_xor_sync(0xffffffffu, t, 2);
                        if (g == 0 && row >= ndesc && d != kZeroRow) keep[row - r0] += t;
                        if (rb - w0 >= ndesc) continue;
                    }
                    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
                    m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
                    if (dual) {
                        mv = max(mv, __shfl_xor_sync(0xffffffffu, mv, 1));
                        mv = max(mv, __shfl_xor_sync(0xffffffffu, mv, 2));
                    }
                    if (g == 0 && row < ndesc && d != kZeroRow)
                        mx[row - r0] = make_int2(max(mx[row - r0].x, m), max(mx[row - r0].y, mv));
                }
            }
        }
    }
    __syncthreads();
    for (int r = r0 + threadIdx.x; r < r1; r += kScanThreads) {
        if (r >= ndesc) {
            spart[(size_t)blockIdx.x * nsum + (r - ndesc)] = keep[r - r0];
        } else {
            if (mx[r - r0].x) atomicMax(rowmax + r, mx[r - r0].x);
            if (dual && mx[r - r0].y) atomicMax(rowmax + dual + r, mx[r - r0].y);
        }
    }
}

// sums[i] += the scan blocks' partials: warp w of a CTA adds the blocks w, w + 8, ...
// of 32 sums in order, the eight warp sums are then added in order
__global__ void __launch_bounds__(256) add_sums_kernel(const double* __restrict__ spart, int nsum, int nblocks,
                                                       double* __restrict__ sums)
{
    __shared__ double ws[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    double t = 0.0;
    if (i < nsum)
        for (int b = w; b < nblocks; b += 8) t += spart[(size_t)b * nsum + i];
    ws[w][lane] = t;
    __syncthreads();
    if (w || i >= nsum) return;
#pragma unroll
    for (int k = 1; k < 8; k++) t += ws[k][lane];
    sums[i] += t;
}

// The seven digits of 16 values (register order of read16) into a row's 16-byte
// chunk of each digit's box: the bytes of x + sum 128 256^b, each xor 0x80.
__device__ __forceinline__ void put_digits(const double* o, int hi, int g, uint8_t* p)
{
    const double inv = hi >= 0x7ff00000 ? 0.0 : pow2(55 - row_exp(hi));
    uint32_t w[kDigits][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        uint32_t lo[4], h[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const long long t = __double2ll_rn(o[4 * j + k] * inv) + 0x0080808080808080ll;
            lo[k] = (uint32_t)t ^ 0x80808080u;
            h[k] = (uint32_t)(t >> 32) ^ 0x00808080u;
        }
        // 4 x 4 byte transposes: byte b of the four values becomes one word
        const uint32_t l01 = __byte_perm(lo[0], lo[1], 0x5140), l23 = __byte_perm(lo[2], lo[3], 0x5140);
        const uint32_t m01 = __byte_perm(lo[0], lo[1], 0x7362), m23 = __byte_perm(lo[2], lo[3], 0x7362);
        w[6][j] = __byte_perm(l01, l23, 0x5410);
        w[5][j] = __byte_perm(l01, l23, 0x7632);
        w[4][j] = __byte_perm(m01, m23, 0x5410);
        w[3][j] = __byte_perm(m01, m23, 0x7632);
        const uint32_t h01 = __byte_perm(h[0], h[1], 0x5140), h23 = __byte_perm(h[2], h[3], 0x5140);
        const uint32_t n01 = __byte_perm(h[0], h[1], 0x7362), n23 = __byte_perm(h[2], h[3], 0x7362);
        w[2][j] = __byte_perm(h01, h23, 0x5410);
        w[1][j] = __byte_perm(h01, h23, 0x7632);
        w[0][j] = __byte_perm(n01, n23, 0x5410);
    }
#pragma unroll
    for (int i = 0; i < kDigits; i++)     // half 1 holds its samples as 8..15, 0..7
        *reinterpret_cast<uint4*>(p + i * kBox) =
            g ? make_uint4(w[i][2], w[i][3], w[i][0], w[i][1]) : make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// CTA (x, y): the 32 samples of block x, rows of chunk y (`per` rows, a multiple of 4).
// Two kernels, and V read from the table like any factor: with V's 16 values kept in
// registers too it spilled (hexamer, 2^16 samples direct 264 us, now 229, the operand's
// 1.1 GB alone 172; gradient, 2^15 samples 309 us, now 270, of 206).
template <bool kDual>
__global__ void __launch_bounds__(kDigitThreads, 2)
    digits_kernel(const int16_t* __restrict__ entries, int v_entry, int trows, const uint32_t* __restrict__ xdesc,
                  int ndesc, int dual, int per, int nm, const double* __restrict__ q, const double* __restrict__ v,
                  const double* __restrict__ vq, const int* __restrict__ rowmax, const uint32_t* __restrict__ heavy,
                  int64_t nkb_alloc, uint8_t* __restrict__ x)
{
    extern __shared__ __align__(16) double tab[];
    build_table<kDigitThreads, false>(entries, v_entry, nm, q, v, vq, (int64_t)blockIdx.x * kS, tab);
    __syncthreads();
    if (const uint32_t hw = __ldg(heavy + blockIdx.x)) {       // their digits are zero: every row's first factor is
        drop_samples(tab, trows, hw);
        __syncthreads();
    }
    const int g = threadIdx.x & 1, rl = threadIdx.x >> 1;
    const int64_t kb = blockIdx.x >> 1;
    const int c = ((blockIdx.x & 1) << 1) | g;          // 16-byte chunk of the box rows
    auto box = [&](int row) {
        const int rin = row & (kTile - 1);
        return x + ((size_t)(row / kTile) * nkb_alloc + kb) * (kDigits * kBox) + rin * kKB +
               ((c ^ ((rin >> 1) & 3)) << 4);
    };
    double fa[16];
    const int r0 = blockIdx.y * per, r1 = min(ndesc, r0 + per);
    for (int rb = r0 + 4 * rl; rb < r1; rb += 2 * kDigitThreads) {
        uint32_t pia = kZeroRow;
        uint4 d4 = __ldg(reinterpret_cast<const uint4*>(xdesc + rb));
        int4 m4 = __ldg(reinterpret_cast<const int4*>(rowmax + rb)), w4 = make_int4(0, 0, 0, 0);
        if (kDual) w4 = __ldg(reinterpret_cast<const int4*>(rowmax + dual + rb));
#pragma unroll 1
        for (int u = 0; u < 4; u++) {
            const int row = rb + u, hi = m4.x, hiw = w4.x;
            const uint32_t d = d4.x;
            d4 = make_uint4(d4.y, d4.z, d4.w, kZeroRow);
            m4 = make_int4(m4.y, m4.z, m4.w, 0), w4 = make_int4(w4.y, w4.z, w4.w, 0);
            if (d == kZeroRow) continue;
            double o[16];
            row16(tab, d, g, pia, fa, o);
            put_digits(o, hi, g, box(row));
            if (kDual) {
                mul16(tab, v_entry, g, o);
                put_digits(o, hiw, g, box(dual + row));
            }
        }
    }
}

size_t digits_smem(const Plan& p) { return sizeof(double) * (size_t)p.trows * kS; }
size_t scan_smem(const Plan& p) { return digits_smem(p) + sizeof(double) * (size_t)p.scan_per + 2 * sizeof(uint32_t); }
int described(const Plan& p) { return p.dual ? p.dual : p.rows; }
int scan_chunks(const Plan& p) { return (described(p) + p.nsum + p.scan_per - 1) / p.scan_per; }
int scan_blocks(const Plan& p, int64_t k)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>(k / kS, p.sms / scan_chunks(p)));
}

}  // namespace

void direct_rows(const std::vector<uint32_t>& desc, int nm, int nb_pad, std::vector<uint32_t>& tspec,
                 std::vector<uint32_t>& xdesc)
{
    std::vector<uint32_t> at((size_t)4 * nm, 0);      // entry of level l of mode m
    tspec = {kOne, kV};
    xdesc.assign(nb_pad, kZeroRow);
    for (size_t r = 0; r < desc.size(); r++) {
        int mm[3], ll[3];
        const int k = decode(desc[r], mm, ll);
        uint32_t d = 0;
        for (int a = 0; a < k; a++) {
            uint32_t& e = at[(size_t)4 * mm[a] + ll[a]];
            if (!e) {
                e = (uint32_t)tspec.size();
                tspec.push_back(kHo | (uint32_t)ll[a] << 4 | (uint32_t)mm[a] << 8);
            }
            d |= e << (10 * a);
        }
        xdesc[r] = d;
    }
}

constexpr int kScanStep = kScanThreads, kMinScanRows = 2048;     // rows a scan CTA keeps a value of, at least
int table_room() { return (int)((227 * 1024 - sizeof(double) * kMinScanRows) / (sizeof(double) * kS)); }

// Clocks of a pass: waves of units, each 136 per sample (34 products of 128 clocks per
// 32 samples) and four drains of 10,000; and 150 a unit for its partial, stored by the first
// drain and summed at read-out.  With 75 (the read-out's traffic alone) bases of one
// and two tiles get more splits and lose: 8192 samples of one tile 122 splits 143.4 us, 86
// (as chosen) 141.0; 4096 of two tiles 61 splits 144.6 and 147.4 us, 43 143.4 and 145.9.
int plan_splits(int ntiles, int64_t chunk, int sms)
{
    int best_m = 1;
    double best = 1e300;
    for (int m = 1; m <= sms; m++) {
        const int64_t units = (int64_t)ntiles * m;
        if (m > 1 && units * kTile * kN * 8 > (4ll << 30)) break;
        const double cost = (double)((units + sms - 1) / sms) * (136.0 * chunk / m + 40000.0) + 150.0 * units;
        if (cost < best) best = cost, best_m = m;
    }
    return best_m;
}

int create(Plan& p, const std::vector<uint32_t>& tspec, const std::vector<uint32_t>& xdesc, int rows, int dual,
           int nsum, int nm, const std::vector<int4>& tiles, int nsplit, int64_t chunk, int sms)
{
    p = Plan{};
    p.rows = rows, p.dual = dual, p.nsum = nsum, p.nm = nm, p.trows = (int)tspec.size();
    p.ntiles = (int)tiles.size(), p.nsplit = nsplit, p.sms = sms;
    p.chunk = chunk, p.nkb = chunk / kKB;
    if (rows % kTile || chunk % kKB || (int)xdesc.size() != described(p) + nsum || p.trows > kMaxTable)
        return fail(SCP3GPU_ERR_ARG, "contract_i8: operand not tiled");
    if (p.trows > table_room()) return fail(SCP3GPU_ERR_ARG, "contract_i8: too many modes for the expansion's table");
    // entry of each kind of each mode
    std::vector<int16_t> entries((size_t)nm * kModeKinds, -1);
    p.v_entry = -1;
    for (int i = 0; i < p.trows; i++) {
        const int kind = tspec[i] & 15, a = (tspec[i] >> 4) & 3, b = (tspec[i] >> 6) & 3, m = tspec[i] >> 8;
        if (kind == kV) p.v_entry = i;
        else if (kind != kOne)
            entries[(size_t)m * kModeKinds + (kind == kHo ? a - 1 : kind == kKa0 ? 2 + a : a == 1 ? 5 + b : a == 2 ? 7 + b : 11)] =
                (int16_t)i;
    }
    std::vector<uint32_t> desc4 = xdesc;
    desc4.resize((xdesc.size() + 3) / 4 * 4, kZeroRow);
    const size_t ndesc4 = desc4.size();
    desc4.insert(desc4.end(), tspec.begin(), tspec.end());
    // rows per scan CTA: what fits beside the table, in whole trips of the CTA
    const int room = (int)((227 * 1024 - digits_smem(p) - 2 * sizeof(uint32_t)) / sizeof(double)) / kScanStep * kScanStep;
    p.scan_per = std::min(room, ((int)xdesc.size() + kScanStep - 1) / kScanStep * kScanStep);
    const size_t xbytes = (size_t)rows * chunk * kDigits;
    int rc;
    if ((rc = upload(&p.entries, entries.data(), entries.size())) || (rc = upload(&p.xdesc, desc4.data(), desc4.size())) ||
        (rc = upload(&p.tiles, tiles.data(), tiles.size())) || (rc = dalloc(&p.x, xbytes)) ||
        (rc = dalloc(&p.rowmax, (size_t)rows + 2 * nm + 1 + chunk / kS + 1)) || (rc = dalloc(&p.filled, (size_t)p.nsplit * p.ntiles + 1)) ||
        (rc = dalloc(&p.partial, (size_t)p.nsplit * p.ntiles * kTile * kN)) ||
        (nsum && ((rc = dalloc(&p.spart, (size_t)scan_blocks(p, chunk) * nsum)) || (rc = dalloc(&p.sums, (size_t)nsum))))) {
        destroy(p);
        return rc;
    }
    p.err = p.filled + (size_t)p.nsplit * p.ntiles;
    for (const int4& t : tiles) p.half_tiles += t.z != 0;
    p.tspec = p.xdesc + ndesc4;
    p.limits = p.rowmax + rows;
    p.heavy = reinterpret_cast<uint32_t*>(p.limits + 2 * nm + 1);
    // padding rows are never written: zero the row blocks that hold any
    const size_t block = (size_t)p.nkb * kDigits * kBox;
    for (int rb = 0; rb < described(p) / kTile; rb++)
        if (std::find(xdesc.begin() + rb * kTile, xdesc.begin() + (rb + 1) * kTile, kZeroRow) != xdesc.begin() + (rb + 1) * kTile) {
            SCP3_CUDA(cudaMemset(p.x + rb * block, 0, block));
            if (dual) SCP3_CUDA(cudaMemset(p.x + (rb + dual / kTile) * block, 0, block));
        }
    SCP3_CUDA(cudaMemset(p.filled, 0, sizeof(int) * ((size_t)p.nsplit * p.ntiles + 1)));
    return SCP3GPU_OK;
}

void destroy(Plan& p)
{
    void* ptrs[] = {p.x, p.rowmax, p.entries, p.xdesc, p.tiles, p.partial, p.spart, p.sums, p.filled};
    for (void* q : ptrs)
        if (q) cudaFree(q);
    p = Plan{};
}

int zero(const Plan& p, cudaStream_t s)
{
    if (p.nsum) SCP3_CUDA(cudaMemsetAsync(p.sums, 0, sizeof(double) * (size_t)p.nsum, s));
    SCP3_CUDA(cudaMemsetAsync(p.filled, 0, sizeof(int) * ((size_t)p.nsplit * p.ntiles + 1), s));     // and err
    return SCP3GPU_OK;
}

// Samples that few_samples_kernel takes at a time, and its shared memory
static size_t few_smem(const Plan& p, int batch) { return sizeof(double) * (size_t)batch * (kTile + kN + p.trows); }
static int few_batch(const Plan& p) { return few_smem(p, 32) <= 227 * 1024 ? 32 : 16; }

// Sample ranges (of at least 8) of a pass of k samples in FP64 (few_samples_kernel), 0 where
// the digits are faster.  Both sides in clocks, fitted to passes of 64 to 8192 samples of 28
// bases: an SM's units in turn, 1400 a sample and tile (910 in one of a single B panel),
// beside the summed rows, 27 a sample; against limits, scan and digits, then waves of units
// with four drains.  The choice was slower than the other by more than 6 % in four of 224.
// Time of a whole pass with the digits always and as chosen: dimer, one tile, 256 samples
// 73.0 and 35.2 us (with FP64 tiles, before the digits, 49.7), 4096 72.9 and 41.9 (70.7); a
// trimer with triples, three tiles, 1024 90.3 and 48.2 (64.3); hexamer, 28 tiles, 256 105.3
// and 78.9 (98.1), 512 111.7 and 116.3 (115.3) and so left to the digits.
int few_ranges(int ntiles, int half_tiles, int nsplit, int nsum, int sms, int64_t k)
{
    const int64_t ranges = std::max<int64_t>(1, std::min<int64_t>(nsplit, k / 8));
    auto per_sm = [&](int64_t units) { return (double)((units + sms - 1) / sms); };
    const double tile = 1400.0 - 490.0 * half_tiles / ntiles;
    const double few = 12000.0 + std::max(per_sm(ntiles * ranges) * (5000.0 + tile * k / ranges), nsum ? 27.0 * k : 0.0);
    const double digits = (half_tiles == ntiles ? 35000.0 : 73000.0) +
                          per_sm((int64_t)ntiles * nsplit) * (50000.0 + 136.0 * k / nsplit);
    return few < digits ? (int)ranges : 0;
}
static int few_ranges(const Plan& p, int64_t k) { return few_ranges(p.ntiles, p.half_tiles, p.nsplit, p.nsum, p.sms, k); }

int prepare(const Plan& p, const double* q, const double* v, const double* vq, int64_t k, cudaStream_t s)
{
    if (k <= 0) return SCP3GPU_OK;
    if (k > p.chunk || k % kKB) return fail(SCP3GPU_ERR_ARG, "contract_i8: pass not in k-blocks");
    if (few_ranges(p, k)) return SCP3GPU_OK;       // contract() forms the rows itself
    const int ndesc = described(p), nblk = (int)(k / kS), nx = scan_blocks(p, k);
    uint32_t* any = p.heavy + p.chunk / kS;
    const int lblocks = (1 + p.nm * (vq ? 2 : 1) + kLimitValues - 1) / kLimitValues;
    limits_kernel<<<lblocks + (p.rows + kLimitThreads - 1) / kLimitThreads, kLimitThreads, 0, s>>>(
        q, v, vq, p.nm, k, p.limits, any, lblocks, p.rowmax, p.rows);
    SCP3_CUDA(cudaGetLastError());
    const auto digits = p.dual ? digits_kernel<true> : digits_kernel<false>;
    if (int rc = allow_smem(scan_kernel)) return rc;
    if (int rc = allow_smem(digits)) return rc;
    scan_kernel<<<dim3(nx, scan_chunks(p)), kScanThreads, scan_smem(p), s>>>(p.entries, p.v_entry, p.trows, p.xdesc,
                                                                            ndesc, p.dual, p.nsum, p.scan_per, p.nm, q,
                                                                            v, vq, nblk, p.rowmax, p.spart,
                                                                            p.limits, p.heavy, any);
    SCP3_CUDA(cudaGetLastError());
    if (p.nsum) add_sums_kernel<<<(p.nsum + 31) / 32, 256, 0, s>>>(p.spart, p.nsum, nx, p.sums);
    SCP3_CUDA(cudaGetLastError());
    // all rows of a block in one CTA (the table is built once) where there are blocks enough
    const int want = std::max(1, 4 * p.sms / nblk);
    const int per = std::max(kDigitThreads, ((ndesc + want - 1) / want + 3) / 4 * 4);
    digits<<<dim3(nblk, (ndesc + per - 1) / per), kDigitThreads, digits_smem(p), s>>>(
        p.entries, p.v_entry, p.trows, p.xdesc, ndesc, p.dual, per, p.nm, q, v, vq, p.rowmax, p.heavy, p.nkb, p.x);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

int contract(const Plan& p, const double* q, const double* v, const double* vq, int64_t k, cudaStream_t s)
{
    if (k <= 0) return SCP3GPU_OK;
    const int units = p.ntiles * p.nsplit;
    const HeavyArgs ha{p.heavy, p.heavy + p.chunk / kS, p.tspec, p.xdesc, p.dual, p.nm, q, v, vq};
    if (const int ranges = few_ranges(p, k)) {
        if (int rc = allow_smem(few_samples_kernel)) return rc;
        constexpr int kWarps = kFewThreads / 32;
        const int batch = few_batch(p);
        few_samples_kernel<<<p.ntiles * ranges + (p.nsum + kWarps - 1) / kWarps, kFewThreads, few_smem(p, batch), s>>>(
            p.tiles, p.ntiles, ranges, (int)k, p.trows, batch, described(p), p.nsum, p.sums, p.partial, p.filled, ha);
        SCP3_CUDA(cudaGetLastError());
        return SCP3GPU_OK;
    }
    if (int rc = allow_smem(contract_i8_kernel)) return rc;
    contract_i8_kernel<<<std::min(units, p.sms), kThreads, kSmem, s>>>(p.x, (long long)p.nkb, p.rowmax, p.tiles, p.ntiles,
                                                                       p.nsplit, (int)(k / kKB), units, p.partial, p.filled, p.err, ha);
    SCP3_CUDA(cudaGetLastError());
    return SCP3GPU_OK;
}

int check(const Plan& p, cudaStream_t s)
{
    int err = 0;
    SCP3_CUDA(cudaMemcpyAsync(&err, p.err, sizeof(int), cudaMemcpyDeviceToHost, s));
    SCP3_CUDA(cudaStreamSynchronize(s));
    return err ? fail(SCP3GPU_ERR_TIMEOUT, "integer contraction: a bounded pipeline wait expired") : SCP3GPU_OK;
}

}  // namespace i8
}  // namespace scp3

// Host-only view of the limits' samples, for tests: sample j of a pass of k, -1 past the last.
extern "C" int64_t scp3gpu_internal_limit_sample(int j, int64_t k)
{
    const int ns = (int)std::min<int64_t>(scp3::i8::kLimitSamples, k);
    return j < 0 || j >= ns ? -1 : scp3::i8::limit_sample(j, ns, k);
}

// Host-only view of the rule for passes of few samples, for tests: the sample ranges of a
// pass of k samples in FP64, 0 for the digits.
extern "C" int scp3gpu_internal_few_ranges(int ntiles, int half_tiles, int nsplit, int nsum, int sms, int64_t k)
{
    return ntiles < 1 || nsplit < 1 || sms < 1 || k < 1 ? -1 : scp3::i8::few_ranges(ntiles, half_tiles, nsplit, nsum, sms, k);
}

// Host-only view of the contraction's digit sweeps, for tests: the digit of step e of
// sweep t (0..3) and whether its sum with step e - 1 is the sweep's larger one; returns
// the digits of the sweep, negative on bad arguments.
extern "C" int scp3gpu_internal_digit_chain(int t, int e, int* digit, int* large)
{
    using namespace scp3::i8;
    if (t < 0 || t > 3 || e < 0 || e >= sweep_digits(t) || !digit || !large) return -1;
    *digit = chain_digit(t, e);
    *large = in_large(t, e);
    return sweep_digits(t);
}
