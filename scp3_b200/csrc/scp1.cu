// SCP1 thermal averages (SCP1.cpp:34-90, SCP1::average) on the GPU.
//
// For Sobol points i of the unscrambled sequence at offset `skip` (dimension
// dim = 9 nw, every Cartesian coordinate), each sample is
//
//   y  = std_normal(dim) % sqrt(d)                       (SCP1.cpp:54-58)
//   dq = isqrtM_U y,   r = bohr (q + dq)                  (SCP1.cpp:60-61)
//   V  = pes(r) / autokcal,  g = dV/dr * bohr / autokcal  (SCP1.cpp:62-63)
//
// and the call returns the sums over its points of V, g and g dq^T (the
// reference's per-rank partials before its MPI_Allreduce, SCP1.cpp:65-80).
//
// Two kernels per chunk of samples:
//   scp1_samples_kernel   (sampling.cu, beside the potentials' constant tables)
//                         four samples per warp (contiguous, balanced ranges
//                         per warp, Gray-code Sobol walk), isqrtM_U staged in
//                         shared memory, the potential's energy and gradient
//                         (the same warp code as the gradient estimator); writes
//                         V, g and dq per sample.
//   scp1_reduce_kernel    R = sum_s [g_s, V_s] [dq_s, 1]^T, a (dim+1)^2 grid of
//                         FP64 sums: every block owns a fixed sample range and
//                         adds into its own partial, so the result does not
//                         depend on scheduling; a last kernel adds the block
//                         partials in block order.
#include "common.cuh"
#include "internal.h"

#include <algorithm>
#include <cmath>
#include <vector>

struct scp3gpu_scp1 {
    int pes = 0, nw = 0, dim = 0, device = 0;
    int64_t chunk = 0;
    int blocks = 0;                 // reduction blocks (fixed per handle)
    cudaStream_t stream = nullptr;
    int64_t* vdir = nullptr;        // [62][dim] direction numbers
    double* q = nullptr;            // [dim]
    double* sqd = nullptr;          // [dim] sqrt(d)
    double* U = nullptr;            // [dim*dim] isqrtM_U, column-major
    double* V = nullptr;            // [chunk]
    double* G = nullptr;            // [chunk][dim]
    double* D = nullptr;            // [chunk][dim]
    double* P = nullptr;            // [blocks][(dim+1)^2] block partials
    double* R = nullptr;            // [(dim+1)^2]
    unsigned long long* capped = nullptr;   // [1] TTM3-F samples at the sweep cap, all calls
    long long not_converged = 0;
};

namespace scp3 {
namespace {

constexpr int kRedThreads = 256, kRedRows = 32, kRedTile = 8, kRedLd = 80;   // dim + 1 <= 80
constexpr int kRedStage = 2 * kRedRows * kRedLd;     // rows of [g, V], then of [dq, 1]
constexpr size_t kRedSmem = sizeof(double) * 2 * kRedStage;
static_assert(kRedLd * kRedLd <= 2 * kRedStage && kRedTile * kRedTile * kRedThreads / 2 <= 2 * kRedStage,
              "the sums go over the stages");

// P[block] += sum over the block's samples of [g, V] [dq, 1]^T, column-major
// (dim+1) x (dim+1).  nt = ceil((dim+1) / 8): thread (ti, tj) of a group of nt^2 threads
// owns the 64 elements (ti + nt a, tj + nt b), and the CTA's groups take the staged rows
// in turn, so a row costs a thread 16 conflict-free reads for 64 FMAs; the groups' sums
// are added in pairs.  It was 16 elements per thread on pairs of reads each, bound by
// shared memory: hexamer, 141 us per 2^16 samples.
__global__ void __launch_bounds__(kRedThreads) scp1_reduce_kernel(int dim, int64_t n, const double* __restrict__ V,
                                                                  const double* __restrict__ G,
                                                                  const double* __restrict__ D, double* __restrict__ P)
{
    extern __shared__ double sm[];                 // two stages; later the sums
    const int E1 = dim + 1, E = E1 * E1, nt = (E1 + kRedTile - 1) / kRedTile;
    const int t = threadIdx.x, groups = kRedThreads / (nt * nt), g = t / (nt * nt), u = t - g * nt * nt;
    const int ti = u % nt, tj = u / nt, lane = t & 31;
    double acc[kRedTile][kRedTile] = {};
    // columns past E1 stay zero, the last column of dq's rows 1
    for (int e = t; e < 2 * kRedStage; e += kRedThreads)
        sm[e] = e % kRedStage >= kRedRows * kRedLd && e % kRedLd == dim ? 1.0 : 0.0;
    __syncthreads();
    const int64_t s0 = n * blockIdx.x / gridDim.x, s1 = n * (blockIdx.x + 1) / gridDim.x;
    auto copy8 = [](double* dst, const double* src) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                     : "memory");
    };
    auto fetch = [&](int64_t c0, int stage) {
        double *sg = sm + stage * kRedStage, *sd = sg + kRedRows * kRedLd;
        for (int r = t >> 5; r < kRedRows && c0 + r < s1; r += kRedThreads / 32) {
            const int64_t s = c0 + r;
            for (int c = lane; c < dim; c += 32) {
                copy8(sg + r * kRedLd + c, G + s * dim + c);
                copy8(sd + r * kRedLd + c, D + s * dim + c);
            }
            if (lane == 0) copy8(sg + r * kRedLd + dim, V + s);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(s0, 0);
    int stage = 0;
    for (int64_t c0 = s0; c0 < s1; c0 += kRedRows, stage ^= 1) {
        const int rows = (int)(s1 - c0 < kRedRows ? s1 - c0 : kRedRows);
        fetch(c0 + kRedRows, stage ^ 1);           // an empty group past the end
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        const double *sg = sm + stage * kRedStage, *sd = sg + kRedRows * kRedLd;
        if (g < groups)
            for (int r = g; r < rows; r += groups) {
                double a[kRedTile], b[kRedTile];
#pragma unroll
                for (int k = 0; k < kRedTile; k++) a[k] = sg[r * kRedLd + ti + nt * k], b[k] = sd[r * kRedLd + tj + nt * k];
#pragma unroll
                for (int i = 0; i < kRedTile; i++)
#pragma unroll
                    for (int j = 0; j < kRedTile; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
            }
        __syncthreads();                           // the stage is free for the next fetch
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    // the upper half of the groups hands its sums to the lower, until one is left
    for (int left = groups; left > 1;) {
        const int low = (left + 1) / 2;
        __syncthreads();
        if (g >= low && g < left)
#pragma unroll
            for (int e = 0; e < kRedTile * kRedTile; e++)
                sm[e * (kRedThreads / 2) + t - low * nt * nt] = acc[e / kRedTile][e % kRedTile];
        __syncthreads();
        if (g < left - low)
#pragma unroll
            for (int e = 0; e < kRedTile * kRedTile; e++)
                acc[e / kRedTile][e % kRedTile] += sm[e * (kRedThreads / 2) + t];
        left = low;
    }
    __syncthreads();
    if (g == 0)
#pragma unroll
        for (int i = 0; i < kRedTile; i++)
#pragma unroll
            for (int j = 0; j < kRedTile; j++) sm[(tj + nt * j) * kRedLd + ti + nt * i] = acc[i][j];
    __syncthreads();
    double* Pb = P + (size_t)blockIdx.x * E;
    for (int e = t; e < E; e += kRedThreads) {
        const int j = e / E1;
        Pb[e] += sm[j * kRedLd + (e - j * E1)];
    }
}

// R[e] = sum of the block partials: warp w of a CTA adds the blocks w, w + 8, ... of 32
// elements in order, the eight warp sums are then added in order
__global__ void __launch_bounds__(256) scp1_sum_kernel(int E, int blocks, const double* __restrict__ P,
                                                       double* __restrict__ R)
{
    __shared__ double ws[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (e < E)
        for (int b = w; b < blocks; b += 8) s += P[(size_t)b * E + e];
    ws[w][lane] = s;
    __syncthreads();
    if (w || e >= E) return;
#pragma unroll
    for (int k = 1; k < 8; k++) s += ws[k][lane];
    R[e] = s;
}

void free_all(scp3gpu_scp1* h)
{
    void* p[] = {h->vdir, h->q, h->sqd, h->U, h->V, h->G, h->D, h->P, h->R, h->capped};
    for (void* x : p)
        if (x) cudaFree(x);
    if (h->stream) cudaStreamDestroy(h->stream);
}

}  // namespace
}  // namespace scp3

using namespace scp3;

extern "C" {

int scp3gpu_scp1_create(int pes, int nw, int64_t chunk, int device, scp3gpu_scp1** out)
{
    (void)cudaGetLastError();
    if (!out) return fail(SCP3GPU_ERR_ARG, "scp1_create: null handle pointer");
    *out = nullptr;
    if (pes != SCP3GPU_PES_QTIP4PF && pes != SCP3GPU_PES_TTM3F) return fail(SCP3GPU_ERR_ARG, "unknown potential");
    if (nw < 1 || nw > 8) return fail(SCP3GPU_ERR_ARG, "scp1: 1 <= nw <= 8");
    if (chunk < 0) return fail(SCP3GPU_ERR_ARG, "scp1: negative chunk");
    int rc = check_device(device);
    if (rc) return rc;
    DeviceGuard guard(device);
    if (pes == SCP3GPU_PES_TTM3F && (rc = ttm_init_device())) return rc;
    scp3gpu_scp1* h = new scp3gpu_scp1;
    h->pes = pes;
    h->nw = nw;
    h->dim = 9 * nw;
    h->device = device;
    h->chunk = chunk > 0 ? (chunk + 31) / 32 * 32 : (1 << 16);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    h->blocks = sms;
    const int dim = h->dim, E = (dim + 1) * (dim + 1);
    std::vector<int64_t> v;
    std::vector<uint64_t> sh;
    if ((rc = sobol_tables(dim, 0, 0, v, sh)) || (rc = upload(&h->vdir, v.data(), v.size())) ||
        (rc = dalloc(&h->q, dim)) || (rc = dalloc(&h->sqd, dim)) ||
        (rc = dalloc(&h->U, (size_t)dim * dim)) || (rc = dalloc(&h->V, h->chunk)) ||
        (rc = dalloc(&h->G, (size_t)h->chunk * dim)) || (rc = dalloc(&h->D, (size_t)h->chunk * dim)) ||
        (rc = dalloc(&h->P, (size_t)h->blocks * E)) || (rc = dalloc(&h->R, E)) || (rc = dalloc(&h->capped, 1))) {
        free_all(h);
        delete h;
        return rc;
    }
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMemsetAsync(h->capped, 0, sizeof(*h->capped), h->stream) != cudaSuccess ||
        cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {     // the table's copy
        free_all(h);
        delete h;
        return fail(SCP3GPU_ERR_CUDA, "scp1: stream creation failed");
    }
    *out = h;
    return SCP3GPU_OK;
}

int scp3gpu_scp1_average(scp3gpu_scp1* h, const double* q, const double* d, const double* isqrtM_U, int64_t skip,
                         int64_t i0, int64_t i1, double* Upot, double* UX, double* UX_q)
{
    (void)cudaGetLastError();
    if (!h || !q || !d || !isqrtM_U || !Upot || !UX || !UX_q)
        return fail(SCP3GPU_ERR_ARG, "scp1_average: null handle or pointer");
    if (skip < 0 || i0 < 0 || i1 < i0 || skip + i1 >= (1ll << kLogMax))
        return fail(SCP3GPU_ERR_ARG, "scp1_average: bad Sobol range");
    DeviceGuard guard(h->device);
    const int dim = h->dim, E1 = dim + 1, E = E1 * E1;
    std::vector<double> sqd(dim);
    for (int k = 0; k < dim; k++) {
        if (!(d[k] >= 0.0)) return fail(SCP3GPU_ERR_ARG, "scp1_average: d must be >= 0");
        sqd[k] = std::sqrt(d[k]);
    }
    cudaStream_t s = h->stream;
    SCP3_CUDA(cudaMemcpyAsync(h->q, q, sizeof(double) * dim, cudaMemcpyHostToDevice, s));
    SCP3_CUDA(cudaMemcpyAsync(h->sqd, sqd.data(), sizeof(double) * dim, cudaMemcpyHostToDevice, s));
    SCP3_CUDA(cudaMemcpyAsync(h->U, isqrtM_U, sizeof(double) * dim * dim, cudaMemcpyHostToDevice, s));
    SCP3_CUDA(cudaMemsetAsync(h->P, 0, sizeof(double) * (size_t)h->blocks * E, s));
    int rc = SCP3GPU_OK;
    for (int64_t c0 = i0; c0 < i1; c0 += h->chunk) {
        const int64_t n = std::min<int64_t>(h->chunk, i1 - c0);
        Scp1Args a{h->nw, dim, h->q, h->sqd, h->U, h->vdir, skip + c0, n, h->V, h->G, h->D, h->capped};
        if ((rc = launch_scp1_samples(h->pes, a, s))) return rc;
        if ((rc = allow_smem(scp1_reduce_kernel))) return rc;
        scp1_reduce_kernel<<<h->blocks, kRedThreads, kRedSmem, s>>>(dim, n, h->V, h->G, h->D, h->P);
        SCP3_CUDA(cudaGetLastError());
    }
    scp1_sum_kernel<<<(E + 31) / 32, 256, 0, s>>>(E, h->blocks, h->P, h->R);
    SCP3_CUDA(cudaGetLastError());
    std::vector<double> R(E);
    unsigned long long capped = 0;
    SCP3_CUDA(cudaMemcpyAsync(R.data(), h->R, sizeof(double) * E, cudaMemcpyDeviceToHost, s));
    if (h->pes == SCP3GPU_PES_TTM3F)
        SCP3_CUDA(cudaMemcpyAsync(&capped, h->capped, sizeof(capped), cudaMemcpyDeviceToHost, s));
    SCP3_CUDA(cudaStreamSynchronize(s));
    h->not_converged = (long long)capped;
    for (int j = 0; j < dim; j++)
        for (int i = 0; i < dim; i++) UX_q[(size_t)j * dim + i] = R[(size_t)j * E1 + i];
    for (int i = 0; i < dim; i++) UX[i] = R[(size_t)dim * E1 + i];
    *Upot = R[(size_t)dim * E1 + dim];
    return SCP3GPU_OK;
}

int scp3gpu_scp1_status(const scp3gpu_scp1* h, int64_t* not_converged)
{
    if (!h || !not_converged) return fail(SCP3GPU_ERR_ARG, "scp1_status: null handle or pointer");
    *not_converged = h->not_converged;
    return SCP3GPU_OK;
}

void scp3gpu_scp1_destroy(scp3gpu_scp1* h)
{
    if (!h) return;
    DeviceGuard guard(h->device);
    free_all(h);
    delete h;
}

}  // extern "C"
