// Copies out of the device into pageable host memory go through pinned buffers and are
// stored by a few threads: a program's fresh result array has no pages yet, and one
// thread faulting them in is what such a copy costs (12 MB Mout: 2.04 ms by one
// cudaMemcpy, of which the PCIe copy is 0.2 ms and the faults 0.7 to 1.1; 1.51 ms through
// four workers here, 0.56 against 0.93 ms into memory already there).  Small calls of the
// potentials keep their device memory and pinned buffer between calls (a Hessian's 108
// gradients: 970 us a call before, cudaMalloc and cudaFree most of it, 83 us now).
#include "staging.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "internal.h"

namespace scp3 {
namespace staging {

namespace {
struct Idle {
    char* pinned;
    char* dev;
    size_t dev_bytes;
    int device;
};
constexpr size_t kMaxIdle = 8;
std::mutex& mu()
{
    static std::mutex* m = new std::mutex;      // outlives every static object's user
    return *m;
}
std::vector<Idle>& idle()
{
    static std::vector<Idle>* v = new std::vector<Idle>;
    return *v;
}
void drop(const Idle& s)
{
    if (s.pinned) cudaFreeHost(s.pinned);
    if (s.dev) {
        DeviceGuard g(s.device);
        cudaFree(s.dev);
    }
}
}  // namespace

int Slot::acquire()
{
    SCP3_CUDA(cudaGetDevice(&device_));
    {
        std::lock_guard<std::mutex> lock(mu());
        std::vector<Idle>& v = idle();
        for (size_t k = v.size(); k-- > 0;)
            if (v[k].device == device_) {
                pinned_ = v[k].pinned, dev_ = v[k].dev, dev_bytes_ = v[k].dev_bytes;
                v.erase(v.begin() + (long)k);
                return SCP3GPU_OK;
            }
    }
    const cudaError_t e = cudaHostAlloc((void**)&pinned_, kPinned, cudaHostAllocPortable);
    if (e != cudaSuccess) {
        pinned_ = nullptr;
        (void)cudaGetLastError();
        return cuda_fail(e, "pinned staging buffer");
    }
    return SCP3GPU_OK;
}

Slot::~Slot()
{
    if (!pinned_) return;
    Idle mine{pinned_, dev_, dev_bytes_, device_}, spare[kMaxIdle + 1];
    size_t n = 0;
    {
        std::lock_guard<std::mutex> lock(mu());
        size_t held = mine.dev_bytes;
        for (Idle& s : idle())
            if ((held += s.dev_bytes) > kScratchMax) {         // its device memory, not the buffer
                held -= s.dev_bytes;
                spare[n++] = Idle{nullptr, s.dev, s.dev_bytes, s.device};
                s.dev = nullptr, s.dev_bytes = 0;
            }
        if (idle().size() < kMaxIdle) idle().push_back(mine);
        else spare[n++] = mine;
    }
    for (size_t k = 0; k < n; k++) drop(spare[k]);
}

int Slot::scratch(size_t bytes, char** p)
{
    if (bytes > dev_bytes_) {
        if (dev_) cudaFree(dev_);
        dev_ = nullptr, dev_bytes_ = 0;
        size_t want = 1u << 20;
        while (want < bytes) want *= 2;
        if (int rc = dalloc(&dev_, want)) return rc;
        dev_bytes_ = want;
    }
    *p = dev_;
    return SCP3GPU_OK;
}

void trim()
{
    std::vector<Idle> v;
    {
        std::lock_guard<std::mutex> lock(mu());
        v.swap(idle());
    }
    for (const Idle& s : v) drop(s);
}

int copy_out(void* dst, size_t pitch, const void* src, size_t width, size_t rows, cudaStream_t s)
{
    constexpr size_t kPiece = 1u << 20, kPieces = kPinned / kPiece;
    const bool flat = pitch == width;
    const size_t total = width * rows;
    if (!total) return SCP3GPU_OK;
    const size_t per = flat ? kPiece : std::max<size_t>(1, kPiece / width) * width;     // bytes per piece
    const size_t pieces = (total + per - 1) / per;
    Slot slot;
    // Memory the driver knows (pinned above all) takes one DMA; only pageable memory gains
    // from the pool (12 MB of Mout: pageable 2.04 ms plain, 1.51 staged; pinned, in a
    // build of 2^20 host normals, 6.3 ms a step plain, 6.9 staged).
    auto known = [&] {
        cudaPointerAttributes at{};
        const cudaError_t ea = cudaPointerGetAttributes(&at, dst);
        if (ea != cudaSuccess) (void)cudaGetLastError();
        return ea == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    };
    // so do small copies, rows longer than a piece, or where there is no pinned memory
    if (total < 2 * kPiece || per > kPiece || known() || slot.acquire() != SCP3GPU_OK) {
        if (flat) SCP3_CUDA(cudaMemcpyAsync(dst, src, total, cudaMemcpyDeviceToHost, s));
        else SCP3_CUDA(cudaMemcpy2DAsync(dst, pitch, src, width, width, rows, cudaMemcpyDeviceToHost, s));
        SCP3_CUDA(cudaStreamSynchronize(s));
        return SCP3GPU_OK;
    }
    int dev = 0;
    SCP3_CUDA(cudaGetDevice(&dev));
    // worker w takes an n-th of the pieces, in a row, through its own two pinned pieces
    // (eight workers with half-size pieces: 2.37 ms)
    const size_t n = std::min<size_t>(kPieces / 2, std::max<size_t>(1, pieces / 2));
    std::atomic<int> failed{(int)cudaSuccess};
    auto work = [&](size_t w) {
        cudaEvent_t ev[2] = {nullptr, nullptr};
        cudaError_t e = cudaSetDevice(dev);
        for (int b = 0; b < 2 && e == cudaSuccess; b++) e = cudaEventCreateWithFlags(ev + b, cudaEventDisableTiming);
        char* const buf[2] = {slot.pinned() + 2 * w * kPiece, slot.pinned() + (2 * w + 1) * kPiece};
        auto issue = [&](size_t k, int b) {
            e = cudaMemcpyAsync(buf[b], (const char*)src + k * per, std::min(per, total - k * per),
                                cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(ev[b], s);
        };
        auto store = [&](size_t k, const char* from) {
            const size_t o = k * per, bytes = std::min(per, total - o);
            if (flat) std::memcpy((char*)dst + o, from, bytes);
            else
                for (size_t i = 0; i < bytes; i += width) std::memcpy((char*)dst + (o + i) / width * pitch, from + i, width);
        };
        const size_t k0 = pieces * w / n, k1 = pieces * (w + 1) / n;
        if (e == cudaSuccess) issue(k0, 0);
        int b = 0;
        for (size_t k = k0; k < k1 && e == cudaSuccess; k++, b ^= 1) {
            if (k + 1 < k1) issue(k + 1, b ^ 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(ev[b]);
            if (e == cudaSuccess) store(k, buf[b]);
        }
        if (e != cudaSuccess) {
            failed = (int)e;
            cudaStreamSynchronize(s);      // no copy into the slot's buffers in flight when it goes back
        }
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
    };
    std::vector<std::thread> others;
    try {
        others.reserve(n);
        while (others.size() + 1 < n) others.emplace_back(work, others.size() + 1);
    } catch (...) {
        // no more threads: their pieces fall to this one
    }
    const size_t started = others.size() + 1;
    work(0);
    for (size_t w = started; w < n; w++) work(w);
    for (std::thread& t : others) t.join();
    const cudaError_t e = (cudaError_t)failed.load();
    return e == cudaSuccess ? SCP3GPU_OK : cuda_fail(e, "copy to host memory");
}

}  // namespace staging
}  // namespace scp3

// For tests: idle slots of the pool and the device memory they hold.
extern "C" int scp3gpu_internal_staging_idle(size_t* device_bytes)
{
    using namespace scp3::staging;
    std::lock_guard<std::mutex> lock(mu());
    size_t held = 0;
    for (const Idle& s : idle()) held += s.dev_bytes;
    if (device_bytes) *device_bytes = held;
    return (int)idle().size();
}
