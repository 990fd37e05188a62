// Host transfers: a bounded pool of pinned buffers and small device scratch.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace scp3 {
namespace staging {

constexpr size_t kPinned = 8u << 20;       // pinned bytes of a slot
constexpr size_t kScratchMax = 32u << 20;  // device bytes of a slot, and of all idle ones together

// One call's exclusive buffers on the current device, from the pool and back to it.  At
// most eight idle slots are kept (64 MB pinned) with kScratchMax of device memory between
// them, and all of them are freed when an allocation of the library fails (trim; the
// libraries it calls and others on the same GPU do not know of them).
class Slot {
public:
    Slot() = default;
    ~Slot();
    Slot(const Slot&) = delete;
    Slot& operator=(const Slot&) = delete;
    int acquire();                         // SCP3GPU_OK or an error
    char* pinned() const { return pinned_; }
    int scratch(size_t bytes, char** p);   // device memory of this slot, bytes <= kScratchMax

private:
    friend void trim();
    char* pinned_ = nullptr;
    char* dev_ = nullptr;
    size_t dev_bytes_ = 0;
    int device_ = -1;
};

void trim();

// rows x width bytes from device memory (contiguous) to host memory with the given row
// pitch, ordered on stream s; returns when the host memory is written.
int copy_out(void* dst, size_t pitch, const void* src, size_t width, size_t rows, cudaStream_t s);

}  // namespace staging
}  // namespace scp3
