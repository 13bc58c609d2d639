// Host memory that kernels can reach: caller buffers that are pinned, or a bounded pinned staging
// buffer for those that are not. Small transfers of particle state go through it in one launch
// instead of one copy per array and a kernel.
#pragma once

#include <cstddef>
#include <cstdint>

namespace lsp {

// Device address of the memory [p, p + bytes) when all of it is one pinned, mapped allocation of the
// host; null otherwise. *host says whether the host may touch p: false for device memory, which
// callers may pass as well, and when the driver cannot be asked.
void* pinned_view(const void* p, size_t bytes, bool* host);

// Pinned memory of a solver, kept between calls and at most kMaxBytes.
class HostStage {
public:
    static constexpr size_t kMaxBytes = 1 << 20;
    ~HostStage();
    // At least `bytes` of pinned memory, null when that is above the limit or cannot be had.
    char* get(size_t bytes);

private:
    char* p_ = nullptr;
    size_t n_ = 0;
};

// The arrays of one transfer: each gets a device address in the caller's memory or in the stage;
// finish() copies staged results out (after the stream has been waited for).
class HostTransfer {
public:
    // to_device: the caller's data is read (staged arrays are copied in), else written.
    HostTransfer(HostStage& stage, bool to_device) : stage_(stage), in_(to_device) {}
    void add(const void* p, size_t bytes);
    // False when some array can be reached neither way (device memory goes by copies); the device
    // addresses are view(k).
    bool ready();
    void* view(int k) const { return e_[k].dev; }
    void finish();

private:
    static constexpr int kMost = 5;
    struct Entry {
        void* host;
        size_t bytes;
        void* dev;
        char* staged;
    };
    HostStage& stage_;
    bool in_;
    bool host_ = true;   // every array is the host's
    int n_ = 0;
    Entry e_[kMost];
};

// Largest transfer that goes through kernels directly: its kernels reach 50 GB/s of PCIe where the
// copy engines reach 54, but start at once (62 KB of state in five arrays: 53 -> 16 us; 5.3 MB: 143 ->
// 122 us; 51.6 MB: 1.00 -> 1.03 ms).
constexpr size_t kDirectTransferBytes = 8u << 20;

}  // namespace lsp
