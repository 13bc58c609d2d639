// Pinned host memory as kernels see it (host_view.h).
#include "host_view.h"

#include <cstring>

#include <cuda.h>
#include <cuda_runtime.h>

namespace lsp {

namespace {
using GetAttributes = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);

GetAttributes pointer_attributes()
{
    static const GetAttributes fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &p, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<GetAttributes>(p);
    }();
    return fn;
}
}  // namespace

void* pinned_view(const void* p, size_t bytes, bool* host)
{
    const GetAttributes get = pointer_attributes();
    *host = false;
    if (!get || !p) return nullptr;
    unsigned type = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[4] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                   CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* to[4] = {&type, &dev, &start, &size};
    const CUdeviceptr a = (CUdeviceptr)(uintptr_t)p;
    if (get(4, what, to, a) != CUDA_SUCCESS) return nullptr;
    *host = type == 0 || type == CU_MEMORYTYPE_HOST;   // 0: not known to the driver, pageable
    if (type != CU_MEMORYTYPE_HOST || !dev) return nullptr;
    // The whole array lies in the allocation (its start is reported in the address space of p or of dev).
    const bool inside = (a >= start && a - start <= size && bytes <= size - (a - start)) ||
                        (dev >= start && dev - start <= size && bytes <= size - (dev - start));
    return inside ? (void*)(uintptr_t)dev : nullptr;
}

HostStage::~HostStage()
{
    if (p_) cudaFreeHost(p_);
}

char* HostStage::get(size_t bytes)
{
    if (bytes > kMaxBytes) return nullptr;
    if (bytes > n_) {
        if (p_) cudaFreeHost(p_);
        p_ = nullptr;
        n_ = 0;
        if (cudaMallocHost((void**)&p_, kMaxBytes) != cudaSuccess) {
            cudaGetLastError();
            p_ = nullptr;
            return nullptr;
        }
        n_ = kMaxBytes;
    }
    return p_;
}

void HostTransfer::add(const void* p, size_t bytes)
{
    if (!host_) return;
    e_[n_++] = Entry{const_cast<void*>(p), bytes, pinned_view(p, bytes, &host_), nullptr};
}

bool HostTransfer::ready()
{
    if (!host_) return false;
    auto padded = [](size_t b) { return (b + 127) / 128 * 128; };
    size_t need = 0;
    for (int k = 0; k < n_; k++)
        if (!e_[k].dev) need += padded(e_[k].bytes);
    if (!need) return true;
    char* s = stage_.get(need);
    if (!s) return false;
    void* dev = nullptr;
    if (cudaHostGetDevicePointer(&dev, s, 0) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    size_t at = 0;
    for (int k = 0; k < n_; k++) {
        Entry& e = e_[k];
        if (e.dev) continue;
        e.staged = s + at;
        e.dev = (char*)dev + at;
        if (in_) std::memcpy(e.staged, e.host, e.bytes);
        at += padded(e.bytes);
    }
    return true;
}

void HostTransfer::finish()
{
    if (in_) return;
    for (int k = 0; k < n_; k++)
        if (e_[k].staged) std::memcpy(e_[k].host, e_[k].staged, e_[k].bytes);
}

}  // namespace lsp
