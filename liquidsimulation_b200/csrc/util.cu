// Caller-order read-back and write-back: the device keeps particles sorted by cell and
// slot_of_id[id] tells where caller particle `id` sits. These kernels replace the
// reference's blocking sorted read-back (SPHSolver::onEndUpdate, SPHSolver.cpp:400-427)
// and its full re-upload on change (SPHSolver::initParallelBuffers, :791-886).
#include "lsp_device.cuh"
#include "lsp_kernels.h"

#include <atomic>

namespace lsp {

constexpr int kThreads = 256;
static inline unsigned blocks_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// Rows of three floats between caller order (packed) and device slots: a thread moves a row of up to
// four arrays and its first-step flag. Packed arrays in the host's memory go through shared memory (the
// _host kernels), 256 rows at a time, so that they are read and written contiguously, 16 bytes at a
// time where every array's alignment allows: a row at a time it would be three strided accesses, each a
// request of its own over PCIe. In device memory L2 merges those, and the block's wait for its slowest
// row costs more than it saves: a field of 990,000 positions 25 us a row at a time, 35 through shared
// memory, the state 88 and 106.
struct RowArrays {
    const float4* slots[4];
    float* rows[4];
    int count;
    const float4* flag_slots;   // w != 0 is the flag, null when there are no flags
    int32_t* flags;
};

// Moves `floats` floats between shared and packed memory (kStore: to packed).
template <bool kVector, bool kStore>
__device__ __forceinline__ void move_rows(float* packed, float* sm, int floats)
{
    int done = 0;
    if (kVector) {
        done = floats & ~3;
        for (int k = 4 * threadIdx.x; k < done; k += 4 * blockDim.x) {
            if (kStore) *reinterpret_cast<float4*>(packed + k) = *reinterpret_cast<const float4*>(sm + k);
            else *reinterpret_cast<float4*>(sm + k) = *reinterpret_cast<const float4*>(packed + k);
        }
    }
    for (int k = done + threadIdx.x; k < floats; k += blockDim.x) {
        if (kStore) packed[k] = sm[k];
        else sm[k] = packed[k];
    }
}

template <int kCount>
__global__ void __launch_bounds__(kThreads) k_gather_rows(RowArrays a, const int32_t* __restrict__ slot_of_id, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (id >= n) return;
    const int32_t s = slot_of_id[id];
    float4 v[kCount];
#pragma unroll
    for (int c = 0; c < kCount; c++) v[c] = __ldg(a.slots[c] + s);
    const float flag = a.flag_slots ? __ldg(&a.flag_slots[s].w) : 0.f;
#pragma unroll
    for (int c = 0; c < kCount; c++) {
        float* to = a.rows[c] + 3 * id;
        to[0] = v[c].x;
        to[1] = v[c].y;
        to[2] = v[c].z;
    }
    if (a.flag_slots) a.flags[id] = flag != 0.f ? 1 : 0;
}

template <bool kVector>
__global__ void __launch_bounds__(kThreads) k_gather_rows_host(RowArrays a, const int32_t* __restrict__ slot_of_id, int64_t n)
{
    __shared__ alignas(16) float sm[4][3 * kThreads];
    const int64_t base = (int64_t)blockIdx.x * kThreads, id = base + threadIdx.x;
    if (id < n) {
        const int32_t s = slot_of_id[id];
        for (int c = 0; c < a.count; c++) {
            const float4 v = a.slots[c][s];
            sm[c][3 * threadIdx.x] = v.x;
            sm[c][3 * threadIdx.x + 1] = v.y;
            sm[c][3 * threadIdx.x + 2] = v.z;
        }
        if (a.flag_slots) a.flags[id] = a.flag_slots[s].w != 0.f ? 1 : 0;
    }
    __syncthreads();
    const int floats = 3 * (int)min((int64_t)kThreads, n - base);
    for (int c = 0; c < a.count; c++) move_rows<kVector, true>(a.rows[c] + 3 * base, sm[c], floats);
}

// The other way for the whole state: positions (w: caller id), velocities (w: flag), half and old
// half velocities (w kept).
__global__ void __launch_bounds__(kThreads) k_scatter_state(RowArrays a, float4* __restrict__ pos, float4* __restrict__ vel,
                                                            float4* __restrict__ hv, float4* __restrict__ ov,
                                                            const int32_t* __restrict__ slot_of_id, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (id >= n) return;
    const int32_t s = slot_of_id[id], flag = __ldg(a.flags + id);
    auto row = [&](int c, float w) {
        const float* from = a.rows[c] + 3 * id;
        return make_float4(__ldg(from), __ldg(from + 1), __ldg(from + 2), w);
    };
    const float hw = hv[s].w, ow = ov[s].w;
    pos[s] = row(0, __int_as_float((int)id));
    vel[s] = row(1, flag ? 1.f : 0.f);
    hv[s] = row(2, hw);
    ov[s] = row(3, ow);
}

template <bool kVector>
__global__ void __launch_bounds__(kThreads) k_scatter_state_host(RowArrays a, float4* pos, float4* vel, float4* hv, float4* ov,
                                                                 const int32_t* __restrict__ slot_of_id, int64_t n)
{
    __shared__ alignas(16) float sm[4][3 * kThreads];
    const int64_t base = (int64_t)blockIdx.x * kThreads, id = base + threadIdx.x;
    const int floats = 3 * (int)min((int64_t)kThreads, n - base);
#pragma unroll
    for (int c = 0; c < 4; c++) move_rows<kVector, false>(a.rows[c] + 3 * base, sm[c], floats);
    const int32_t flag = id < n ? a.flags[id] : 0;
    const int32_t s = id < n ? slot_of_id[id] : 0;
    __syncthreads();
    if (id >= n) return;
    auto row = [&](int c, float w) {
        return make_float4(sm[c][3 * threadIdx.x], sm[c][3 * threadIdx.x + 1], sm[c][3 * threadIdx.x + 2], w);
    };
    pos[s] = row(0, __int_as_float((int)id));
    vel[s] = row(1, flag ? 1.f : 0.f);
    hv[s] = row(2, hv[s].w);
    ov[s] = row(3, ov[s].w);
}

static bool aligned_rows(const RowArrays& a)
{
    for (int c = 0; c < a.count; c++)
        if ((uintptr_t)a.rows[c] % sizeof(float4)) return false;
    return true;
}
static void gather_rows_host(const RowArrays& a, const int32_t* slot_of_id, int64_t n, cudaStream_t s)
{
    if (!n) return;
    if (aligned_rows(a)) k_gather_rows_host<true><<<blocks_for(n), kThreads, 0, s>>>(a, slot_of_id, n);
    else k_gather_rows_host<false><<<blocks_for(n), kThreads, 0, s>>>(a, slot_of_id, n);
}

__global__ void k_gather_w(const float4* __restrict__ src, const int32_t* __restrict__ slot_of_id,
                           float* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    out[id] = src[slot_of_id[id]].w;
}

__global__ void k_gather_sqlen(const float4* __restrict__ src, const int32_t* __restrict__ slot_of_id,
                               float* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    out[id] = sqmag(v3(src[slot_of_id[id]]));
}

__global__ void k_gather_scalar(const float* __restrict__ src, const int32_t* __restrict__ slot_of_id,
                                float* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    out[id] = src[slot_of_id[id]];
}

__global__ void k_gather_count(const int32_t* __restrict__ count, const int32_t* __restrict__ slot_of_id,
                               float* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    out[id] = (float)count[slot_of_id[id]];
}

__global__ void k_slots_of_ids(const float4* __restrict__ pos, int32_t* __restrict__ slot_of_id, int64_t n)
{
    const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot < n) slot_of_id[id_of(pos[slot])] = (int32_t)slot;
}

void launch_slots_of_ids(const float4* pos, int32_t* slot_of_id, int64_t n, cudaStream_t s)
{
    if (n) k_slots_of_ids<<<blocks_for(n), kThreads, 0, s>>>(pos, slot_of_id, n);
}

void launch_gather_field(const void* src, int comps, int mode, const int32_t* slot_of_id, float* out, bool host, int64_t n,
                         cudaStream_t s)
{
    if (!n) return;
    if (comps == 3) {
        RowArrays a{};
        a.slots[0] = (const float4*)src;
        a.rows[0] = out;
        a.count = 1;
        if (host) gather_rows_host(a, slot_of_id, n, s);
        else k_gather_rows<1><<<blocks_for(n), kThreads, 0, s>>>(a, slot_of_id, n);
    } else if (mode == 1)
        k_gather_w<<<blocks_for(n), kThreads, 0, s>>>((const float4*)src, slot_of_id, out, n);
    else if (mode == 2)
        k_gather_sqlen<<<blocks_for(n), kThreads, 0, s>>>((const float4*)src, slot_of_id, out, n);
    else
        k_gather_scalar<<<blocks_for(n), kThreads, 0, s>>>((const float*)src, slot_of_id, out, n);
}

void launch_gather_count(const int32_t* count, const int32_t* slot_of_id, float* out, int64_t n, cudaStream_t s)
{
    if (n) k_gather_count<<<blocks_for(n), kThreads, 0, s>>>(count, slot_of_id, out, n);
}

void launch_gather_particles(const float4* pos, const float4* vel, const int32_t* slot_of_id, float* x, float* v,
                             int64_t n, cudaStream_t s)
{
    RowArrays a{};
    a.slots[0] = pos;
    a.slots[1] = vel;
    a.rows[0] = x;
    a.rows[1] = v;
    a.count = 2;
    gather_rows_host(a, slot_of_id, n, s);
}

void launch_scatter_state(const float* x, const float* v, const float* half, const float* old, const int32_t* first,
                          const int32_t* slot_of_id, float4* pos, float4* vel, float4* hvel, float4* oldv,
                          bool host, int64_t n, cudaStream_t s)
{
    if (!n) return;
    RowArrays a{};
    const float* rows[4] = {x, v, half, old};
    for (int c = 0; c < 4; c++) a.rows[c] = const_cast<float*>(rows[c]);
    a.count = 4;
    a.flags = const_cast<int32_t*>(first);
    const unsigned blocks = blocks_for(n);
    if (!host) k_scatter_state<<<blocks, kThreads, 0, s>>>(a, pos, vel, hvel, oldv, slot_of_id, n);
    else if (aligned_rows(a)) k_scatter_state_host<true><<<blocks, kThreads, 0, s>>>(a, pos, vel, hvel, oldv, slot_of_id, n);
    else k_scatter_state_host<false><<<blocks, kThreads, 0, s>>>(a, pos, vel, hvel, oldv, slot_of_id, n);
}

__global__ void k_scatter_vec(const float* __restrict__ in, const int32_t* __restrict__ slot_of_id,
                              float4* __restrict__ dst, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    dst[slot_of_id[id]] = make_float4(in[3 * id], in[3 * id + 1], in[3 * id + 2], 0.f);
}

void launch_scatter_vec(const float* in, const int32_t* slot_of_id, float4* dst, int64_t n, cudaStream_t s)
{
    if (n) k_scatter_vec<<<blocks_for(n), kThreads, 0, s>>>(in, slot_of_id, dst, n);
}

void launch_gather_state(const float4* pos, const float4* vel, const float4* hvel, const float4* oldv,
                         const int32_t* slot_of_id, float* x, float* v, float* half, float* old, int32_t* first,
                         bool host, int64_t n, cudaStream_t s)
{
    if (!n) return;
    RowArrays a{};
    const float4* slots[4] = {pos, vel, hvel, oldv};
    float* rows[4] = {x, v, half, old};
    for (int c = 0; c < 4; c++) {
        a.slots[c] = slots[c];
        a.rows[c] = rows[c];
    }
    a.count = 4;
    a.flag_slots = vel;
    a.flags = first;
    if (host) gather_rows_host(a, slot_of_id, n, s);
    else k_gather_rows<4><<<blocks_for(n), kThreads, 0, s>>>(a, slot_of_id, n);
}

__global__ void k_neighbor_export(const int32_t* __restrict__ nbr, const int32_t* __restrict__ count, int64_t stride,
                                  const float4* __restrict__ pos, const int32_t* __restrict__ slot_of_id,
                                  const int64_t* __restrict__ offsets, int32_t* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    int32_t s = slot_of_id[id];
    int c = count[s];
    int64_t o = offsets[id];
    for (int e = 0; e < c; e++) out[o + e] = id_of(pos[list_entry(nbr, stride, s, e)]);
}

void launch_neighbor_export(const int32_t* nbr, const int32_t* count, int64_t stride, const float4* pos,
                            const int32_t* slot_of_id, const int64_t* offsets, int32_t* out, int64_t n,
                            cudaStream_t s)
{
    if (n) k_neighbor_export<<<blocks_for(n), kThreads, 0, s>>>(nbr, count, stride, pos, slot_of_id, offsets, out, n);
}

__global__ void k_scale(const float* __restrict__ src, float* __restrict__ dst, int64_t n, float f)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i] * f;
}

void launch_scale(const float* src, float* dst, int64_t n, float factor, cudaStream_t s)
{
    if (n) k_scale<<<blocks_for(n), kThreads, 0, s>>>(src, dst, n, factor);
}

__global__ void k_gather_rows(const float* __restrict__ src, int width, const int32_t* __restrict__ slot_of_id,
                              float* __restrict__ out, int64_t n)
{
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const int64_t s = slot_of_id[id];
    for (int c = 0; c < width; c++) out[id * width + c] = src[s * width + c];
}

void launch_gather_rows(const float* src, int width, const int32_t* slot_of_id, float* out, int64_t n, cudaStream_t s)
{
    if (n) k_gather_rows<<<blocks_for(n), kThreads, 0, s>>>(src, width, slot_of_id, out, n);
}

// Float min/max through order-preserving integer images (atomicMin/Max on ints).
__device__ __forceinline__ int32_t ordered(float f)
{
    int32_t i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}

__global__ void k_bounds(const float4* __restrict__ pos, int64_t n, int32_t* out)
{
    int32_t lo[3] = {INT32_MAX, INT32_MAX, INT32_MAX}, hi[3] = {INT32_MIN, INT32_MIN, INT32_MIN};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float4 p = pos[i];
        float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (!isfinite(c[a])) continue;
            int32_t o = ordered(c[a]);
            lo[a] = min(lo[a], o);
            hi[a] = max(hi[a], o);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        for (int off = 16; off > 0; off >>= 1) {
            lo[a] = min(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
            hi[a] = max(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; a++) {
            atomicMin(&out[a], lo[a]);
            atomicMax(&out[3 + a], hi[a]);
        }
    }
}

void launch_bounds(const float4* pos, int64_t n, int32_t* out, cudaStream_t s)
{
    if (n) k_bounds<<<148 * 4, kThreads, 0, s>>>(pos, n, out);
}

int device_sm_count()
{
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cached[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    int v = cached[dev].load(std::memory_order_relaxed);
    if (v <= 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        v = sms > 0 ? sms : 148;
        cached[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

}  // namespace lsp
