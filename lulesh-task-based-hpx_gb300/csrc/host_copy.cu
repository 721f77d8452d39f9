// Copies between device arrays and the caller's host arrays, many small ones
// in one launch.
//
// A copy-engine transfer costs the host about 2.5 us to queue and the stream
// as much again between two of them, whatever its size, so the 23 arrays of
// a small Domain take 60 us to download and the drop-in call's slabs, with
// some 200 copies, take longer to queue than to run. Arrays in page-locked
// memory can be reached by kernels over the same link at the same rate
// (193 GB/s down, 211 up measured either way), so one kernel copies a whole
// list of them.
#include <cuda.h>
#include <cuda_runtime.h>

#include "lulesh_dev.h"

namespace lulesh {
namespace {

constexpr int kCopyBlock = 256;
constexpr int kCopyMax = 24;     // segments of a launch
constexpr int kPerThread = 4;    // vectors in flight per thread

struct Segments {
    void* dst[kCopyMax];
    const void* src[kCopyMax];
    size_t bytes[kCopyMax];
};

template <class V>
__device__ __forceinline__ void copy_range(V* dst, const V* src, size_t n) {
    const size_t step = size_t(gridDim.x) * kCopyBlock;
    for (size_t i = size_t(blockIdx.x) * kCopyBlock + threadIdx.x; i < n; i += kPerThread * step) {
        V v[kPerThread];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k)
            if (i + k * step < n) v[k] = src[i + k * step];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k)
            if (i + k * step < n) dst[i + k * step] = v[k];
    }
}

// Segment blockIdx.y, in the widest vectors that both its ends allow (its
// bytes are a multiple of 4, copy_segments).
__global__ void __launch_bounds__(kCopyBlock) k_copy(const __grid_constant__ Segments s) {
    const int k = blockIdx.y;
    const size_t bytes = s.bytes[k];
    const unsigned long long at =
        reinterpret_cast<unsigned long long>(s.dst[k]) | reinterpret_cast<unsigned long long>(s.src[k]) | bytes;
    if ((at & 15) == 0)
        copy_range(static_cast<int4*>(s.dst[k]), static_cast<const int4*>(s.src[k]), bytes / 16);
    else if ((at & 7) == 0)
        copy_range(static_cast<int2*>(s.dst[k]), static_cast<const int2*>(s.src[k]), bytes / 8);
    else
        copy_range(static_cast<int*>(s.dst[k]), static_cast<const int*>(s.src[k]), bytes / 4);
}

using PointerAttributes = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);

// cuPointerGetAttributes of the loaded driver, or null.
PointerAttributes pointer_attributes() {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &fn, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
        return nullptr;
    return reinterpret_cast<PointerAttributes>(fn);
}

}  // namespace

bool host_mapped(const HostCopy* c, int n) {
    static const PointerAttributes attributes = pointer_attributes();
    if (!attributes) return false;
    for (int k = 0; k < n; ++k) {
        unsigned type = 0;
        CUdeviceptr dev = 0, start = 0;
        size_t size = 0;
        CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                      CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
        void* out[] = {&type, &dev, &start, &size};
        const CUdeviceptr p = reinterpret_cast<CUdeviceptr>(c[k].host);
        if (attributes(4, what, out, p) != CUDA_SUCCESS) return false;
        // page-locked, at the same address for the device, the whole array in one range
        if (type != CU_MEMORYTYPE_HOST || dev != p || p < start || c[k].bytes > size - (p - start)) return false;
    }
    return true;
}

int copy_segments(const HostCopy* c, int n, bool to_device, bool mapped, size_t limit, cudaStream_t s,
                  int64_t* launches) {
    size_t total = 0, most = 0;
    bool words = true;
    for (int k = 0; k < n; ++k) {
        total += c[k].bytes;
        most = c[k].bytes > most ? c[k].bytes : most;
        words &= ((reinterpret_cast<unsigned long long>(c[k].dev) | reinterpret_cast<unsigned long long>(c[k].host) |
                   c[k].bytes) & 3) == 0;
    }
    if (!mapped || !words || n < 2 || total > n * limit) {
        for (int k = 0; k < n; ++k) {
            const cudaError_t e = to_device
                                      ? cudaMemcpyAsync(c[k].dev, c[k].host, c[k].bytes, cudaMemcpyHostToDevice, s)
                                      : cudaMemcpyAsync(c[k].host, c[k].dev, c[k].bytes, cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess) return LULESH_ECUDA;
        }
        return LULESH_OK;
    }
    for (int first = 0; first < n; first += kCopyMax) {
        const int m = n - first < kCopyMax ? n - first : kCopyMax;
        Segments seg{};
        for (int k = 0; k < m; ++k) {
            const HostCopy& h = c[first + k];
            seg.dst[k] = to_device ? h.dev : h.host;
            seg.src[k] = to_device ? h.host : h.dev;
            seg.bytes[k] = h.bytes;
        }
        const size_t per_block = size_t(kCopyBlock) * kPerThread * 16;
        const int blocks = int(most / per_block + 1 < 16 ? most / per_block + 1 : 16);
        k_copy<<<dim3(blocks, m), kCopyBlock, 0, s>>>(seg);
        if (launches) ++*launches;
    }
    return cudaGetLastError() == cudaSuccess ? LULESH_OK : LULESH_ECUDA;
}

}  // namespace lulesh
