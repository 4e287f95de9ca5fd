// Host-side CUDA helpers: status check, device allocation, host to device copy, small results on
// the host and the grid of elementwise kernels.
#pragma once

#include <cuda_runtime.h>
#include <unistd.h>
#include <algorithm>
#include <cstdlib>
#include <new>
#include <string>
#include "host/capi_common.hpp"

namespace spn {
namespace cuh {

inline void check_cuda(cudaError_t e, const char *what) {
    if (e != cudaSuccess) throw Error(ErrorType::Cuda, std::string(what) + ": " + cudaGetErrorString(e));
}

// count elements of T (at least one) plus 16 bytes of slack for vector tail reads
template <class T>
T *dalloc(size_t count, const char *what) {
    void *p = nullptr;
    check_cuda(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T) + 16), what);
    return static_cast<T *>(p);
}

template <class T>
void h2d(T *dst, const T *src, size_t count, cudaStream_t s) {
    if (count) check_cuda(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyHostToDevice, s), "cudaMemcpyAsync H2D");
}

// Host memory that a handle's small results (a measurement, the status word) are copied to, in one copy each: four copies take 39 us,
// one 14, and 12.4 to page-locked memory.  It is taken with the first copy, so a flow whose results are not fetched by itself (a batch's)
// has none, and pages of its own are locked in place: cudaHostAlloc and cudaFreeHost cost 240 us a handle, which a flow of a few
// steps does not earn back; registering and unregistering 16.
class HostResults {
  public:
    HostResults() = default;
    HostResults(const HostResults &) = delete;
    HostResults &operator=(const HostResults &) = delete;
    ~HostResults() { release(); }
    // `count` elements from the device, once the stream's work so far is done; valid until the next fetch
    template <class T>
    const T *fetch(const T *src, size_t count, cudaStream_t s) {
        reserve(count * sizeof(T));
        if (count) check_cuda(cudaMemcpyAsync(p_, src, count * sizeof(T), cudaMemcpyDeviceToHost, s), "D2H");
        check_cuda(cudaStreamSynchronize(s), "D2H sync");
        return static_cast<const T *>(p_);
    }

  private:
    void reserve(size_t bytes) {
        if (p_ && bytes <= size_) return;
        release();
        const size_t page = size_t(sysconf(_SC_PAGESIZE));
        const size_t size = (std::max<size_t>(bytes, 1) + page - 1) / page * page;
        p_ = std::aligned_alloc(page, size);
        if (!p_) throw std::bad_alloc();
        size_ = size;
        locked_ = cudaHostRegister(p_, size, cudaHostRegisterDefault) == cudaSuccess;
        if (!locked_) cudaGetLastError();  // the copies are staged by the driver then
    }
    void release() {
        if (locked_) cudaHostUnregister(p_);
        std::free(p_);
        p_ = nullptr;
        size_ = 0;
        locked_ = false;
    }
    void *p_ = nullptr;
    size_t size_ = 0;
    bool locked_ = false;
};

// blocks of 256 threads for an elementwise kernel over n items (grid-stride beyond 4096 blocks)
inline int copy_grid(long long n) { return int(std::min<long long>((n + 255) / 256, 4096)); }

// The frequency mesh of a diagnostic read: 2 <= n <= max_n positive, strictly ascending values.
inline void check_mesh(const float *pos, int n, int max_n) {
    if (!pos || n < 2 || n > max_n)
        throw Error(ErrorType::Argument, "mesh: need 2 <= n <= " + std::to_string(max_n) + " values");
    for (int i = 0; i < n; ++i)
        if (!(pos[i] > 0.0f) || (i > 0 && !(pos[i] > pos[i - 1])))
            throw Error(ErrorType::Argument, "mesh: values must be positive and strictly ascending");
}

// The index of the mesh value |w| (the channel's own frequency of an access buffer).
inline int mesh_index_of(const float *pos, int n, float w) {
    const float a = w < 0.0f ? -w : w;
    for (int i = 0; i < n; ++i)
        if (pos[i] == a) return i;
    throw Error(ErrorType::Argument, "the channel's own frequency must be a mesh value");
}

}  // namespace cuh
}  // namespace spn
