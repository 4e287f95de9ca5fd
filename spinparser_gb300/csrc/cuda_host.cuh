// Host-side CUDA helpers of the XYZ and TRI cores: status check, device allocation, host to
// device copy and the grid of elementwise kernels.
#pragma once

#include <cuda_runtime.h>
#include <algorithm>
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

// Page-locked memory that a handle's small results are copied to.  The driver stages a copy to pageable memory and waits for
// each by itself; a measurement's four or five arrays come in one copy here (square r2, N = 16: 277 -> 214 us for a cutoff
// step, two measurements and the state in and out).
class Pinned {
  public:
    Pinned() = default;
    Pinned(const Pinned &) = delete;
    Pinned &operator=(const Pinned &) = delete;
    ~Pinned() { release(); }
    void alloc(size_t bytes) { check_cuda(cudaHostAlloc(&p_, std::max<size_t>(bytes, 16), cudaHostAllocDefault), "cudaHostAlloc"); }
    void release() {
        if (p_) cudaFreeHost(p_);
        p_ = nullptr;
    }
    // `count` elements from the device, once the stream's work so far is done
    template <class T>
    const T *fetch(const T *src, size_t count, cudaStream_t s) {
        if (count) check_cuda(cudaMemcpyAsync(p_, src, count * sizeof(T), cudaMemcpyDeviceToHost, s), "D2H");
        check_cuda(cudaStreamSynchronize(s), "D2H sync");
        return static_cast<const T *>(p_);
    }

  private:
    void *p_ = nullptr;
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
