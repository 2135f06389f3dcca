// Error types, CUDA call checking and a grow-only device array shared by the host-side code.
#pragma once

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>
#include <vector>

namespace smx {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct ArgError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

#define SMX_CUDA(expr)                                                                              \
    do {                                                                                            \
        cudaError_t err__ = (expr);                                                                 \
        if (err__ != cudaSuccess) {                                                                 \
            cudaGetLastError(); /* reported here, not again by the next launch check */             \
            throw ::smx::CudaError(std::string(#expr) + ": " + cudaGetErrorString(err__));          \
        }                                                                                           \
    } while (0)

// Kernels of one evaluation follow one another on a stream and are short for small structures, so the drain-and-launch gap
// between them matters. There they are launched with programmatic stream serialization (Launcher::overlap): a kernel may become
// resident while its predecessor runs, and chain_begin(), the first statement of every kernel launched this way, waits until
// the predecessor has finished and its writes are visible, then lets the successor come in (without the attribute both
// instructions do nothing).
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
struct Launcher {
    cudaStream_t stream = nullptr;
    bool overlap = false;
};
// `cluster`: CTAs of a thread-block cluster (1: no clusters).
template <typename... P, typename... A>
inline void chain_launch(const Launcher& on, void (*kern)(P...), dim3 grid, int block, size_t smem, int cluster, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = on.stream;
    cudaLaunchAttribute at[2]{};
    unsigned n = 0;
    if (on.overlap) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = 1; at[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = at; cfg.numAttrs = n;
    SMX_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

// Grow-only device array. `n` is the logical length, `cap` the allocated one.
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t cap = 0, n = 0;
    ~DevBuf() { if (p) cudaFree(p); }
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    // Set the logical length to `count`, reallocating if needed; contents survive only if `keep`.
    void resize(size_t count, cudaStream_t s, bool keep = false) {
        if (count > cap) {
            T* q = nullptr;
            const size_t newcap = count + count / 8 + 16;
            SMX_CUDA(cudaMalloc(&q, newcap * sizeof(T)));
            if (keep && p && n) SMX_CUDA(cudaMemcpyAsync(q, p, n * sizeof(T), cudaMemcpyDeviceToDevice, s));
            if (p) { SMX_CUDA(cudaStreamSynchronize(s)); cudaFree(p); }
            p = q;
            cap = newcap;
        }
        n = count;
    }
    void upload(const std::vector<T>& h, cudaStream_t s) {
        resize(h.size(), s);
        if (!h.empty()) SMX_CUDA(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    void zero(cudaStream_t s) { if (n) SMX_CUDA(cudaMemsetAsync(p, 0, n * sizeof(T), s)); }
};

}  // namespace smx
