// lp_scratch.cuh - growable device scratch of a translation unit.
#pragma once

#include <vector>

#include "lp_common.cuh"

namespace lp {

// Scratch that a translation unit owns. A buffer that has been handed to a launch may be baked into a captured
// CUDA graph (its address and the tensor maps built from it), so a buffer is never freed when a larger one is
// needed: superseded buffers are kept until laplace_cuda_shutdown. Growing calls the allocator, which is illegal
// while the call's stream is being captured: such a call is refused and the capture stays valid.
struct Scratch {
    void*  p = nullptr;
    size_t cap = 0;
    std::vector<void*> retired;
    int ensure(size_t n, cudaStream_t st) {
        if (n <= cap) return LAPLACE_OK;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone)
            return fail(LAPLACE_ERR_STATE, "the call needs %zu bytes of scratch but only %zu are allocated, and its stream is being "
                                           "captured: make the same call once before the capture begins", n, cap);
        if (p) retired.push_back(p);
        p = nullptr; cap = 0;
        cudaError_t e = cudaMalloc(&p, n + n / 8);
        if (e != cudaSuccess) return cuda_check(e, "cudaMalloc scratch");
        cap = n + n / 8;
        return LAPLACE_OK;
    }
    void release() {
        if (p) cudaFree(p);
        for (void* q : retired) cudaFree(q);
        retired.clear();
        p = nullptr; cap = 0;
    }
};

Scratch& gemm_scratch();       // of the dense matmuls with more than 8 rows (lp_gemm_sa.cu)

}  // namespace lp
