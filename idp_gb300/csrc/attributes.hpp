// Launch attributes of kernels (dynamic shared memory, cluster sizes) belong to a
// device: a process with contexts on two devices has to set them on both. Every
// context keeps one of these and sets what its launches need once.
#pragma once
#include <cuda_runtime_api.h>
#include <vector>

namespace idp {

struct KernelAttributes {
    std::vector<const void*> done;  // kernels whose attribute is set
    cudaError_t set(const void* kernel, cudaFuncAttribute what, int value) {
        for (const void* k : done)
            if (k == kernel) return cudaSuccess;
        const cudaError_t e = cudaFuncSetAttribute(kernel, what, value);
        if (e == cudaSuccess) done.push_back(kernel);
        return e;
    }
};

}  // namespace idp
