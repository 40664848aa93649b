// Driver entry points by name: the library links the CUDA runtime only.
#pragma once
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

namespace olv {

// The driver's `name` as of CUDA `version`, or null where the driver lacks it.
template <class Fn>
Fn driver_entry(const char *name, unsigned version) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion(name, &fn, version, cudaEnableDefault, &found) !=
            cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return reinterpret_cast<Fn>(fn);
}

}  // namespace olv
