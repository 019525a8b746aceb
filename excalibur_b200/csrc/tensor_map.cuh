// The driver's tensor-map encoder, looked up once (no link against libcuda).
#pragma once
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

namespace exb {

inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
        return PFN_cuTensorMapEncodeTiled_v12000(nullptr);
    }();
    return fn;
}

}  // namespace exb
