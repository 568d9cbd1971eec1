// The tables of the correctly rounded single-precision functions
// (device/lg_crfloat.cuh) on the device, one copy for every module the
// library compiles: a module holds a pointer to them.  Inside the modules'
// sources they were most of the text that NVRTC read for each model.

#include <cuda_runtime.h>

#include "lg_internal.h"

#define LG_CRF_TABLE(name, n) __device__ const __align__(16) unsigned long long name[n]
#include "../device/lg_crf_tables.cuh"

namespace lg {

// Stores the tables' address on the current device in module mod.
int bind_crf_tables(CUmodule mod, std::string& err)
{
    void* words = nullptr;
    CUdeviceptr base = 0;
    size_t bytes = 0;
    cudaError_t e = cudaGetSymbolAddress(&words, lg_crf_words);
    if (e == cudaSuccess && driver()->moduleGetGlobal(&base, &bytes, mod, "lg_crf_base") != CUDA_SUCCESS)
        e = cudaErrorSymbolNotFound;
    if (e == cudaSuccess) e = cudaMemcpy((void*)base, &words, sizeof words, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) return LG_OK;
    err = std::string("function tables: ") + cudaGetErrorString(e);
    return LG_ERR_CUDA;
}

}  // namespace lg
