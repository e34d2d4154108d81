// pvl_stream_create(): a stream for graph captures that no stream pool also hands out.
#include <cuda_runtime.h>

#include "pvl_status.h"

extern "C" int pvl_stream_create(void** stream)
{
    if (!stream)
        return pvl_fail(PVL_ERR_ARG, "pvl_stream_create: null pointer argument");
    cudaStream_t s = nullptr;
    const cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e != cudaSuccess)
        return pvl_fail(PVL_ERR_CUDA, "pvl_stream_create: %s", cudaGetErrorString(e));
    *stream = s;
    return PVL_OK;
}
