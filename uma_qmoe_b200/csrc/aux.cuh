// Host launchers of the supporting kernels (aux.cu).
#pragma once
#include <cuda_runtime.h>

namespace umaq {
// `chunks` runs of `chunk_elements` values, `chunk_stride` values apart; the codes and scales are written without gaps
int launch_quantize_groups(const void* src_bf16, long long chunk_elements, long long chunks, long long chunk_stride, int enc,
                           void* codes, float* scales, cudaStream_t stream);
}
