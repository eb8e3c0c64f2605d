// Entry points of decoder_kernel_few.cu.
#pragma once
#include <cuda_runtime.h>

#include "runtime_types.h"

cudaError_t mpk_prepare_few(int smem_bytes);
void mpk_launch_few(const mpk::KernelParams &params, int smem_bytes, cudaStream_t stream);
