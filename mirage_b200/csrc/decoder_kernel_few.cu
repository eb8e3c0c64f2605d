// The decoder megakernel for graphs of few tokens on the general instantiation (decoder_kernels.cu).  In a file of its own: beside the other
// instantiations the register allocation of all of them comes out worse.
#include "decoder_kernels.h"
#include "megakernel.cuh"

cudaError_t mpk_prepare_few(int smem_bytes) {
  return cudaFuncSetAttribute(mpk::mpk_megakernel<true, false, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
}
void mpk_launch_few(const mpk::KernelParams &params, int smem_bytes, cudaStream_t stream) {
  mpk::mpk_megakernel<true, false, 0, true><<<params.num_workers, mpk::block_threads(true), smem_bytes, stream>>>(params);
}
