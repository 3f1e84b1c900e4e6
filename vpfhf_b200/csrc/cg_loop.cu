// cg_loop.cu -- the device-side end of the CG loop.  Apart from solver.cu because setting a
// graph condition needs relocatable device code (cudadevrt), and a call of it inside the
// direction kernel would hold that kernel to the calling convention's registers.
#include "cg.cuh"

namespace vfgpu {

namespace {
__global__ void cg_condition_kernel(const CGState* st, cudaGraphConditionalHandle loop) {
  cudaGraphSetConditional(loop, !st->done && st->its < st->yield);
}
__global__ void cg_yield_kernel(CGState* st, int yield) { st->yield = yield; }
}  // namespace

cudaError_t cg_set_condition(const CGState* st, cudaGraphConditionalHandle loop, cudaStream_t s) {
  cg_condition_kernel<<<1, 1, 0, s>>>(st, loop);
  return cudaGetLastError();
}

cudaError_t cg_set_yield(CGState* st, int yield, cudaStream_t s) {
  cg_yield_kernel<<<1, 1, 0, s>>>(st, yield);
  return cudaGetLastError();
}

}  // namespace vfgpu
