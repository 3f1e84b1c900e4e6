// cg_loop.cu -- the device-side end of the CG loop.  Apart from solver.cu because setting a
// graph condition needs relocatable device code (cudadevrt), and a call of it inside the
// direction kernel would hold that kernel to the calling convention's registers.
#include "cg.cuh"

namespace vfgpu {

namespace {
__global__ void cg_condition_kernel(const CGState* st, cudaGraphConditionalHandle loop) {
  cudaGraphSetConditional(loop, !st->done && st->its < st->yield);
}
// End of an iteration of the PCG around the V-cycle: the stopping test on
// ||D^-1 r|| from its block partials.
__global__ void __launch_bounds__(RED_THREADS) mgcg_end_kernel(CGState* st, const double* partial, int nblk,
                                                               int loop, cudaGraphConditionalHandle handle) {
  if (!__syncthreads_or(st->done)) {
    double s[1];
    final_sum<1>(partial, nblk, s);
    if (threadIdx.x == 0) {
      const int its = st->its + 1;
      const double dp = sqrt(s[0]);
      int reason = CG_RUNNING;
      if (!(dp == dp)) reason = CG_DIVERGED_NAN;
      else if (dp <= st->ttol) reason = CG_CONVERGED_RTOL;
      else if (dp >= st->dtol * st->rnorm0) reason = CG_DIVERGED_DTOL;
      else if (its >= st->maxit) reason = CG_DIVERGED_ITS;
      st->its = its;
      st->zz = s[0];
      if (reason) {
        st->reason = reason;
        st->done = 1;
      }
    }
  }
  if (loop && threadIdx.x == 0) cudaGraphSetConditional(handle, !st->done);
}
__global__ void cg_yield_kernel(CGState* st, int yield) { st->yield = yield; }
}  // namespace

cudaError_t cg_set_condition(const CGState* st, cudaGraphConditionalHandle loop, cudaStream_t s) {
  cg_condition_kernel<<<1, 1, 0, s>>>(st, loop);
  return cudaGetLastError();
}

cudaError_t mgcg_end(CGState* st, const double* partial, int64_t n, const cudaGraphConditionalHandle* loop,
                     cudaStream_t s) {
  mgcg_end_kernel<<<1, RED_THREADS, 0, s>>>(st, partial + RED_BLOCKS, cg_blocks(n, 8), loop != nullptr,
                                            loop ? *loop : 0);
  return cudaGetLastError();
}

cudaError_t cg_set_yield(CGState* st, int yield, cudaStream_t s) {
  cg_yield_kernel<<<1, 1, 0, s>>>(st, yield);
  return cudaGetLastError();
}

}  // namespace vfgpu
