// Pieces shared by the kernels of a conjugate-gradient iteration (k_qs.cu,
// k_coarse.cu): the device-resident scalars, sums finished by the last block,
// and the report the host follows.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace pdb {

// What the host follows (mapped pinned memory): iterations done * 8 + state, one
// word, so that no fence to the host has to order it after another.
using CgReport = unsigned long long;
enum CgState { CG_RUNNING = 0, CG_CONVERGED = 1, CG_NONFINITE = 2, CG_ZERO_RHS = 3, CG_MAX_ITERATIONS = 4 };

// Device state of one solve.
struct CgCtl {
  double rz, pq, beta, rr0;  // r.z, p.q, r.z / (r.z before), |r|^2 at the start
  double tol, rel;           // the stopping test and |r| / |r| of the start
  long long max_it, it;
  int state;              // CgState; every kernel of a later iteration returns at once when it is not 0
  unsigned int ticket[2];  // blocks finished, of the p.q sum and of the dot products (wrap to 0)
  CgReport* report;
  int waits;  // ST_TIMEOUT when a block of the one-launch solve gave up waiting
};

// Block sums of NV values per thread (T threads), a fixed tree: warp shuffles,
// then the warps' sums in order. Every thread gets the totals.
template <int NV, int T>
__device__ __forceinline__ void cg_block_sum(double (&v)[NV], double (*sh)[T / 32]) {
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][threadIdx.x >> 5] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double s = sh[k][0];
#pragma unroll
    for (int w = 1; w < T / 32; ++w) s += sh[k][w];
    v[k] = s;
  }
  __syncthreads();
}

// Grid sums: each block's sums go to partial[NV blk ..]; the block that
// finishes last adds them in block order (thread t takes blocks t, t + T, ..;
// then the block tree) and gets true, with the totals in v. No block waits for
// another.
template <int NV, int T>
__device__ __forceinline__ bool cg_grid_sum(double (&v)[NV], double* partial, unsigned int* ticket) {
  __shared__ double sh[NV][T / 32];
  __shared__ bool last;
  cg_block_sum<NV, T>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) partial[(size_t)NV * blockIdx.x + k] = v[k];
    __threadfence();
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
#pragma unroll 4
  for (unsigned b = threadIdx.x; b < gridDim.x; b += T)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += __ldcg(partial + (size_t)NV * b + k);
  cg_block_sum<NV, T>(v, sh);
  return true;
}

// The iteration's scalars from r.z and r.r of the new residual (one thread):
// at the start of a solve the reference residual, else beta and the stopping
// test on sqrt(r.r / r.r of the start).
__device__ __forceinline__ void cg_scalars(CgCtl* c, double rz, double rr, bool first) {
  int state = CG_RUNNING;
  double rel = 1.0;
  if (first) {
    c->rr0 = rr;
    c->beta = 0.0;
    c->it = 0;
    if (rr == 0.0) state = CG_ZERO_RHS, rel = 0.0;
  } else {
    c->beta = rz / c->rz;
    rel = sqrt(rr) / sqrt(c->rr0);
    c->it += 1;
    if (!isfinite(rel)) state = CG_NONFINITE;
    else if (rel <= c->tol) state = CG_CONVERGED;
    else if (c->it >= c->max_it) state = CG_MAX_ITERATIONS;
  }
  c->rz = rz;
  c->state = state;
  c->rel = rel;
  if (c->report) *(volatile CgReport*)c->report = (unsigned long long)c->it * 8 + state;
}

}  // namespace pdb
