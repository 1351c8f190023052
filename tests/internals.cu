// What tests reach past the C interface: fields of a context that no caller
// sets, and the arithmetic of fp64_math.cuh beside the built-in functions.
#include "fp64_math.cuh"
#include "pd_internal.cuh"

using namespace pdb;

namespace {
struct Counts {
  unsigned long long roots, quotients, bad_root, bad_quotient, bad_by_m;
};

__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

// The numerators for which quotient_d is the rounded quotient.
__device__ bool numerator_in_range(double a) { return a == 0.0 || (fabs(a) >= 0x1p-500 && fabs(a) < 0x1p500); }

// a: numerators, c: |Y|^2 of the divisors (and m).
__global__ void k_compare(int64_t n, const double* a, const double* c, Counts* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (root_in_range(c[i])) {
      const RootD r = root_d(c[i]);
      atomicAdd(&out->roots, 1ull);
      if (!same(r.root, __dsqrt_rn(c[i]))) atomicAdd(&out->bad_root, 1ull);
      if (recip_in_range(r.root) && numerator_in_range(a[i])) {
        const double rd = recip_d(r.root, r.inv);
        atomicAdd(&out->quotients, 1ull);
        if (!same(quotient_d(a[i], r.root, rd), __ddiv_rn(a[i], r.root))) atomicAdd(&out->bad_quotient, 1ull);
      }
    }
    if (divisor_in_range(c[i]) && numerator_in_range(a[i]) &&
        !same(quotient_d(a[i], c[i], __drcp_rn(c[i])), __ddiv_rn(a[i], c[i])))
      atomicAdd(&out->bad_by_m, 1ull);
  }
}
}  // namespace

extern "C" int compare_fp64(int64_t n, const double* a, const double* c, unsigned long long* counts) {
  double *da = nullptr, *dc = nullptr;
  Counts* out = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&da, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&dc, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(Counts));
  if (e == cudaSuccess) e = cudaMemset(out, 0, sizeof(Counts));
  if (e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dc, c, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_compare<<<1184, 256>>>(n, da, dc, out);
    e = cudaMemcpy(counts, out, sizeof(Counts), cudaMemcpyDeviceToHost);
  }
  cudaFree(da);
  cudaFree(dc);
  cudaFree(out);
  return (int)e;
}

// The arrivals of the kernels that loop in one launch are counted from one that
// no wait's target is reached from, or from zero as ever.
extern "C" void set_waits_run_out(pd_ctx* c, int on) { c->bar_fill = on ? 0x80 : 0; }

// More shared memory than a block can have: the driver refuses the one launch
// of the time steps and of the CG solve.
extern "C" void ask_too_much(pd_ctx* c) { c->small_bytes = c->cg_bytes = 512 << 10; }
extern "C" int small_step_threads(pd_ctx* c) { return c->small_threads; }
