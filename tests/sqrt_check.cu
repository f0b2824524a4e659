// Compares the square roots of csrc/phase_math.cuh with sqrtf over bit patterns.
#include <cuda_runtime.h>

#include "../pystamps_b200/csrc/phase_math.cuh"

using namespace ps2;

// Patterns first .. first + count - 1, a grid-stride loop. sqrt_rn: every pattern;
// sqrt_newton2: those of its range, the pattern beside it in the other half. NaN
// equals NaN. bad[0], bad[1]: mismatches.
__global__ void k_compare(unsigned first, unsigned long long count, unsigned long long* bad) {
  unsigned long long one = 0, two = 0;
  for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
    const unsigned u = first + static_cast<unsigned>(i);
    const float q = __uint_as_float(u), want = sqrtf(q), got = sqrt_rn(q);
    const bool both_nan = want != want && got != got;
    if (!both_nan && __float_as_uint(want) != __float_as_uint(got)) ++one;
    if (u - kSqrtLo < kSqrtSpan) {
      const unsigned v = u ^ 1u;  // the range starts at an even pattern and ends before one
      const float2 r = sqrt_newton2(make_float2(q, __uint_as_float(v)));
      if (__float_as_uint(r.x) != __float_as_uint(want) ||
          __float_as_uint(r.y) != __float_as_uint(sqrtf(__uint_as_float(v))))
        ++two;
    }
  }
  if (one) atomicAdd(bad, one);
  if (two) atomicAdd(bad + 1, two);
}

extern "C" int sqrt_check(unsigned first, unsigned long long count, unsigned long long* mismatches) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 2 * sizeof(*d));
  if (e == cudaSuccess) e = cudaMemset(d, 0, 2 * sizeof(*d));
  if (e == cudaSuccess) {
    k_compare<<<148 * 8, 256>>>(first, count, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, 2 * sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return static_cast<int>(e);
}
