// Checks of the in-range division and square root (jc_exact.cuh) against the
// IEEE operations, on the device.
#include <cuda_runtime.h>

#include "jc_common.h"
#include "jc_exact.cuh"

namespace jc {
namespace {

constexpr float ONES = 1.99999988079071045f;  // 2 - 2^-23, an all-ones significand

__device__ __forceinline__ uint64_t mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// 1.f times 2^e, e uniform in [lo, hi].
__device__ __forceinline__ float draw(uint32_t r, uint32_t s, int lo, int hi) {
  return ldexpf(__uint_as_float(0x3F800000u | (r & 0x7FFFFFu)), lo + (int)(s % (uint32_t)(hi - lo + 1)));
}

__device__ __forceinline__ void count(unsigned long long* out, uint32_t bad) {
  bad = __reduce_add_sync(0xFFFFFFFFu, bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(out, (unsigned long long)bad);
}

// bad[0]: roots of every f32 in [2^-40, 2^60); bad[1]: every smaller one, whose
// root only has to stay under the 1e-6 clamp (NaN is dropped by it).
__global__ void __launch_bounds__(256) k_check_roots(unsigned long long* bad) {
  const uint32_t step = gridDim.x * blockDim.x, lo = (127u - 40u) << 23, hi = (127u + 60u) << 23;
  uint32_t wrong = 0, loose = 0;
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < hi; b += step) {
    const float s = __uint_as_float(b), r = dev::sqrt_in_range(s);
    if (b >= lo) wrong += __float_as_uint(r) != __float_as_uint(__fsqrt_rn(s)) ? 1u : 0u;
    else if (s < 1e-12f) loose += fmaxf(r, 1e-6f) != 1e-6f ? 1u : 0u;
  }
  count(bad, wrong);
  count(bad + 1, loose);
}

// Quotients. bad[2]: every numerator significand over the all-ones divisor and its
// neighbours; bad[3]: random pairs over the whole contract; bad[4]: the stress
// sweep's operands (numerators from 2^-69, divisors from 1e-6 to 2^29); bad[5]:
// numerators at the halfway points between two quotients and beside them.
__global__ void __launch_bounds__(256) k_check_quotients(uint64_t pairs, unsigned long long* bad) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x, t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t wrong[4] = {};
  auto check = [&](int k, float n, float d) {
    wrong[k] += __float_as_uint(dev::div_in_range(n, d)) != __float_as_uint(__fdiv_rn(n, d)) ? 1u : 0u;
  };
  for (uint64_t t = t0; t < (1ull << 23); t += step)
    for (int k = 0; k < 4; ++k) check(0, __uint_as_float(0x3F800000u | (uint32_t)t), __uint_as_float(__float_as_uint(ONES) - k));
  for (uint64_t t = t0; t < pairs; t += step) {
    const uint64_t a = mix(2 * t), b = mix(2 * t + 1);
    const float sign = b >> 63 ? -1.0f : 1.0f;
    check(1, sign * draw((uint32_t)a, (uint32_t)(b >> 32) & 0xFFFFu, -60, 59), draw((uint32_t)(a >> 32), (uint32_t)b & 0xFFFFu, -60, 59));
    check(2, sign * draw((uint32_t)a, (uint32_t)(b >> 32) & 0xFFFFu, -69, 28),
          fmaxf(draw((uint32_t)(a >> 32), (uint32_t)b & 0xFFFFu, -20, 28), 1e-6f));
    // d (q + half an ulp), rounded, and the numerators beside it
    const float d = draw((uint32_t)(a >> 32), (uint32_t)b & 0xFFFFu, -20, 28), q = draw((uint32_t)a, 0u, 0, 0);
    const float n = (float)((double)d * ((double)q + 5.9604644775390625e-8));
    for (int k = -1; k <= 1; ++k) check(3, __uint_as_float(__float_as_uint(n) + k), d);
  }
  for (int k = 0; k < 4; ++k) count(bad + 2 + k, wrong[k]);
}

}  // namespace
}  // namespace jc

extern "C" jc_status jc_selftest_exact(uint64_t pairs, uint64_t* mismatches) {
  using namespace jc;
  if (!mismatches) return JC_ERR_ARG;
  unsigned long long* bad = nullptr;
  jc_status rc = JC_OK;
  try {
    JC_CUDA_CHECK(cudaMalloc(&bad, 6 * sizeof(*bad)));
    JC_CUDA_CHECK(cudaMemset(bad, 0, 6 * sizeof(*bad)));
    k_check_roots<<<148 * 8, 256>>>(bad);
    k_check_quotients<<<148 * 8, 256>>>(pairs, bad);
    JC_CUDA_CHECK(cudaGetLastError());
    JC_CUDA_CHECK(cudaMemcpy(mismatches, bad, 6 * sizeof(*bad), cudaMemcpyDeviceToHost));
  } catch (const Error& e) {
    rc = e.code;
  } catch (...) {
    rc = JC_ERR_ARG;
  }
  if (bad) cudaFree(bad);
  return rc;
}
