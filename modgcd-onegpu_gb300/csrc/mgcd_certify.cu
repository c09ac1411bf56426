// mgcd_certify.cu -- exhaustive certification of the float quotient steps of the modular
// inverse (inv_euclid) on the device it runs on (the reference certifies its quoRem<QUASI>
// the same way, per device, certifyQuoRemQuasi.cu:25-48).
//
// Each step takes the quotient Q = rint(f0 * rcp(f1)) from fma_rn(f0, rcp(f1), 1.5 * 2^23) and
// the remainder fma_rn(-Q, f1, f0); it makes progress (|remainder| < |f1|) and is exact iff Q
// is within 1 of f0 / f1 (at most 1 at multiples: Q exact) and the remainder is representable:
//   first part, quotients from integer remainders rounded to float: f1 of every 24-bit
//            significand, f0 any float with f1 < f0 < 2^13 f1.  Scaling both by a power of two
//            changes nothing (one reciprocal of a normal number, products and sums well
//            inside the range), so f1 in [2^23, 2^24) covers every exponent.  (Larger
//            quotients have an error of up to 2^-22 of themselves besides: the remainder is
//            then within 2^-20 of the dividend, which is progress all the same.)
//   second part, exact operands: 2 <= f1 < f0 < 2^23 with Q below 2^22, and f0 < f1 (the first
//            step of the part may start there): Q of 0 or 1.
// On [k f1, (k+1) f1 - 1] the allowed quotients are k at f0 = k f1 and {k, k + 1} above it.
// For a fixed f1 the estimate is non-decreasing in f0 (every operation is monotone and
// rcp(f1) is fixed), so it is allowed on the whole interval iff it is at the two ends (the
// lowest and the highest float in it): checking both ends of every interval, for every f1,
// covers every pair.  First part: ~1.4e11 end points; second part: ~2.7e8.  The steps run on
// signed remainders; the estimate is odd in each operand (a reciprocal and
// round-to-nearest-even products), so the positive operands checked here cover the negative
// ones too.
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/modgcd.h"
#include "mgcd_device.cuh"
#include "mgcd_plan.h"

namespace mgcd {

namespace {

struct CertOut {
  unsigned long long checked;
  unsigned long long failures;
  uint32_t first_r0, first_r1;
};

// Q allowed for r0 in [k r1, (k+1) r1): k at the bottom end, k or k + 1 above it.
__device__ __forceinline__ bool quot_ok(uint64_t r0, uint32_t r1, uint32_t k, uint32_t Q)
{
  return r0 == (uint64_t)k * r1 ? Q == k : (Q == k || Q == k + 1u);
}

// A step on (f0, f1), f0 in [k f1, (k+1) f1) as integers: an allowed quotient and the exact
// signed remainder.
__device__ __forceinline__ bool step_ok(uint64_t r0, uint32_t r1, uint32_t k)
{
  const float f0 = __ull2float_rn(r0), f1 = __uint2float_rn(r1);   // both exact
  const float nq = INV_MAGIC - inv_quot(f0, f1);
  const int32_t Q = -(int32_t)nq;
  if (!quot_ok(r0, r1, k, (uint32_t)Q)) return false;
  return (int64_t)__fmaf_rn(nq, f1, f0) == (int64_t)r0 - (int64_t)Q * (int64_t)r1;
}

__device__ void fail(CertOut* o, uint64_t r0, uint32_t r1)
{
  if (atomicAdd(&o->failures, 1ull) == 0ull) {
    o->first_r0 = (uint32_t)r0;
    o->first_r1 = r1;
  }
}

__global__ void __launch_bounds__(256) certify_kernel(CertOut* out)
{
  const uint32_t stride = gridDim.x * blockDim.x;
  unsigned long long n = 0;
  // second part: 2 <= r1 < r0 < 2^23
  constexpr uint32_t C_TOP = (1u << 23) - 1u;
  for (uint32_t r1 = 2u + blockIdx.x * blockDim.x + threadIdx.x; r1 <= C_TOP; r1 += stride) {
    for (uint32_t k = 1; k <= C_TOP / r1; ++k) {
      const uint32_t lo = k == 1 ? r1 + 1u : k * r1;
      const uint32_t hi = min((k + 1) * r1 - 1u, C_TOP);
      if (lo > hi) continue;
      n += 2;
      if (!step_ok(lo, r1, k)) fail(out, lo, r1);
      if (!step_ok(hi, r1, k)) fail(out, hi, r1);
    }
    n += 2;                                            // k = 0: r0 in [1, r1 - 1]
    if (!step_ok(1u, r1, 0u)) fail(out, 1u, r1);
    if (!step_ok(r1 - 1u, r1, 0u)) fail(out, r1 - 1u, r1);
  }
  // first part: f1 in [2^23, 2^24), f0 below 2^13 f1 on the float grid
  constexpr uint32_t K_MAX = (1u << 13) - 1u;
  for (uint32_t r1 = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x; r1 < (1u << 24); r1 += stride) {
    for (uint32_t k = 1; k <= K_MAX; ++k) {
      const uint64_t base = (uint64_t)k * r1;
      const uint64_t lo = (uint64_t)__ull2float_ru(k == 1 ? base + 1 : base);
      const uint64_t hi = (uint64_t)__ull2float_rd(base + r1 - 1);
      if (lo > hi) continue;
      n += 2;
      if (!step_ok(lo, r1, k)) fail(out, lo, r1);
      if (!step_ok(hi, r1, k)) fail(out, hi, r1);
    }
  }
  atomicAdd(&out->checked, n);
}

}  // namespace

}  // namespace mgcd

extern "C" int mgcd_certify_inverse(mgcd_context* c, uint64_t* checked, uint64_t* failures, uint32_t* first_r0,
                                    uint32_t* first_r1)
{
  using namespace mgcd;
  if (!c || !checked || !failures) return MGCD_ERR_INVALID_ARG;
  if (c->serving) return MGCD_ERR_BUSY;
  if (cudaSetDevice(c->device) != cudaSuccess) return MGCD_ERR_CUDA;
  cudaStream_t s = c->main.stream;
  DevBuf buf;
  if (buf.grow(sizeof(CertOut), c->pool, s) != cudaSuccess) return MGCD_ERR_CUDA;
  CertOut h = {};
  int rc = MGCD_OK;
  if (cudaMemsetAsync(buf.p, 0, sizeof(CertOut), s) != cudaSuccess) rc = MGCD_ERR_CUDA;
  if (rc == MGCD_OK) {
    certify_kernel<<<c->sms * 8, 256, 0, s>>>(buf.as<CertOut>());
    if (cudaGetLastError() != cudaSuccess) rc = MGCD_ERR_CUDA;
  }
  if (rc == MGCD_OK && (cudaMemcpyAsync(&h, buf.p, sizeof(CertOut), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                        cudaStreamSynchronize(s) != cudaSuccess))
    rc = MGCD_ERR_CUDA;
  buf.release(s);
  cudaStreamSynchronize(s);
  if (rc != MGCD_OK) return rc;
  *checked = h.checked;
  *failures = h.failures;
  if (first_r0) *first_r0 = h.first_r0;
  if (first_r1) *first_r1 = h.first_r1;
  return MGCD_OK;
}
