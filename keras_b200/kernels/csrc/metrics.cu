// Running means of a training loop, one launch an operation: their totals and counts are single numbers on the device, and each elementwise
// operation on one costs a launch and a gap of some two microseconds, at every step.  The same roundings as those operations, one by one.
#include "common.cuh"

namespace {
__global__ void mean_update_kernel(float* total, float* count, const float* value, float weight) {
  *total = __fadd_rn(*total, __fmul_rn(*value, weight));
  *count = __fadd_rn(*count, weight);
}
__global__ void mean_result_kernel(const float* total, const float* count, float* out) {
  const float t = *total, n = *count;
  *out = n == 0.f ? 0.f : __fdiv_rn(t, n);
}
__global__ void mean_clear_kernel(float* total, float* count) { *total = *count = 0.f; }
}  // namespace

// total += value * weight, count += weight
KB_API int kb200_mean_update(float* total, float* count, const float* value, float weight, cudaStream_t stream) {
  mean_update_kernel<<<1, 1, 0, stream>>>(total, count, value, weight);
  KB_CHECK_LAUNCH("mean_update");
  return 0;
}
// out = total / count, zero without a count
KB_API int kb200_mean_result(const float* total, const float* count, float* out, cudaStream_t stream) {
  mean_result_kernel<<<1, 1, 0, stream>>>(total, count, out);
  KB_CHECK_LAUNCH("mean_result");
  return 0;
}
KB_API int kb200_mean_clear(float* total, float* count, cudaStream_t stream) {
  mean_clear_kernel<<<1, 1, 0, stream>>>(total, count);
  KB_CHECK_LAUNCH("mean_clear");
  return 0;
}
