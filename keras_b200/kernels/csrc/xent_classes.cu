// Softmax cross-entropy of a classifier, fewer than 64 classes: the row kernels of xent_rows.cuh with exponentials and logarithms in full
// accuracy (this file is compiled without fast math), which a float32 model's loss shows.  log_softmax, its loss and their two gradients, with
// casts around them for bf16, were eight launches of the library: [100352, 21] bf16 10.7 + 7.9 us for the two softmax kernels alone, here
// 6.3 + 5.7.
#define XE_EXP expf
#include "xent_rows.cuh"

int kb200_xent_classes_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, long long ld, int vec, int dtype,
                           int* outside, cudaStream_t stream) {
  if (dtype == 1) xe_narrow_fwd<__nv_bfloat16>((const __nv_bfloat16*)logits, labels, loss, lse, rows, V, ld, vec, stream, 1, outside);
  else xe_narrow_fwd<float>((const float*)logits, labels, loss, lse, rows, V, ld, vec, stream, 1, outside);
  KB_CHECK_LAUNCH("xent_classes_fwd");
  return 0;
}

int kb200_xent_classes_bwd(const void* logits, const long long* labels, const float* lse, const float* dloss, int dloss_stride, void* dlogits, long long rows, int V,
                           long long ld, int zero_to, int vec, int dtype, cudaStream_t stream) {
  if (dtype == 1)
    xe_narrow_bwd<__nv_bfloat16>((const __nv_bfloat16*)logits, labels, lse, dloss, dloss_stride, (__nv_bfloat16*)dlogits, rows, V, ld, zero_to, vec, stream, 1);
  else
    xe_narrow_bwd<float>((const float*)logits, labels, lse, dloss, dloss_stride, (float*)dlogits, rows, V, ld, zero_to, vec, stream, 1);
  KB_CHECK_LAUNCH("xent_classes_bwd");
  return 0;
}
