// What the BatchNorm backward passes share: dx = a dy' + b x + c with per-channel coefficients from the reduction's sums.  Every thread
// of an apply pass works its channels' coefficients out for itself: 2 C values out of L2, where a launch of its own between the two passes
// cost 2 us and a gap ([7776, 384], seven layers: 26 us a step).
#pragma once

struct BnCoef {
  const float* sums;  // [2 C]: sum of dy', and of dy' * normalised x
  const float* gamma;
  const float* mean;
  const float* invstd;
  float inv_m;
  float* dgamma_acc;  // persistent gradient storage that the sums are added to, by one block; either may be null
  float* dbeta_acc;
};

__device__ __forceinline__ void bn_coefficients(const BnCoef& q, int C, int c, float& a, float& b, float& cc) {
  const float g = q.gamma ? q.gamma[c] : 1.f, is = q.invstd[c], mu = q.mean[c];
  const float s1 = q.sums[c] * q.inv_m, s2 = q.sums[C + c] * q.inv_m;
  a = g * is;
  b = -a * is * s2;
  cc = a * (mu * is * s2 - s1);
}
__device__ __forceinline__ void bn_keep_sums(const BnCoef& q, int C, int c) {
  if (q.dgamma_acc != nullptr) q.dgamma_acc[c] += q.sums[C + c];
  if (q.dbeta_acc != nullptr) q.dbeta_acc[c] += q.sums[c];
}
