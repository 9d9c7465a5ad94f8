// Soft-max probability of a logit, from its row's log-sum-exp times log2(e).  One expression for every kernel that turns the language-model
// head's logits into their gradient: which of them runs depends on the memory that is free, the bits must not.
#pragma once

namespace mcb {

constexpr float CE_LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ce_prob(float logit, float lse_log2e) {
  return exp2f(fmaf(logit, CE_LOG2E, -lse_log2e));
}

}  // namespace mcb
