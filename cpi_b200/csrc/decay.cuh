// The decays of the recurrent mixers, one function for every kernel that takes them.
#pragma once
#include "common.cuh"

namespace cpi {

__device__ __forceinline__ float softplus_f(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float log_sigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
// a = sigmoid(z + b)^(1 / tau); one function for the kernel that prepares a prompt's decays and for the recurrence
// that computes a decoded token's own, so that both give the same bits
// (kind 1: a = exp(-rate * softplus(z + b)), rate = exp(A_log) of the row's head)
__device__ __forceinline__ float row_decay_f(float z, float b, float inv_tau, int kind = 0, float rate = 0.f) {
  if (kind == 1) return expf(-rate * softplus_f(z + b));
  return expf(log_sigmoid_f(z + b) * inv_tau);
}

}  // namespace cpi
