// The sum-product rule's functions for the generic decoders (sparse.cu, sparse_chain.cu).
#pragma once
#include "atanh2.cuh"
#include "decode_common.cuh"

namespace cbk {
namespace {

// TANH_BOUND of ldpc.rs:93; it rounds to 1 in f32, where the bound is the largest
// float below 1 (1 - 2^-24)
template <typename T>
__device__ __forceinline__ T tanh_bound();
template <>
__device__ __forceinline__ double tanh_bound<double>() { return 0.999999999999; }
template <>
__device__ __forceinline__ float tanh_bound<float>() { return __uint_as_float(0x3f7fffffu); }

__device__ __forceinline__ double tanh_t(double x) { return tanh(x); }
__device__ __forceinline__ float tanh_t(float x) { return tanhf(x); }

// f64::clamp(lo, hi)
template <typename T>
__device__ __forceinline__ T clamp_t(T x, T lo, T hi) {
  return x < lo ? lo : (x > hi ? hi : x);
}

// the check-node output 2 atanh(clamp(p, -TANH_BOUND, TANH_BOUND)) (ldpc.rs:451-466)
__device__ __forceinline__ double twice_atanh_t(double p) { return at2::twice_atanh(p, tanh_bound<double>()); }
__device__ __forceinline__ float twice_atanh_t(float p) {
  return mul_rn(2.0f, atanhf(clamp_t(p, -tanh_bound<float>(), tanh_bound<float>())));
}

}  // namespace
}  // namespace cbk
