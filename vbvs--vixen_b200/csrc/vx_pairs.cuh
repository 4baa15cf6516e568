// vx_pairs.cuh - binary32 arithmetic on pairs (one instruction for two values),
// each half rounded as the scalar operation rounds it.
//
// A packed product whose result goes into a packed sum is fused into one
// rounding by the assembler, with -fmad=false too (and the intrinsics' _rn
// names, and a product written as fma(a, b, -0) with a constant -0).  Here the
// kernels must round twice, so mul2 is fma(a, b, z) with z = -0 handed to the
// kernel at run time, which nothing can fold: a * b + -0 is a * b rounded, its
// sign of zero included.  Checked against __fmul_rn and __fadd_rn on 10^8
// random triples: no difference (one in four with the fused form).
#pragma once

namespace vx {
namespace {

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
// a * b; neg_zero: -0 in a register or parameter the compiler knows nothing about
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float neg_zero) { return __ffma2_rn(a, b, dup2(neg_zero)); }
// b - a: the product by -1 is exact
__device__ __forceinline__ float2 sub2(float2 b, float2 a) { return __ffma2_rn(a, dup2(-1.0f), b); }

}  // namespace
}  // namespace vx
