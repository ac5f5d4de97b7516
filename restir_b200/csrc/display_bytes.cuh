// The tone mapping's short forms, equal to the ABI's conventions for every value
// that reaches them (tests/test_numeric.py tries them all).
#pragma once

#include "common.cuh"

namespace restir
{

// x / 16.5 (the stops from minEv to maxEv), rounded as the division: a product
// with the reciprocal and one correction by its remainder, exact (Brisebarre,
// Muller and Raina, "Accelerating correctly rounded floating-point division
// when the divisor is known in advance"). Equal for every float from 4e-37
// to 17; x is 0 or at least 4e-7 here.
__device__ __forceinline__ float agxShare(float x)
{
	constexpr float kShare = 1.0f / 16.5f;
	const float q = x * kShare;
	return __fmaf_rn(__fmaf_rn(-q, 16.5f, x), kShare, q);
}

// A channel of the display: rn_unorm8(rn_pow(color, 1 / 2.2)), color itself
// raised to 2.2 first when agx.
static __device__ __noinline__ uint32_t gammaByteExact(float color, bool agx)
{
	return rn_unorm8(rn_pow(fabsf(agx ? rn_pow(color, 2.2f) : color), 1.0f / 2.2f));
}

// The same, from an approximation where its rounding cannot be wrong: the
// powers were a quarter of the pixel's instructions. AgX's two powers undo
// each other, so color itself is the approximation; the other operators take
// __powf. For every float of [0, 1] (of [0, inf] with __powf) the bytes differ
// within 3.1e-5 of the edge between two bytes, if at all, and only there the
// powers decide, as for NaN. (kGammaEdge 1e-3 sent 6 pixels of 1,000 and so a
// sixth of the warps to them: 0.384 ms where 1e-4 took 0.335, all powers 0.423.)
constexpr float kGammaEdge = 1e-4f;

__device__ __forceinline__ uint32_t gammaByte(float color, bool agx)
{
	const float value = agx ? color : __powf(fabsf(color), 1.0f / 2.2f);
	const float t = (value > 1.0f ? 1.0f : value) * 255.0f + 0.5f;
	const float part = t - floorf(t);
	return part > kGammaEdge && part < 1.0f - kGammaEdge ? uint32_t(t) : gammaByteExact(color, agx);
}

} // namespace restir
