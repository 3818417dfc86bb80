// 2-D simplex noise and its fractal sum on sm_103a, shared by the
// multi-biome heightfield and the splatmap kernels
// (SuperTerrain+/SuperAlgorithm+/Device/Private/STPSimplexNoise.cu:5-110).
#pragma once

#include "internal.hpp"

namespace stpgb {
namespace simplex {

// STPSimplexNoise.cu:5-7
constexpr float kF2 = 0.3660254038f;
constexpr float kG2 = 0.2113248654f;
constexpr float kH2 = -1.0f + 2.0f * kG2;

// STPSimplexNoise.cu:14-16: not floorf (an exact negative integer maps one lower)
__device__ __forceinline__ int floori(const float x) {
	return x > 0.0f ? static_cast<int>(x) : static_cast<int>(x - 1.0f);
}

// A corner's share from its weight before the power, half less its squared
// distance, and the dot product of its gradient and offset.  Outside its reach
// the share is 0, by a choice and not a branch, which the lanes of a warp would
// take differently, nor by a weight of 0: a sample so far out that its offsets
// or their product overflow has a share of 0 as well.  The roundings are spelled out, here and in the
// weights and dot products, so that no change of the code around moves a height.
__device__ __forceinline__ float corner(const float w, const float dot) {
	const float w2 = __fmul_rn(w, w);
	return w <= 0.0f ? 0.0f : __fmul_rn(__fmul_rn(w2, w2), dot);
}

// Heights and splatmaps round the squared offset of the middle corner
// differently, by at most an ulp of the weight; both stay as they are.
enum class Rounding { heights, splatmap };

// What a block keeps in shared memory for the noise: for every permutation
// slot j, its value and the next slot's as byte offsets into the gradients
// (value * 8 in the low and the high half), and for every slot the gradient
// perm[k] % Gradient2DSize picks, already looked up.  A cell's three corners
// hash with slots j and j + 1 alone, so a sample takes one lookup for all
// three and adds offsets for the rest.
struct Tables {
	uint32_t pair[256];
	float2 gradient[512];
};

__device__ __forceinline__ void load_tables(const stpgb_permutation& perm, Tables& T) {
	const uint32_t n = blockDim.x * blockDim.y;
	for (uint32_t k = threadIdx.y * blockDim.x + threadIdx.x; k < 512u; k += n) {
		const uint32_t p = perm.Permutation[k];
		const uint32_t g = p % perm.Gradient2DSize;
		T.gradient[k] = make_float2(perm.Gradient2D[2u * g], perm.Gradient2D[2u * g + 1u]);
		if (k < 256u) {
			T.pair[k] = (p << 3) | (static_cast<uint32_t>(perm.Permutation[k + 1u]) << 19);
		}
	}
}

// STPSimplexNoise.cu:18-82.  The skew and unskew (x + (x+y)*F2 and
// i - (i+j)*G2) are written with separately rounded operations: fused into
// one multiply-add they shift the cell origin by up to an ulp of the sample
// coordinate, which at world offsets of 10^4-10^5 pixels is a visible error.
// i + j is added as floats: exact wherever i and j are, below 2^24.
template<Rounding R>
__device__ __forceinline__ float simplex2d(const Tables& T, const float x, const float y) {
	const float s = __fmul_rn(__fadd_rn(x, y), kF2);
	const int i = floori(__fadd_rn(x, s)), j = floori(__fadd_rn(y, s));
	const float fi = static_cast<float>(i), fj = static_cast<float>(j);
	const float t = __fmul_rn(__fadd_rn(fi, fj), kG2);
	const float dx0 = __fsub_rn(x, __fsub_rn(fi, t));
	const float dy0 = __fsub_rn(y, __fsub_rn(fj, t));
	const bool east = dx0 > dy0;
	const float dx1 = (east ? dx0 - 1.0f : dx0) + kG2, dy1 = (east ? dy0 : dy0 - 1.0f) + kG2;
	const float dx2 = dx0 + kH2, dy2 = dy0 + kH2;
	const uint32_t pair = T.pair[static_cast<uint32_t>(j) & 255u];
	const uint32_t here = (static_cast<uint32_t>(i) & 255u) * 8u;
	const char* const g = reinterpret_cast<const char*>(T.gradient);
	const uint32_t a0 = here + (pair & 0xFFFFu), a1 = here + (pair >> 16);
	const float2 g0 = *reinterpret_cast<const float2*>(g + a0);
	const float2 g1 = *reinterpret_cast<const float2*>(g + (east ? a0 + 8u : a1));
	const float2 g2 = *reinterpret_cast<const float2*>(g + a1 + 8u);
	const float x1 = R == Rounding::heights ? __fsub_rn(0.5f, __fmul_rn(dx1, dx1)) : __fmaf_rn(-dx1, dx1, 0.5f);
	const float c0 = corner(__fmaf_rn(-dy0, dy0, __fmaf_rn(-dx0, dx0, 0.5f)), __fmaf_rn(g0.y, dy0, __fmul_rn(g0.x, dx0)));
	const float c1 = corner(__fmaf_rn(-dy1, dy1, x1), __fmaf_rn(g1.x, dx1, __fmul_rn(g1.y, dy1)));
	const float c2 = corner(__fmaf_rn(-dy2, dy2, __fmaf_rn(-dx2, dx2, 0.5f)), __fmaf_rn(g2.x, dx2, __fmul_rn(g2.y, dy2)));
	return __fmul_rn(70.0f, __fadd_rn(__fadd_rn(c0, c1), c2));
}

// STPSimplexNoise.cu:84-110 at sample (ux, uy) = ((x - half) + offset) / Scale:
// the saturated, normalised fractal sum in [0, 1].
template<Rounding R>
__device__ __forceinline__ float fractal(const Tables& T, const float ux, const float uy, const uint32_t octave,
	const float persistence, const float lacunarity) {
	float sum = 0.0f, amplitude = 1.0f, frequency = 1.0f, range = 0.0f;
	for (uint32_t o = 0u; o < octave; o++) {
		sum = __fmaf_rn(simplex2d<R>(T, __fmul_rn(ux, frequency), __fmul_rn(uy, frequency)), amplitude, sum);
		range += amplitude;
		amplitude *= persistence;
		frequency *= lacunarity;
	}
	return __saturatef((sum + range) / (2.0f * range));
}

} // namespace simplex
} // namespace stpgb
