// Multi-biome fractal simplex heightfield on sm_103a.
//
// Per pixel (x, y) of a chunk:  h = sum_bins Weight * (fractal(x, y) * Variation + Depth)
// (SuperDemo+/Script/STPMultiHeightGenerator.cu:35-72), with the 2D simplex
// noise and its fractal sum of SuperTerrain+/SuperAlgorithm+/Device/Private/
// STPSimplexNoise.cu:18-110.  The kernel is FP32-pipe bound.  Two exact
// rewrites take work out of the inner loop without changing a result:
//  * the reference hashes a corner as perm[a] % Gradient2DSize and then reads
//    the gradient; here a 512-entry table of the already-reduced gradient for
//    every perm slot lives in shared memory, so a corner costs one lookup;
//  * ((x - half) + offset) / Scale is the same for every octave (the
//    reference multiplies it by the octave frequency afterwards), so the IEEE
//    division is done once per bin instead of once per octave.
#include "noise.cuh"
#include "simplex.cuh"

#include <algorithm>

namespace stpgb {

namespace {

constexpr uint32_t kNoiseBlock = 256u;

// resident blocks of 256 threads per SM (48 registers)
constexpr uint32_t kNoiseBlocksPerSM = 5u;
// most strips of pixels a block takes: past a few the tables' share is gone
constexpr uint32_t kNoiseStrips = 8u;

// One pixel per thread and strip; a block takes the strips blockIdx.x,
// blockIdx.x + gridDim.x, ... so that building the tables (two lookups per
// slot, a modulo) is shared by several strips where a launch has them: 144
// chunks of 512^2 1.57 ms with one strip a block, 1.29 with up to eight.  A
// strip's offsets are loaded before the tables are waited for, or while the
// strip before is computed.  The block size (128, 256 or 512) is the batch
// tuner's choice.  Bound by instruction issue: about 90 per octave of a bin.
template<uint32_t Block>
__global__ void __launch_bounds__(Block, kNoiseBlocksPerSM * 256u / Block) multibiome_kernel(
	const NoiseJob* __restrict__ jobs, const NoiseJob single, const stpgb_permutation perm,
	const stpgb_biome_property* __restrict__ table, const uint32_t biome_count) {
	chain_begin();
	__shared__ simplex::Tables tables;
	const NoiseJob& J = jobs ? jobs[blockIdx.y] : single;
	const uint64_t npix = static_cast<uint64_t>(J.W) * J.H;
	const uint64_t stride = static_cast<uint64_t>(gridDim.x) * Block;
	uint64_t idx = static_cast<uint64_t>(blockIdx.x) * Block + threadIdx.x;
	const uint2* const bins = reinterpret_cast<const uint2*>(J.bins);
	uint32_t b0 = 0u, b1 = 0u;
	auto load = [&](const uint64_t i) {
		b0 = b1 = 0u;
		if (i < npix) {
			b0 = J.offsets[i];
			b1 = J.offsets[i + 1u];
		}
	};
	load(idx);
	simplex::load_tables(perm, tables);
	__syncthreads();
	// HalfDimension = vec2(MapSize) / 2 (SuperDemo+/World/Biomes/STPCommonCompiler.cpp:236)
	const float half_x = static_cast<float>(J.W) / 2.0f, half_y = static_cast<float>(J.H) / 2.0f;
	// the first pixel's place by 32-bit divisions (more than 2^32 pixels have no 32-bit offsets
	// either), the next ones' by the stride's
	const uint32_t W = J.W, step = gridDim.x * Block, step_y = step / W, step_x = step - step_y * W;
	uint32_t y = static_cast<uint32_t>(idx) / W, x = static_cast<uint32_t>(idx) - y * W;
	for (; idx < npix; x += step_x, y += step_y) {
		if (x >= W) {
			x -= W;
			y++;
		}
		const float fx = (1.0f * x - half_x) + J.off_x, fy = (1.0f * y - half_y) + J.off_y;
		const uint32_t begin = b0, end = b1;
		idx += stride;
		load(idx);
		float height = 0.0f;
		for (uint32_t b = begin; b < end; b++) {
			const uint2 raw = __ldg(bins + b);
			const uint32_t id = raw.x & 0xFFFFu;
			const float weight = __uint_as_float(raw.y);
			if (id >= biome_count) {
				continue;
			}
			const stpgb_biome_property p = table[id];
			const float f = simplex::fractal<simplex::Rounding::heights>(tables, fx / p.Scale, fy / p.Scale, p.Octave, p.Persistence,
				p.Lacunarity);
			height += weight * (f * p.Variation + p.Depth);
		}
		J.out[static_cast<uint64_t>(y) * J.pitch + x] = height;
	}
}

} // namespace

int noise_launch(const NoiseJob* jobs, const NoiseJob& single, uint32_t njobs, uint64_t max_pixels,
	const stpgb_permutation& perm, const stpgb_biome_property* table, uint32_t biome_count, cudaStream_t stream,
	const uint32_t block) {
	const uint32_t b = block == 0u ? kNoiseBlock : block;
	const uint64_t strips = (max_pixels + b - 1u) / b;
	const uint64_t resident = static_cast<uint64_t>(current_sm_count()) * (kNoiseBlocksPerSM * 256u / b);
	const uint64_t per = std::min<uint64_t>(std::max<uint64_t>(strips * njobs / resident, 1u), kNoiseStrips);
	const dim3 grid(static_cast<uint32_t>((strips + per - 1u) / per), njobs);
	// Blocks that come up while the kernel before still runs take the SMs that it leaves free: that
	// saves the gap where every block finds an SM of its own (128^2 heights 13.1 us, early 11.8) or
	// where they fill most of the GPU anyway (400^2, 4.1 blocks per SM, 24.1 and 22.4; 512^2 39.6 and
	// 37.4), but piles up the blocks of launches between (256^2 17.1 and 21.9; 350^2, 3.2 per SM, 25.2
	// and 27.9).
	const bool early = njobs == 1u && (grid.x <= current_sm_count() || 5u * grid.x >= 4u * resident);
	switch (b) {
	case 128u:
		return launch_chained(early, multibiome_kernel<128u>, grid, 128u, 0u, stream, jobs, single, perm, table, biome_count);
	case 256u:
		return launch_chained(early, multibiome_kernel<256u>, grid, 256u, 0u, stream, jobs, single, perm, table, biome_count);
	case 512u:
		return launch_chained(early, multibiome_kernel<512u>, grid, 512u, 0u, stream, jobs, single, perm, table, biome_count);
	default:
		return inval("noise_launch: block size must be 128, 256 or 512");
	}
}

} // namespace stpgb

using namespace stpgb;

extern "C" int stpgb_multibiome_heightmap(float* heightmap, uint32_t pitch, const uint32_t* offsets,
	const stpgb_bin* bins, uint32_t map_x, uint32_t map_y, float offset_x, float offset_y,
	const stpgb_permutation* perm, const stpgb_biome_property* biome_table, uint32_t biome_count, void* stream) {
	if (!heightmap || !offsets || !perm || !perm->Permutation || !perm->Gradient2D || !biome_table) {
		return inval("stpgb_multibiome_heightmap: null pointer argument");
	}
	if (perm->Gradient2DSize == 0u) {
		return inval("stpgb_multibiome_heightmap: empty gradient table");
	}
	if (pitch < map_x) {
		return inval("stpgb_multibiome_heightmap: pitch below map width");
	}
	if (map_x == 0u || map_y == 0u) {
		return STPGB_OK;
	}
	NoiseJob job { heightmap, pitch, offsets, bins, map_x, map_y, offset_x, offset_y };
	return noise_launch(nullptr, job, 1u, static_cast<uint64_t>(map_x) * map_y, *perm, biome_table, biome_count,
		as_stream(stream));
}
