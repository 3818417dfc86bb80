// Free-slip particle hydraulic erosion in shared-memory tiles on sm_103a.
//
// The kernels of erosion.cu keep the map in the L2 and are bound by its
// atomic unit: an eroding step of a brush of radius 4 costs 16.5 returning
// 16-byte atomics.  Here a block owns a T x T tile of the map in shared memory
// and erodes the droplets inside it there; nobody else touches the tile's
// cells while it does, so the tile is read and written back with plain loads
// and stores.  A droplet takes a step only while everything the step reads or
// writes (the brush, the corners of the old and of the new cell) lies inside
// its tile; a droplet that comes nearer to the tile's edge leaves, and is
// picked up in the next phase by the tile of a shifted grid (shifts of half a
// tile in x, y or both, so a droplet near an edge of one grid is well inside a
// tile of the next).  A phase is two launches:
//
//   tile_scatter  sorts the phase's droplets by tile and lists the tiles that
//                 hold any
//   tile_erode    persistent blocks take tiles from the list: load, erode,
//                 write back the changed cells, and file every droplet that
//                 left under its tile of the next phase's grid
//
// before which tile_measure looks over the map and the brush and tile_bin
// files the first starts; tile_finish then takes the few droplets left after
// the last phase through the map in global memory.
//
// Droplets race as in the kernels of erosion.cu, and their order matters as
// much: the starts enter in index order, a small group of them a phase (tile_plan),
// in tiles that a droplet crosses in few phases, and a tile alternates fresh
// droplets with those that came from other tiles.  With groups of 0.4 droplets
// per pixel and tiles that put every SM to work the RMS against the FP64 serial
// result was 1.1 to 2.2 times that of the kernels of erosion.cu; it is 0.67 to
// 1.05 times theirs.  (Most of either is not the races': a serial run in 32 bits
// is as far from the one in 64, 0.00117 on a 2048^2 field where the kernels of
// erosion.cu are at 0.00119 and the tiles at 0.00123.)
//
// Inside a tile a height is a 32-bit integer, h * 2^k with 2^k such that the
// map's largest magnitude lies in [2^26, 2^27): shared memory adds integers
// natively, floats only by compare-and-swap (measured for radius-4 brushes at
// random places of a 48^2 tile, 1024 threads per SM: 9.2 SM cycles per brush
// with returning integer adds, 15.3 with returning float adds, 18.6 with
// compare-and-swap; 9.2, 29.9 and 38.1 when all brushes meet in a 12^2 area).
// The unit is no coarser than the spacing of the floats from an eighth of the
// map's largest height up, where the mean height lies (tile_measure); amounts
// are rounded to the nearest unit, sums of units are exact, and a cell's
// fraction below a unit is kept and added back when the tile is written.
// Differences of heights are taken in units, exactly.
// A brush point takes its amount w with one returning add and gives back what
// the cell lacked, so a droplet removes min(max(cell, 0), w) of the cell's
// exact current value (STPRainDrop.cu:146-157) whoever races it.
//
// No sum leaves 32 bits: nothing is put on a cell that was seen at kCellLimit
// (2^29 units, at least four times the map's largest height) or above, no more
// than kMoveLimit (2^21) at a time, and a block holds at most 768 droplets, so a
// cell stays below 2^29 + 768 * 2^21 = 2^31.  A droplet that meets a cell at
// the limit goes to tile_finish.
//
// Maps this arithmetic does not suit (a value that is not finite, a largest
// magnitude above 8 times the mean one, so that the unit would be coarser than
// the floats of most of the map) and brushes that reach further than their radius are left
// to the kernels of erosion.cu: tile_measure finds that out per job, and those
// kernels, launched after, return at once for the jobs eroded here.
#include "erosion.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

namespace stpgb {

namespace {

// Threads of an eroding block, one block per SM, by the brush points that a
// lane keeps in registers: 768 (80 registers) took the 4096^2 field's erosion,
// 9 points, to 36.1 ms, 640 to 36.9 and 512 to 38.8; 14 points spill at 768
// (1000^2 chunks of radius 6 3.16 ms, at 640 2.93).
constexpr uint32_t tile_threads(const uint32_t points) {
	return points <= 9u ? 768u : 640u;
}
constexpr uint32_t kTileLeast = 128u, kTileMost = 200u; // sides of a tile
// A tile's rows lie `side` rounded up to 12 more than a multiple of 32 words
// apart: rows of the brush up to radius 6 then start in different banks.
constexpr uint32_t kTilePitchMost = 204u;
constexpr uint32_t kTileBrushLanes = 8u;  // lanes that take one brush
constexpr uint32_t kTileBrushes = 32u / kTileBrushLanes; // brushes a warp takes at a time
constexpr uint32_t kTileMostPoints = 14u; // brush points per lane: up to radius 6
constexpr uint32_t kTileMostRadius = 6u;
// least starts' area, brushes of 4 and more, and lifetime: see erosion_tile_pays
constexpr double kTileLeastArea = 1024.0 * 1024.0;
constexpr uint32_t kTileLeastSteps = 30u;
constexpr uint32_t kTileMostTiles = 48u * 1024u; // tile_scatter keeps a word of each in shared memory
constexpr uint32_t kBinThreads = 256u;
constexpr uint32_t kScanThreads = 1024u;
constexpr uint32_t kFinishThreads = 128u;
// Few: what is left is few, or droplets that pile up in one place and would race there.
constexpr uint32_t kFinishBlocks = 16u;
constexpr int32_t kCellLimit = 1 << 29;
constexpr int32_t kMoveUnits = 1 << 21;
static_assert(kCellLimit - 1 + int64_t { tile_threads(0u) } * kMoveUnits <= INT32_MAX, "a cell's sum leaves 32 bits");
constexpr float kMoveLimit = static_cast<float>(kMoveUnits);
// what others may put on a corner beside a droplet, in multiples of what it puts there itself
constexpr int32_t kMostPuts = 3;
// adding 1.5 * 2^23 leaves a float's nearest integer in its low bits (|x| < 2^22)
constexpr float kMagic = 12582912.0f;
constexpr int32_t kMagicBits = 0x4B400000;
// lanes without a droplet that make a warp fetch more (4096^2 field: 2 of them
// 35.9 ms, 4 35.8, 8 36.1, 12 37.0)
constexpr uint32_t kRefill = 4u;
constexpr uint32_t kNoJob = 0xFFFFFFFFu, kNoTile = 0xFFFFFFFFu;

struct TileJob {
	uint32_t drop0;  // first droplet of the job in the launch's arrays
	uint32_t tile0;  // first tile of the job
	uint32_t nx, ny; // tiles of a grid
};

// what tile_measure finds out about a job
struct TileStat {
	double sum;        // of |h|
	uint32_t peak;     // bits of the largest |h|
	uint32_t odd;      // a value or a brush that the tiles do not take
	uint32_t max_bw;   // bits of the brush's largest weight
	uint32_t pad;
};

struct TileWork {
	uint32_t tile, base, count, job;
};

// zeroed before a launch; what a phase reads was written in the one before, so each comes twice
struct TileControl {
	uint32_t carried[2]; // places of `filed` for the droplets that tiles hand to an even / odd phase
	uint32_t fresh[2];   // and after them for its starts
	uint32_t nwork;     // tiles that hold droplets
	uint32_t cursor[2]; // next tile of the list
};

struct TileArgs {
	const ErosionJob* jobs; // device array, or null for `single`
	ErosionJob single;
	const TileJob* geom; // device array, or null for `one`
	TileJob one;
	uint32_t njobs, tiles;
	uint32_t T, pitch;
	uint32_t groups; // the starts of a job come in this many groups, one a phase
	RainParams p;    // what all jobs have alike (all but BrushRadius, minWaterVolume and MaxSteps)
	int32_t minus1; // -1, unknown to the compiler: see pipe_add
	TileStat* stat;
	TileControl* ctl;
	uint32_t* count[2]; // droplets per tile for an even / odd phase
	TileWork* work;
	float4* pos;   // x, y, direction
	float4* flow;  // speed, volume, sediment, steps
	uint4* filed;  // filed droplets: which, in which tile (kNoTile: none), at which place there
	uint32_t* order; // droplets by tile
	uint32_t* left;  // per job from its drop0 on: droplets left for tile_finish
	uint32_t* nleft; // per job
	uint32_t* taken; // per job: 1 if it is eroded here
};

__device__ __forceinline__ const ErosionJob& job_of(const TileArgs& A, const uint32_t j) {
	return A.jobs ? A.jobs[j] : A.single;
}
__device__ __forceinline__ const TileJob& geom_of(const TileArgs& A, const uint32_t j) {
	return A.geom ? A.geom[j] : A.one;
}

// k of the unit 2^-k, or false where the tiles do not take the job: odd values, or a largest
// height of more than 8 times the mean one (whose spacing as a float the unit then exceeds)
__device__ __forceinline__ bool unit_of(const TileStat& s, const uint64_t cells, int& k) {
	const float peak = __uint_as_float(s.peak);
	if (s.odd || !(peak >= 1e-30f && peak <= 1e30f) || !(s.sum * 8.0 >= static_cast<double>(peak) * cells)) {
		return false;
	}
	k = 26 - ilogbf(peak);
	return true;
}
__device__ __forceinline__ float power2(const int k) {
	return __int_as_float((127 + k) << 23);
}

// point p of a brush as (dx, dy) from its map offset
__device__ __forceinline__ int2 brush_point(const ErosionJob& J, const uint32_t p) {
	const int32_t at = J.brush_index[p], pitch = static_cast<int32_t>(J.pitch);
	const int32_t half = pitch / 2, shifted = at + half;
	const int32_t dy = shifted >= 0 ? shifted / pitch : -((-shifted + pitch - 1) / pitch);
	return make_int2(at - dy * pitch, dy);
}

// ---------------------------------------------------------------- measure --

// Largest magnitude and mean magnitude of a job's map, and its brush.  Bound
// by reading the map once.
__global__ void __launch_bounds__(kBinThreads) tile_measure(const TileArgs A) {
	chain_begin();
	const ErosionJob& J = job_of(A, blockIdx.y);
	TileStat& S = A.stat[blockIdx.y];
	const uint64_t cells = static_cast<uint64_t>(J.dim_x) * J.dim_y;
	float peak = 0.0f, sum = 0.0f;
	double total = 0.0;
	bool odd = false;
	uint32_t since = 0u;
	auto take = [&](const float h) {
		const float m = fabsf(h);
		odd = odd || !(m <= 3.0e38f);
		peak = fmaxf(peak, m);
		sum += m;
	};
	const uint64_t first = static_cast<uint64_t>(blockIdx.x) * kBinThreads + threadIdx.x,
				   stride = static_cast<uint64_t>(gridDim.x) * kBinThreads;
	if (J.pitch == J.dim_x && (reinterpret_cast<uintptr_t>(J.map) & 15u) == 0u) {
		const float4* const m4 = reinterpret_cast<const float4*>(J.map);
		for (uint64_t i = first; i < cells / 4u; i += stride) {
			const float4 v = __ldcg(m4 + i);
			take(v.x);
			take(v.y);
			take(v.z);
			take(v.w);
			if (++since == 16u) {
				total += sum;
				sum = 0.0f;
				since = 0u;
			}
		}
		for (uint64_t i = cells / 4u * 4u + first; i < cells; i += stride) {
			take(__ldcg(J.map + i));
		}
	} else {
		for (uint64_t i = first; i < cells; i += stride) {
			take(__ldcg(J.map + i / J.dim_x * J.pitch + i % J.dim_x));
			if (++since == 64u) {
				total += sum;
				sum = 0.0f;
				since = 0u;
			}
		}
	}
	total += sum;
	float max_bw = 0.0f;
	if (blockIdx.x == 0u) {
		const int32_t reach = static_cast<int32_t>(J.p.BrushRadius) - 1;
		for (uint32_t p = threadIdx.x; p < J.brush_size; p += kBinThreads) {
			const int2 d = brush_point(J, p);
			const float w = J.brush_weight[p];
			odd = odd || abs(d.x) > reach || abs(d.y) > reach || !(w >= 0.0f && w <= 1.0f);
			max_bw = fmaxf(max_bw, w);
		}
	}
	__shared__ float s_peak[kBinThreads / 32u], s_bw[kBinThreads / 32u];
	__shared__ double s_sum[kBinThreads / 32u];
	for (int o = 16; o > 0; o >>= 1) {
		peak = fmaxf(peak, __shfl_xor_sync(0xFFFFFFFFu, peak, o));
		max_bw = fmaxf(max_bw, __shfl_xor_sync(0xFFFFFFFFu, max_bw, o));
		total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
	}
	odd = __any_sync(0xFFFFFFFFu, odd);
	if ((threadIdx.x & 31u) == 0u) {
		s_peak[threadIdx.x >> 5] = peak;
		s_bw[threadIdx.x >> 5] = max_bw;
		s_sum[threadIdx.x >> 5] = total;
		if (odd) {
			atomicOr(&S.odd, 1u);
		}
	}
	__syncthreads();
	if (threadIdx.x == 0u) {
		for (uint32_t w = 1u; w < kBinThreads / 32u; w++) {
			peak = fmaxf(peak, s_peak[w]);
			max_bw = fmaxf(max_bw, s_bw[w]);
			total += s_sum[w];
		}
		atomicMax(&S.peak, __float_as_uint(peak));
		atomicMax(&S.max_bw, __float_as_uint(max_bw));
		atomicAdd(&S.sum, total);
	}
}

// -------------------------------------------------------------------- bin --

struct TilePhase {
	uint32_t phase;
	uint32_t shift_x, shift_y; // of this phase's grid
	uint32_t next_x, next_y;   // of the next one's
	bool last;
};

__device__ __forceinline__ uint32_t tile_at(const TileJob& G, const uint32_t cx, const uint32_t cy, const uint32_t T,
	const uint32_t shift_x, const uint32_t shift_y) {
	return G.tile0 + (cy + shift_y) / T * G.nx + (cx + shift_x) / T;
}

// first droplet of a job's group g
__device__ __forceinline__ uint32_t group_first(const uint32_t count, const uint32_t groups, const uint32_t g) {
	return static_cast<uint32_t>(static_cast<uint64_t>(count) * g / groups);
}

// Files the starts of a group under their tiles, thread `first` of `stride`,
// behind the droplets that the tiles hand over.  A start has a place of its own,
// as a tile's droplets have: places handed out by one counter kept a million
// droplets of a batch's phase waiting at one address.
__device__ __forceinline__ void file_group(const TileArgs& A, const uint32_t group, const uint32_t shift_x,
	const uint32_t shift_y, const uint32_t first, const uint32_t stride) {
	const uint32_t to = group & 1u;
	uint32_t at = A.ctl->carried[to];
	uint32_t starts = 0u;
	for (uint32_t j = 0u; j < A.njobs; j++) {
		const ErosionJob& J = job_of(A, j);
		const TileJob& G = geom_of(A, j);
		int k;
		if (!unit_of(A.stat[j], static_cast<uint64_t>(J.dim_x) * J.dim_y, k)) {
			continue;
		}
		const uint32_t d0 = group_first(J.count, A.groups, group), d1 = group_first(J.count, A.groups, group + 1u);
		for (uint32_t d = d0 + first; d < d1; d += stride) {
			const float px = J.starts[2u * d], py = J.starts[2u * d + 1u];
			// a start whose 2x2 bilinear footprint is not inside the map dies at once
			const bool in = px >= 0.0f && px < J.dim_x - 1.0f && py >= 0.0f && py < J.dim_y - 1.0f;
			uint4 f = make_uint4(0u, kNoTile, 0u, 0u);
			if (in) {
				const uint32_t key = tile_at(G, static_cast<uint32_t>(px), static_cast<uint32_t>(py), A.T, shift_x,
					shift_y);
				f = make_uint4(G.drop0 + d, key, atomicAdd(A.count[to] + key, 1u), 0u);
			}
			A.filed[at + starts + (d - d0)] = f;
		}
		starts += d1 - d0;
	}
	if (first == 0u) {
		A.ctl->fresh[to] = starts;
	}
}

__global__ void __launch_bounds__(kBinThreads) tile_bin(const TileArgs A) {
	chain_begin();
	for (uint32_t j = blockIdx.x * kBinThreads + threadIdx.x; j < A.njobs; j += gridDim.x * kBinThreads) {
		const ErosionJob& J = job_of(A, j);
		int k;
		A.taken[j] = unit_of(A.stat[j], static_cast<uint64_t>(J.dim_x) * J.dim_y, k) ? 1u : 0u;
	}
	file_group(A, 0u, 0u, 0u, blockIdx.x * kBinThreads + threadIdx.x, gridDim.x * kBinThreads);
}

// ---------------------------------------------------------------- scatter --

// Every block scans the droplets per tile for itself (a few thousand words out
// of the L2) and sorts its share of the filed droplets by tile; the first
// block also lists the tiles that hold any.
__global__ void __launch_bounds__(kScanThreads) tile_scatter(const TileArgs A, const uint32_t phase) {
	chain_begin();
	extern __shared__ uint32_t s_base[]; // per tile
	__shared__ uint32_t s_sum[32], s_bucket[256];
	TileControl& C = *A.ctl;
	const uint32_t now = phase & 1u;
	const uint32_t* const count = A.count[now];
	const uint32_t n = C.carried[now] + C.fresh[now];
	const uint32_t per = (A.tiles + kScanThreads - 1u) / kScanThreads;
	const uint32_t lo = min(A.tiles, threadIdx.x * per), hi = min(A.tiles, lo + per);
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	if (threadIdx.x < 256u) {
		s_bucket[threadIdx.x] = 0u;
	}
	uint32_t sum = 0u;
	for (uint32_t t = lo; t < hi; t++) {
		sum += count[t];
	}
	uint32_t isum = sum;
#pragma unroll
	for (uint32_t d = 1u; d < 32u; d <<= 1) {
		const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, isum, d);
		if (lane >= d) {
			isum += a;
		}
	}
	if (lane == 31u) {
		s_sum[warp] = isum;
	}
	__syncthreads();
	if (warp == 0u) {
		uint32_t a = s_sum[lane];
#pragma unroll
		for (uint32_t d = 1u; d < 32u; d <<= 1) {
			const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, a, d);
			if (lane >= d) {
				a += x;
			}
		}
		s_sum[lane] = a;
	}
	__syncthreads();
	uint32_t at = isum - sum + (warp ? s_sum[warp - 1u] : 0u);
	for (uint32_t t = lo; t < hi; t++) {
		s_base[t] = at;
		at += count[t];
	}
	if (blockIdx.x == 0u) {
		// the list of the tiles that hold any, those with most droplets first (by eighths of powers of
		// two), so that no block starts on a full tile when the others are done
		auto bucket = [](const uint32_t c) {
			const uint32_t z = static_cast<uint32_t>(__clz(c));
			return 8u * z + 7u - ((c << z) >> 28 & 7u);
		};
		for (uint32_t t = lo; t < hi; t++) {
			const uint32_t c = count[t];
			if (c != 0u) {
				atomicAdd(&s_bucket[bucket(c)], 1u);
			}
		}
		__syncthreads();
		if (threadIdx.x < 32u) {
			uint32_t mine = 0u;
			for (uint32_t b = 8u * lane; b < 8u * lane + 8u; b++) {
				mine += s_bucket[b];
			}
			uint32_t run = mine;
#pragma unroll
			for (uint32_t d = 1u; d < 32u; d <<= 1) {
				const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, run, d);
				run += lane >= d ? a : 0u;
			}
			if (lane == 31u) {
				C.nwork = run;
			}
			run -= mine;
			for (uint32_t b = 8u * lane; b < 8u * lane + 8u; b++) {
				const uint32_t c = s_bucket[b];
				s_bucket[b] = run;
				run += c;
			}
		}
		__syncthreads();
		uint32_t job = 0u;
		for (uint32_t t = lo; t < hi; t++) {
			const uint32_t c = count[t];
			if (c != 0u) {
				while (job + 1u < A.njobs && geom_of(A, job + 1u).tile0 <= t) {
					job++;
				}
				A.work[atomicAdd(&s_bucket[bucket(c)], 1u)] = TileWork { t, s_base[t], c, job };
			}
		}
	}
	// the words the coming tile_erode writes for the next phase, and its cursor
	for (uint32_t t = blockIdx.x * kScanThreads + threadIdx.x; t < A.tiles; t += gridDim.x * kScanThreads) {
		A.count[now ^ 1u][t] = 0u;
	}
	if (blockIdx.x == 0u && threadIdx.x == 0u) {
		C.carried[now ^ 1u] = s_sum[31]; // a place for every droplet of this phase
		C.fresh[now ^ 1u] = 0u;
		C.cursor[now] = 0u;
	}
	__syncthreads();
	for (uint32_t i = blockIdx.x * kScanThreads + threadIdx.x; i < n; i += gridDim.x * kScanThreads) {
		const uint4 f = A.filed[i];
		if (f.y == kNoTile) {
			continue;
		}
		A.order[s_base[f.y] + f.z] = f.x;
	}
}

// ------------------------------------------------------------------ erode --

// a * one + b on the multiply-add pipe: integer adds, minima and compares share
// the other one, which runs at half the rate of issue and bounds the step
__device__ __forceinline__ int32_t pipe_add(const int32_t a, const int32_t one, const int32_t b) {
	int32_t r;
	asm("mad.lo.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(one), "r"(b));
	return r;
}
__device__ __forceinline__ int32_t shared_add(const int32_t address, const int32_t v) {
	int32_t old;
	asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(address), "r"(v) : "memory");
	return old;
}

// At most kMoveLimit units over the corners of a cell; what it put, nothing where a corner has
// reached kCellLimit.
__device__ __noinline__ int32_t deposit_part(int32_t* const c, const int32_t pitch, const float part, const float ox,
	const float oy) {
	volatile const int32_t* const v = c;
	if (max(max(v[0], v[1]), max(v[pitch], v[pitch + 1])) >= kCellLimit) {
		return 0;
	}
	const int32_t d00 = __float2int_rn(part * (1.0f - ox) * (1.0f - oy)), d10 = __float2int_rn(part * ox * (1.0f - oy)),
				  d01 = __float2int_rn(part * (1.0f - ox) * oy), d11 = __float2int_rn(part * ox * oy);
	atomicAdd(c, d00);
	atomicAdd(c + 1, d10);
	atomicAdd(c + pitch, d01);
	atomicAdd(c + pitch + 1, d11);
	return (d00 + d10) + (d01 + d11);
}

// A droplet per lane, as the warp-cooperative kernel of erosion.cu; a warp
// fetches more droplets of the tile when kRefill of its lanes have none.  A
// step is straight-line code for all lanes (those without a droplet, or whose
// droplet stops, compute on the tile's first cells), since the instructions a
// step issues bound the kernel, not the shared memory's atomics.  The brushes
// of a warp's eroding droplets are taken four at a time, 8 lanes each; a lane
// keeps the tile offsets and the weights of its (at most Points) points of
// the brush in registers, with weight 0 past the brush's last point, and leaves
// what it took in shared memory for the droplet's lane to sum.  (Two at a time,
// 16 lanes each and a warp reduction per pair, spent 1.7 times the instructions
// on a brush of radius 4 or 5: the 4096^2 field 41.1 ms, now 35.6, the
// production batch's erosion 18.0 and 15.7.)
template<uint32_t Points, bool Mixed>
__global__ void __launch_bounds__(tile_threads(Points), 1) tile_erode(const TileArgs A, const TilePhase F) {
	constexpr uint32_t kThreads = tile_threads(Points);
	chain_begin();
	extern __shared__ int32_t cells[];
	__shared__ int2 s_brush[kThreads / 32u][32];    // cell, amount in units (float bits)
	__shared__ __align__(16) int32_t s_taken[kThreads / 32u][32u * kTileBrushLanes]; // units each lane took for each
	__shared__ uint32_t s_work, s_next, s_left;
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint32_t T = A.T;
	const int32_t pitch = static_cast<int32_t>(A.pitch);
	volatile int32_t* const vcells = cells;
	const uint32_t now = F.phase & 1u, to = now ^ 1u;
	// the starts of the next phase
	if (F.phase + 1u < A.groups) {
		file_group(A, F.phase + 1u, F.next_x, F.next_y, blockIdx.x * kThreads + threadIdx.x,
			gridDim.x * kThreads);
	}
	const uint32_t nwork = A.ctl->nwork;
	uint32_t job = kNoJob;
	int32_t off[Points]; // in bytes
	float bw[Points];
	uint32_t mypoints = 0u; // points of the brush this lane takes
	const int32_t cells_at = static_cast<int32_t>(__cvta_generic_to_shared(cells));
	while (true) {
		if (threadIdx.x == 0u) {
			s_work = atomicAdd(&A.ctl->cursor[now], 1u);
			s_next = 0u;
			s_left = 0u;
		}
		__syncthreads();
		const uint32_t wi = s_work;
		if (wi >= nwork) {
			return;
		}
		const TileWork W = A.work[wi];
		const ErosionJob& J = job_of(A, W.job);
		const TileJob& G = geom_of(A, W.job);
		const RainParams& P = A.p;
		const float min_volume = J.p.minWaterVolume;
		const uint32_t max_steps = J.p.MaxSteps;
		int k = 0;
		unit_of(A.stat[W.job], static_cast<uint64_t>(J.dim_x) * J.dim_y, k);
		const float scale = power2(k), unit = power2(-k);
		const float max_amount = kMoveLimit / fmaxf(__uint_as_float(A.stat[W.job].max_bw), 1e-30f);
		if (job != W.job) {
			job = W.job;
			mypoints = 0u;
#pragma unroll
			for (uint32_t j = 0u; j < Points; j++) {
				const uint32_t p = lane % kTileBrushLanes + j * kTileBrushLanes;
				off[j] = 0;
				bw[j] = 0.0f;
				if (p < J.brush_size) {
					const int2 q = brush_point(J, p);
					off[j] = 4 * (q.y * pitch + q.x);
					bw[j] = J.brush_weight[p];
					mypoints = j + 1u;
				}
			}
		}
		// the tile's cells inside the map: [x0, x1) x [y0, y1), and the cells a step may start from
		const uint32_t tx = (W.tile - G.tile0) % G.nx, ty = (W.tile - G.tile0) / G.nx;
		const int32_t ox0 = static_cast<int32_t>(tx * T) - static_cast<int32_t>(F.shift_x),
					  oy0 = static_cast<int32_t>(ty * T) - static_cast<int32_t>(F.shift_y);
		const int32_t dim_x = static_cast<int32_t>(J.dim_x), dim_y = static_cast<int32_t>(J.dim_y);
		const int32_t x0 = max(ox0, 0), y0 = max(oy0, 0);
		const int32_t x1 = min(ox0 + static_cast<int32_t>(T), dim_x), y1 = min(oy0 + static_cast<int32_t>(T), dim_y);
		const int32_t R = static_cast<int32_t>(J.p.BrushRadius);
		const int32_t keep_lo = max(R - 1, 2), keep_hi = max(R - 1, 3);
		const int32_t in_x0 = x0 == 0 ? 0 : x0 + keep_lo, in_y0 = y0 == 0 ? 0 : y0 + keep_lo;
		const uint32_t in_w = static_cast<uint32_t>((x1 == dim_x ? dim_x : x1 - keep_hi) - in_x0),
					   in_h = static_cast<uint32_t>((y1 == dim_y ? dim_y : y1 - keep_hi) - in_y0);
		const int32_t origin = y0 * pitch + x0; // of the tile-local index y * pitch + x
		const uint32_t width = static_cast<uint32_t>(x1 - x0), area = width * static_cast<uint32_t>(y1 - y0);
		float* const map = J.map + static_cast<uint64_t>(y0) * J.pitch + x0;
		for (uint32_t c = threadIdx.x; c < area; c += kThreads) {
			const uint32_t y = c / width, x = c - y * width;
			cells[y * pitch + x] = __float2int_rd(__ldcg(map + static_cast<uint64_t>(y) * J.pitch + x) * scale);
		}
		__syncthreads();

		// a droplet can die at the map's border here
		const bool border = x0 < R || y0 < R || x1 > dim_x - R || y1 > dim_y - R;
		const float inertia = P.Inertia, turn = unit * (1.0f - P.Inertia);
		const uint32_t fresh = G.drop0 + group_first(J.count, A.groups, min(F.phase, A.groups));
		bool has = false, drained = false;
		uint32_t id = 0u, step = 0u;
		float px = static_cast<float>(x0), py = static_cast<float>(y0), dirx = 0.0f, diry = 0.0f, speed = 0.0f,
			  vol = 0.0f, sed = 0.0f;
		double residual = 0.0;
		uint32_t steps_done = 0u, erode_steps = 0u;
		bool capped = false;
		while (true) {
			const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !has);
			const uint32_t nidle = static_cast<uint32_t>(__popc(idle));
			if (!drained && nidle >= kRefill) {
				uint32_t from = 0u;
				if (lane == 0u) {
					from = atomicAdd(&s_next, nidle);
				}
				from = __shfl_sync(0xFFFFFFFFu, from, 0);
				drained = from + nidle >= W.count;
				const uint32_t mine = from + static_cast<uint32_t>(__popc(idle & ((1u << lane) - 1u)));
				if (!has && mine < W.count) {
					has = true;
					id = A.order[W.base + (mine & 1u ? W.count - 1u - (mine >> 1) : mine >> 1)];
					if (id >= fresh) {
						px = J.starts[2u * (id - G.drop0)];
						py = J.starts[2u * (id - G.drop0) + 1u];
						dirx = diry = 0.0f;
						speed = P.initSpeed;
						vol = P.initWaterVolume;
						sed = 0.0f;
						step = 0u;
					} else {
						const float4 a = __ldcg(A.pos + id), b = __ldcg(A.flow + id);
						px = a.x;
						py = a.y;
						dirx = a.z;
						diry = a.w;
						speed = b.x;
						vol = b.y;
						sed = b.z;
						step = __float_as_uint(b.w);
					}
				}
			}
			if (!__any_sync(0xFFFFFFFFu, has)) {
				break;
			}
			// dries up, reaches the step cap, or leaves the tile's inner part
			const bool dry = !(vol >= min_volume), over = step >= max_steps;
			const int32_t cx = static_cast<int32_t>(px), cy = static_cast<int32_t>(py);
			const bool inside = static_cast<uint32_t>(cx - in_x0) < in_w && static_cast<uint32_t>(cy - in_y0) < in_h;
			bool dies = dry || over;
			capped = capped || (has && over && !dry);
			const bool leaves = has && !dies && !inside;
			bool going = has && !dies && inside;
			// corners of the current cell (STPRainDrop.cu:23-51), in units and above q00
			const int32_t at = going ? cy * pitch + cx - origin : 0;
			const int32_t q00 = vcells[at], q10 = vcells[at + 1], q01 = vcells[at + pitch], q11 = vcells[at + pitch + 1];
			const float ox = px - static_cast<float>(cx), oy = py - static_cast<float>(cy);
			const float left = static_cast<float>(q01 - q00);
			const float gx = static_cast<float>(q10 - q00) * (1.0f - oy) + static_cast<float>(q11 - q01) * oy;
			const float gy = left * (1.0f - ox) + static_cast<float>(q11 - q10) * ox;
			const float rel = oy * left + ox * gx;
			float ndx = dirx * inertia - gx * turn, ndy = diry * inertia - gy * turn;
			const float len2 = ndx * ndx + ndy * ndy;
			const float inv = len2 != 0.0f ? rsqrtf(len2) : 1.0f;
			ndx *= inv;
			ndy *= inv;
			const float npx = px + ndx, npy = py + ndy;
			bool stays = ndx != 0.0f || ndy != 0.0f;
			const int32_t nx = static_cast<int32_t>(npx), ny = static_cast<int32_t>(npy);
			if (border) {
				// the reference's border test, R <= npx < dim - R, and a brush inside the map
				stays = stays && static_cast<uint32_t>(nx - R) < static_cast<uint32_t>(dim_x - 2 * R)
					&& static_cast<uint32_t>(ny - R) < static_cast<uint32_t>(dim_y - 2 * R)
					&& static_cast<uint32_t>(cx - (R - 1)) <= static_cast<uint32_t>(dim_x - max(R, 2) - (R - 1))
					&& static_cast<uint32_t>(cy - (R - 1)) <= static_cast<uint32_t>(dim_y - max(R, 2) - (R - 1));
			}
			dies = dies || (going && !stays);
			going = going && stays;
			// corners of the new cell
			const int32_t at2 = going ? ny * pitch + nx - origin : 0;
			const int32_t r00 = vcells[at2], r10 = vcells[at2 + 1], r01 = vcells[at2 + pitch],
						  r11 = vcells[at2 + pitch + 1];
			const float cx2 = npx - static_cast<float>(nx), cy2 = npy - static_cast<float>(ny);
			const float gx2 = static_cast<float>(r10 - r00) * (1.0f - cy2) + static_cast<float>(r11 - r01) * cy2;
			const float dh = (static_cast<float>(r00 - q00) + (cy2 * static_cast<float>(r01 - r00) + cx2 * gx2 - rel)) * unit;
			const float cap = fmaxf(-dh * speed * vol * P.SedimentCapacityFactor, P.minSedimentCapacity);
			const bool deposit = going && (sed > cap || dh > 0.0f);
			const float dep = fmaxf((dh > 0.0f ? fminf(dh, sed) : (sed - cap) * P.DepositSpeed) * scale, 0.0f);
			const float amount = fminf((cap - sed) * P.ErodeSpeed, -dh) * scale;
			// all four corners in [0, kCellLimit), or each within its bounds
			bool fits = amount < max_amount;
			if (deposit) {
				fits = dep < 1e9f
					&& (static_cast<uint32_t>((q00 | q10) | (q01 | q11)) < static_cast<uint32_t>(kCellLimit)
						|| (max(max(q00, q10), max(q01, q11)) < kCellLimit && min(min(q00, q10), min(q01, q11)) > -kCellLimit));
			}
			const bool unfit = going && !fits;
			going = going && fits;
			if (deposit && going) {
				const float part = fminf(dep, kMoveLimit);
				const float up = part * (1.0f - oy), down = part * oy;
				const int32_t d00 = __float_as_int(up * (1.0f - ox) + kMagic) - kMagicBits,
							  d10 = __float_as_int(up * ox + kMagic) - kMagicBits,
							  d01 = __float_as_int(down * (1.0f - ox) + kMagic) - kMagicBits,
							  d11 = __float_as_int(down * ox + kMagic) - kMagicBits;
				const int32_t s00 = atomicAdd(cells + at, d00) - q00, s10 = atomicAdd(cells + at + 1, d10) - q10,
							  s01 = atomicAdd(cells + at + pitch, d01) - q01,
							  s11 = atomicAdd(cells + at + pitch + 1, d11) - q11;
				int32_t put = (d00 + d10) + (d01 + d11);
				// What others have put on a corner since it was read is not put on it again, as a later
				// droplet of the serial order would find it there, past kMostPuts times the droplet's own:
				// droplets that meet in a hollow, in lockstep in one warp even, would otherwise all fill it in
				// full and raise a mound.  (From the first on, what droplets put while others pass is taken
				// back too: RMS of a 1024^2 field 0.00125, this way 0.00123, erosion.cu's 0.00122.)
				if (max(max(s00, s10), max(s01, s11)) > 0) {
					const int32_t e00 = min(max(s00 - kMostPuts * d00, 0), d00), e10 = min(max(s10 - kMostPuts * d10, 0), d10),
								  e01 = min(max(s01 - kMostPuts * d01, 0), d01), e11 = min(max(s11 - kMostPuts * d11, 0), d11);
					atomicAdd(cells + at, -e00);
					atomicAdd(cells + at + 1, -e10);
					atomicAdd(cells + at + pitch, -e01);
					atomicAdd(cells + at + pitch + 1, -e11);
					put -= (e00 + e10) + (e01 + e11);
				}
				// the rest of more than kMoveLimit units in parts, while the cells are low enough
				for (float rest = dep - part; rest > 0.0f; rest -= kMoveLimit) {
					put += deposit_part(cells + at, pitch, fminf(rest, kMoveLimit), ox, oy);
				}
				sed -= static_cast<float>(put) * unit;
			}
			// the brushes of the warp's eroding droplets, four at a time
			const bool erode = going && !deposit;
			const uint32_t emask = __ballot_sync(0xFFFFFFFFu, erode);
			if (emask != 0u) {
				const uint32_t n = static_cast<uint32_t>(__popc(emask));
				const uint32_t mine = static_cast<uint32_t>(__popc(emask & ((1u << lane) - 1u)));
				if (erode) {
					s_brush[warp][mine] = make_int2(cells_at + 4 * at, __float_as_int(amount));
				}
				if (lane < (0u - n) % kTileBrushes) {
					s_brush[warp][n + lane] = make_int2(cells_at + 4 * (R - 1) * (pitch + 1), 0); // nothing to take
				}
				__syncwarp();
				const int2* mybrush = &s_brush[warp][lane / kTileBrushLanes];
				int32_t* mytaken = &s_taken[warp][lane];
#pragma unroll 1
				for (uint32_t b = 0u; b < n; b += kTileBrushes, mybrush += kTileBrushes, mytaken += 32) {
					const int2 B = *mybrush;
					const float e = __int_as_float(B.y);
					int32_t bits[Points], old[Points];
#pragma unroll
					for (uint32_t j = 0u; j < Points; j++) {
						bits[j] = __float_as_int(fmaf(e, bw[j], kMagic)); // kMagicBits + w
						old[j] = kCellLimit;
						if (Mixed || j + 1u == Points ? j < mypoints : true) {
							old[j] = shared_add(B.x + off[j], pipe_add(bits[j], A.minus1, kMagicBits));
						}
					}
					uint32_t sum = static_cast<uint32_t>(bits[0]);
					int32_t least = old[0];
#pragma unroll
					for (uint32_t j = 1u; j < Points; j++) {
						sum += static_cast<uint32_t>(bits[j]);
						least = min(least, old[j]);
					}
					int32_t part = static_cast<int32_t>(sum - Points * static_cast<uint32_t>(kMagicBits));
					// an amount is at most kMoveUnits: only a cell below that can have lacked some of it
					if (least < kMoveUnits) {
#pragma unroll
						for (uint32_t j = 0u; j < Points; j++) {
							const int32_t w = bits[j] - kMagicBits, lack = min(w - old[j], w);
							if (lack > 0) {
								shared_add(B.x + off[j], lack); // w was taken: give back what the cell lacked
								part -= lack;
							}
						}
					}
					*mytaken = part;
				}
				__syncwarp();
				if (erode) {
					// the droplet's eight lanes, two reads apart in the order that leaves no bank twice
					const int4* const taken = reinterpret_cast<const int4*>(&s_taken[warp][mine * kTileBrushLanes]);
					const int4 a = taken[(mine >> 2) & 1u], c = taken[((mine >> 2) & 1u) ^ 1u];
					sed += static_cast<float>(((a.x + a.y) + (a.z + a.w)) + ((c.x + c.y) + (c.z + c.w))) * unit;
				}
				__syncwarp();
			}
			if (going) {
				px = npx;
				py = npy;
				dirx = ndx;
				diry = ndy;
				speed = sqrtf(fmaxf(0.0f, speed * speed + dh * P.Gravity)) * (1.0f - P.Friction);
				vol *= 1.0f - P.EvaporateSpeed;
				step++;
				steps_done++;
				erode_steps += erode ? 1u : 0u;
			}
			const bool ends = has && dies; // the carried sediment leaves with the droplet
			const bool parts = leaves || unfit;
			if (__any_sync(0xFFFFFFFFu, ends || parts)) {
				if (ends) {
					residual += sed;
				}
				if (unfit || (leaves && F.last)) {
					A.left[G.drop0 + atomicAdd(A.nleft + W.job, 1u)] = id;
				}
				// file the droplets that left
				const uint32_t out = __ballot_sync(0xFFFFFFFFu, leaves && !F.last);
				uint32_t from = 0u;
				if (out != 0u && lane == 0u) {
					from = atomicAdd(&s_left, static_cast<uint32_t>(__popc(out)));
				}
				from = __shfl_sync(0xFFFFFFFFu, from, 0);
				if (leaves && !F.last) {
					const uint32_t key = tile_at(G, static_cast<uint32_t>(px), static_cast<uint32_t>(py), T, F.next_x,
						F.next_y);
					A.filed[W.base + from + static_cast<uint32_t>(__popc(out & ((1u << lane) - 1u)))] = make_uint4(id, key,
						atomicAdd(A.count[to] + key, 1u), 0u);
				}
				if (parts) {
					A.pos[id] = make_float4(px, py, dirx, diry);
					A.flow[id] = make_float4(speed, vol, sed, __uint_as_float(step));
				}
				has = has && !ends && !parts;
			}
		}
		if (J.counters) {
			uint32_t s = steps_done, e = erode_steps;
			for (int o = 16; o > 0; o >>= 1) {
				s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
				e += __shfl_xor_sync(0xFFFFFFFFu, e, o);
			}
			if (lane == 0u && s != 0u) {
				atomicAdd(J.counters, static_cast<unsigned long long>(s));
				atomicAdd(J.counters + 1, static_cast<unsigned long long>(e));
			}
		}
		if (J.residual) {
			for (int o = 16; o > 0; o >>= 1) {
				residual += __shfl_xor_sync(0xFFFFFFFFu, residual, o);
			}
			if (lane == 0u && residual != 0.0) {
				atomicAdd(J.residual, residual);
			}
		}
		if (capped && J.status) {
			atomicOr(J.status, STATUS_TIMEOUT);
		}
		__syncthreads();
		// the places of the droplets that went no further
		for (uint32_t i = s_left + threadIdx.x; i < W.count; i += kThreads) {
			A.filed[W.base + i].y = kNoTile;
		}
		// the changed cells, each with its fraction of a unit
		for (uint32_t c = threadIdx.x; c < area; c += kThreads) {
			const uint32_t y = c / width, x = c - y * width;
			float* const cell = map + static_cast<uint64_t>(y) * J.pitch + x;
			const float h = __ldcg(cell) * scale;
			const int32_t before = __float2int_rd(h), after = cells[y * pitch + x];
			if (after != before) {
				*cell = (static_cast<float>(after) + (h - static_cast<float>(before))) * unit;
			}
		}
		__syncthreads();
	}
}

// ----------------------------------------------------------------- finish --

// The droplets left after the last phase and those the tiles could not hold
// (a few), a warp each on the map in global memory: the corners in one round
// trip, the brush in one per 32 points, each point taken by a returning add
// that gives back what the cell lacked.
__global__ void __launch_bounds__(kFinishThreads) tile_finish(const TileArgs A) {
	chain_begin();
	const uint32_t job = blockIdx.y;
	const uint32_t n = A.nleft[job];
	if (n == 0u) {
		return;
	}
	const ErosionJob& J = job_of(A, job);
	const RainParams& P = J.p;
	float* const map = J.map;
	const uint64_t pitch = J.pitch;
	const uint32_t lane = threadIdx.x & 31u;
	const uint64_t corner = (lane & 2u ? pitch : 0u) + (lane & 1u);
	const float lo = static_cast<float>(P.BrushRadius);
	const float hi_x = 1.0f * J.dim_x - P.BrushRadius, hi_y = 1.0f * J.dim_y - P.BrushRadius;
	const int32_t R = static_cast<int32_t>(P.BrushRadius);
	const int32_t safe_lo = R - 1, safe_hx = static_cast<int32_t>(J.dim_x) - max(R, 2),
				  safe_hy = static_cast<int32_t>(J.dim_y) - max(R, 2);
	const uint32_t warps = gridDim.x * (kFinishThreads / 32u);
	for (uint32_t i = (blockIdx.x * kFinishThreads + threadIdx.x) / 32u; i < n; i += warps) {
		const uint32_t id = A.left[geom_of(A, job).drop0 + i];
		const float4 a = A.pos[id], b = A.flow[id];
		float px = a.x, py = a.y, dirx = a.z, diry = a.w, speed = b.x, vol = b.y, sed = b.z;
		uint32_t step = __float_as_uint(b.w), steps_done = 0u, erode_steps = 0u;
		while (vol >= P.minWaterVolume) {
			if (step++ >= P.MaxSteps) {
				if (lane == 0u && J.status) {
					atomicOr(J.status, STATUS_TIMEOUT);
				}
				break;
			}
			const int32_t cx = static_cast<int32_t>(px), cy = static_cast<int32_t>(py);
			const bool safe = cx >= safe_lo && cx <= safe_hx && cy >= safe_lo && cy <= safe_hy;
			float* const c = map + static_cast<uint64_t>(cy) * pitch + cx;
			const float ox = px - static_cast<float>(cx), oy = py - static_cast<float>(cy);
			float v = __ldcg(c + corner);
			const float h00 = __shfl_sync(0xFFFFFFFFu, v, 0), h10 = __shfl_sync(0xFFFFFFFFu, v, 1),
						h01 = __shfl_sync(0xFFFFFFFFu, v, 2), h11 = __shfl_sync(0xFFFFFFFFu, v, 3);
			const float h = h00 * (1.0f - ox) * (1.0f - oy) + h10 * ox * (1.0f - oy) + h01 * (1.0f - ox) * oy
				+ h11 * ox * oy;
			const float gx = (h10 - h00) * (1.0f - oy) + (h11 - h01) * oy, gy = (h01 - h00) * (1.0f - ox) + (h11 - h10) * ox;
			dirx = (-gx) * (1.0f - P.Inertia) + dirx * P.Inertia;
			diry = (-gy) * (1.0f - P.Inertia) + diry * P.Inertia;
			const float len = sqrtf(dirx * dirx + diry * diry);
			if (len != 0.0f) {
				dirx /= len;
				diry /= len;
			}
			px += dirx;
			py += diry;
			if ((dirx == 0.0f && diry == 0.0f) || !(px >= lo && px < hi_x && py >= lo && py < hi_y) || !safe) {
				break;
			}
			const int32_t nx = static_cast<int32_t>(px), ny = static_cast<int32_t>(py);
			const float cx2 = px - static_cast<float>(nx), cy2 = py - static_cast<float>(ny);
			v = __ldcg(map + static_cast<uint64_t>(ny) * pitch + nx + corner);
			const float h2 = __shfl_sync(0xFFFFFFFFu, v, 0) * (1.0f - cx2) * (1.0f - cy2)
				+ __shfl_sync(0xFFFFFFFFu, v, 1) * cx2 * (1.0f - cy2) + __shfl_sync(0xFFFFFFFFu, v, 2) * (1.0f - cx2) * cy2
				+ __shfl_sync(0xFFFFFFFFu, v, 3) * cx2 * cy2;
			const float dh = h2 - h;
			const float cap = fmaxf(-dh * speed * vol * P.SedimentCapacityFactor, P.minSedimentCapacity);
			if (sed > cap || dh > 0.0f) {
				const float dep = (dh > 0.0f) ? fminf(dh, sed) : (sed - cap) * P.DepositSpeed;
				sed -= dep;
				if (lane < 4u) {
					atomicAdd(c + corner, dep * (lane & 1u ? ox : 1.0f - ox) * (lane & 2u ? oy : 1.0f - oy));
				}
			} else {
				erode_steps++;
				const float ero = fminf((cap - sed) * P.ErodeSpeed, -dh);
				float part = 0.0f;
				for (uint32_t p = lane; p < J.brush_size; p += 32u) {
					float* const cell = c + J.brush_index[p];
					const float w = ero * J.brush_weight[p];
					const float took = fminf(fmaxf(atomicAdd(cell, -w), 0.0f), w);
					part += took;
					if (took < w) {
						atomicAdd(cell, w - took);
					}
				}
				for (int o = 16; o > 0; o >>= 1) {
					part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
				}
				sed += part;
			}
			__syncwarp();
			speed = sqrtf(fmaxf(0.0f, speed * speed + dh * P.Gravity));
			speed *= 1.0f - P.Friction;
			vol *= 1.0f - P.EvaporateSpeed;
			steps_done++;
		}
		if (lane == 0u) {
			if (J.residual) {
				atomicAdd(J.residual, static_cast<double>(sed));
			}
			if (J.counters) {
				atomicAdd(J.counters, static_cast<unsigned long long>(steps_done));
				atomicAdd(J.counters + 1, static_cast<unsigned long long>(erode_steps));
			}
		}
	}
}

size_t up(const size_t v) {
	return (v + 255u) & ~static_cast<size_t>(255u);
}

uint32_t tiles_along(const uint32_t dim, const uint32_t T) {
	return (dim + T - 1u) / T + 1u; // one more for the shifted grids
}

struct TileLayout {
	size_t stat, ctl, nleft, count, zeroed, work, pos, flow, filed, order, left, taken, total;
	uint32_t tiles;
};

TileLayout tile_layout(const ErosionJob* jobs, const uint32_t njobs, const uint32_t T) {
	TileLayout L {};
	uint64_t droplets = 0u, tiles = 0u;
	for (uint32_t j = 0u; j < njobs; j++) {
		droplets += jobs[j].count;
		tiles += static_cast<uint64_t>(tiles_along(jobs[j].dim_x, T)) * tiles_along(jobs[j].dim_y, T);
	}
	L.tiles = static_cast<uint32_t>(tiles);
	L.stat = 0u;
	L.ctl = up(L.stat + njobs * sizeof(TileStat));
	L.nleft = up(L.ctl + sizeof(TileControl));
	L.count = up(L.nleft + njobs * sizeof(uint32_t));
	L.zeroed = up(L.count + tiles * sizeof(uint32_t));
	L.work = up(L.zeroed + tiles * sizeof(uint32_t));
	L.pos = up(L.work + tiles * sizeof(TileWork));
	L.flow = up(L.pos + droplets * sizeof(float4));
	L.filed = up(L.flow + droplets * sizeof(float4));
	L.order = up(L.filed + droplets * sizeof(uint4));
	L.left = up(L.order + droplets * sizeof(uint32_t));
	L.taken = up(L.left + droplets * sizeof(uint32_t));
	L.total = up(L.taken + njobs * sizeof(uint32_t));
	return L;
}

int tile_smem_attributes() {
	const int bytes = static_cast<int>(kTileMost * kTilePitchMost * sizeof(int32_t));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
		static_cast<int>(kTileMostTiles * sizeof(uint32_t))));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<2u, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<4u, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<6u, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<9u, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<14u, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<9u, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(tile_erode<14u, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	return STPGB_OK;
}

} // namespace

// A tile for every SM out of the starts' areas (the droplets spread a little
// past them), but no smaller than kTileLeast: a droplet moves a pixel a step, so
// in small tiles it leaves after a few steps and takes many phases, while later
// droplets overtake it.  Measured, ms and RMS against the FP64 serial result, in
// groups of 0.05 per pixel: a 1024^2 field (brush 5, 64 steps) in tiles of 80, 100,
// 128, 160 5.70 / 5.53 / 7.16 / 9.33 and 0.00145 / 0.00131 / 0.00124 / 0.00121
// (erosion.cu 9.00, 0.00123); a 2048^2 field in tiles of 100, 128, 160, 200 13.0 /
// 12.9 / 13.1 / 14.4 and 0.00136 / 0.00128 / 0.00125 / 0.00123 (34.9, 0.00119).
uint32_t erosion_tile_side(const ErosionJob* jobs, const uint32_t njobs) {
	double area = 0.0, tiles = 0.0;
	for (uint32_t j = 0u; j < njobs; j++) {
		const ErosionJob& J = jobs[j];
		if (J.brush_size == 0u || J.brush_size > kTileMostPoints * kTileBrushLanes || J.p.BrushRadius > kTileMostRadius
			|| J.p.MaxSteps > kTileMaxSteps || J.start_area == 0u) {
			return 0u;
		}
		// the droplets' settings are kernel parameters: all jobs' alike but for these three
		RainParams p = J.p;
		p.BrushRadius = jobs[0].p.BrushRadius;
		p.minWaterVolume = jobs[0].p.minWaterVolume;
		p.MaxSteps = jobs[0].p.MaxSteps;
		if (std::memcmp(&p, &jobs[0].p, sizeof(p)) != 0) {
			return 0u;
		}
		area += J.start_area;
	}
	const double side = std::sqrt(area / (1.1 * current_sm_count()));
	const uint32_t T = std::min(kTileMost, std::max(kTileLeast, static_cast<uint32_t>(side / 4.0 + 1.0) * 4u));
	for (uint32_t j = 0u; j < njobs; j++) {
		tiles += static_cast<double>(tiles_along(jobs[j].dim_x, T)) * tiles_along(jobs[j].dim_y, T);
	}
	return tiles <= kTileMostTiles ? T : 0u;
}

namespace {

// Whether a map's width keeps erosion.cu from taking brush rows as 16-byte blocks.
bool no_rows(const ErosionJob* jobs, const uint32_t njobs) {
	return std::any_of(jobs, jobs + njobs, [](const ErosionJob& j) { return (j.pitch & 3u) != 0u; });
}

} // namespace

// Brush points enough that either way's time is worth choosing; below, either takes under 3 ms.
bool erosion_tile_many(const ErosionJob* jobs, const uint32_t njobs) {
	double points = 0.0;
	for (uint32_t j = 0u; j < njobs; j++) {
		points += static_cast<double>(jobs[j].count) * jobs[j].p.MaxSteps * jobs[j].brush_size;
	}
	return points >= 1e9;
}

// Where the tiles are the better way and follow the serial order as closely.
// A phase lasts as long as a tile's droplets take for their steps, however few
// tiles hold any, so the tiles want wide starts' areas, and more so the fewer points
// a brush has.  erosion.cu against the tiles, ms (3x3 chunks, 1 droplet per
// pixel, 40 steps): 768^2 brush 5 3.78 / 4.52, 1024^2 brush 3 3.51 / 3.97, brush 4 4.76 /
// 4.16, brush 5 6.13 / 4.70; fields at 0.95: 1448^2 brush 2 6.96 / 3.97, brush 3 6.28
// / 4.30, 2048^2 brush 5 21.1 / 10.7.  Short lifetimes gain less, the launches'
// share being larger (1024^2 brush 4 20 steps 2.39 / 2.45, 3000^2 brush 3 20 steps 4.08 / 4.22).
// Without erosion.cu's rows (no_rows) the tiles gain more: 1025^2 brush 3 7.69 / 4.91; brushes of
// 2 have no rows anyway.
bool erosion_tile_pays(const ErosionJob* jobs, const uint32_t njobs) {
	double area = 0.0;
	uint32_t radius = kTileMostRadius, steps = 0u;
	for (uint32_t j = 0u; j < njobs; j++) {
		area += jobs[j].start_area;
		radius = std::min(radius, jobs[j].p.BrushRadius);
		steps = std::max(steps, jobs[j].p.MaxSteps);
	}
	const bool wide_brush = radius >= (no_rows(jobs, njobs) ? 3u : 4u);
	return erosion_tile_many(jobs, njobs) && steps >= kTileLeastSteps && area >= (wide_brush ? kTileLeastArea : 2.0 * kTileLeastArea);
}

namespace {

// groups the starts come in, and phases in all
struct TilePlan {
	uint32_t groups, phases;
};

TilePlan tile_plan(const ErosionJob* jobs, const uint32_t njobs, const uint32_t T) {
	uint32_t steps = 0u;
	double droplets = 0.0, area = 1.0;
	for (uint32_t j = 0u; j < njobs; j++) {
		steps = std::max(steps, jobs[j].p.MaxSteps);
		droplets += jobs[j].count;
		area += jobs[j].start_area;
	}
	TilePlan p;
	// A droplet is under way for a few phases, and what then starts beside it is what departs from the
	// serial order: groups of 0.05 droplets per pixel, of fewer the larger the map, where the kernels of
	// erosion.cu hold fewer per pixel under way, too.  Measured, ms and RMS against the FP64 serial result,
	// in groups of 0.2, 0.1, 0.05, 0.025, 0.0125 per pixel: a 4096^2 field (brush 5, 64 steps) 35.0 / 36.7 /
	// 39.6 / 45.7 / 52.1 and 0.00142 / 0.00130 / 0.00125 / 0.00124 / 0.00123 (erosion.cu 136.6, 0.00120).
	// Past 48 groups the launches cost more than the order gains: sixteen 3x3 x 512^2 chunks in 48, 64 and
	// 92 groups 24, 27.5 and 32.0 ms, 0.00043 each way (erosion.cu 59.5, 0.00042).
	// Where erosion.cu goes without rows it is slower and follows the serial order more closely, and so do
	// groups of half as many: a 1201^2 field (brush 4, 30 steps) in groups of 0.043, 0.025, 0.0125
	// 3.45 / 4.16 / 7.50 and 0.00115 / 0.00112 / 0.00108 (erosion.cu 10.4, 0.00106).
	const double wide = no_rows(jobs, njobs) ? 0.5 : 1.0;
	const double per_group = wide * std::clamp(0.05 * 1024.0 / std::sqrt(area), 0.0125, 0.05);
	p.groups = static_cast<uint32_t>(std::min(48.0 / wide, std::max(4.0, std::ceil(droplets / area / per_group))));
	// a droplet that walks straight on crosses steps / T tiles; one that meanders comes back
	p.phases = p.groups + 3u + (5u * steps + T - 1u) / T;
	return p;
}

} // namespace

uint32_t erosion_tile_kernels(const ErosionJob* jobs, const uint32_t njobs, const uint32_t T) {
	return 3u + 2u * tile_plan(jobs, njobs, T).phases;
}

size_t erosion_tile_bytes(const ErosionJob* jobs, const uint32_t njobs, const uint32_t T) {
	return tile_layout(jobs, njobs, T).total + up(njobs * sizeof(TileJob));
}

int erosion_tile_prepare(const ErosionJob* jobs, const uint32_t njobs, const uint32_t T, void* workspace) {
	const TileLayout L = tile_layout(jobs, njobs, T);
	std::vector<TileJob> geom;
	uint32_t drop0 = 0u, tile0 = 0u;
	for (uint32_t j = 0u; j < njobs; j++) {
		const TileJob g { drop0, tile0, tiles_along(jobs[j].dim_x, T), tiles_along(jobs[j].dim_y, T) };
		geom.push_back(g);
		drop0 += jobs[j].count;
		tile0 += g.nx * g.ny;
	}
	STPGB_CUDA_TRY(cudaMemcpy(static_cast<unsigned char*>(workspace) + L.total, geom.data(), njobs * sizeof(TileJob),
		cudaMemcpyHostToDevice));
	return STPGB_OK;
}

int erosion_tile_launch(const ErosionJob* host_jobs, const ErosionJob* jobs, const uint32_t njobs, const uint32_t T,
	void* workspace, const uint32_t** taken, cudaStream_t stream) {
	STPGB_TRY(once_per_device(SETUP_EROSION_TILE_SMEM, tile_smem_attributes));
	const TileLayout L = tile_layout(host_jobs, njobs, T);
	const TilePlan plan = tile_plan(host_jobs, njobs, T);
	const uint32_t groups = plan.groups, phases = plan.phases;
	unsigned char* const ws = static_cast<unsigned char*>(workspace);
	TileArgs A {};
	A.jobs = jobs;
	A.single = host_jobs[0];
	A.njobs = njobs;
	A.tiles = L.tiles;
	A.T = T;
	A.pitch = (T + 19u) / 32u * 32u + 12u;
	A.p = host_jobs[0].p;
	A.minus1 = -1;
	A.groups = groups;
	A.stat = reinterpret_cast<TileStat*>(ws + L.stat);
	A.ctl = reinterpret_cast<TileControl*>(ws + L.ctl);
	A.count[0] = reinterpret_cast<uint32_t*>(ws + L.count);
	A.count[1] = reinterpret_cast<uint32_t*>(ws + L.zeroed);
	A.work = reinterpret_cast<TileWork*>(ws + L.work);
	A.pos = reinterpret_cast<float4*>(ws + L.pos);
	A.flow = reinterpret_cast<float4*>(ws + L.flow);
	A.filed = reinterpret_cast<uint4*>(ws + L.filed);
	A.order = reinterpret_cast<uint32_t*>(ws + L.order);
	A.left = reinterpret_cast<uint32_t*>(ws + L.left);
	A.nleft = reinterpret_cast<uint32_t*>(ws + L.nleft);
	A.taken = reinterpret_cast<uint32_t*>(ws + L.taken);
	*taken = A.taken;
	uint32_t max_count = 0u, max_brush = 0u;
	uint64_t max_cells = 0u, droplets = 0u;
	for (uint32_t j = 0u; j < njobs; j++) {
		max_count = std::max(max_count, host_jobs[j].count);
		droplets += host_jobs[j].count;
		max_brush = std::max(max_brush, host_jobs[j].brush_size);
		max_cells = std::max(max_cells, static_cast<uint64_t>(host_jobs[j].dim_x) * host_jobs[j].dim_y);
	}
	A.geom = jobs ? reinterpret_cast<const TileJob*>(ws + L.total) : nullptr;
	A.one = TileJob { 0u, 0u, tiles_along(host_jobs[0].dim_x, T), tiles_along(host_jobs[0].dim_y, T) };
	const uint32_t sms = current_sm_count();
	STPGB_CUDA_TRY(cudaMemsetAsync(ws, 0, L.zeroed, stream));
	const uint32_t mblocks = static_cast<uint32_t>(std::min<uint64_t>((max_cells / 4u + kBinThreads - 1u) / kBinThreads,
		std::max(1u, 8u * sms / njobs)));
	STPGB_TRY(launch_chained(true, tile_measure, dim3(std::max(1u, mblocks), njobs), kBinThreads, 0u, stream, A));
	const uint64_t group = droplets / groups + 1u;
	STPGB_TRY(launch_chained(true, tile_bin,
		static_cast<uint32_t>(std::min<uint64_t>(8u * sms, (group + kBinThreads - 1u) / kBinThreads)), kBinThreads, 0u, stream,
		A));
	const uint32_t sblocks = static_cast<uint32_t>(std::min<uint64_t>(sms, (2u * group + kScanThreads - 1u) / kScanThreads));
	const size_t smem = static_cast<size_t>(T) * A.pitch * sizeof(int32_t);
	const uint32_t points = (max_brush + kTileBrushLanes - 1u) / kTileBrushLanes;
	bool mixed = false;
	for (uint32_t j = 0u; j < njobs; j++) {
		mixed = mixed || (host_jobs[j].brush_size + kTileBrushLanes - 1u) / kTileBrushLanes != points;
	}
	const uint32_t eblocks = std::min(sms, L.tiles);
	const uint32_t half = T / 8u * 4u;
	for (uint32_t p = 0u; p < phases; p++) {
		auto sx = [&](const uint32_t q) { return (q & 3u) == 1u || (q & 3u) == 2u ? half : 0u; };
		auto sy = [&](const uint32_t q) { return (q & 3u) == 1u || (q & 3u) == 3u ? half : 0u; };
		const TilePhase F { p, sx(p), sy(p), sx(p + 1u), sy(p + 1u), p + 1u == phases };
		STPGB_TRY(launch_chained(true, tile_scatter, sblocks, kScanThreads, L.tiles * sizeof(uint32_t), stream, A, p));
		auto go = [&](auto kernel, const uint32_t most) {
			return launch_chained(true, kernel, eblocks, tile_threads(most), smem, stream, A, F);
		};
		int rc = STPGB_OK;
		switch (mixed ? 0u : points) {
		case 2u:
			rc = go(tile_erode<2u, false>, 2u);
			break;
		case 4u:
			rc = go(tile_erode<4u, false>, 4u);
			break;
		case 6u:
			rc = go(tile_erode<6u, false>, 6u);
			break;
		case 9u:
			rc = go(tile_erode<9u, false>, 9u);
			break;
		case 14u:
			rc = go(tile_erode<14u, false>, 14u);
			break;
		default:
			rc = points <= 9u ? go(tile_erode<9u, true>, 9u) : go(tile_erode<14u, true>, 14u);
			break;
		}
		STPGB_TRY(rc);
	}
	return launch_chained(true, tile_finish, dim3(kFinishBlocks, njobs), kFinishThreads, 0u, stream, A);
}

namespace {

// A pool per device behind erosion_tile_call: it keeps at most kPoolKeeps bytes
// between calls and gives what exceeds that back when its stream is next
// waited for; stream-ordered, so calls on any streams and threads share it.
constexpr uint64_t kPoolKeeps = 64ull << 20;
constexpr int kPoolDevices = 64;
std::mutex g_pool_mutex;
cudaMemPool_t g_pool[kPoolDevices] = {};

// Allocations are refused, and end the capture, while this thread or another captures a stream,
// unless the thread says that it knows what it does: here they are on a stream that is not captured.
class CaptureElsewhere {
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;

public:
	CaptureElsewhere() {
		cudaThreadExchangeStreamCaptureMode(&mode);
	}
	~CaptureElsewhere() {
		cudaThreadExchangeStreamCaptureMode(&mode);
	}
	CaptureElsewhere(const CaptureElsewhere&) = delete;
	CaptureElsewhere& operator=(const CaptureElsewhere&) = delete;
};

cudaMemPool_t tile_pool() {
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kPoolDevices) {
		cudaGetLastError();
		return nullptr;
	}
	const std::lock_guard<std::mutex> lock(g_pool_mutex);
	if (!g_pool[dev]) {
		cudaMemPoolProps props {};
		props.allocType = cudaMemAllocationTypePinned;
		props.location.type = cudaMemLocationTypeDevice;
		props.location.id = dev;
		cudaMemPool_t pool = nullptr;
		uint64_t keeps = kPoolKeeps;
		if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
			cudaGetLastError();
			return nullptr;
		}
		if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keeps) != cudaSuccess) {
			cudaGetLastError();
		}
		g_pool[dev] = pool;
	}
	return g_pool[dev];
}

} // namespace

int erosion_tile_call(const ErosionJob& job, const bool force, void** workspace, const uint32_t** taken, cudaStream_t stream) {
	*workspace = nullptr;
	*taken = nullptr;
	const uint32_t T = force || erosion_tile_pays(&job, 1u) ? erosion_tile_side(&job, 1u) : 0u;
	cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
	if (T == 0u) {
		return STPGB_OK;
	}
	if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
		cudaGetLastError();
		return STPGB_OK;
	}
	const CaptureElsewhere guard;
	const cudaMemPool_t pool = tile_pool();
	void* ws = nullptr;
	if (!pool || cudaMallocFromPoolAsync(&ws, erosion_tile_bytes(&job, 1u, T), pool, stream) != cudaSuccess) {
		cudaGetLastError();
		return STPGB_OK;
	}
	const int rc = erosion_tile_launch(&job, nullptr, 1u, T, ws, taken, stream);
	if (rc != STPGB_OK) {
		cudaFreeAsync(ws, stream);
		return rc;
	}
	*workspace = ws;
	return STPGB_OK;
}

int erosion_tile_release(void* workspace, cudaStream_t stream) {
	if (workspace) {
		const CaptureElsewhere guard;
		STPGB_CUDA_TRY(cudaFreeAsync(workspace, stream));
	}
	return STPGB_OK;
}

} // namespace stpgb
