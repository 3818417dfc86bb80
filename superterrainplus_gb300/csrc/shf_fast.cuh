// Single histogram filter, few-values path: device helpers shared by its two
// formulations (shf_fast.cu: sequential slides in packed form for launches of
// many chunks; shf_band.cu: row bands with prefix scans for launches of few).
//
// A chunk qualifies when its read region ((H+2r) x (W+2r) samples) holds at
// most kShfFastItems distinct values (biome maps: a Voronoi map of 8 biomes,
// the demo's layer chain).  Values are renamed to local indices 0..7 (their
// rank in the chunk's palette), so a histogram lives in registers: eight byte
// counts in one 64-bit word (or eight 16-bit fields in four words), and the
// reference accumulator's order (STPSingleHistogramFilter.cpp:400-450:
// insertion order with erase-compaction) as eight 4-bit indices in one
// 32-bit word.
#pragma once

#include "shf.cuh"

namespace stpgb {
namespace shfx {

constexpr uint32_t kNoValue = 0xFFFFFFFFu;
// words per palette: {count, kNoValue past kShfWideItems; 0; values as uint16 pairs x8; 0, 0}
constexpr uint32_t kSlotWords = 12u;
// Rows and columns of the read region per palette tile: a panel's palette is
// the union of the tiles it touches, so a tile is a fraction of its width.
constexpr uint32_t kTileRows = 16u, kTileCols = 256u;
// the byte counts hold 2r+2 (add before remove), the 16-bit fields
// (2r+1)(2r+2), a column's ring of local indices 2r+2
constexpr uint32_t kFastMaxRadius = 126u;

__device__ __forceinline__ const ShfJob& pick(const ShfJob* jobs, const ShfJob& single) {
	return jobs ? jobs[blockIdx.y] : single;
}

__device__ __forceinline__ uint32_t tile_rows(const ShfJob& J) {
	return (J.H + 2u * J.r + kTileRows - 1u) / kTileRows;
}
__device__ __forceinline__ uint32_t tile_cols(const ShfJob& J) {
	return (J.W + 2u * J.r + kTileCols - 1u) / kTileCols;
}

// The tiles' palettes lie at the start of the workspace (vbuf, and vn behind
// it), which every path writes only after the routing has read them.
__device__ __forceinline__ uint32_t* tile_slot(const ShfJob& J, const uint32_t i) {
	return J.vbuf + static_cast<size_t>(kSlotWords) * i;
}
// the panels' palettes lie in vn, which only the general slides use
__device__ __forceinline__ uint32_t* panel_slot(const ShfJob& J, const uint32_t i) {
	return reinterpret_cast<uint32_t*>(J.vn) + static_cast<size_t>(kSlotWords) * i;
}

__device__ __forceinline__ uint64_t vbuf_bytes(const ShfJob& J) {
	return 4ull * J.kcap_v * J.H * (J.W + 2u * J.r);
}
__device__ __forceinline__ uint64_t vn_bytes(const ShfJob& J) {
	return 2ull * J.H * (J.W + 2u * J.r);
}
__device__ __forceinline__ uint64_t tiles_bytes(const ShfJob& J) {
	return 4ull * kSlotWords * tile_rows(J) * tile_cols(J);
}
// The others go the general slides without a palette: those read their workspace by words of four
// bytes, these kernels by words of eight, and a caller's workspace may begin at any word.
__device__ __forceinline__ bool has_palette(const ShfJob& J) {
	return J.r <= kFastMaxRadius && (reinterpret_cast<uintptr_t>(J.vbuf) & 7u) == 0u
		&& tiles_bytes(J) <= vbuf_bytes(J) + vn_bytes(J);
}

// A job's panels: panel p covers the columns [p * step, p * step + cols) of the
// read region and the pixels [p * step + (p ? 1 : 0), p * step + step], so that
// it also holds the columns of the last window before its first pixel's.
// (Radius at most kFastMaxRadius and cols above 2r + 1.)
struct Panels {
	uint32_t step, count;
	uint64_t columns; // of all panels: the columns of the read region, 2r+1 more per further panel
	__device__ __forceinline__ Panels(const ShfJob& J, const uint32_t cols) {
		step = cols - 2u * J.r - 1u;
		count = J.W > 1u ? (J.W - 1u + step - 1u) / step : 1u;
		columns = J.W + 2u * J.r + static_cast<uint64_t>(count - 1u) * (2u * J.r + 1u);
	}
};

// first sample of the read region: row sy - r, column sx - r
__device__ __forceinline__ const uint16_t* read_region(const ShfJob& J) {
	return J.samplemap + static_cast<uint64_t>(J.sy - J.r) * J.pitch + (J.sx - J.r);
}

// number of nonzero bytes (present items)
__device__ __forceinline__ uint32_t nonzero_bytes(const uint64_t v) {
	const uint64_t low7 = 0x7F7F7F7F7F7F7F7Full;
	return static_cast<uint32_t>(__popcll((((v & low7) + low7) | v) & 0x8080808080808080ull));
}

// place of item j in an order word (j is in its first nonzero_bytes nibbles):
// the lowest zero nibble of order ^ (j in every nibble)
__device__ __forceinline__ uint32_t place_of(const uint32_t order, const uint32_t j) {
	const uint32_t x = order ^ (j * 0x11111111u);
	const uint32_t z = (x - 0x11111111u) & ~x & 0x88888888u;
	return static_cast<uint32_t>(__ffs(z) - 1) >> 2;
}

// the reference accumulator's add of one sample of item a: appended when absent
__device__ __forceinline__ void hist_add(uint64_t& cnt, uint32_t& order, const uint32_t a) {
	const uint32_t sh = 8u * a;
	if (((cnt >> sh) & 0xFFull) == 0ull) {
		order |= a << (4u * nonzero_bytes(cnt));
	}
	cnt += 1ull << sh;
}

// its remove: an item whose count drops to zero is erased, later ones close up
__device__ __forceinline__ void hist_sub(uint64_t& cnt, uint32_t& order, const uint32_t b) {
	const uint32_t sh = 8u * b;
	cnt -= 1ull << sh;
	if (((cnt >> sh) & 0xFFull) == 0ull) {
		const uint32_t low = (1u << (4u * place_of(order, b))) - 1u;
		order = (order & low) | ((order >> 4) & ~low);
	}
}

// The palette as eight 16-bit fields (value j in word j/2, half j%2),
// ascending, 0xFFFF past the count.
using Palette = uint4;

// local index of a palette value: the number of palette values below it
// (a padding field, 0xFFFF, is never below a 16-bit value)
__device__ __forceinline__ uint32_t local_index(const Palette p, const uint32_t v) {
	const uint32_t vv = v * 0x00010001u;
	return (__popc(__vcmpgtu2(vv, p.x)) + __popc(__vcmpgtu2(vv, p.y)) + __popc(__vcmpgtu2(vv, p.z))
			   + __popc(__vcmpgtu2(vv, p.w)))
		>> 4;
}

// The palette of a job routed to the dense path, from its record.
__device__ __forceinline__ Palette record_palette(const ShfFastRecord* const rec) {
	const uint32_t n = rec->count;
	const uint32_t* const rw = reinterpret_cast<const uint32_t*>(rec->item);
	auto half = [&](const uint32_t j) {
		return j < n ? ((rw[j / 2u] >> (16u * (j & 1u))) & 0xFFFFu) : 0xFFFFu;
	};
	return make_uint4(half(0) | (half(1) << 16), half(2) | (half(3) << 16), half(4) | (half(5) << 16),
		half(6) | (half(7) << 16));
}

// the job's path record (the routing kernel writes it)
__device__ __forceinline__ void write_record(const ShfJob& J, const uint32_t mode, const uint32_t count,
	const uint32_t* const vals, const uint32_t form) {
	ShfFastRecord* const rec = reinterpret_cast<ShfFastRecord*>(J.fast);
	rec->mode = mode;
	rec->count = count;
	rec->form = mode == kShfModeFast ? form : 0u;
	for (uint32_t j = 0u; j < kShfFastItems; j++) {
		rec->item[j] = static_cast<uint16_t>(j < count ? vals[j] : 0u);
	}
}

// ----------------------------------------------------- eight 16-bit fields --

__device__ __forceinline__ uint4 add4(const uint4 a, const uint4 b) {
	return make_uint4(__vadd2(a.x, b.x), __vadd2(a.y, b.y), __vadd2(a.z, b.z), __vadd2(a.w, b.w));
}
__device__ __forceinline__ uint4 sub4(const uint4 a, const uint4 b) {
	return make_uint4(__vsub2(a.x, b.x), __vsub2(a.y, b.y), __vsub2(a.z, b.z), __vsub2(a.w, b.w));
}
// eight byte counts -> eight 16-bit fields (item j in word j/2, half j%2)
__device__ __forceinline__ uint4 widen(const uint64_t c) {
	const uint32_t lo = static_cast<uint32_t>(c), hi = static_cast<uint32_t>(c >> 32);
	return make_uint4(__byte_perm(lo, 0u, 0x4140u), __byte_perm(lo, 0u, 0x4342u), __byte_perm(hi, 0u, 0x4140u),
		__byte_perm(hi, 0u, 0x4342u));
}

// bit j set where field j is nonzero
__device__ __forceinline__ uint32_t present_mask(const uint4 v) {
	const uint32_t a = __vcmpne2(v.x, 0u), b = __vcmpne2(v.y, 0u), c = __vcmpne2(v.z, 0u), d = __vcmpne2(v.w, 0u);
	return (a & 1u) | ((a >> 15) & 2u) | ((b & 1u) << 2) | ((b >> 13) & 8u) | ((c & 1u) << 4) | ((c >> 11) & 32u)
		| ((d & 1u) << 6) | ((d >> 9) & 128u);
}

__device__ __forceinline__ uint32_t field(const uint4 v, const uint32_t j) {
	const uint32_t w = (j & 4u) ? ((j & 2u) ? v.w : v.z) : ((j & 2u) ? v.y : v.x);
	return (w >> (16u * (j & 1u))) & 0xFFFFu;
}

// fields of a that are zero, as 0xFFFF halves
__device__ __forceinline__ uint4 zero4(const uint4 a) {
	return make_uint4(__vcmpeq2(a.x, 0u), __vcmpeq2(a.y, 0u), __vcmpeq2(a.z, 0u), __vcmpeq2(a.w, 0u));
}

// a hint to bring the line of p into L1 (callers keep p inside the buffer)
__device__ __forceinline__ void prefetch_l1(const void* p) {
	asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

} // namespace shfx
} // namespace stpgb
