// Single histogram filter, row-band formulation, on sm_103a:
// the one for launches of few chunks, where a thread per row or column would
// leave most of the GPU idle.  Same output as the reference filter
// (SuperTerrain+/SuperAlgorithm+/Host/Private/STPSingleHistogramFilter.cpp),
// bin order included.
//
// Horizontally the order follows from a rule that makes every pixel
// independent of the slide: when column k's vertical histogram is added, an
// item is inserted iff none of columns [max(0, k-2r-1), k-1] holds it (before
// the add, the window holds exactly those columns; the initial fill is the
// case k <= 2r).  An item present at pixel x was last inserted at the latest
// such column k0 <= x+2r, in the place it has in column k0's vertical
// histogram, and erasures keep the relative order of what remains, so the bins
// of pixel x are its present items sorted by (k0, place in column k0's
// histogram).  Windowed counts and "latest insertion column" are prefix scans
// over the columns of a row: one sum scan and one max scan of eight 16-bit
// fields per column, so a block computes a whole row at once.
//
//   shf_band_carry thread per (column, group of bands): the column's vertical
//                  histogram at each band's first row, from its window, a
//                  sweep up and steps down.
//   shf_band_rows  block per (band of rows, job), thread per column and pixel
//                  of a panel, panel after panel: per row, the vertical step,
//                  the count scan, the insertion scan and the pixels' bins
//                  (COUNT: bins per row; WRITE: offsets and bins, from the
//                  counts of the rows above).
//
// A row wider than a block is cut into panels.  A panel's items inserted before
// it keep, by the same rule, the order they have in the last window before its
// first pixel's, which the panel before leaves per row; so a panel needs only
// its own columns and, as no more values than its own occur in it, may have a
// palette of its own.  That is how a chunk of many values takes the bands: its
// panels hold few.  Both kernels come for 8 and for 16 values: a histogram is
// then eight or sixteen byte counts and as many 4-bit indices, a row's tables
// one or two uint4 per column.
#include "shf_fast.cuh"

#include <algorithm>

namespace stpgb {

using namespace shfx;

namespace {

constexpr uint32_t kCarryBlock = 64u;
// Most columns of a panel.  Panels overlap by 2r+1 columns, so wide ones waste
// less: 4096^2, radius 64, 1.40 ms, with 512 columns 1.64.
constexpr uint32_t kPanelCols = 1024u;
// rows of a column the carry loads together (64^2 44 us, with 32 of them 53)
constexpr uint32_t kAhead = 8u;
// A carry thread's group: as many bands as leave this many threads per SM, and
// at most this many rows (a palette covers the group).  A step down costs a
// fraction of a window and a sweep: with a group per band the carry was 499 of
// the 4096^2 chunk's 1656 us, so it is 138.
constexpr uint32_t kCarryThreadsPerSM = 128u;
constexpr uint32_t kCarryRows = 64u;
constexpr uint32_t kCarryBlocksPerSM = 32u;
constexpr uint32_t kBandMaxRows = 64u;
// past every row, with room to subtract one
constexpr int32_t kNoRow = 1 << 30;

// ------------------------------------------------- palettes and histograms --

// Local indices of a palette's values: the number of palette values below.
template<uint32_t K>
struct BandPalette;

template<>
struct BandPalette<kShfFastItems> {
	Palette p;
	__device__ __forceinline__ uint32_t index(const uint32_t v) const {
		return local_index(p, v);
	}
	__device__ __forceinline__ uint32_t value(const uint32_t i) const {
		return field(p, i);
	}
};

template<>
struct BandPalette<kShfWideItems> {
	Palette lo, hi;
	__device__ __forceinline__ uint32_t index(const uint32_t v) const {
		return local_index(lo, v) + local_index(hi, v);
	}
	__device__ __forceinline__ uint32_t value(const uint32_t i) const {
		return field(i < 8u ? lo : hi, i & 7u);
	}
};

// the values at slot + 2 of a panel's palette
__device__ __forceinline__ Palette slot_palette(const uint32_t* const w) {
	return make_uint4(w[0], w[1], w[2], w[3]);
}

// A column's vertical histogram: byte counts and the order as 4-bit indices.
// Kept in vbuf at `at` of `all` (band, panel and column): the counts of the
// first eight items, the orders (32 bits with one palette for the chunk) and
// the other counts.
template<uint32_t K>
struct BandHist;

template<>
struct BandHist<kShfFastItems> {
	using Order = uint32_t;
	uint64_t cnt = 0ull;
	Order order = 0u;
	__device__ __forceinline__ void count(const uint32_t j, const uint32_t n) {
		cnt += static_cast<uint64_t>(n) << (8u * j);
	}
	__device__ __forceinline__ bool has(const uint32_t j) const {
		return ((cnt >> (8u * j)) & 0xFFull) != 0ull;
	}
	__device__ __forceinline__ void put(const uint32_t place, const uint32_t j) {
		order |= j << (4u * place);
	}
	__device__ __forceinline__ void step(const uint32_t in, const uint32_t out) {
		hist_add(cnt, order, in);
		hist_sub(cnt, order, out);
	}
	__device__ __forceinline__ void widened(uint4 (&w)[1]) const {
		w[0] = widen(cnt);
	}
	__device__ __forceinline__ void store(const ShfJob& J, const bool wide, const size_t all, const size_t at) const {
		uint64_t* const counts = reinterpret_cast<uint64_t*>(J.vbuf);
		counts[at] = cnt;
		if (wide) {
			counts[all + at] = order;
		} else {
			reinterpret_cast<uint32_t*>(counts + all)[at] = order;
		}
	}
	__device__ __forceinline__ void load(const ShfJob& J, const bool wide, const size_t all, const size_t at) {
		const uint64_t* const counts = reinterpret_cast<const uint64_t*>(J.vbuf);
		cnt = counts[at];
		order = wide ? static_cast<uint32_t>(counts[all + at]) : reinterpret_cast<const uint32_t*>(counts + all)[at];
	}
	static __device__ __forceinline__ uint32_t place(const Order order, const uint32_t j) {
		return place_of(order, j);
	}
};

template<>
struct BandHist<kShfWideItems> {
	using Order = uint64_t;
	uint64_t lo = 0ull, hi = 0ull; // items 0-7, 8-15
	Order order = 0ull;
	__device__ __forceinline__ void count(const uint32_t j, const uint32_t n) {
		const uint64_t add = static_cast<uint64_t>(n) << (8u * (j & 7u));
		lo += j < 8u ? add : 0ull;
		hi += j < 8u ? 0ull : add;
	}
	__device__ __forceinline__ bool has(const uint32_t j) const {
		return (((j < 8u ? lo : hi) >> (8u * (j & 7u))) & 0xFFull) != 0ull;
	}
	__device__ __forceinline__ void put(const uint32_t place, const uint32_t j) {
		order |= static_cast<uint64_t>(j) << (4u * place);
	}
	__device__ __forceinline__ void step(const uint32_t in, const uint32_t out) {
		if (!has(in)) {
			put(nonzero_bytes(lo) + nonzero_bytes(hi), in);
		}
		count(in, 1u);
		const uint64_t one = 1ull << (8u * (out & 7u));
		lo -= out < 8u ? one : 0ull;
		hi -= out < 8u ? 0ull : one;
		if (!has(out)) {
			const uint64_t low = (1ull << (4u * place(order, out))) - 1ull;
			order = (order & low) | ((order >> 4) & ~low);
		}
	}
	__device__ __forceinline__ void widened(uint4 (&w)[2]) const {
		w[0] = widen(lo);
		w[1] = widen(hi);
	}
	__device__ __forceinline__ void store(const ShfJob& J, const bool, const size_t all, const size_t at) const {
		uint64_t* const counts = reinterpret_cast<uint64_t*>(J.vbuf);
		counts[at] = lo;
		counts[all + at] = order;
		counts[2u * all + at] = hi;
	}
	__device__ __forceinline__ void load(const ShfJob& J, const bool, const size_t all, const size_t at) {
		const uint64_t* const counts = reinterpret_cast<const uint64_t*>(J.vbuf);
		lo = counts[at];
		order = counts[all + at];
		hi = counts[2u * all + at];
	}
	// the lowest zero nibble of order ^ (j in every nibble)
	static __device__ __forceinline__ uint32_t place(const Order order, const uint32_t j) {
		const uint64_t x = order ^ (j * 0x1111111111111111ull);
		const uint64_t z = (x - 0x1111111111111111ull) & ~x & 0x8888888888888888ull;
		return static_cast<uint32_t>(__ffsll(static_cast<long long>(z)) - 1) >> 2;
	}
};

// ------------------------------------------------------------------ carry --

// Thread per (column of a panel, group of bands): the vertical histogram of
// rows [y0, y0+2r] (relative to the region) at each band's first row y0, as the
// reference's slide (:522-563) leaves it there.  At the group's first band the
// counts are the window's; the order is that of the starts of the present
// items' current runs (an item stays present while its occurrences are at most
// 2r+1 rows apart: the slide adds before it removes).  A sweep up from the
// window finds them, and ends when all runs but one are known to have started:
// that one started above the others.  Windows of one item, most of them, need
// no sweep.  Both go by stretches of equal samples, a comparison and an add per
// row.  The group's further bands are the slide's own steps from there.
template<uint32_t K>
__device__ __forceinline__ void band_carry(const ShfJob& J, const ShfBandShape& shape, const uint32_t group,
	const bool wide, const size_t all, const size_t column, const size_t columns, const uint32_t k,
	const BandPalette<K>& pal, int32_t* const first) {
	const uint64_t pitch = J.pitch;
	const uint32_t y0 = group * shape.group * shape.rows, y1 = min(J.H, y0 + shape.group * shape.rows);
	const int32_t r2 = static_cast<int32_t>(2u * J.r), top = static_cast<int32_t>(y0);
	const uint16_t* const col = read_region(J) + k;
	// rows from `from` up to (not past) `to`, kAhead loaded together
	auto rows_up = [&](const int32_t from, const int32_t to, auto&& each, auto&& done) {
		for (int32_t q0 = from; q0 >= to; q0 -= static_cast<int32_t>(kAhead)) {
			uint32_t v[kAhead];
#pragma unroll
			for (int32_t u = 0; u < static_cast<int32_t>(kAhead); u++) {
				v[u] = q0 - u >= to ? __ldg(col + static_cast<uint64_t>(q0 - u) * pitch) : 0u;
			}
#pragma unroll
			for (int32_t u = 0; u < static_cast<int32_t>(kAhead); u++) {
				if (q0 - u >= to) {
					each(q0 - u, v[u]);
				}
			}
			if (done(max(q0 - static_cast<int32_t>(kAhead) + 1, to))) {
				break;
			}
		}
	};
	// first row of item j's current run as far as seen, at first[j * kCarryBlock]
#pragma unroll
	for (uint32_t j = 0u; j <= K; j++) {
		first[j * kCarryBlock] = kNoRow;
	}
	BandHist<K> hist;
	// the last sample, its index, and the length of its stretch
	uint32_t seen = kNoValue, li = 0u, stretch = 0u;
	rows_up(top + r2, top, [&](const int32_t q, const uint32_t v) {
		if (v != seen) {
			if (stretch != 0u) {
				hist.count(li, stretch);
				first[li * kCarryBlock] = q + 1;
			}
			seen = v;
			li = pal.index(v);
			stretch = 0u;
		}
		stretch++;
	}, [](const int32_t) { return false; });
	hist.count(li, stretch);
	first[li * kCarryBlock] = top;
	uint32_t present = 0u;
#pragma unroll
	for (uint32_t j = 0u; j < K; j++) {
		present |= hist.has(j) ? 1u << j : 0u;
	}
	const uint32_t n = static_cast<uint32_t>(__popc(present));
	if (n == 1u) {
		hist.put(0u, li);
	} else {
		// whether the stretch belongs to its item's run, and up to which row
		bool joined = true;
		int32_t reached = top;
		rows_up(top - 1, 0, [&](const int32_t q, const uint32_t v) {
			if (v != seen) {
				if (joined) {
					first[li * kCarryBlock] = reached;
				}
				seen = v;
				// above the band's windows there may be values that its palette does not hold; item K
				// and the items past its count have no run to join
				const uint32_t i = pal.index(v);
				li = i < K && pal.value(i) == v ? i : K;
				joined = first[li * kCarryBlock] - q <= r2 + 1;
			}
			reached = joined ? q : reached;
		}, [&](const int32_t q) {
			if (joined) {
				first[li * kCarryBlock] = reached;
			}
			// a run whose first row seen so far is more than 2r+1 rows below the next row has started
			uint32_t open = 0u;
#pragma unroll
			for (uint32_t j = 0u; j < K; j++) {
				open += first[j * kCarryBlock] - (q - 1) <= r2 + 1 ? 1u : 0u;
			}
			return open <= 1u;
		});
		// the items by the starts of their runs (distinct rows)
		for (uint32_t m = 0u; m < n; m++) {
			int32_t least = kNoRow;
			uint32_t at = 0u;
#pragma unroll
			for (uint32_t j = 0u; j < K; j++) {
				const int32_t f = first[j * kCarryBlock];
				at = f < least ? j : at;
				least = min(least, f);
			}
			first[at * kCarryBlock] = kNoRow;
			hist.put(m, at);
		}
	}
	size_t at = static_cast<size_t>(group) * shape.group * columns + column;
	hist.store(J, wide, all, at);
	for (uint32_t y = y0 + shape.rows; y < y1; y += shape.rows) {
		for (uint32_t q = y - shape.rows + 1u; q <= y; q++) {
			// to row q: region row q+2r enters, row q-1 leaves
			const uint32_t in = __ldg(col + static_cast<uint64_t>(q + 2u * J.r) * pitch);
			const uint32_t out = __ldg(col + static_cast<uint64_t>(q - 1u) * pitch);
			if (in != out) {
				hist.step(pal.index(in), pal.index(out));
			}
		}
		at += columns;
		hist.store(J, wide, all, at);
	}
}

// Block (64 columns of a panel of a group of bands, job).
__global__ void __launch_bounds__(kCarryBlock) shf_band_carry(const ShfJob* __restrict__ jobs, const ShfJob single,
	const ShfBandShape shape, const uint32_t panels, const uint32_t works) {
	chain_begin();
	const ShfJob& J = pick(jobs, single);
	const uint32_t mode = shf_job_mode(J);
	if (mode == kShfModeSlide) {
		return;
	}
	__shared__ int32_t firsts[kShfWideItems + 1u][kCarryBlock];
	const Panels P(J, shape.cols);
	const uint32_t NC = J.W + 2u * J.r;
	const uint32_t bands = (J.H + shape.rows - 1u) / shape.rows;
	const uint32_t blocks = (shape.cols + kCarryBlock - 1u) / kCarryBlock;
	for (uint32_t w = blockIdx.x; w < works; w += gridDim.x) {
		const uint32_t c = w % blocks * kCarryBlock + threadIdx.x;
		const uint32_t panel = w / blocks % panels, group = w / blocks / panels;
		const uint32_t k = panel * P.step + c;
		if (panel >= P.count || group * shape.group >= bands || c >= shape.cols || k >= NC) {
			continue;
		}
		const size_t columns = P.columns, all = static_cast<size_t>(bands) * columns;
		const size_t column = static_cast<size_t>(panel) * shape.cols + c;
		int32_t* const first = &firsts[0][threadIdx.x];
		if (mode == kShfModeFast) {
			band_carry<kShfFastItems>(J, shape, group, false, all, column, columns, k,
				BandPalette<kShfFastItems> { record_palette(reinterpret_cast<const ShfFastRecord*>(J.fast)) }, first);
			continue;
		}
		const uint32_t* const pal = panel_slot(J, group * P.count + panel);
		if (pal[0] <= kShfFastItems) {
			band_carry<kShfFastItems>(J, shape, group, true, all, column, columns, k,
				BandPalette<kShfFastItems> { slot_palette(pal + 2u) }, first);
		} else {
			band_carry<kShfWideItems>(J, shape, group, true, all, column, columns, k,
				BandPalette<kShfWideItems> { slot_palette(pal + 2u), slot_palette(pal + 6u) }, first);
		}
	}
}

// ------------------------------------------------------------------- rows --

__device__ __forceinline__ uint4 max4(const uint4 a, const uint4 b) {
	return make_uint4(__vmaxu2(a.x, b.x), __vmaxu2(a.y, b.y), __vmaxu2(a.z, b.z), __vmaxu2(a.w, b.w));
}
__device__ __forceinline__ uint4 shfl_up4(const uint4 v, const uint32_t d) {
	return make_uint4(__shfl_up_sync(0xFFFFFFFFu, v.x, d), __shfl_up_sync(0xFFFFFFFFu, v.y, d),
		__shfl_up_sync(0xFFFFFFFFu, v.z, d), __shfl_up_sync(0xFFFFFFFFu, v.w, d));
}

struct AddOp {
	__device__ __forceinline__ uint4 operator()(const uint4 a, const uint4 b) const {
		return add4(a, b);
	}
};
struct MaxOp {
	__device__ __forceinline__ uint4 operator()(const uint4 a, const uint4 b) const {
		return max4(a, b);
	}
};

// Exclusive scan over the block (identity 0) of V uint4 and, with `Extra`, one
// integer sum per thread, with `wt` (32 * V entries) and `we` (32) for the warp
// totals; `total` and `extra_total` get the whole block's.  One barrier: every
// warp then scans the warp totals for itself.  The caller has a barrier
// between two scans that use the same `wt`.
template<uint32_t V, bool Extra, class Op>
__device__ __forceinline__ void block_exscan(uint4 (&v)[V], uint4 (&total)[V], uint4* const wt, const Op op,
	uint32_t& extra, uint32_t& extra_total, uint32_t* const we) {
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
	const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
	uint4 ex[V];
	uint32_t exe = 0u;
	auto warp_scan = [&](uint4 (&x)[V], uint32_t& e) {
#pragma unroll
		for (uint32_t d = 1u; d < 32u; d <<= 1) {
#pragma unroll
			for (uint32_t i = 0u; i < V; i++) {
				const uint4 t = shfl_up4(x[i], d);
				if (lane >= d) {
					x[i] = op(x[i], t);
				}
			}
			if constexpr (Extra) {
				const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, e, d);
				e += lane >= d ? t : 0u;
			}
		}
	};
	uint32_t inc = extra;
	warp_scan(v, inc);
#pragma unroll
	for (uint32_t i = 0u; i < V; i++) {
		ex[i] = shfl_up4(v[i], 1u);
		if (lane == 0u) {
			ex[i] = zero;
		}
		if (lane == 31u) {
			wt[32u * i + warp] = v[i];
		}
	}
	if constexpr (Extra) {
		exe = inc - extra;
		if (lane == 31u) {
			we[warp] = inc;
		}
	}
	__syncthreads();
	uint4 s[V];
	uint32_t se = 0u;
#pragma unroll
	for (uint32_t i = 0u; i < V; i++) {
		s[i] = lane < nw ? wt[32u * i + lane] : zero;
	}
	if constexpr (Extra) {
		se = lane < nw ? we[lane] : 0u;
	}
	warp_scan(s, se);
	auto from = [&](const uint4 x, const uint32_t l) {
		return make_uint4(__shfl_sync(0xFFFFFFFFu, x.x, l), __shfl_sync(0xFFFFFFFFu, x.y, l),
			__shfl_sync(0xFFFFFFFFu, x.z, l), __shfl_sync(0xFFFFFFFFu, x.w, l));
	};
	const uint32_t before = warp ? warp - 1u : 0u;
#pragma unroll
	for (uint32_t i = 0u; i < V; i++) {
		total[i] = from(s[i], nw - 1u);
		const uint4 b = from(s[i], before);
		v[i] = warp ? op(b, ex[i]) : ex[i];
	}
	if constexpr (Extra) {
		extra_total = __shfl_sync(0xFFFFFFFFu, se, nw - 1u);
		const uint32_t b = __shfl_sync(0xFFFFFFFFu, se, before);
		extra = (warp ? b : 0u) + exe;
	}
}

// Bound by the instructions of the scans (a warp's row is some 800, of which
// the two scans are nearly half) and by their four barriers a row: 0.58
// instructions per cycle and scheduler on a 4096^2 chunk, DRAM at 6 %.  So a
// block takes as many columns as it has threads for, and a thread two columns
// where a row is several panels anyway.  Before, a chunk wider than 4096
// columns or of more than 8 values took the general slides: 4096^2 of 32
// biomes, radius 64, 2.95 ms, now 1.20; 1024^2 of 16, radius 48, 923 us, now 220.

// What a block keeps of its rows from panel to panel.
struct BandRows {
	uint32_t bins[kBandMaxRows];          // bins of the panels so far
	uint32_t items[kBandMaxRows];         // items of the last window,
	uint16_t order[kBandMaxRows][kShfWideItems]; // their values in their order
	uint32_t sums[32];                    // warp totals
	uint64_t base[kBandMaxRows + 1u];     // WRITE: bins of the rows above
	uint64_t parts[32];
	uint16_t value[kShfWideItems];        // the panel's palette
	uint16_t seed[kShfWideItems];         // 1 + place of its items in the last window of the panel before
};

// The rows [y0, y1) of a band and one panel of them; thread c owns its column
// c and, where its window lies in the panel, its pixel c.
// Shared memory: counts prefix C[cols+1] and insertion scan M[cols] (V uint4
// each: 8 V 16-bit fields), the warp totals of both, orders[cols].
// Per row y: C[k] = counts of columns < k (the window of pixel x is
// C[x+2r+1] - C[x]); column k inserts item j iff it holds j and columns
// [max(0, k-2r-1), k-1] do not; M[k] = 17 + the latest such column <= k, per
// item, or 1 + its place in the panel before's last window.
template<bool Write, uint32_t Cols, uint32_t K>
__device__ __forceinline__ void band_panel(const ShfJob& J, const ShfBandShape& shape, const Panels& panels,
	const uint32_t band, const uint32_t panel, const bool wide, const BandPalette<K>& pal, BandRows& keep, uint4* const fsm) {
	constexpr uint32_t V = K / 8u;
	constexpr uint32_t kColumn = kShfWideItems + 1u; // of M: the first column's
	using Hist = BandHist<K>;
	using Order = typename Hist::Order;
	const uint32_t y0 = band * shape.rows, y1 = min(J.H, y0 + shape.rows);
	const uint32_t r2 = 2u * J.r, k0 = panel * panels.step;
	const uint32_t ncols = min(J.W + r2 - k0, shape.cols);
	const bool more = panel + 1u < panels.count;
	const uint32_t first = threadIdx.x * Cols;
	uint4* const C = fsm;
	uint4* const M = C + static_cast<size_t>(shape.cols + 1u) * V;
	uint4* const wc = M + static_cast<size_t>(shape.cols) * V;
	uint4* const wm = wc + 32u * V;
	Order* const ord = reinterpret_cast<Order*>(wm + 32u * V);
	const uint16_t* const C16 = reinterpret_cast<const uint16_t*>(C);
	const uint16_t* const M16 = reinterpret_cast<const uint16_t*>(M);
	const uint32_t bands = (J.H + shape.rows - 1u) / shape.rows;
	const uint16_t* const base = read_region(J) + k0 + first;
	const uint64_t pitch = J.pitch;
	auto column = [&](const uint32_t t) {
		return first + t < ncols;
	};
	auto pixel = [&](const uint32_t t) {
		return first + t + r2 < ncols && (panel == 0u || first + t != 0u);
	};
	Hist hist[Cols];
	// samples of the next row: they enter and leave
	uint32_t in[Cols], out[Cols];
#pragma unroll
	for (uint32_t t = 0u; t < Cols; t++) {
		if (column(t)) {
			hist[t].load(J, wide, static_cast<size_t>(bands) * panels.columns,
				static_cast<size_t>(band) * panels.columns + static_cast<size_t>(panel) * shape.cols + first + t);
		}
		in[t] = out[t] = 0u;
	}
	// for row y: region row y+2r enters, row y-1 leaves
	auto load_row = [&](const uint32_t y) {
		if (y < y1) {
#pragma unroll
			for (uint32_t t = 0u; t < Cols; t++) {
				if (column(t)) {
					in[t] = __ldg(base + static_cast<uint64_t>(y + r2) * pitch + t);
					out[t] = __ldg(base + static_cast<uint64_t>(y - 1u) * pitch + t);
				}
			}
		}
	};
	load_row(y0 + 1u);
	const uint32_t side = r2 + 1u;
	const float norm = __fdiv_rn(1.0f, static_cast<float>(side * side));
	uint2* const bins = reinterpret_cast<uint2*>(J.bins);
	const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

	for (uint32_t y = y0; y < y1; y++) {
		if (y > y0) {
#pragma unroll
			for (uint32_t t = 0u; t < Cols; t++) {
				if (in[t] != out[t]) {
					hist[t].step(pal.index(in[t]), pal.index(out[t]));
				}
			}
			load_row(y + 1u);
		}
		if constexpr (Write) {
			if (threadIdx.x < K && panel != 0u) {
				uint32_t seed = 0u;
				for (uint32_t i = 0u; i < keep.items[y - y0]; i++) {
					seed = keep.order[y - y0][i] == keep.value[threadIdx.x] ? i + 1u : seed;
				}
				keep.seed[threadIdx.x] = static_cast<uint16_t>(seed);
			}
		}
		// counts prefix
		uint4 acc[V], total[V], own[V];
#pragma unroll
		for (uint32_t i = 0u; i < V; i++) {
			acc[i] = zero;
		}
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			hist[t].widened(own); // no counts past the panel's columns
#pragma unroll
			for (uint32_t i = 0u; i < V; i++) {
				acc[i] = add4(acc[i], own[i]);
			}
		}
		uint32_t none = 0u, none_total = 0u;
		block_exscan<V, false>(acc, total, wc, AddOp {}, none, none_total, keep.sums);
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			if (column(t)) {
				hist[t].widened(own);
#pragma unroll
				for (uint32_t i = 0u; i < V; i++) {
					C[(first + t) * V + i] = acc[i];
					acc[i] = add4(acc[i], own[i]);
				}
				ord[first + t] = hist[t].order;
			}
		}
		if (threadIdx.x == 0u) {
#pragma unroll
			for (uint32_t i = 0u; i < V; i++) {
				C[ncols * V + i] = total[i];
			}
		}
		__syncthreads();
		// the pixels' present items
		uint32_t mask[Cols], mine = 0u, all = 0u;
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			mask[t] = 0u;
			if (pixel(t)) {
				const uint32_t c = first + t;
#pragma unroll
				for (uint32_t i = 0u; i < V; i++) {
					mask[t] |= present_mask(sub4(C[(c + r2 + 1u) * V + i], C[c * V + i])) << (8u * i);
				}
				mine += __popc(mask[t]);
			}
		}
		if constexpr (!Write) {
			mine = __reduce_add_sync(0xFFFFFFFFu, mine);
			if ((threadIdx.x & 31u) == 0u) {
				keep.sums[threadIdx.x >> 5] = mine;
			}
			__syncthreads();
			if (threadIdx.x < 32u) {
				all = __reduce_add_sync(0xFFFFFFFFu, threadIdx.x < (blockDim.x >> 5) ? keep.sums[threadIdx.x] : 0u);
				if (threadIdx.x == 0u) {
					all += panel ? keep.bins[y - y0] : 0u;
					if (more) {
						keep.bins[y - y0] = all;
					} else {
						J.rows[y] = all;
					}
				}
			}
			continue; // the next row's scan has a barrier before the sums are written again
		}
		// insertion columns and their running maximum, with the pixels' bins before this thread's
		// beside it (thread 0's stand in for those of the panels before)
		auto inserts = [&](const uint32_t t, const uint32_t i) {
			const uint32_t c = first + t;
			uint4 ins = zero;
			if (column(t) && (panel == 0u || c > r2)) {
				const uint32_t key = (c + kColumn) * 0x00010001u;
				const uint4 win = sub4(C[c * V + i], C[(c > r2 ? c - r2 - 1u : 0u) * V + i]);
				ins = make_uint4(__vcmpeq2(win.x, 0u) & __vcmpne2(own[i].x, 0u) & key,
					__vcmpeq2(win.y, 0u) & __vcmpne2(own[i].y, 0u) & key, __vcmpeq2(win.z, 0u) & __vcmpne2(own[i].z, 0u) & key,
					__vcmpeq2(win.w, 0u) & __vcmpne2(own[i].w, 0u) & key);
			} else if (c == 0u) {
				const uint32_t* const w = reinterpret_cast<const uint32_t*>(keep.seed) + 4u * i;
				ins = make_uint4(w[0], w[1], w[2], w[3]);
			}
			return ins;
		};
		uint4 ins[Cols][V];
#pragma unroll
		for (uint32_t i = 0u; i < V; i++) {
			acc[i] = zero;
		}
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			hist[t].widened(own);
#pragma unroll
			for (uint32_t i = 0u; i < V; i++) {
				ins[t][i] = inserts(t, i);
				acc[i] = max4(acc[i], ins[t][i]);
			}
		}
		uint32_t before = 0u, rank = mine;
		if (threadIdx.x == 0u && panel != 0u) {
			before = keep.bins[y - y0];
			rank += before;
		}
		block_exscan<V, true>(acc, total, wm, MaxOp {}, rank, all, keep.sums);
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			if (column(t)) {
#pragma unroll
				for (uint32_t i = 0u; i < V; i++) {
					acc[i] = max4(acc[i], ins[t][i]);
					M[(first + t) * V + i] = acc[i];
				}
			}
		}
		__syncthreads();
		if (threadIdx.x == 0u) {
			rank = before;
			if (more) {
				keep.bins[y - y0] = all;
			}
		}
		uint64_t o = keep.base[y - y0] + rank;
#pragma unroll
		for (uint32_t t = 0u; t < Cols; t++) {
			if (!pixel(t)) {
				continue;
			}
			const uint32_t c = first + t;
			J.offsets[static_cast<size_t>(y) * J.W + k0 + c] = static_cast<uint32_t>(o);
			const bool last = more && c + r2 + 1u == ncols; // the next panel starts from its order
			uint32_t place = 0u;
			auto put = [&](const uint32_t j) {
				if (o < J.bins_capacity) {
					const uint32_t n = static_cast<uint32_t>(C16[(c + r2 + 1u) * K + j]) - C16[c * K + j];
					const float weight = __fmul_rn(__uint2float_rn(n & 0xFFFFu), norm);
					bins[o] = make_uint2(keep.value[j], __float_as_uint(weight));
				}
				o++;
				if (last) {
					keep.order[y - y0][place++] = keep.value[j];
				}
			};
			// present items by (insertion column, place in its vertical histogram), after those of
			// before the panel by place; most pixels hold one or two
			uint32_t left = mask[t];
			while (left & (left - 1u)) {
				uint32_t best = 0u, least = 0xFFFFFFFFu;
				for (uint32_t m = left; m != 0u; m &= m - 1u) {
					const uint32_t j = static_cast<uint32_t>(__ffs(m) - 1);
					const uint32_t at = M16[(c + r2) * K + j];
					// every present item has an entry (the clamp only keeps a broken invariant inside
					// the tables)
					uint32_t key = at << 4;
					if (at >= kColumn) {
						key |= Hist::place(ord[min(at - kColumn, ncols - 1u)], j);
					}
					if (key < least) {
						least = key;
						best = j;
					}
				}
				left &= ~(1u << best);
				put(best);
			}
			if (left != 0u) {
				put(static_cast<uint32_t>(__ffs(left) - 1));
			}
			if (last) {
				keep.items[y - y0] = place;
			}
		}
	}
}

// The bins of the rows above each of [y0, y1), from the counts of all rows: no
// launch of its own scans them, which saves 1.6 us (of some 48 at 64^2, 74 at
// 512^2).  The last band's block writes the total.
__device__ __forceinline__ void band_bases(const ShfJob& J, const uint32_t y0, const uint32_t y1, BandRows& keep) {
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint64_t sum = 0u;
	for (uint32_t y = threadIdx.x; y < y0; y += blockDim.x) {
		sum += J.rows[y];
	}
	for (uint32_t d = 16u; d > 0u; d >>= 1) {
		sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
	}
	if (lane == 0u) {
		keep.parts[warp] = sum;
	}
	__syncthreads();
	if (threadIdx.x == 0u) {
		uint64_t base = 0u;
		for (uint32_t w = 0u; w < blockDim.x >> 5; w++) {
			base += keep.parts[w];
		}
		for (uint32_t y = y0; y < y1; y++) {
			keep.base[y - y0] = base;
			base += J.rows[y];
		}
		if (y1 == J.H) {
			const uint64_t most = 0xFFFFFFFFull;
			J.offsets[static_cast<size_t>(J.W) * J.H] = static_cast<uint32_t>(min(base, most));
			if (base > J.bins_capacity || base > most) {
				atomicOr(J.status, STATUS_CAPACITY);
			}
		}
	}
}

// Block (band, job).
template<bool Write, uint32_t Cols>
__global__ void __launch_bounds__(kPanelCols / Cols, Cols) shf_band_rows(const ShfJob* __restrict__ jobs, const ShfJob single,
	const ShfBandShape shape) {
	chain_begin();
	const ShfJob& J = pick(jobs, single);
	const uint32_t mode = shf_job_mode(J), band = blockIdx.x;
	if (mode == kShfModeSlide || band * shape.rows >= J.H) {
		return;
	}
	extern __shared__ uint4 fsm[];
	__shared__ __align__(16) BandRows keep;
	const ShfFastRecord* const rec = reinterpret_cast<const ShfFastRecord*>(J.fast);
	const Panels panels(J, shape.cols);
	if constexpr (Write) {
		band_bases(J, band * shape.rows, min(J.H, band * shape.rows + shape.rows), keep);
	}
	for (uint32_t p = 0u; p < panels.count; p++) {
		const uint32_t* const pal = panel_slot(J, band / shape.group * panels.count + p);
		__syncthreads(); // the panel before is done with the tables and the palette
		if (mode == kShfModeFast) {
			if (threadIdx.x < kShfFastItems) {
				keep.value[threadIdx.x] = rec->item[threadIdx.x];
			}
			__syncthreads();
			band_panel<Write, Cols, kShfFastItems>(J, shape, panels, band, p, false,
				BandPalette<kShfFastItems> { record_palette(rec) }, keep, fsm);
			continue;
		}
		if (threadIdx.x < kShfWideItems) {
			keep.value[threadIdx.x] = reinterpret_cast<const uint16_t*>(pal + 2u)[threadIdx.x];
		}
		__syncthreads();
		if (pal[0] <= kShfFastItems) {
			band_panel<Write, Cols, kShfFastItems>(J, shape, panels, band, p, true,
				BandPalette<kShfFastItems> { slot_palette(pal + 2u) }, keep, fsm);
		} else {
			band_panel<Write, Cols, kShfWideItems>(J, shape, panels, band, p, true,
				BandPalette<kShfWideItems> { slot_palette(pal + 2u), slot_palette(pal + 6u) }, keep, fsm);
		}
	}
}

int band_set_smem_attributes() {
	const int bytes = 100 * 1024;
	STPGB_CUDA_TRY(cudaFuncSetAttribute(shf_band_rows<false, 1u>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(shf_band_rows<false, 2u>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(shf_band_rows<true, 1u>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	STPGB_CUDA_TRY(cudaFuncSetAttribute(shf_band_rows<true, 2u>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
	return STPGB_OK;
}

template<bool Write>
int launch_rows(const ShfJob* jobs, const ShfJob& single, const uint32_t njobs, const ShfBandLaunch& cfg,
	cudaStream_t stream) {
	const dim3 grid(cfg.bands, njobs);
	// a column per thread where a row is one panel (64^2 44 us, with two columns 52; 300^2 of 20 biomes
	// 84 and 105), two where it is several (1024^2 of 8 biomes 182 us, with two columns 149; 4096^2 of
	// 32 1.30 ms and 1.20): half the scans per column, and two or three blocks per SM
	const bool one = cfg.panels == 1u;
	const uint32_t threads = one ? cfg.shape.cols : cfg.shape.cols / 2u;
	// Blocks that come up while the kernel before still runs pile up on the SMs that it leaves free,
	// unless an SM holds one of them (64 registers a thread) or they are few: 512^2 82 us, early 76;
	// 64^2 46 and 44; but 300^2 of 20 biomes 75 and 84, 4096^2 1.16 ms and 1.20.
	const bool early = threads > 512u || 2ull * cfg.bands * njobs <= current_sm_count();
	return one ? launch_chained(early, shf_band_rows<Write, 1u>, grid, threads, cfg.smem, stream, jobs, single, cfg.shape)
			   : launch_chained(early, shf_band_rows<Write, 2u>, grid, threads, cfg.smem, stream, jobs, single, cfg.shape);
}

uint32_t ceil_div(const uint32_t a, const uint32_t b) {
	return (a + b - 1u) / b;
}

} // namespace

ShfBandLaunch shf_band_config(const uint32_t njobs, const uint32_t max_W, const uint32_t max_H, const uint32_t max_r) {
	ShfBandLaunch cfg {};
	// panels of equal width, as few as kPanelCols allows (wider radii never take the bands)
	const uint32_t reach = 2u * std::min(max_r, kFastMaxRadius) + 1u;
	const uint32_t across = std::max(max_W, 2u) - 1u;
	const uint32_t fewest = ceil_div(across, kPanelCols - reach);
	cfg.shape.cols = ceil_div(ceil_div(across, fewest) + reach, 64u) * 64u;
	cfg.panels = ceil_div(across, cfg.shape.cols - reach);
	// about three blocks per SM over the launch; bands of kShfBandMinRows to kBandMaxRows rows
	const uint64_t want = (3ull * current_sm_count() + njobs - 1u) / std::max(njobs, 1u);
	const uint64_t rows = (static_cast<uint64_t>(max_H) + want - 1u) / std::max<uint64_t>(want, 1u);
	cfg.shape.rows = static_cast<uint32_t>(std::min<uint64_t>(std::max<uint64_t>(rows, kShfBandMinRows), kBandMaxRows));
	cfg.bands = ceil_div(max_H, cfg.shape.rows);
	const uint64_t columns = static_cast<uint64_t>(njobs) * cfg.bands * cfg.panels * cfg.shape.cols;
	cfg.shape.group = static_cast<uint32_t>(std::clamp<uint64_t>(
		columns / (static_cast<uint64_t>(kCarryThreadsPerSM) * current_sm_count()), 1u, std::max(1u, kCarryRows / cfg.shape.rows)));
	cfg.groups = ceil_div(cfg.bands, cfg.shape.group);
	// the tables of 16 values; of 8 they need less
	cfg.smem = (2u * cfg.shape.cols + 1u + 64u) * 2u * sizeof(uint4) + cfg.shape.cols * sizeof(uint64_t);
	return cfg;
}

int shf_band_carry_launch(const ShfJob* jobs, const ShfJob& single, const uint32_t njobs, const ShfBandLaunch& cfg,
	cudaStream_t stream) {
	const uint32_t works = ceil_div(cfg.shape.cols, kCarryBlock) * cfg.panels * cfg.groups;
	// blocks loop over the works: where the job goes the slides, 30000 that return at once took 32 us
	const uint32_t blocks = std::min(works, ceil_div(kCarryBlocksPerSM * current_sm_count(), njobs));
	return launch_chained(true, shf_band_carry, dim3(blocks, njobs), kCarryBlock, 0u, stream, jobs, single, cfg.shape,
		cfg.panels, works);
}

int shf_band_rows_launch(const ShfJob* jobs, const ShfJob& single, const uint32_t njobs, const ShfBandLaunch& cfg,
	const bool write, cudaStream_t stream) {
	STPGB_TRY(once_per_device(SETUP_SHF_BAND_SMEM, band_set_smem_attributes));
	return write ? launch_rows<true>(jobs, single, njobs, cfg, stream) : launch_rows<false>(jobs, single, njobs, cfg, stream);
}

} // namespace stpgb
