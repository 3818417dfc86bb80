// Single histogram filter: job descriptor and batched launch entry shared by
// the per-chunk C ABI (shf.cu) and the batched pipeline.
#pragma once

#include "internal.hpp"

namespace stpgb {

// Library bound on the number of distinct sample values inside one filter
// window; it sizes the per-thread accumulators in shared memory.
constexpr uint32_t kShfMaxItems = 256u;

// Most segments a column (vertical pass) or row (horizontal pass) is cut
// into; the workspace holds one bin count per (row, segment).
constexpr uint32_t kShfMaxSegments = 16u;

// One filter invocation over one chunk.  `samplemap` points at the top-left
// pixel of the chunk's nearest-neighbour region (TotalMapSize), rows `pitch`
// elements apart; the central chunk starts at (sx, sy).
struct ShfJob {
	const uint16_t* samplemap;
	uint64_t pitch;
	uint32_t W, H, sx, sy, r;
	uint32_t kcap_v; // accumulator capacity of the vertical pass (<= 2r+1)
	// workspace
	uint32_t* vbuf;  // [W+2r][kcap_v][H] packed (item << 16 | count), column-major
	uint16_t* vn;    // [W+2r][H] entries per vertical histogram
	uint32_t* rows;  // [H*segments+1] bins per (row, segment), then exclusive prefix + total
	uint32_t* fast;  // [8] path record (ShfFastRecord)
	// output
	uint32_t* offsets;  // [W*H+1]
	stpgb_bin* bins;
	uint64_t bins_capacity;
	uint32_t* status;
};

// The few-values path (shf_fast.cu, shf_band.cu) filters a chunk whose read
// region holds at most kShfFastItems distinct sample values; its row bands also
// take chunks of more whose panels hold at most kShfWideItems each; the others
// take the general slides.  Its packed vertical histograms (12 bytes per
// column and row, or per band; 24 with a palette per panel) overlay `vbuf`,
// which that chunk does not otherwise use.
constexpr uint32_t kShfFastItems = 8u;
// A job's path: the general slides, the few-values path, or the row bands with
// a palette of up to kShfWideItems values per panel (a chunk of more values of
// which no panel holds more).
constexpr uint32_t kShfWideItems = 16u;
constexpr uint32_t kShfModeSlide = 0u, kShfModeFast = 1u, kShfModeWide = 2u;
// Widest chunk (W + 2r) that the row bands take with one palette.
constexpr uint32_t kShfBandMaxCols = 4096u;
// Fewest rows of a band, unless the chunk has fewer.
constexpr uint32_t kShfBandMinRows = 2u;

// Record of the path a job takes, written by the routing kernel: words
// {mode, distinct values, formulation (kShfForm*, 0 outside the few-values
// path), 1 where a panel turned out to hold too many values for mode Wide, then
// the values as 8 uint16, ascending}.
struct ShfFastRecord {
	uint32_t mode, count, form, crowded;
	uint16_t item[kShfFastItems];
};
static_assert(sizeof(ShfFastRecord) == 32u, "record is 8 words");

__device__ __forceinline__ uint32_t shf_job_mode(const ShfJob& J) {
	const volatile ShfFastRecord* const rec = reinterpret_cast<const volatile ShfFastRecord*>(J.fast);
	const uint32_t mode = rec->mode;
	return mode == kShfModeWide && rec->crowded != 0u ? kShfModeSlide : mode;
}

// the general slides' kernels filter only the jobs routed to them
__device__ __forceinline__ bool shf_job_general(const ShfJob& J) {
	return shf_job_mode(J) == kShfModeSlide;
}

struct ShfLayout {
	size_t vbuf, vn, rows, fast, total;
};

// Workspace layout for one job (256-byte aligned sub-buffers).
ShfLayout shf_layout(uint32_t W, uint32_t H, uint32_t r, uint32_t kcap_v);
// Points the job's workspace fields at the sub-buffers of `ws` (laid out by shf_layout).
void shf_bind_workspace(ShfJob& job, unsigned char* ws, const ShfLayout& l);
uint32_t shf_kcap_v(uint32_t r, uint32_t max_items);
uint32_t shf_kcap_h(uint32_t r, uint32_t max_items);

// Runs the whole filter for `njobs` jobs (device array `jobs`, or `single`
// when jobs == nullptr). max_W/max_H/max_r bound the grids.
// `segments`: the general slides' columns and rows cut into this many
// segments (clamped to [1, kShfMaxSegments] and the slide length); 0 = chosen
// from the launch size.  `path`: 0 = the process-wide choice
// (stpgb_shf_set_path, by size by default), else that choice for this launch
// (1 packed slides, 2 row bands, 3 general slides).  `clear_status`: zero each
// job's status word first.
int shf_launch(const ShfJob* jobs, const ShfJob& single, uint32_t njobs, uint32_t max_W, uint32_t max_H,
	uint32_t max_r, uint32_t kcap_v, uint32_t kcap_h, cudaStream_t stream, uint32_t segments = 0u,
	uint32_t path = 0u, bool clear_status = false);

// The few-values path's launches around the general slides: palette and
// vertical histograms, then the bin count per row (before the row scan), and
// the write pass (after it).  Jobs that do not qualify return at once.  Two
// formulations: sequential slides in packed form (a thread per column, then
// per row) for launches of many chunks, row bands with prefix scans (a block
// per band of rows) for launches of few.
// A launch's cut into bands and panels: bands of `rows` rows, the carry's
// groups of `group` bands, panels of `cols` columns of the read region.
struct ShfBandShape {
	uint32_t rows, group, cols;
};
struct ShfBandLaunch {
	ShfBandShape shape;
	uint32_t bands, groups, panels; // of the largest chunk
	size_t smem;
};
struct ShfFastPlan {
	bool bands;
	uint32_t max_cols; // widest chunk (W + 2r) the few-values path takes; 0: none
	bool wide; // chunks of more values may take the bands with a palette per panel
	ShfBandLaunch band;
};
// stpgb_shf_set_path's choice (0 = by size)
uint32_t shf_path_override();
// the record's form: the few-values formulation that filtered the job
constexpr uint32_t kShfFormSlides = 1u, kShfFormBands = 2u;
ShfFastPlan shf_fast_plan(uint32_t njobs, uint32_t max_W, uint32_t max_H, uint32_t max_r, uint32_t path = 0u);
int shf_fast_prepare(const ShfJob* jobs, const ShfJob& single, uint32_t njobs, uint32_t max_W, uint32_t max_H,
	uint32_t max_r, uint32_t kcap_h, const ShfFastPlan& plan, bool clear_status, cudaStream_t stream);
int shf_fast_pass(const ShfJob* jobs, const ShfJob& single, uint32_t njobs, uint32_t max_H, const ShfFastPlan& plan,
	bool write, cudaStream_t stream);
// the row-band formulation (shf_band.cu)
ShfBandLaunch shf_band_config(uint32_t njobs, uint32_t max_W, uint32_t max_H, uint32_t max_r);
int shf_band_carry_launch(const ShfJob* jobs, const ShfJob& single, uint32_t njobs, const ShfBandLaunch& cfg,
	cudaStream_t stream);
int shf_band_rows_launch(const ShfJob* jobs, const ShfJob& single, uint32_t njobs, const ShfBandLaunch& cfg,
	bool write, cudaStream_t stream);

} // namespace stpgb
