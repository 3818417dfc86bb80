// Copies of rectangles between host arrays and a merged device map by one
// kernel.  The generator's callers hand it nine (or more) chunk arrays in
// pageable host memory; where the GPU reads and writes such memory itself
// (through the host's page tables, as beside a Grace CPU), one launch moves
// them all: nine 2D copies of a 512^2 uint16 neighbourhood took 266 us, each
// staged by the driver; the launch takes 20 us for the part the filter reads
// (one 512^2 generate call 420 -> 142 us).  Bound by the link between the two
// memories.
#include "host_rects.hpp"

#include <algorithm>

namespace stpgb {

namespace {

constexpr uint32_t kRectThreads = 256u;
constexpr uint32_t kRectBlocksPerSM = 4u;

struct RectList {
	HostRect rect[kMaxRects];
};

template<typename Word>
__device__ __forceinline__ void copy_rect(const HostRect& R, const uint32_t first, const uint32_t stride) {
	const uint32_t words = R.width / static_cast<uint32_t>(sizeof(Word));
	for (uint32_t i = first; i < words * R.rows; i += stride) {
		const uint32_t y = i / words, x = i - y * words;
		const char* const src = static_cast<const char*>(R.src) + static_cast<size_t>(y) * R.src_pitch;
		char* const dst = static_cast<char*>(R.dst) + static_cast<size_t>(y) * R.dst_pitch;
		reinterpret_cast<Word*>(dst)[x] = reinterpret_cast<const Word*>(src)[x];
	}
}

// grid.y: the rectangle.  The widest word that divides its addresses, pitches and width.
__global__ void __launch_bounds__(kRectThreads) rects_kernel(const RectList L) {
	const HostRect& R = L.rect[blockIdx.y];
	const uint64_t all = reinterpret_cast<uintptr_t>(R.src) | reinterpret_cast<uintptr_t>(R.dst) | R.src_pitch | R.dst_pitch
		| R.width;
	const uint32_t first = blockIdx.x * kRectThreads + threadIdx.x, stride = gridDim.x * kRectThreads;
	if ((all & 15u) == 0u) {
		copy_rect<uint4>(R, first, stride);
	} else if ((all & 3u) == 0u) {
		copy_rect<uint32_t>(R, first, stride);
	} else {
		copy_rect<uint16_t>(R, first, stride);
	}
}

} // namespace

bool host_memory_direct() {
	// through the host's page tables: a GPU that takes faults on such memory instead would move the
	// caller's arrays to itself and back with every call
	int dev = 0, yes = 0;
	if (cudaGetDevice(&dev) != cudaSuccess
		|| cudaDeviceGetAttribute(&yes, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	return yes != 0;
}

int copy_host_rects(const HostRect* const rects, const uint32_t count, cudaStream_t stream) {
	for (uint32_t r0 = 0u; r0 < count; r0 += kMaxRects) {
		RectList L {};
		const uint32_t n = std::min(kMaxRects, count - r0);
		std::copy(rects + r0, rects + r0 + n, L.rect);
		const uint32_t across = std::max(1u, kRectBlocksPerSM * current_sm_count() / n);
		rects_kernel<<<dim3(across, n), kRectThreads, 0, stream>>>(L);
		STPGB_CUDA_TRY(cudaGetLastError());
	}
	return STPGB_OK;
}

} // namespace stpgb
