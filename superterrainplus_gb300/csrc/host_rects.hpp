// Rectangles copied between host and device memory by one kernel.
#pragma once

#include "internal.hpp"

namespace stpgb {

// rectangles of one launch (kernel parameters)
constexpr uint32_t kMaxRects = 64u;

// `rows` rows of `width` bytes, an even number as are the addresses and pitches (bytes)
struct HostRect {
	const void* src;
	void* dst;
	uint32_t src_pitch, dst_pitch, width, rows;
};

// Whether the current device reads and writes pageable host memory itself, where it lies.
bool host_memory_direct();
// Enqueues the copies; host arrays must stay until the stream is waited for.
int copy_host_rects(const HostRect* rects, uint32_t count, cudaStream_t stream);

} // namespace stpgb
