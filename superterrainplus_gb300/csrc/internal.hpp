// Internal helpers shared by the translation units of libstpgb.so.
#pragma once

#include "stpgb.h"

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

namespace stpgb {

// Thread-local message behind stpgb_last_error().
void set_error(const std::string& msg);
void clear_error();

// Device status word bits (set by kernels with atomicOr, read by stpgb_status_check).
enum : uint32_t {
	STATUS_CAPACITY = 1u << 0, // a caller-sized output or a per-window item bound was exceeded
	STATUS_TIMEOUT = 1u << 1   // a droplet reached the step cap
};

inline int cuda_fail(cudaError_t e, const char* what) {
	set_error(std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
	return STPGB_ECUDA;
}

inline int inval(const std::string& msg) {
	set_error(msg);
	return STPGB_EINVAL;
}

inline cudaStream_t as_stream(void* s) {
	return static_cast<cudaStream_t>(s);
}

// SM count of the current device, queried once per device (152 if the query fails).
uint32_t current_sm_count();

// Keys of one-time per-device set-up steps (function attributes are per device).
enum : unsigned { SETUP_SHF_SMEM = 0u, SETUP_SHF_BAND_SMEM = 1u, SETUP_EROSION_TILE_SMEM = 2u };

// Runs `setup` on the current device the first time `key` is asked for there and it succeeds;
// serialised under a lock, so concurrent first calls from several host threads set up once.
int once_per_device(unsigned key, int (*setup)());

// Launches `kernel` so that its blocks may be brought to the SMs while the
// kernel before it in the stream still runs: every block of such a kernel
// begins with chain_begin(), which waits until all work before it is complete
// and visible, and lets the next kernel's blocks be brought up in turn.  What
// is saved is the gap between two kernels of a chain of short ones (one
// 64^2 chunk's filter, nine launches: 68 -> 53 us).  Without `early_up` the
// launch is an ordinary one: blocks that wait hold their shared memory, and a
// full launch of many chunks that lives on its L1 pays for that (the packed
// slides of a 144-chunk batch 1.53 -> 2.7 ms).
template<class... Params, class... Args>
int launch_chained(const bool early_up, void (*kernel)(Params...), const dim3 grid, const dim3 block, const size_t smem,
	const cudaStream_t stream, Args&&... args) {
	cudaLaunchAttribute early {};
	early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	early.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t config {};
	config.gridDim = grid;
	config.blockDim = block;
	config.dynamicSmemBytes = smem;
	config.stream = stream;
	config.attrs = &early;
	config.numAttrs = early_up ? 1u : 0u;
	const cudaError_t e = cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
	if (e != cudaSuccess) {
		cudaGetLastError();
		return cuda_fail(e, "cudaLaunchKernelEx");
	}
	return STPGB_OK;
}

#ifdef __CUDACC__
__device__ __forceinline__ void chain_begin() {
	asm volatile("griddepcontrol.launch_dependents;");
	asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

} // namespace stpgb

#define STPGB_CUDA_TRY(expr)                                   \
	do {                                                       \
		const cudaError_t stpgb_e_ = (expr);                   \
		if (stpgb_e_ != cudaSuccess) {                         \
			return ::stpgb::cuda_fail(stpgb_e_, #expr);        \
		}                                                      \
	} while (0)

#define STPGB_TRY(expr)                                        \
	do {                                                       \
		const int stpgb_rc_ = (expr);                          \
		if (stpgb_rc_ != STPGB_OK) {                           \
			return stpgb_rc_;                                  \
		}                                                      \
	} while (0)
