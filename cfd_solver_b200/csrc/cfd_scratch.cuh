// cfd_scratch.cuh -- device scratch of the seams' calls.
//
// A seam call needs scratch for its own duration only. cudaMalloc and cudaFree per call cost
// 0.7 to 3 ms on a busy host (they synchronise the device and take the driver's locks), more
// than the solve itself; here the scratch comes from a pool of the library, one per device,
// stream-ordered on the caller's stream, so calls from several threads and streams share it
// safely. The pool keeps at most kScratchKeep bytes between calls and gives anything above back
// to the device at the next synchronisation. A pool dies with its context (cudaDeviceReset), so
// it is kept with the context's id.
#pragma once
#include <cuda_runtime.h>

namespace cfd {
constexpr unsigned long long kScratchKeep = 256ull << 20;
constexpr unsigned kSeamPolls = 1u << 24;  // polls of the gauss solve's barrier before it gives up (about 10 s)
// scratch of `bytes` bytes on the current device, usable by work on `st`; nullptr: no memory
void* scratch_take(size_t bytes, cudaStream_t st);
// gives it back once the work queued on `st` so far is done
void scratch_give(void* p, cudaStream_t st);
// id of the calling thread's context, never used again by another one; 0: none, or the query failed
unsigned long long context_id();
}  // namespace cfd
