// uploads.h -- plain host-to-device copies before work on a non-blocking stream.
#pragma once
#include <cuda_runtime.h>

namespace falcon {

// A cudaMemcpy from pageable memory may return once the data is staged, and nothing orders
// it before work on the library's non-blocking streams: called after the last of a group
// of such copies, before the work that reads them is queued.
inline cudaError_t uploads_arrived() { return cudaStreamSynchronize(cudaStreamLegacy); }

}  // namespace falcon
