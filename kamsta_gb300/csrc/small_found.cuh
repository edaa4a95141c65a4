// small_found.cuh -- one small graph solved by one CTA, forest in the order
// the rounds find it (small_solve.cuh): the allocation-free entry point and
// the device entry points' smallest inputs.
#pragma once
#include <cuda_runtime.h>

#include "small_solve.cuh"

namespace kamsta {
namespace small {

// CTA size by input: a small graph's phases are as short as the barriers of a
// large CTA (1000 vertices, 8000 entries: 33 us on 1024 threads, 26 on 256).
constexpr int kFoundThreads = 1024, kFoundThreadsFew = 256;
constexpr uint64_t kFoundFewMd = 1ull << 14;

// Launches the solve on `st`; scratch holds kScratchBytes and starts with the
// Result.  Ids are checked against n, the order when check_order is set.
// found_setup() first, once per device.
cudaError_t found_setup();
cudaError_t found_launch(const uint32_t* in, uint32_t md, uint32_t n, unsigned char* scratch,
                         uint32_t* out, bool check_order, cudaStream_t st);

}  // namespace small
}  // namespace kamsta
