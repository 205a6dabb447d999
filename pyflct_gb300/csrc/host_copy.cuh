// host_copy.cuh -- copies between a caller's host arrays and the device for
// the host-buffer entry points.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace flct {

// Arrays up to this size go in one kernel that reads or writes the host memory
// itself, where the GPU shares the host's page tables: the rate is the copy
// engine's (150-165 GB/s either way), and one launch replaces two to five
// copies of about 10 us of latency each.  A call on 201 x 101 frames 147 ->
// 105 us, 512^2 -s 3i 225 -> 178, 1024^2 -s 4i 532 -> 490.  Larger arrays
// gain nothing by it, and pages that were never touched cost a kernel more
// than the copy engine.  Arrays off an 8-byte boundary, and results that share
// memory, go to the runtime.
constexpr size_t kHostKernelBytes = 1u << 24;
// Copies in of up to this many bytes in all are taken by the runtime as they
// are enqueued, while a kernel would first have to fetch them: 2-3 us of a
// 60 us call (shift of 17 x 17 63.6 -> 60.4 us, velocity of 24 x 24 66.3 ->
// 63.6); three arrays of 18 KB gain nothing.
constexpr size_t kHostStagedBytes = 1u << 15;

// `count` arrays of n doubles, src[k] to dst[k], ordered on st.  direct: the
// GPU may use pageable host addresses (cudaDevAttrPageableMemoryAccess with
// the host's page tables).
cudaError_t copy_arrays(const double* const* src, double* const* dst, int count, size_t n, cudaMemcpyKind kind,
                        bool direct, cudaStream_t st);

// Makes a caller's output pages present while the GPU computes: 8 MB of fresh
// pages cost a copy 377 us through GPU faults, 52 us once they are there.
// Leaves the contents as they are.  False where the host may not write them (or
// the system cannot tell): a copy kernel must not either, a store to such a page
// is a fault of the device where the runtime's copy returns an error.  (Results
// of less than a page are touched: without permission that is the host's own
// fault, as a copy by the host would be.)
bool populate_output(void* p, size_t bytes);

}  // namespace flct
