// dcm_hostcopy.h -- copies between pageable host arrays and device memory.
//
// The driver moves pageable memory through one thread's copy into its own
// page-locked buffer; page-locked memory moves at 55 GB/s.  Here several
// threads copy between the caller's array and a ring of page-locked buffers
// while the DMA of another buffer runs.  GB/s on a B200's host (16 cores),
// driver -> here: to the device 19 -> 35 at 6.6 MB, 15 -> 45 at 69 MB; back
// 19 -> 26 and 21 -> 50, and 2.2 -> 13 into 69 MB of pages never touched.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace dcm {

// A handle's share of the process' one copier: its threads and buffers (four
// of 4 MB) are made by the first transfer that uses it and given back with the
// last handle.
void hostcopy_retain();
void hostcopy_release();

// dst (device) <- src (host) on st, n bytes; back when src has been read.
cudaError_t hostcopy_h2d(void* dst, const void* src, size_t n, cudaStream_t st);
// dst (host) <- src (device) on st, n bytes.  Page-locked dst: queued on st;
// pageable: back when dst is written.
cudaError_t hostcopy_d2h(void* dst, const void* src, size_t n, cudaStream_t st);

}  // namespace dcm
