// How many CTAs of a kernel an SM holds at once.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>

namespace msda {

// CTAs of `threads` threads and `smem` bytes of dynamic shared memory that one SM of the current
// device holds at once (at least 1); lets the kernel use that much shared memory. Asked of the
// runtime once per kernel, size and device: the query costs more host time than a launch. May be
// called by several threads.
cudaError_t resident_ctas(const void* kernel, int threads, size_t smem, int* per_sm);

}  // namespace msda
