// Copies between pageable host memory and the device through page-locked slots, several threads at once.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace tg {

// host <-> device copy of `bytes` behind the work of stream s; on success the copy has ended (host buffer and
// device buffer may be used).  Page-locked host memory, short copies, the first copies since an owner came, the
// per-thread default stream and a stream in capture go through cudaMemcpyAsync.
cudaError_t host_copy(void* dst, const void* src, size_t bytes, bool to_device, int device, cudaStream_t s);

// the owners of the copying threads and their slots (contexts, servers): the last one to leave gives them back
void host_copy_retain();
void host_copy_release();

}  // namespace tg
