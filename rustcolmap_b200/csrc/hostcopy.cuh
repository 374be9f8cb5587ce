// hostcopy.cuh — large copies between the caller's (pageable) memory and the device.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace rcmvs {

// Queues a copy on st, of the current device.  Upload: a pageable source may
// change on return (a pinned one once st has passed the copy).
cudaError_t host_upload(void* dev, const void* host, size_t n, cudaStream_t st);
// The destination is filled on return, with all that was queued on st done.
cudaError_t host_download(void* host, const void* dev, size_t n, cudaStream_t st);

// Contexts that may copy; what the copies keep (threads, pinned buffers) is
// given back with the last one.  false: no memory, nothing attached.
bool host_copy_attach();
void host_copy_detach();

}  // namespace rcmvs
