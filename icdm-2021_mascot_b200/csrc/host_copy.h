// Copies between pageable host memory and the GPU through a pinned staging ring, with several host threads.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace mascot {

struct CopySpan {
    void* host;
    void* dev;
    size_t bytes;
};

// Host -> device on `st`.  On return the host buffer has been read (it may change); the device side is complete in
// stream order.  Pinned source buffers are copied directly and must stay unchanged until the stream has passed.
cudaError_t copy_to_device(void* dev, const void* host, size_t bytes, cudaStream_t st);
// Device -> host after everything queued on `st`; the host buffers are complete on return.
cudaError_t copy_to_host(const CopySpan* spans, int n_spans, cudaStream_t st);
// Gives idle staging rings back to the system (they are allocated again at the next large copy).
void release_copy_rings();

}  // namespace mascot
