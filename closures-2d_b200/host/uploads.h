// uploads.h -- order between uploads on the legacy stream and the library's own
// streams.
//
// cudaMemcpy from pageable memory returns when the source has been read, before
// the last bytes have arrived, and the library's streams do not wait for the
// legacy one.
#pragma once

#include <cuda_runtime.h>

namespace clb {

// Waits until the copies and fills made on the legacy stream are done.
inline cudaError_t uploads_arrived() { return cudaStreamSynchronize(cudaStreamLegacy); }

// Lets work that is queued on `stream` from now on wait for them (the host does
// not wait: 36 x 74 P2 host-state step 100 us with uploads_arrived(), 92 with this).
inline cudaError_t order_after_uploads(cudaStream_t stream)
{
    cudaEvent_t ev;
    cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess)
        return e;
    e = cudaEventRecord(ev, cudaStreamLegacy);
    if (e == cudaSuccess)
        e = cudaStreamWaitEvent(stream, ev, 0);
    cudaEventDestroy(ev);   // (released once the wait is over)
    return e;
}

}  // namespace clb
