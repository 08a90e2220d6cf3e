// Grow-only device buffers of a context (DeviceBuffer, common.cuh). Host code that needs nothing but the runtime's
// allocation calls, so that running out of memory can be tested without a GPU.
#include "common.cuh"

namespace yscv {

// Is the stream being captured? (A query that fails, as on the legacy stream while another thread captures,
// is not this call's failure: the launch that follows reports it.)
bool stream_capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return st != cudaStreamCaptureStatusNone;
}

// The new block first: when there is no memory for it the old one stays as it is, unless nobody can be using it
// (no graph holds its address, no call has it in hand) and its own bytes are what is missing.
cudaError_t DeviceBuffer::grow(size_t want, bool in_use) {
    const size_t least = want < 256 ? 256 : want;
    size_t sz = in_graph && ptr && least < bytes + bytes / 2 ? bytes + bytes / 2 : least;
    void *fresh = nullptr;
    cudaError_t e = cudaMalloc(&fresh, sz);
    if (e == cudaErrorMemoryAllocation && sz > least) {
        cudaGetLastError();
        e = cudaMalloc(&fresh, sz = least);
    }
    if (e == cudaErrorMemoryAllocation && ptr && !in_graph && !in_use) {
        cudaGetLastError();
        e = cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
        if (e == cudaSuccess) e = cudaMalloc(&fresh, sz);
    }
    if (e != cudaSuccess) return e;
    if (ptr && in_graph) captured.push_back(ptr);
    else if (ptr) e = cudaFree(ptr);
    ptr = fresh;
    bytes = sz;
    in_graph = false;
    return e;
}

int DeviceBuffer::reserve(size_t want) {
    if (want > bytes || !ptr) YSCV_CUDA_TRY(grow(want, false));
    return YSCV_CUDA_OK;
}

int DeviceBuffer::reserve(size_t want, cudaStream_t stream) {
    const bool capturing = stream_capturing(stream);
    const int rc = reserve(want);
    in_graph = in_graph || (capturing && rc == YSCV_CUDA_OK);
    return rc;
}

bool DeviceBuffer::try_reserve(size_t want, cudaStream_t stream, bool in_use) {
    const bool capturing = stream_capturing(stream);
    if (want > bytes || !ptr) {
        if (capturing) return false;
        if (grow(want, in_use) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    }
    in_graph = in_graph || capturing;
    return true;
}

void DeviceBuffer::release() {
    if (ptr) cudaFree(ptr);
    for (void *p : captured) cudaFree(p);
    captured.clear();
    ptr = nullptr;
    bytes = 0;
    in_graph = false;
}

}  // namespace yscv
