// DeviceBuffer (yscv_b200/csrc/device_buffer.cu) on a runtime whose memory runs out on request.
#include <cstdlib>
#include <set>

#include "../yscv_b200/csrc/common.cuh"

static std::set<void *> live;
static size_t room;          // bytes a request may have
static bool capturing;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (n > room) return cudaErrorMemoryAllocation;
    live.insert(*p = malloc(1));
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (p && !live.erase(p)) abort();   // freed twice, or never given
    free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
}
namespace yscv {
int fail(int status, const char *, ...) { return status; }
}

#define CHECK(c) \
    if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }

int main() {
    yscv::DeviceBuffer b;
    room = 1000;
    CHECK(b.reserve(600, nullptr) == YSCV_CUDA_OK);
    void *const first = b.ptr;
    // a call that works on the block: whatever the answer, the block is there and as large
    CHECK(!b.try_reserve(2000, nullptr, true) && b.ptr == first && b.bytes == 600 && live.count(first));
    capturing = true;
    CHECK(!b.try_reserve(900, nullptr, true) && b.ptr == first && live.count(first));
    capturing = false;
    CHECK(b.try_reserve(900, nullptr, true) && b.ptr != first && b.bytes == 900 && live.size() == 1);
    // nobody works on it: its bytes may make room, and a failure leaves an empty buffer that a later call fills
    CHECK(!b.try_reserve(2000, nullptr) && !b.ptr && b.bytes == 0 && live.empty());
    CHECK(b.reserve(2000, nullptr) != YSCV_CUDA_OK && !b.ptr);
    CHECK(b.reserve(300, nullptr) == YSCV_CUDA_OK && live.count(b.ptr));
    // a graph holds its address: kept when outgrown, kept when there is no room
    capturing = true;
    CHECK(b.try_reserve(300, nullptr));
    capturing = false;
    void *const held = b.ptr;
    CHECK(!b.try_reserve(2000, nullptr) && b.ptr == held);
    CHECK(b.try_reserve(400, nullptr, true) && b.ptr != held && live.count(held) && live.size() == 2);
    b.release();
    CHECK(live.empty());
    return 0;
}
