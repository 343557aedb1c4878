/*
 * csrc/upload.hpp on a runtime that test_uploads.py can watch: built without the CUDA runtime, with
 * the calls it makes defined here.  Host memory stands in for the device's; copies from pinned
 * buffers are carried out late, by the next wait for their event, as a copy engine may.
 */
#include <mutex>
#include <vector>

#include "upload.hpp"

namespace {

struct Late {
    char *dst;
    const char *src;
    size_t n;
};
std::mutex mu;
std::vector<Late> late;
char *pinned = nullptr;
size_t pinned_bytes = 0;
long long made = 0, freed = 0, plain = 0, staged = 0, refuse_alloc = 0, fail_copy = 0;
const char *registered = nullptr;
size_t registered_bytes = 0;

void finish() {
    for (const Late &c : late) std::memcpy(c.dst, c.src, c.n);
    late.clear();
}

}  // namespace

extern "C" {

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) {
    if (refuse_alloc) return cudaErrorMemoryAllocation;
    ++made;
    *p = pinned = new char[bytes];
    pinned_bytes = bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    ++freed;
    delete[] static_cast<char *>(p);
    pinned = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new int(0)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<int *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    std::lock_guard<std::mutex> lock(mu);
    finish();
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> lock(mu);
    const char *from = static_cast<const char *>(src);
    if (pinned && from >= pinned && from < pinned + pinned_bytes) {
        if (fail_copy) return cudaErrorUnknown;
        ++staged;
        late.push_back({static_cast<char *>(dst), from, n});
    } else {
        ++plain;
        std::memcpy(dst, src, n);
    }
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    const char *at = static_cast<const char *>(p);
    a->type = at >= registered && at < registered + registered_bytes ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}

Uploader *uploader_new() { return new Uploader(); }
void uploader_release(Uploader *u) { u->release(); }
void uploader_delete(Uploader *u) { delete u; }
int uploader_copy(Uploader *u, void *dst, const void *src, size_t bytes) {
    const cudaError_t e = u->copy(dst, src, bytes, nullptr);
    std::lock_guard<std::mutex> lock(mu);
    finish();   // the stream's end
    return e;
}
void set_registered(const void *p, size_t bytes) { registered = static_cast<const char *>(p); registered_bytes = bytes; }
void set_failures(int alloc, int copy) { refuse_alloc = alloc; fail_copy = copy; }
/* buffers made, given back, plain copies, staged pieces since the last call */
void counts(long long *out) {
    const long long now[4] = {made, freed, plain, staged};
    std::memcpy(out, now, sizeof now);
    made = freed = plain = staged = 0;
}

}
