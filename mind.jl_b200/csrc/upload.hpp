/*
 * Copies of large arrays from a caller's pageable memory to the device.
 *
 * The runtime stages a pageable copy through pinned memory on one thread, at the rate of one
 * thread's memory copies.  Here a few threads take 512 KB pieces of the array in turn, each through two
 * pinned buffers of its own, so that their copies to the buffers run side by side and
 * the DMA engine is always fed: 20,000 rows of 645 inputs (51.6 MB) are predicted in 2.2 ms in
 * place of 4.4, 100,000 in 10.2 in place of 23.5.  At 5 MB both take 0.43 ms, which is where the line
 * between them lies.  Making the pinned buffers takes 2-4 ms, which a network that is used
 * once would lose: they are made by the copy with which the large ones so far come to 256 MB, where
 * even a host whose plain copies are fast (51.6 MB in 2.9 ms a call in place of 2.2) has it back.
 * Like a pageable cudaMemcpyAsync, the call returns when the source has been read, and the data is
 * there for what follows on the stream.
 */
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <thread>

class Uploader {
  public:
    static constexpr size_t kPiece = 512 * 1024;
    static constexpr int kThreads = 4;
    static constexpr size_t kStagedBytes = 8 * kPiece;   // smaller arrays go as they are
    static constexpr size_t kRepaidBytes = (size_t)256 << 20;   // buffers are made for this much

    Uploader() = default;
    Uploader(const Uploader &) = delete;
    Uploader &operator=(const Uploader &) = delete;

    /* dst (device) = src (host), `bytes` of it, on `stream`; one call at a time per object. */
    cudaError_t copy(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
        if (bytes < kStagedBytes || !pageable(src) || !buffers(bytes))
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
        int device = 0;
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        std::atomic<size_t> next{0};
        std::atomic<int> failed{cudaSuccess};
        auto work = [&](int t) {
            cudaError_t s = cudaSetDevice(device);
            for (int turn = 0; s == cudaSuccess && failed.load() == cudaSuccess; turn ^= 1) {
                const size_t at = next.fetch_add(1) * kPiece;
                if (at >= bytes) return;
                const size_t n = bytes - at < kPiece ? bytes - at : kPiece;
                char *buffer = staging_ + (2 * t + turn) * kPiece;
                s = cudaEventSynchronize(read_[2 * t + turn]);   // the buffer's last copy has left it
                if (s != cudaSuccess) break;
                std::memcpy(buffer, static_cast<const char *>(src) + at, n);
                s = cudaMemcpyAsync(static_cast<char *>(dst) + at, buffer, n, cudaMemcpyHostToDevice, stream);
                if (s == cudaSuccess) s = cudaEventRecord(read_[2 * t + turn], stream);
            }
            if (s != cudaSuccess) failed.store(s);
        };
        std::thread helpers[kThreads - 1];
        try {
            for (int t = 1; t < kThreads; ++t) helpers[t - 1] = std::thread(work, t);
        } catch (...) {
            // no more threads: those that run, this one at least, take all pieces
        }
        work(0);
        for (std::thread &h : helpers)
            if (h.joinable()) h.join();
        return static_cast<cudaError_t>(failed.load());
    }

    /* Gives the pinned buffers back; the streams that were copied on have been waited for. */
    void release() {
        for (cudaEvent_t &e : read_) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (staging_) cudaFreeHost(staging_);
        staging_ = nullptr;
        seen_ = 0;
    }

  private:
    /* Whether the runtime would stage a copy from p itself. */
    static bool pageable(const void *p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }

    /* Whether there are pinned buffers (4 MB) for a copy of `bytes`; makes them when it is time.  Where
     * they cannot be had, copies go as they are for as much again. */
    bool buffers(size_t bytes) {
        if (staging_) return true;
        seen_ = bytes < kRepaidBytes - seen_ ? seen_ + bytes : kRepaidBytes;
        if (seen_ < kRepaidBytes) return false;
        void *p = nullptr;
        bool made = cudaHostAlloc(&p, 2 * kThreads * kPiece, cudaHostAllocDefault) == cudaSuccess;
        staging_ = made ? static_cast<char *>(p) : nullptr;
        for (cudaEvent_t &e : read_)
            if (made) made = cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
        if (!made) {
            (void)cudaGetLastError();
            release();
        }
        return made;
    }

    size_t seen_ = 0;   // large copies so far, until the buffers are made
    char *staging_ = nullptr;
    cudaEvent_t read_[2 * kThreads] = {};
};
