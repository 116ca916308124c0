// Copies between pageable host matrices and device matrices through pinned
// staging, by several host threads.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace tns {

// The driver's own copy of pageable memory is one thread through one staging
// buffer: 134 MB took 12.0 ms to the device and 7.9 ms back, against 2.4 ms
// either way from pinned memory; one thread's memcpy moves 15 GB/s, four 50,
// and pages touched for the first time cost more still (61 ms by one thread,
// 9.5 by eight). Here every thread packs (or unpacks) pieces of up to kPiece
// bytes through two pinned slots of its own while the others' pieces cross the
// bus: 3.0 ms to the device and 3.3 ms back (8 threads, pieces of 1 MiB; 4.4
// and 6 with pieces of 256 KiB, 3.5 and 4.4 with four threads). One per
// Context, made at its first large copy and given back with it: at most
// kMaxThreads - 1 helper threads and 2 * kMaxThreads * kPiece pinned bytes.
class HostCopier {
public:
    static constexpr size_t kPiece = size_t(1) << 20;
    static constexpr int kMaxThreads = 8;
    // Below this many bytes the driver's copy is as fast: norms of square matrices
    // took, with it and with pieces, 124 and 125 us at 262 KB, 89 and 90 at 320 KB,
    // 103 and 90 at 387 KB, 117 and 95 at 500 KB, 148 and 130 at 1.4 MB.
    static constexpr size_t kLeast = size_t(256) << 10;

    explicit HostCopier(int device);
    ~HostCopier();
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;

    // False when the pinned memory is not to be had (the caller copies plainly).
    bool usable() const { return pinned_ != nullptr; }
    // rows x cols elements of `esz` bytes. `device` is the padded side: ld_dev
    // >= rows, its padding zero (to_device writes it so). Both return when the
    // host side is done with; to_device's last pieces may still be in flight on
    // `stream`. Errors: a CUDA error code.
    cudaError_t to_device(cudaStream_t stream, char* device, size_t ld_dev, const char* host, size_t ld_host, size_t rows,
                          size_t cols, size_t esz);
    cudaError_t to_host(cudaStream_t stream, char* host, size_t ld_host, const char* device, size_t ld_dev, size_t rows,
                        size_t cols, size_t esz);

private:
    struct Slot {
        char* p = nullptr;
        cudaEvent_t done = nullptr;
    };
    void run(int threads, const std::function<void(int)>& work);
    void helper(int index);
    void release();

    int device_;
    char* pinned_ = nullptr;
    Slot slots_[kMaxThreads][2];
    std::vector<std::thread> helpers_;
    std::mutex mutex_;
    std::condition_variable start_, finish_;
    const std::function<void(int)>* work_ = nullptr;
    int wanted_ = 0;   // helpers that the current run takes
    int pending_ = 0;  // of them not yet done
    unsigned long long run_ = 0;
    bool stop_ = false;
};

}  // namespace tns
