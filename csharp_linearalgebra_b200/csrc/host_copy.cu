// Staged copies between pageable host memory and the device (host_copy.h).

#include "host_copy.h"

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace tns {

HostCopier::HostCopier(int device) : device_(device) {
    const int cores = (int)std::thread::hardware_concurrency();
    const int threads = std::clamp(cores / 2, 1, kMaxThreads);
    if (cudaHostAlloc(reinterpret_cast<void**>(&pinned_), 2 * kPiece * threads, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();  // not sticky; the plain copies still work
        pinned_ = nullptr;
        return;
    }
    for (int t = 0; t < threads; ++t)
        for (int b = 0; b < 2; ++b) {
            slots_[t][b].p = pinned_ + (size_t)(2 * t + b) * kPiece;
            if (cudaEventCreateWithFlags(&slots_[t][b].done, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                release();
                return;
            }
        }
    try {
        helpers_.reserve(threads - 1);
        for (int t = 1; t < threads; ++t) helpers_.emplace_back([this, t] { helper(t); });
    } catch (const std::exception&) {
        // No thread (system_error) or no memory for one (bad_alloc): fewer
        // helpers then, the calling thread alone in the worst case. Nothing may
        // leave here, since the destructor that joins them would not run.
    }
}

HostCopier::~HostCopier() {
    {
        std::lock_guard<std::mutex> lock(mutex_);
        stop_ = true;
    }
    start_.notify_all();
    for (auto& h : helpers_) h.join();
    release();
}

void HostCopier::release() {
    for (auto& pair : slots_)
        for (auto& s : pair)
            if (s.done) {
                cudaEventDestroy(s.done);
                s.done = nullptr;
            }
    if (pinned_) cudaFreeHost(pinned_);
    pinned_ = nullptr;
}

void HostCopier::helper(int index) {
    cudaSetDevice(device_);
    unsigned long long seen = 0;
    std::unique_lock<std::mutex> lock(mutex_);
    for (;;) {
        start_.wait(lock, [&] { return stop_ || run_ != seen; });
        if (stop_) return;
        seen = run_;
        if (index > wanted_) continue;
        const std::function<void(int)>* work = work_;
        lock.unlock();
        (*work)(index);
        lock.lock();
        if (--pending_ == 0) finish_.notify_one();
    }
}

// work(0) here and work(1..threads-1) on the helpers; `work` does not throw.
void HostCopier::run(int threads, const std::function<void(int)>& work) {
    const int helpers = std::min(threads - 1, (int)helpers_.size());
    if (helpers > 0) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            work_ = &work;
            wanted_ = pending_ = helpers;
            ++run_;
        }
        start_.notify_all();
    }
    work(0);
    if (helpers > 0) {
        std::unique_lock<std::mutex> lock(mutex_);
        finish_.wait(lock, [&] { return pending_ == 0; });
        work_ = nullptr;
    }
}

namespace {

// memcpy into a pinned slot past the caches: the bus read lines that were
// dirty in the packing cores' caches at 19 GB/s, lines in memory at 55.
void pack(char* dst, const char* src, size_t bytes) {
#if defined(__SSE2__)
    const size_t head = std::min(bytes, (size_t)(-reinterpret_cast<uintptr_t>(dst) & 15));
    std::memcpy(dst, src, head);
    dst += head;
    src += head;
    bytes -= head;
    for (; bytes >= 64; bytes -= 64, dst += 64, src += 64) {
        const __m128i* from = reinterpret_cast<const __m128i*>(src);
        __m128i* to = reinterpret_cast<__m128i*>(dst);
        const __m128i a = _mm_loadu_si128(from), b = _mm_loadu_si128(from + 1);
        const __m128i c = _mm_loadu_si128(from + 2), d = _mm_loadu_si128(from + 3);
        _mm_stream_si128(to, a);
        _mm_stream_si128(to + 1, b);
        _mm_stream_si128(to + 2, c);
        _mm_stream_si128(to + 3, d);
    }
#endif
    std::memcpy(dst, src, bytes);
}

// Orders the streaming stores of `pack` before the copy that reads them.
void pack_fence() {
#if defined(__SSE2__)
    _mm_sfence();
#endif
}

// The padded side cut into pieces of whole columns or, where a column is
// longer than a piece, of parts of one.
struct Pieces {
    size_t rows, cols, ld_dev, esz;
    size_t cols_per, parts, part;  // columns per piece; pieces and bytes per column
    size_t count;
    Pieces(size_t rows_, size_t cols_, size_t ld_, size_t esz_) : rows(rows_), cols(cols_), ld_dev(ld_), esz(esz_) {
        const size_t column = ld_dev * esz;
        cols_per = std::max<size_t>(1, HostCopier::kPiece / column);
        // At least four pieces, so that packing and the bus overlap.
        cols_per = std::min(cols_per, std::max<size_t>(1, (cols + 3) / 4));
        part = std::clamp(column * cols / 4, HostCopier::kLeast, HostCopier::kPiece);
        parts = (column + part - 1) / part;
        count = parts > 1 ? cols * parts : (cols + cols_per - 1) / cols_per;
    }
    // Piece i: `bytes` of the padded side from `offset` on.
    void at(size_t i, size_t& offset, size_t& bytes) const {
        const size_t column = ld_dev * esz;
        if (parts > 1) {
            const size_t within = i % parts * part;
            offset = i / parts * column + within;
            bytes = std::min(part, column - within);
        } else {
            offset = i * cols_per * column;
            bytes = std::min(cols_per, cols - i * cols_per) * column;
        }
    }
    // The piece's host bytes, column by column: f(host column, byte within
    // it, byte within the piece, host bytes, padding bytes behind them).
    template <class F>
    void each(size_t i, F&& f) const {
        const size_t column = ld_dev * esz, host = rows * esz;
        size_t offset, bytes;
        at(i, offset, bytes);
        for (size_t done = 0; done < bytes;) {
            const size_t col = (offset + done) / column, within = (offset + done) % column;
            const size_t span = std::min(column - within, bytes - done);
            const size_t real = within < host ? std::min(span, host - within) : 0;
            f(col, within, done, real, span - real);
            done += span;
        }
    }
};

}  // namespace

cudaError_t HostCopier::to_device(cudaStream_t stream, char* device, size_t ld_dev, const char* host, size_t ld_host,
                                  size_t rows, size_t cols, size_t esz) {
    const Pieces pieces(rows, cols, ld_dev, esz);
    std::atomic<size_t> next{0};
    std::atomic<int> error{(int)cudaSuccess};
    run((int)std::min<size_t>(pieces.count, kMaxThreads), [&](int t) {
        int b = 0;
        for (size_t i; (i = next.fetch_add(1)) < pieces.count; b ^= 1) {
            Slot& s = slots_[t][b];
            cudaError_t e = cudaEventSynchronize(s.done);  // the slot's last copy
            if (e == cudaSuccess) {
                pieces.each(i, [&](size_t col, size_t within, size_t at, size_t real, size_t pad) {
                    pack(s.p + at, host + col * ld_host * esz + within, real);
                    if (pad) std::memset(s.p + at + real, 0, pad);
                });
                pack_fence();
                size_t offset, bytes;
                pieces.at(i, offset, bytes);
                e = cudaMemcpyAsync(device + offset, s.p, bytes, cudaMemcpyHostToDevice, stream);
                if (e == cudaSuccess) e = cudaEventRecord(s.done, stream);
            }
            if (e != cudaSuccess) {
                error = (int)e;
                return;
            }
        }
    });
    return (cudaError_t)error.load();
}

cudaError_t HostCopier::to_host(cudaStream_t stream, char* host, size_t ld_host, const char* device, size_t ld_dev,
                                size_t rows, size_t cols, size_t esz) {
    // One thread waits for what the copies follow, instead of all of them.
    cudaError_t e0 = cudaStreamSynchronize(stream);
    if (e0 != cudaSuccess) return e0;
    const Pieces pieces(rows, cols, ld_dev, esz);
    std::atomic<size_t> next{0};
    std::atomic<int> error{(int)cudaSuccess};
    run((int)std::min<size_t>(pieces.count, kMaxThreads), [&](int t) {
        // One piece on the bus while the one before it is unpacked.
        size_t waiting[2];
        int queued = 0;  // slots in flight, the older at `head`
        int head = 0;
        cudaError_t e = cudaSuccess;
        for (;;) {
            size_t i = pieces.count;
            if (queued < 2) i = next.fetch_add(1);
            if (i < pieces.count) {
                Slot& s = slots_[t][(head + queued) & 1];
                size_t offset, bytes;
                pieces.at(i, offset, bytes);
                e = cudaMemcpyAsync(s.p, device + offset, bytes, cudaMemcpyDeviceToHost, stream);
                if (e == cudaSuccess) e = cudaEventRecord(s.done, stream);
                if (e != cudaSuccess) break;
                waiting[(head + queued) & 1] = i;
                if (++queued < 2) continue;
            }
            if (queued == 0) break;
            Slot& s = slots_[t][head];
            e = cudaEventSynchronize(s.done);
            if (e != cudaSuccess) break;
            pieces.each(waiting[head], [&](size_t col, size_t within, size_t at, size_t real, size_t) {
                std::memcpy(host + col * ld_host * esz + within, s.p + at, real);
            });
            head ^= 1;
            --queued;
        }
        if (e != cudaSuccess) error = (int)e;
    });
    return (cudaError_t)error.load();
}

}  // namespace tns
