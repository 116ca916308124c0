// The staged host copies against a runtime that copies in place: what happens
// when the host refuses memory while a copier is made, and that every byte
// arrives whatever number of helper threads there are.

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "host_copy.cu"

// The runtime calls that host_copy.cu makes.
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
}

// The allocation that fails, counted down; negative: none.
static std::atomic<int> g_fail{-1};
void* operator new(size_t bytes) {
    if (g_fail.load() >= 0 && g_fail.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void* p = std::malloc(bytes ? bytes : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main() {
    const size_t rows = 1000, cols = 301, ld = 1024, esz = 8;
    std::vector<char> host(rows * cols * esz), device(ld * cols * esz, 1), back(rows * cols * esz);
    for (size_t i = 0; i < host.size(); ++i) host[i] = (char)(i * 31 + i / 977);
    for (int k = -1; k < 40; ++k) {
        g_fail = k;
        tns::HostCopier copier(0);
        g_fail = -1;
        if (!copier.usable()) continue;
        if (copier.to_device(nullptr, device.data(), ld, host.data(), rows, rows, cols, esz) != cudaSuccess) return 1;
        for (size_t c = 0; c < cols; ++c) {
            if (std::memcmp(&device[c * ld * esz], &host[c * rows * esz], rows * esz)) return 2;
            for (size_t b = rows * esz; b < ld * esz; ++b)
                if (device[c * ld * esz + b]) return 3;
        }
        std::memset(back.data(), 0, back.size());
        if (copier.to_host(nullptr, back.data(), rows, device.data(), ld, rows, cols, esz) != cudaSuccess) return 4;
        if (back != host) return 5;
    }
    std::puts("ok");
    return 0;
}
