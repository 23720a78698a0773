// Small device-memory helpers shared by the CUDA translation units.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "hdd_common.h"

namespace hdd {
namespace dev {

inline void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw Error(HDD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
T* upload(const std::vector<T>& h, cudaStream_t s, size_t& bytes) {
    if (h.empty()) return nullptr;
    T* p = nullptr;
    cudaError_t e = cudaMalloc(&p, h.size() * sizeof(T));
    if (e != cudaSuccess) throw Error(HDD_ERR_OUT_OF_MEMORY, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    ck(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s), "upload");
    bytes += h.size() * sizeof(T);
    return p;
}

// Zeroed on the caller's stream: a legacy-stream memset would not be ordered
// before work on the solver's non-blocking stream.
template <class T>
T* alloc_zero(size_t n, size_t& bytes, cudaStream_t s) {
    if (n == 0) return nullptr;
    T* p = nullptr;
    cudaError_t e = cudaMalloc(&p, n * sizeof(T));
    if (e != cudaSuccess) throw Error(HDD_ERR_OUT_OF_MEMORY, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    ck(cudaMemsetAsync(p, 0, n * sizeof(T), s), "memset");
    bytes += n * sizeof(T);
    return p;
}

// A device array of `total` floats made of n items, item i at at(i) (ascending;
// it ends where the next begins) and written by pack(i, dst) in parallel.  The
// items go through two pinned staging buffers in turn, each copied to the device
// while the next is packed: the gigabytes of a large solve plan then cross at
// pinned-copy speed and the packing overlaps the copy.  Returns once the
// staging buffers are free again.
template <class At, class Pack>
void upload_packed(size_t n, long long total, At at, Pack pack, cudaStream_t s, float*& d, size_t& bytes) {
    const long long alloc = std::max<long long>(total, 4);
    d = nullptr;
    if (cudaMalloc(&d, (size_t)alloc * sizeof(float)) != cudaSuccess)
        throw Error(HDD_ERR_OUT_OF_MEMORY, "cudaMalloc: supernodal coefficients");
    auto end_of = [&](size_t i) { return i + 1 < n ? (long long)at(i + 1) : total; };
    long long biggest = 4;
    for (size_t i = 0; i < n; ++i) biggest = std::max(biggest, end_of(i) - (long long)at(i));
    // Floats per staging buffer: 32 MB (pinning costs about as much as the
    // copy, so the buffers stay small), or the largest item.
    const long long chunk = std::max<long long>(biggest, 8ll << 20);
    float* stage[2] = {nullptr, nullptr};
    cudaEvent_t copied[2] = {nullptr, nullptr};
    auto cleanup = [&]() {
        for (int i = 0; i < 2; ++i) {
            if (copied[i]) { cudaEventSynchronize(copied[i]); cudaEventDestroy(copied[i]); }
            if (stage[i]) cudaFreeHost(stage[i]);
        }
    };
    try {
        for (int i = 0; i < 2; ++i) {
            ck(cudaMallocHost(&stage[i], (size_t)std::min(chunk, alloc) * sizeof(float)), "pinned staging");
            ck(cudaEventCreateWithFlags(&copied[i], cudaEventDisableTiming), "event");
        }
        size_t g0 = 0;
        int buf = 0;
        bool used[2] = {false, false};
        while (g0 < n) {
            // Items g0 .. g1-1 fill this chunk (at least one item).
            const long long base = at(g0);
            size_t g1 = g0 + 1;
            while (g1 < n && end_of(g1) - base <= chunk) ++g1;
            const long long end = end_of(g1 - 1);
            if (used[buf]) ck(cudaEventSynchronize(copied[buf]), "staging reuse");
            float* st = stage[buf];
#pragma omp parallel for schedule(dynamic)
            for (size_t g = g0; g < g1; ++g) pack(g, st + ((long long)at(g) - base));
            if (end > base)
                ck(cudaMemcpyAsync(d + base, st, (size_t)(end - base) * sizeof(float), cudaMemcpyHostToDevice, s),
                   "coefficient upload");
            ck(cudaEventRecord(copied[buf], s), "event");
            used[buf] = true;
            buf ^= 1;
            g0 = g1;
        }
        if (total < alloc)  // an empty plan's placeholder
            ck(cudaMemsetAsync(d + total, 0, (size_t)(alloc - total) * sizeof(float), s), "memset");
    } catch (...) {
        cleanup();
        throw;
    }
    cleanup();
    bytes += (size_t)alloc * sizeof(float);
}

template <class T>
void release(T*& p) {
    if (p) cudaFree(p);
    p = nullptr;
}

}  // namespace dev
}  // namespace hdd
