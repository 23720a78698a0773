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

// Two pinned buffers through which a setup's plans go to the device in turn.
// Pinning and unpinning a pair for every plan was most of a small domain's
// set-up (sparse 128^3, sub 32: 375 ms so, 152 ms with one pair), so one pair
// serves all plans of a setup and grows as they need it.
class Staging {
public:
    Staging() = default;
    Staging(const Staging&) = delete;
    Staging& operator=(const Staging&) = delete;
    ~Staging() {
        free_buffers();
        for (cudaEvent_t e : copied_)
            if (e) cudaEventDestroy(e);
    }
    void reserve(size_t floats) {
        for (cudaEvent_t& e : copied_)
            if (!e) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
        if (floats <= size_) return;
        free_buffers();
        for (float*& b : buf_) ck(cudaMallocHost(&b, floats * sizeof(float)), "pinned staging");
        size_ = floats;
    }
    size_t size() const { return size_; }
    // The next buffer, once its last copy has been made.
    float* next() {
        at_ ^= 1;
        ck(cudaEventSynchronize(copied_[at_]), "staging reuse");
        return buf_[at_];
    }
    // Copies the buffer next() gave.
    void copy(float* dst, size_t floats, cudaStream_t s) {
        if (floats > 0)
            ck(cudaMemcpyAsync(dst, buf_[at_], floats * sizeof(float), cudaMemcpyHostToDevice, s), "coefficient upload");
        ck(cudaEventRecord(copied_[at_], s), "event");
    }

private:
    void free_buffers() {
        for (cudaEvent_t e : copied_)
            if (e) cudaEventSynchronize(e);
        for (float*& b : buf_) {
            if (b) cudaFreeHost(b);
            b = nullptr;
        }
        size_ = 0;
    }
    float* buf_[2] = {nullptr, nullptr};
    cudaEvent_t copied_[2] = {nullptr, nullptr};
    size_t size_ = 0;
    int at_ = 0;
};

// A device array of `total` floats made of n items, item i at at(i) (ascending;
// it ends where the next begins) and written by pack(i, dst) in parallel: one
// staging buffer is copied while the next is packed.
template <class At, class Pack>
void upload_packed(size_t n, long long total, At at, Pack pack, Staging& stage, cudaStream_t s, float*& d, size_t& bytes) {
    const long long alloc = std::max<long long>(total, 4);
    d = nullptr;
    if (cudaMalloc(&d, (size_t)alloc * sizeof(float)) != cudaSuccess)
        throw Error(HDD_ERR_OUT_OF_MEMORY, "cudaMalloc: supernodal coefficients");
    try {
        auto end_of = [&](size_t i) { return i + 1 < n ? (long long)at(i + 1) : total; };
        long long biggest = 4;
        for (size_t i = 0; i < n; ++i) biggest = std::max(biggest, end_of(i) - (long long)at(i));
        // Floats per chunk: 16 MB, or the largest item.
        const long long chunk = std::max<long long>(biggest, 4ll << 20);
        stage.reserve((size_t)std::min(chunk, alloc));
        for (size_t g0 = 0, g1; g0 < n; g0 = g1) {
            // Items g0 .. g1-1 fill this chunk (at least one item).
            const long long base = at(g0);
            for (g1 = g0 + 1; g1 < n && end_of(g1) - base <= chunk; ++g1) {}
            float* st = stage.next();
#pragma omp parallel for schedule(dynamic)
            for (size_t g = g0; g < g1; ++g) pack(g, st + ((long long)at(g) - base));
            stage.copy(d + base, (size_t)(end_of(g1 - 1) - base), s);
        }
        if (total < alloc)  // an empty plan's placeholder
            ck(cudaMemsetAsync(d + total, 0, (size_t)(alloc - total) * sizeof(float), s), "memset");
    } catch (...) {
        cudaStreamSynchronize(s);
        cudaFree(d);
        d = nullptr;
        throw;
    }
    bytes += (size_t)alloc * sizeof(float);
}

template <class T>
void release(T*& p) {
    if (p) cudaFree(p);
    p = nullptr;
}

}  // namespace dev
}  // namespace hdd
