// Internal declarations shared by the host and device sources of libsgr.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/sgr.h"

namespace sgr {

struct Error : std::runtime_error {
    sgr_status code;
    Error(sgr_status c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] inline void fail(sgr_status c, const std::string& m) { throw Error(c, m); }

#define SGR_CUDA(call)                                                                                   \
    do {                                                                                                 \
        cudaError_t e_ = (call);                                                                         \
        if (e_ != cudaSuccess) {                                                                         \
            if (e_ == cudaErrorMemoryAllocation) {                                                       \
                cudaGetLastError();                                                                      \
                ::sgr::fail(SGR_ERR_OUT_OF_MEMORY, std::string(#call) + ": " + cudaGetErrorString(e_));  \
            }                                                                                            \
            ::sgr::fail(SGR_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_) + " (" +        \
                                          __FILE__ + ":" + std::to_string(__LINE__) + ")");              \
        }                                                                                                \
    } while (0)

#define SGR_LAUNCH_CHECK() SGR_CUDA(cudaGetLastError())

// Lets a kernel take up to `most` bytes of dynamic shared memory.  The limit is the kernel's, not the
// launch's: `most` is the largest size that any launch asks for, so that contexts in several threads do not
// lower it under one another's launches.
template <class K>
inline void allow_smem(K kern, size_t most) {
    SGR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
}

// The same for kernels whose launches take what the trained reference needs: all that a CTA can have next to the
// kernel's own shared arrays.
template <class K>
inline void allow_most_smem(K kern) {
    constexpr size_t kBlock = 227 * 1024;
    cudaFuncAttributes at;
    SGR_CUDA(cudaFuncGetAttributes(&at, kern));
    allow_smem(kern, kBlock - at.sharedSizeBytes);
}

// Device memory of one context in slabs: buffers up to 16 MiB are carved from 64 MiB slabs instead of a
// cudaMalloc and a cudaFree each (0.33 ms a call here, about 100 buffers per context: 10 of 22 ms of a whole
// drop-in run on 1,900 x 800 cells).  A context's arena is used by the thread that is in a call on the
// context.  A released block is handed out again only after settle(), which the context calls when its
// streams have finished, so no queued work can still use it; the slabs are freed with the context.  Where less
// than kSpare of the device's memory is free, a slab's unused part would be missed, and buffers are cudaMalloc'ed
// at their own size.
class DevArena {
public:
    static constexpr size_t kSlab = (size_t)64 << 20, kLargest = (size_t)16 << 20, kSpare = (size_t)1 << 30;
    DevArena() = default;
    DevArena(const DevArena&) = delete;
    DevArena& operator=(const DevArena&) = delete;
    ~DevArena() {
        for (char* s : slabs_) cudaFree(s);
    }
    // bytes is rounded up to what the block holds; null (bytes as given) where memory is short
    void* alloc(size_t& bytes) {
        const int c = size_class(bytes);
        if (!free_[c].empty()) {
            char* p = free_[c].back();
            free_[c].pop_back();
            bytes = class_bytes(c);
            return p;
        }
        const size_t n = class_bytes(c);
        if (slabs_.empty() || used_ + n > kSlab) {
            size_t left = 0, total = 0;
            SGR_CUDA(cudaMemGetInfo(&left, &total));
            if (left < kSpare) return nullptr;
            char* s = nullptr;
            SGR_CUDA(cudaMalloc(reinterpret_cast<void**>(&s), kSlab));
            slabs_.push_back(s);
            used_ = 0;
        }
        char* p = slabs_.back() + used_;
        used_ += n;
        bytes = n;
        return p;
    }
    void release(void* p, size_t bytes) { pending_.push_back({size_class(bytes), static_cast<char*>(p)}); }
    void settle() {
        for (auto& b : pending_) free_[b.first].push_back(b.second);
        pending_.clear();
    }
    // The arena of the call that this thread is in (nullptr: none, buffers are cudaMalloc'ed).
    static DevArena*& current() {
        static thread_local DevArena* a = nullptr;
        return a;
    }

private:
    static constexpr int kClasses = 66;
    // sizes 256 x {4, 5, 6, 7} / 4 x 2^k: multiples of 256 from 1 KiB on
    static size_t class_bytes(int c) { return ((size_t)(4 + (c & 3)) << (c >> 2)) * 256; }
    static int size_class(size_t bytes) {
        int c = 0;
        while (class_bytes(c) < bytes) ++c;
        return c;
    }
    std::vector<char*> slabs_;
    size_t used_ = 0;
    std::vector<char*> free_[kClasses];
    std::vector<std::pair<int, char*>> pending_;
};

// Owning device buffer (from the calling context's arena, or cudaMalloc'ed; grows, never shrinks unless
// freed).
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevArena* home = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), home(o.home) { o.p = nullptr; o.n = 0; o.home = nullptr; }
    ~DevBuf() { release(); }
    void release() {
        if (p && home) home->release(p, n * sizeof(T));  // n elements fill the block's size class
        else if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        home = nullptr;
    }
    T* ensure(size_t count) {
        if (count > n) {
            release();
            size_t bytes = count * sizeof(T);
            DevArena* a = DevArena::current();
            if (a && bytes <= DevArena::kLargest) p = static_cast<T*>(a->alloc(bytes));
            if (p) home = a;
            else SGR_CUDA(cudaMalloc(reinterpret_cast<void**>(&p), bytes));
            n = bytes / sizeof(T);
        }
        return p;
    }
    void upload(const T* h, size_t count, cudaStream_t s) {
        ensure(count);
        if (count) SGR_CUDA(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    void upload(const std::vector<T>& h, cudaStream_t s) { upload(h.data(), h.size(), s); }
};

// ---- host marker training (train.cpp) ---------------------------------------------------------

struct HostCsr {
    uint32_t n_rows = 0, n_cols = 0;
    const float* data = nullptr;
    const int32_t* indices = nullptr;
    const int32_t* indptr = nullptr;
};

struct Markers {
    uint32_t n_labels = 0;
    uint32_t W = 0;                    // gene space = reference column count as given
    bool filter_genes = false;
    std::vector<int32_t> ref_colmap;   // reference column -> gene id (identity or intersection rank)
    std::vector<int32_t> qry_colmap;   // query column -> gene id, -1 when dropped
    std::vector<uint32_t> ref_order;   // regrouped row -> original reference row
    std::vector<uint32_t> ctidx;       // (start, len) per label in the regrouped reference
    std::vector<uint32_t> common;      // score-step marker genes, ascending
    std::vector<uint32_t> thre;        // fine-tune gene pool, ascending
    std::vector<uint32_t> pair_genes;  // positive-difference genes per ordered pair, concatenated
    std::vector<uint32_t> pair_idx;    // (start, len) per ordered pair, diagonal (0, 0)
    std::vector<uint32_t> ft_genes;    // pair lists restricted to thre, as thre-compact ids
    std::vector<uint32_t> ft_idx;      // (start, len) per ordered pair
};

// Gene-name intersection, label regrouping and marker training on the host (see train.cpp):
// prepare_markers (intersection, regrouping: colmaps, ref_order, ctidx) then rank_markers_host
// (medians, per-pair lists, gene sets).
void train_markers(const HostCsr& ref, const int32_t* celltypes, uint32_t n_labels,
                   const char* const* ref_genes, const char* const* qry_genes, uint32_t n_qry_genes,
                   int cores, Markers& out);
void prepare_markers(const HostCsr& ref, const int32_t* celltypes, uint32_t n_labels,
                     const char* const* ref_genes, const char* const* qry_genes, uint32_t n_qry_genes, Markers& m);
void rank_markers_host(const HostCsr& ref, int cores, Markers& m);
// From pair_genes / pair_idx and the score-step and fine-tune gene flags (W each): the gene sets
// common and thre and the fine-tune pair lists.
void finish_markers(Markers& m, const uint8_t* in_common, const uint8_t* in_thre);
// The medians and per-pair lists on the device (train_gpu.cu) from the label-grouped reference CSR
// in device memory (rows in m.ref_order order, original columns); fills pair_genes, pair_idx and,
// through finish_markers, the gene sets.
void rank_markers_device(const float* data, const int32_t* indices, const int32_t* indptr, uint32_t R,
                         uint32_t ref_cols, int64_t nnz, Markers& m, cudaStream_t s);

// Reference's marker-count formula round(500 * (2/3)^log2(n)) (src/io.cpp:209,
// src/cusingler.cu:1142).
int marker_count(size_t n_labels);

}  // namespace sgr
