// Allocation-free variant of the score-step label selection (per-label quantile, first label,
// candidate flags) for callers that must not allocate device memory.
//
// Who needs it: code that runs while another runtime owns the device memory (a serving process
// whose framework allocates everything from its own pool and budget), code that is being recorded
// into a CUDA graph, or latency-bound code where a cudaMalloc/cudaFree would synchronise the device
// and stall every other stream.  Such callers pass device buffers they already own for the inputs
// and outputs; this entry point itself calls no cudaMalloc, cudaFree or allocating library routine.
//
// The only temporary space the selection needs is a sort buffer for score lists that hold NaN
// (constant rows).  It lives in one file-scope device array of kNoallocScratchFloats floats
// (1,048,576 floats, 4 MiB) that every GPU loading this library holds until the process exits.  Host code cannot pass
// the array's name to a kernel (in host code it is only a stand-in, not a device address), so the
// first call on each device looks its address up with cudaGetSymbolAddress, with that device
// current, and caches it.

#include <algorithm>
#include <mutex>

#include "device_util.cuh"
#include "kernels.cuh"
#include "sgr_internal.h"

namespace sgr {
namespace {

constexpr int kNoallocScratchFloats = 1 << 20;
constexpr int kMaxDevices = 64;

static __device__ __align__(256) float g_noalloc_scratch[kNoallocScratchFloats];

struct LabelTable {
    LabelQ q[256];
    uint8_t order[256];  // longest label first
};

constexpr int ITEMS_NW = 8;                   // warps of a CTA of the item kernel
constexpr uint32_t kSortMark = 0x7fa5a5a5u;  // a NaN that no arithmetic gives: a list to be sorted

// One warp per (label, score row), label by label, longest first (as the score step's select_items_kernel, with
// the extremes in a pass of their own): every list without NaN.  The fixed scratch is not used, so the grid is
// sized to the GPU.  A list that the reference would sort with NaN in it is marked.  8,000 rows x 20,000 scores in
// 30 labels: 1.56 ms with the scratch-bound grid of select_noalloc_kernel alone (65 CTAs of 8 warps), 0.50 with a
// warp per row, 0.46 so (uneven labels); 300 rows: 160 us with the CTAs, 40 so.
__global__ void __launch_bounds__(ITEMS_NW * 32, 5) select_noalloc_items_kernel(const float* scores, int64_t ld, int nq,
                                                                               int L,
                                                                               const __grid_constant__ LabelTable lt,
                                                                               float p, float* label_scores) {
    __shared__ __align__(16) int hist[ITEMS_NW][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gw = blockIdx.x * ITEMS_NW + warp, n_warps = gridDim.x * ITEMS_NW;
    int i = gw / nq, q = gw % nq;
    while (i < L) {
        const int l = lt.order[i];
        const LabelQ d = lt.q[l];
        const float* v = scores + (size_t)q * ld + d.start;
        float r = v[0] == v[0] ? v[0] : __int_as_float(0x7fffffff);
        if (d.kind != 0) {
            bool nan = false, num = false;
            uint32_t kmin = 0xffffffffu, kmax = 0u;
            int t = lane;
            for (; t + 96 < d.len; t += 128) {  // four independent loads in flight per lane
                const float x0 = v[t], x1 = v[t + 32], x2 = v[t + 64], x3 = v[t + 96];
                nan |= (x0 != x0) | (x1 != x1) | (x2 != x2) | (x3 != x3);
                num |= (x0 == x0) | (x1 == x1) | (x2 == x2) | (x3 == x3);
                const uint32_t u0 = ord_key(x0), u1 = ord_key(x1), u2 = ord_key(x2), u3 = ord_key(x3);
                kmin = min(min(kmin, min(u0, u1)), min(u2, u3));
                kmax = max(max(kmax, max(u0, u1)), max(u2, u3));
            }
            for (; t < d.len; t += 32) {
                const float x = v[t];
                nan |= x != x;
                num |= x == x;
                kmin = min(kmin, ord_key(x));
                kmax = max(kmax, ord_key(x));
            }
            nan = __any_sync(FULL, nan);
            num = __any_sync(FULL, num);
            kmin = __reduce_min_sync(FULL, kmin);
            kmax = __reduce_max_sync(FULL, kmax);
            if (nan) r = __uint_as_float(num ? kSortMark : 0x7fffffffu);  // (all NaN: NaN at every grid position)
            else r = quantile_warp_core(v, d, p, hist[warp], nullptr, lane, nullptr, kmin, kmax, false);
        }
        if (lane == 0) label_scores[(size_t)q * L + l] = r;
        __syncwarp();
        for (q += n_warps; q >= nq; q -= nq) ++i;
    }
}

// Per row, one warp: first label and flags; a row with a marked list is left to select_noalloc_kernel (first = -1).
__global__ void __launch_bounds__(256) noalloc_first_kernel(const float* label_scores, int nq, int L, float thre,
                                                            int32_t* first, uint8_t* flags) {
    __shared__ float ls_all[8][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = blockIdx.x * 8 + warp;
    if (q >= nq) return;
    float* ls = ls_all[warp];
    bool sort = false;
    for (int l = lane; l < L; l += 32) {
        ls[l] = label_scores[(size_t)q * L + l];
        sort |= __float_as_uint(ls[l]) == kSortMark;
    }
    if (__any_sync(FULL, sort)) {
        if (lane == 0) first[q] = -1;
        return;
    }
    __syncwarp();
    int mn = 0, mx = 0;
    if (lane == 0) {
        stl::minmax(ls, L, &mn, &mx);
        first[q] = mx;
    }
    mx = __shfl_sync(FULL, mx, 0);
    if (!flags) return;
    const float t = __fsub_rn(ls[mx], thre);
    for (int l = lane; l < L; l += 32) flags[(size_t)q * L + l] = ls[l] >= t ? 1 : 0;
}

// A CTA per row, with the fixed scratch.  marked: only the rows that noalloc_first_kernel left.
__global__ void __launch_bounds__(256) select_noalloc_kernel(const float* scores, int64_t ld, int nq, int L,
                                                             const __grid_constant__ LabelTable lt, float p,
                                                             float thre, float* label_scores, int32_t* first,
                                                             uint8_t* flags, float* scratch, int spw, bool marked) {
    __shared__ float ls[256];
    __shared__ __align__(16) int hist[8][256];
    __shared__ int s_mx;
    // Status bits of the selection are not reported by this entry point: it only enqueues work and
    // has no context to return them through.  Bit 8 (no sort scratch) cannot arise, the scratch is
    // always present; bit 4 (a NaN-bearing list on which libstdc++ would read outside the array,
    // sorted within bounds instead) is not reported by the main path either.
    __shared__ int ignored_status;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) ignored_status = 0;
    __syncthreads();
    float* my_scratch = scratch + (size_t)(blockIdx.x * 8 + warp) * spw;
    for (int q = blockIdx.x; q < nq; q += gridDim.x) {
        if (marked && first[q] != -1) continue;  // the same for every thread: written by the launch before
        const float* row = scores + (size_t)q * ld;
        for (int l = warp; l < L; l += 8) {
            const LabelQ d = lt.q[l];
            // a constant query row makes every score NaN: the quantile of an all-NaN list is NaN for
            // every grid position, so such lists skip the sort (checked only when the first score is NaN)
            bool all_nan = false;
            if (row[d.start] != row[d.start]) {
                bool any = false;
                for (int i = lane; i < d.len; i += 32) any |= row[d.start + i] == row[d.start + i];
                all_nan = !__any_sync(0xffffffffu, any);
            }
            const float r = all_nan ? __int_as_float(0x7fffffff)
                                    : quantile_warp(row + d.start, d, p, hist[warp], my_scratch, lane, &ignored_status);
            if (lane == 0) ls[l] = r;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int mn, mx;
            stl::minmax(ls, L, &mn, &mx);
            s_mx = mx;
            first[q] = mx;
        }
        __syncthreads();
        const float t = __fsub_rn(ls[s_mx], thre);
        for (int l = threadIdx.x; l < L; l += blockDim.x) {
            label_scores[(size_t)q * L + l] = ls[l];
            if (flags) flags[(size_t)q * L + l] = ls[l] >= t ? 1 : 0;
        }
        __syncthreads();
    }
}

std::mutex g_mu;
float* g_scratch_ptr[kMaxDevices] = {};

// Device address of the scratch array on the current device (looked up once per device).
float* scratch_address(int dev) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch_ptr[dev]) {
        float* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            fail(SGR_ERR_CUDA, std::string("cudaGetSymbolAddress of the selection scratch: ") + cudaGetErrorString(e));
        }
        g_scratch_ptr[dev] = p;
    }
    return g_scratch_ptr[dev];
}

}  // namespace

}  // namespace sgr

extern "C" sgr_status sgr_select_labels_noalloc(const float* d_scores, int64_t ld, uint32_t n_rows,
                                                const uint32_t* label_ranges, uint32_t n_labels, float quantile,
                                                float finetune_thre, float* d_label_scores,
                                                int32_t* d_first_labels, uint8_t* d_flags, void* stream) {
    using namespace sgr;
    if (n_rows == 0) return SGR_OK;
    if (!d_scores || !label_ranges || !d_label_scores || !d_first_labels) return SGR_ERR_INVALID_ARGUMENT;
    if (n_labels == 0 || n_labels > 256) return SGR_ERR_UNSUPPORTED;
    LabelTable lt{};
    uint32_t max_len = 1;
    uint64_t total = 0;
    for (uint32_t l = 0; l < n_labels; ++l) {
        const uint32_t start = label_ranges[2 * l], len = label_ranges[2 * l + 1];
        if (len == 0) return SGR_ERR_EMPTY_LABEL;
        if ((uint64_t)start + len > (uint64_t)ld) return SGR_ERR_INVALID_ARGUMENT;
        max_len = std::max(max_len, len);
        total += len;
        // the reference's float index grid (src/cusingler.cu:947-978 of STOmics/cusingler)
        lt.q[l] = make_lq((int)start, (int)len, quantile);
    }
    // eight warps per block, each with its own max_len-float slice of the fixed scratch array
    const long fit_blocks = (long)kNoallocScratchFloats / (8L * max_len);
    if (fit_blocks < 1) return SGR_ERR_UNSUPPORTED;  // a label with more than 131072 reference cells
    try {
        int dev = 0;
        SGR_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= kMaxDevices) return SGR_ERR_UNSUPPORTED;
        float* scratch = scratch_address(dev);
        const unsigned blocks =
            (unsigned)std::min<long>({(long)n_rows, fit_blocks, (long)device_sm_count() * 2});
        // A CTA takes its row's labels eight at a time, and the scratch allows `blocks` of them.  More rows than
        // that are spread better as items on all SMs, unless they are so short that the CTAs' few turns cost less
        // than the two launches more (us, CTAs / items: 12.4 / 16.6 for 300 x 1,000 scores in 5 labels, 28.5 / 16.6
        // for 1,000 x 1,000; 22.7 / 18.6 for 300 x 3,000 in 20; 97.9 / 30.5 for 100 x 20,000 in 30, 24.9 / 28.9 for 30
        // of them, which fit one turn).
        const bool by_item = n_rows > blocks && (n_rows * (double)total > 5e5 || n_rows > 8L * blocks);
        if (by_item) {
            for (uint32_t l = 0; l < n_labels; ++l) lt.order[l] = (uint8_t)l;
            std::sort(lt.order, lt.order + n_labels,
                      [&](uint8_t x, uint8_t y) { return lt.q[x].len != lt.q[y].len ? lt.q[x].len > lt.q[y].len : x < y; });
            const unsigned item_blocks = (unsigned)std::min<long>(
                ((long)n_rows * n_labels + ITEMS_NW - 1) / ITEMS_NW, (long)device_sm_count() * 5);
            select_noalloc_items_kernel<<<item_blocks, ITEMS_NW * 32, 0, (cudaStream_t)stream>>>(
                d_scores, ld, (int)n_rows, (int)n_labels, lt, quantile, d_label_scores);
            SGR_CUDA(cudaGetLastError());
            count_launch();
            noalloc_first_kernel<<<(n_rows + 7) / 8, 256, 0, (cudaStream_t)stream>>>(
                d_label_scores, (int)n_rows, (int)n_labels, finetune_thre, d_first_labels, d_flags);
            SGR_CUDA(cudaGetLastError());
            count_launch();
        }
        select_noalloc_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(
            d_scores, ld, (int)n_rows, (int)n_labels, lt, quantile, finetune_thre, d_label_scores, d_first_labels,
            d_flags, scratch, (int)max_len, by_item);
        SGR_CUDA(cudaGetLastError());
        count_launch();
    } catch (const Error& e) {
        return e.code;
    }
    return SGR_OK;
}
