// Exact fine-tune by rounds over all cells: the row scan batched by (label, four cells).
//
// Restates the reference's per-cell fine-tune loop (src/cusingler.cu:1138-1333 of
// STOmics/cusingler: finetune_round + cufinetune).  The identity behind the scan is the one stated in
// finetune.cu: with e = d + k (k = stored entries of a row inside the round's gene set S), one pass
// over a reference row's value-sorted entries gives the exact numerator and norm over S.  Here a
// round of every active cell is three launches:
//   ft_step_kernel  per cell: the labels' quantiles of the round before, the keep / drop rule, then
//                   the next round's gene set and the query's e-values;
//   ft_plan_kernel  per quad of four active cells: the labels that at least two of them need, and the
//                   others' entries on the work list of each label;
//   ft_scan_kernel  per quad, then per four cells of a work list: the correlations of the labels' rows.
// The cells of a round are put in an order in which neighbours have nearly the same candidates, so that a
// quad's cells share most labels and one table of e-values serves hundreds of row blocks.
//
// What bounds the scan is one shared-memory lookup per (row entry, cell) and the integer work around
// it.  Four cells share a pass because the entry's load, its address and its run end are then paid
// once, and one 16-byte lookup serves the four.  The table holds each gene's four packed words
// (1 << shift) + e (0 outside S) in C = 8 copies of 16 bytes: a quarter-warp's eight lanes read eight
// different bank groups whatever genes they look up, so no lookup conflicts (a gene pool too wide for
// eight copies takes fewer, and its lookups conflict).  Entries are 16-bit gene ids in groups of four
// padded at run ends (entry 0 of a group ending a run has bit 15 set), so the run's bookkeeping is
// done once per group, with the same instructions for every lane.
//
// Packed sums: P is the running sum of the packed words (count in the high bits, e-sum below bit
// `shift`; the host picks the shift so that neither field of a whole row overflows).  At a run end,
// acc = P - (P at the run end before) holds the run's count b and e-sum s.  With z = 2 a + b (a: kept
// entries before the run), X = sum z s is accumulated as sum z acc modulo 2^32: the count fields add
// (sum z b) << shift = k_r^2 << shift, which is taken off at the end.
//
// Measured (B200, 20,000 reference cells in 30 labels, 100,000 queries of which 48,412 take 117,724 rounds,
// 1.3e9 row correlations of 304 entries): fine-tune 319 -> 98 ms against the per-cell kernels of
// finetune.cu, of it the scan 89 ms (68 ps a correlation; shared-memory pipe 77 % busy, issue 69 %).
// Scanning per label instead of per quad left a third of the warps waiting at the table's barriers
// (82 ps); 12, 24 and 32 warps per CTA were 2 % slower, no different and 9 % slower than 16.

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kernels.cuh"
#include "sgr_internal.h"
#include "stl_order.h"
#include "device_util.cuh"

namespace sgr {
namespace {

constexpr int STEP_NW = 8;             // warps of a step CTA, and of one where a round has few cells
constexpr int STEP_NW_FEW = 32;
constexpr int STEP_CTAS = 8;           // step CTAs per SM
constexpr int SCAN_NW = 16;            // warps of a scan CTA (one CTA per SM: the table fills it)
constexpr uint32_t NAN_KEY = 0xffffffffu;  // extreme of a list with a NaN: above every number's key

// ---- at training: the reference rows in groups --------------------------------------------------

// One warp per reference row: its entries sorted by (value, gene) as gene | run end << 15 at the row's
// CSR positions, and the row's groups (runs padded to multiples of four).  Rows are at most `cap` long.
__global__ void __launch_bounds__(256) row_runs_kernel(const float* data, const int32_t* idx, const int32_t* ptr,
                                                       uint32_t n_rows, int cap, uint16_t* sorted, int32_t* n_groups) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem) + (size_t)warp * cap;
    for (uint32_t row = blockIdx.x * wpb + warp; row < n_rows; row += gridDim.x * wpb) {
        const int beg = ptr[row], k = ptr[row + 1] - beg;
        int n = 1;
        while (n < k) n <<= 1;
        for (int i = lane; i < n; i += 32)
            keys[i] = i < k ? ((uint64_t)ord_key(canon_zero(data[beg + i])) << 32) | (uint32_t)idx[beg + i] : ~0ull;
        __syncwarp();
        if (k > 1) warp_bitonic(keys, n, lane);
        int groups = 0;
        for (int j = lane; j < k; j += 32) {
            const uint64_t key = keys[j];
            const bool last = j + 1 == k || (uint32_t)(keys[j + 1] >> 32) != (uint32_t)(key >> 32);
            sorted[beg + j] = (uint16_t)((uint32_t)key | (last ? 0x8000u : 0u));
            if (last) groups += (j + 1 - lower_hi(keys, k, (uint32_t)(key >> 32)) + 3) / 4;
        }
        groups = __reduce_add_sync(FULL, groups);
        if (lane == 0) n_groups[row] = groups;
        __syncwarp();
    }
}

// One thread per row slot (a row of a 32-row block): writes the row's groups.  Vector v of the block's
// lane t (two groups, 16 bytes) is groups[blk_voff + 32 v + t].  slot_row: the slot's reference row, or
// -1 for a slot past the label's last row.
__global__ void row_groups_kernel(const uint16_t* sorted, const int32_t* ptr, const int32_t* slot_row,
                                  const int32_t* blk_voff, uint32_t n_slots, uint32_t pad, uint4* groups) {
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n_slots) return;
    const int blk = slot >> 5, lane = slot & 31, row = slot_row[slot];
    const int nv = (blk_voff[blk + 1] - blk_voff[blk]) / 32;
    uint16_t* out = reinterpret_cast<uint16_t*>(groups + blk_voff[blk] + lane);
    int j = row >= 0 ? ptr[row] : 0;
    const int end = row >= 0 ? ptr[row + 1] : 0;
    for (int g = 0; g < 2 * nv; ++g) {
        uint32_t e[4] = {pad, pad, pad, pad};
        for (int u = 0; u < 4; ++u) {
            if (j >= end) break;
            const uint32_t s = sorted[j++];
            e[u] = s & 0x7fffu;
            if (s & 0x8000u) {
                e[0] |= 0x8000u;
                break;
            }
        }
        uint16_t* o = out + (size_t)(g >> 1) * 32 * 8 + (g & 1) * 4;
        for (int u = 0; u < 4; ++u) o[u] = (uint16_t)e[u];
    }
}

// Bits of each ordered pair's whole fine-tune list over the gene pool.  One warp per pair.
__global__ void pair_mask_kernel(const uint32_t* ft_genes, const uint32_t* ft_idx, int n_pairs, int nwords,
                                 uint32_t* mask) {
    const int lane = threadIdx.x & 31;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n_pairs; p += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t pos = ft_idx[2 * p], len = ft_idx[2 * p + 1];
        for (uint32_t i = lane; i < len; i += 32) {
            const uint32_t g = ft_genes[pos + i];
            atomicOr(mask + (size_t)p * nwords + (g >> 5), 1u << (g & 31));
        }
    }
}

// The same for the first gene_thre(n) genes of the lists that n candidates cut, n = 2 .. L: row (n - 2) *
// n_pairs + pair.  One warp per pair; gene_thre falls with n.  dynamic shared memory: nwords per warp.
__global__ void cut_mask_kernel(const uint32_t* ft_genes, const uint32_t* ft_idx, int n_pairs, int L, int nwords,
                                const int32_t* gene_thre, uint32_t* mask) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    uint32_t* m = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * nwords;
    for (int p = blockIdx.x * wpb + warp; p < n_pairs; p += gridDim.x * wpb) {
        const uint32_t pos = ft_idx[2 * p];
        const int len = (int)ft_idx[2 * p + 1];
        for (int w = lane; w < nwords; w += 32) m[w] = 0u;
        __syncwarp();
        int done = 0;
        for (int n = L; n >= 2; --n) {
            const int t = gene_thre[n];
            if (t >= len) break;  // not cut, nor by fewer candidates
            for (int i = done + lane; i < t; i += 32) {
                const uint32_t g = ft_genes[pos + i];
                atomicOr(&m[g >> 5], 1u << (g & 31));
            }
            done = max(done, t);
            __syncwarp();
            uint32_t* out = mask + ((size_t)(n - 2) * n_pairs + p) * nwords;
            for (int w = lane; w < nwords; w += 32) out[w] = m[w];
            __syncwarp();
        }
    }
}

// ---- per call: the cells to fine-tune ----------------------------------------------------------

// Cells with fewer than two candidates are decided here; the others are appended to `cells` with the
// first 32-row block of their scores (blk_off).  counter: cells in bits 36..,
// blocks below; cand: candidates of the appended cells, summed.
__global__ void __launch_bounds__(256) ft_cells_kernel(int n, const int32_t* list, const int* n_dev, int L,
                                                       const uint8_t* flags, const uint32_t* ctidx, int32_t* cells, int64_t* blk_off,
                                                       int32_t* final_labels, int32_t* rounds,
                                                       unsigned long long* counter, unsigned long long* cand) {
    __shared__ unsigned long long w_tot[8];
    __shared__ unsigned long long s_base;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n_dev) n = *n_dev;
    int c = 0, only = 0, q = 0;
    unsigned long long mine = 0;
    if (i < n) {
        q = list ? list[i] : i;
        const uint8_t* f = flags + (int64_t)q * L;
        unsigned long long blocks = 0;
        for (int l = 0; l < L; ++l)
            if (f[l]) {
                if (c == 0) only = l;
                ++c;
                blocks += (ctidx[2 * l + 1] + 31) / 32;
            }
        if (c >= 2) mine = (1ull << 36) | blocks;
        else {
            final_labels[q] = c ? only : 0;
            rounds[q] = 0;
        }
    }
    unsigned long long x = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) w_tot[warp] = x;
    const int csum = __reduce_add_sync(FULL, c >= 2 ? c : 0);
    if (lane == 0 && csum) atomicAdd(cand, (unsigned long long)csum);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < 8; ++w) {
            const unsigned long long v = w_tot[w];
            w_tot[w] = t;
            t += v;
        }
        s_base = t ? atomicAdd(counter, t) : 0ull;
    }
    __syncthreads();
    if (mine) {
        const unsigned long long at = s_base + w_tot[warp] + x - mine;
        cells[at >> 36] = q;
        blk_off[at >> 36] = (int64_t)(at & ((1ull << 36) - 1));
    }
}

// The FP32 order refuses a NaN that it ranks.  Which entries it ranks is known per round only, so the sorted
// rows carry the mark: bit 15 of the gene (pools are narrower than 2^15).
constexpr uint32_t NAN_GENE = 0x8000u, GENE = 0x7fffu;

__device__ __forceinline__ bool key_is_nan(uint32_t u) {
    return u > 0xff800000u || u < 0x007fffffu;  // beyond ord_key of the infinities
}

// One warp per row: its pool entries by value (NaN marked), with each entry's run as positions [lo, hi).
// any_nan: set where a row holds a NaN.
__global__ void __launch_bounds__(256) ft_sort_rows_kernel(int n, const float* data, const int32_t* idx,
                                                           const int32_t* ptr, int cap, uint16_t* s_gene,
                                                           uint16_t* s_lo, uint16_t* s_hi, int* any_nan) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem) + (size_t)warp * cap;
    for (int i = blockIdx.x * wpb + warp; i < n; i += gridDim.x * wpb) {
        const int beg = ptr[i], k = ptr[i + 1] - beg;
        int m = 1;
        while (m < k) m <<= 1;
        for (int j = lane; j < m; j += 32)
            keys[j] = j < k ? ((uint64_t)ord_key(canon_zero(data[beg + j])) << 32) | (uint32_t)idx[beg + j] : ~0ull;
        __syncwarp();
        if (k > 1) warp_bitonic(keys, m, lane);
        for (int j = lane; j < k; j += 32) {
            const uint64_t key = keys[j];
            const uint32_t hv = (uint32_t)(key >> 32);
            const bool nan = key_is_nan(hv);
            if (nan) *any_nan = 1;
            s_gene[beg + j] = (uint16_t)((uint32_t)key | (nan ? NAN_GENE : 0u));
            s_lo[beg + j] = (uint16_t)lower_hi(keys, k, hv);
            s_hi[beg + j] = (uint16_t)upper_hi(keys, k, hv);
        }
        __syncwarp();
    }
}

// One CTA per cell: its row's entries in the gene pool, by value, with each entry's run as positions
// [lo, hi), at c * row_stride.  Bound by latency (the row's two dependent loads) where there are few cells
// and by issue where there are many: 48,412 cells of 1,500 entries took 1.45 ms in three kernels (count,
// fill, a bitonic sort by one warp per row) and two host round trips for the sizes.
// Values are counted into 256 buckets of a linear map; an entry's place in its bucket is the smaller values
// plus the equal ones in earlier slots.  A bucket above 128 entries (few distinct values) is sorted instead.
// dynamic shared memory: 2 x cap keys (cap: the pool's genes; a row's columns are distinct).
// mark_nan (FP32 order): NaN entries' genes are marked.
constexpr int ROWS_NT = 256;

__global__ void __launch_bounds__(ROWS_NT) ft_rows_kernel(const int32_t* cells, int n, const float* data,
                                                         const int32_t* indices, const int32_t* indptr,
                                                         uint32_t n_cols, const int32_t* map, int cap, int row_stride,
                                                         uint16_t* s_gene, uint16_t* s_lo, uint16_t* s_hi,
                                                         int32_t* row_len, int* longest, bool mark_nan) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int start[257], w_tot[ROWS_NT / 32];
    __shared__ uint32_t s_min, s_max;
    __shared__ int s_n, s_big;
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem);
    uint64_t* slots = keys + cap;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        const int beg = indptr[cells[c]], end = indptr[cells[c] + 1];
        __syncthreads();  // the previous cell's shared memory is no longer read
        start[tid + 1] = 0;
        if (tid == 0) {
            start[0] = 0;
            s_n = 0;
            s_min = 0xffffffffu;
            s_max = 0u;
            s_big = 0;
        }
        __syncthreads();
        uint32_t kmin = 0xffffffffu, kmax = 0u;
        for (int base = beg; base < end; base += 4 * ROWS_NT) {
            int col[4], g[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int i = base + t * ROWS_NT + tid;
                col[t] = i < end ? __ldg(indices + i) : -1;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) g[t] = (unsigned)col[t] < n_cols ? __ldg(map + col[t]) : -1;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const unsigned m = __ballot_sync(FULL, g[t] >= 0);
                if (!m) continue;
                int at = 0;
                if (lane == 0) at = atomicAdd(&s_n, __popc(m));
                at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
                if (g[t] >= 0 && at < cap) {
                    const uint32_t u = ord_key(canon_zero(__ldg(data + base + t * ROWS_NT + tid)));
                    keys[at] = ((uint64_t)u << 32) | (uint32_t)g[t];
                    kmin = min(kmin, u);
                    kmax = max(kmax, u);
                }
            }
        }
        kmin = __reduce_min_sync(FULL, kmin);
        kmax = __reduce_max_sync(FULL, kmax);
        if (lane == 0) {
            atomicMin(&s_min, kmin);
            atomicMax(&s_max, kmax);
        }
        __syncthreads();
        const int k = min(s_n, cap);
        const float fmin = key_float(s_min), span = key_float(s_max) - fmin;
        const float scale = (span > 0.f && span < 1e30f) ? 256.0f / span : 0.f;
        auto bucket = [&](uint64_t key) {
            const float t = (key_float((uint32_t)(key >> 32)) - fmin) * scale;
            return t >= 0.f ? min(255, (int)t) : 0;
        };
        for (int j = tid; j < k; j += ROWS_NT) atomicAdd(&start[bucket(keys[j]) + 1], 1);
        __syncthreads();
        const int mine = start[tid + 1];
        if (mine > 128) s_big = 1;
        const int incl = warp_incl_scan(mine, lane);
        if (lane == 31) w_tot[warp] = incl;
        __syncthreads();
        int before = incl - mine;
        for (int w = 0; w < warp; ++w) before += w_tot[w];
        auto marked = [&](uint64_t key) {
            return (uint16_t)((uint32_t)key | (mark_nan && key_is_nan((uint32_t)(key >> 32)) ? NAN_GENE : 0u));
        };
        uint16_t* gene = s_gene + (size_t)c * row_stride;
        uint16_t* lo_out = s_lo + (size_t)c * row_stride;
        uint16_t* hi_out = s_hi + (size_t)c * row_stride;
        if (!s_big) {
            start[tid + 1] = before;  // advanced to the bucket's end as its slots are taken
            __syncthreads();
            for (int j = tid; j < k; j += ROWS_NT) {
                const uint64_t key = keys[j];
                slots[atomicAdd(&start[bucket(key) + 1], 1)] = key;
            }
            __syncthreads();
            for (int j = tid; j < k; j += ROWS_NT) {
                const uint64_t key = slots[j];
                const uint32_t u = (uint32_t)(key >> 32);
                const int b = bucket(key), s0 = start[b], s1 = start[b + 1];
                int less = 0, eq = 0, eq_before = 0;
                for (int t = s0; t < s1; ++t) {
                    const uint32_t v = (uint32_t)(slots[t] >> 32);
                    less += v < u;
                    eq += v == u;
                    eq_before += v == u && t < j;
                }
                const int lo = s0 + less, at = lo + eq_before;
                gene[at] = marked(key);
                lo_out[at] = (uint16_t)lo;
                hi_out[at] = (uint16_t)(lo + eq);
            }
        } else {
            int m = 1;
            while (m < k) m <<= 1;  // at most 2 cap
            for (int j = k + tid; j < m; j += ROWS_NT) keys[j] = ~0ull;
            __syncthreads();
            for (int size = 2; size <= m; size <<= 1)
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    for (int t = tid; t < (m >> 1); t += ROWS_NT) {
                        const int i = 2 * t - (t & (stride - 1)), j = i + stride;
                        const uint64_t x = keys[i], y = keys[j];
                        if ((x > y) == ((i & size) == 0)) {
                            keys[i] = y;
                            keys[j] = x;
                        }
                    }
                    __syncthreads();
                }
            for (int j = tid; j < k; j += ROWS_NT) {
                const uint64_t key = keys[j];
                const uint32_t u = (uint32_t)(key >> 32);
                gene[j] = marked(key);
                lo_out[j] = (uint16_t)lower_hi(keys, k, u);
                hi_out[j] = (uint16_t)upper_hi(keys, k, u);
            }
        }
        if (tid == 0) {
            row_len[c] = k;
            atomicMax(longest, k);
        }
    }
}

// ---- a round -------------------------------------------------------------------------------------

// The reference's keep / drop rule (src/cusingler.cu:1270-1295) on the list order: returns the new
// list length, the new list in top.  One warp; tmp holds the new list meanwhile.
__device__ int keep_candidates(const float* lsc, int ntop, uint8_t* top, uint8_t* tmp, float thre, int lane) {
    float lo = __int_as_float(0x7f800000), hi = -lo;
    bool nan = false;
    for (int i = lane; i < ntop; i += 32) {
        lo = fminf(lo, lsc[i]);
        hi = fmaxf(hi, lsc[i]);
        nan |= lsc[i] != lsc[i];
    }
    int n = 0;
    if (__any_sync(FULL, nan)) {  // std::minmax_element's pairwise scan decides what a NaN does
        if (lane == 0) {
            int mn, mx;
            stl::minmax(lsc, ntop, &mn, &mx);
            lo = lsc[mn];
            hi = lsc[mx];
            const float t = __fsub_rn(hi, thre);
            if (!(hi != hi)) {
                for (int i = 0; i < ntop; ++i) {
                    const float s = lsc[i];
                    if (s <= lo || s < t) continue;
                    if (s == hi) {
                        for (int j = n; j > 0; --j) tmp[j] = tmp[j - 1];
                        tmp[0] = top[i];
                    } else {
                        tmp[n] = top[i];
                    }
                    ++n;
                }
            }
        }
        n = __shfl_sync(FULL, n, 0);
    } else {
        lo = key_float(__reduce_min_sync(FULL, ord_key(lo)));
        hi = key_float(__reduce_max_sync(FULL, ord_key(hi)));
        const float t = __fsub_rn(hi, thre);
        // every maximum is moved to the front, so the last of them comes first; the others keep their order
        int n_hi = 0;
        for (int base = 0; base < ntop; base += 32) {
            const int i = base + lane;
            const float s = i < ntop ? lsc[i] : lo;
            n_hi += __popc(__ballot_sync(FULL, !(s <= lo || s < t) && s == hi));
        }
        int hi_seen = 0, others = 0;
        for (int base = 0; base < ntop; base += 32) {
            const int i = base + lane;
            const float s = i < ntop ? lsc[i] : lo;
            const bool keep = !(s <= lo || s < t);
            const unsigned mh = __ballot_sync(FULL, keep && s == hi), mo = __ballot_sync(FULL, keep && s != hi);
            const unsigned lt = (1u << lane) - 1u;
            if (keep) {
                if (s == hi) tmp[n_hi - 1 - (hi_seen + __popc(mh & lt))] = top[i];
                else tmp[n_hi + others + __popc(mo & lt)] = top[i];
            }
            hi_seen += __popc(mh);
            others += __popc(mo);
        }
        n = n_hi + others;
    }
    if (n == 0) {
        if (lane == 0) tmp[0] = top[0];
        n = 1;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) top[i] = tmp[i];
    return n;
}

template <int NW>
struct StepSmem {
    alignas(16) int hist[NW][256];
    float lsc[256];
    uint32_t off[256];  // first 32-row block of each candidate's scores
    uint8_t top[256], tmp[256];
    uint8_t is_cand[256];
    long long red64[NW];
    int red[NW];
    int ntop, kq, nan;
};

// Step k of the batch's cells.  k = 0: candidates from the flags, the first round's setup; k > 0: the
// decisions of round k - 1, then the setup of round k.  A cell that goes on is appended, by `mode`:
//   STEP_ORDER  to `un` with its sort key (bits_key > 0: and counted under the key's leading bits);
//   STEP_QUAD   to `act` with a quad of its own, so that nothing has to be ordered and planned;
//   STEP_LIST   to `act` alone.  dynamic shared memory: eq (eq_stride
// words), bits (nwords), in / before (Wt / 32 + 2 words each).
enum StepMode { STEP_ORDER = 0, STEP_QUAD = 1, STEP_LIST = 2 };

template <int NW>
__global__ void __launch_bounds__(NW * 32, NW == STEP_NW ? 4 : 1) ft_step_kernel(FtRounds a, int k, int mode,
                                                                                int bits_key) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ StepSmem<NW> sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NT = NW * 32;
    uint32_t* eq = reinterpret_cast<uint32_t*>(dyn);
    uint32_t* bits = eq + a.eq_stride;
    uint32_t* in = bits + a.nwords;           // the row's entries inside the gene set, as bits
    uint32_t* before = in + a.Wt / 32 + 2;  // those before each word
    const int cur = k & 1, nxt = cur ^ 1;
    const int n = k == 0 ? a.n_cells : a.n_act[cur];
    unsigned long long my_rounds = 0, my_rows = 0;
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        const int c = k == 0 ? it : a.act[(size_t)cur * a.n_cells + it];
        const int cell = a.cells[c];
        uint8_t* gtop = a.top + (size_t)c * a.L;
        const uint32_t blk0 = (uint32_t)(a.blk_off[c] - a.blk_base0);
        __syncthreads();  // the previous cell's shared memory is no longer read
        if (k == 0) {
            if (warp == 0) {  // the flagged labels in ascending order (src/cusingler.cu:1305-1312)
                int m = 0;
                for (int base = 0; base < a.L; base += 32) {
                    const int l = base + lane;
                    const bool f = l < a.L && a.flags[(size_t)cell * a.L + l] != 0;
                    const unsigned b = __ballot_sync(FULL, f);
                    if (f) sh.top[m + __popc(b & ((1u << lane) - 1u))] = (uint8_t)l;
                    m += __popc(b);
                }
                if (lane == 0) sh.ntop = m;
            }
        } else {
            const int ntop = a.ntop[c];
            for (int i = tid; i < ntop; i += NT) sh.top[i] = gtop[i];
            if (tid == 0) {
                sh.ntop = ntop;
                sh.nan = 0;
            }
            for (int i = tid; i < ntop; i += NT) sh.off[i] = a.blk_of[(size_t)c * a.L + i];
            __syncthreads();
            for (int i = warp; i < ntop; i += NW) {
                const LabelQ q = a.lq[sh.top[i]];
                const float* v = a.scores + (size_t)sh.off[i] * 32;
                const uint32_t kmin = a.ext_min[(size_t)c * a.L + i], kmax = a.ext_max[(size_t)c * a.L + i];
                float r = 0.f;
                if (q.kind == 0) r = v[0];
                else if (kmax == NAN_KEY) {
                    if (lane == 0) sh.nan = 1;
                } else r = quantile_warp_core(v, q, a.p, sh.hist[warp], nullptr, lane, a.status, kmin, kmax, false);
                if (lane == 0) sh.lsc[i] = r;
            }
            __syncthreads();
            if (sh.nan && warp == 0) {
                // lists holding NaN: libstdc++'s order depends on the list's own order, which the scan's
                // block order is mapped back to
                float* scratch = a.nan_scratch + (size_t)blockIdx.x * a.max_label;
                for (int i = 0; i < ntop; ++i) {
                    const LabelQ q = a.lq[sh.top[i]];
                    if (q.kind == 0 || a.ext_max[(size_t)c * a.L + i] != NAN_KEY) continue;
                    const float* v = a.scores + (size_t)sh.off[i] * 32;
                    const uint32_t* perm = a.perm + a.ctidx[2 * sh.top[i]];
                    for (int j = lane; j < q.len; j += 32) scratch[perm[j]] = v[j];
                    __syncwarp();
                    if (lane == 0) {
                        int oob = 0;
                        stl::sort(scratch, q.len, &oob);
                        if (oob) atomicOr(a.status, 4);
                        sh.lsc[i] = q.kind == 1   ? scratch[0]
                                    : q.kind == 2 ? scratch[q.len - 1]
                                                  : interp(a.p, q.prev_index, q.step, scratch[q.k - 1], scratch[q.k]);
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            if (warp == 0) {
                const int m = keep_candidates(sh.lsc, ntop, sh.top, sh.tmp, a.thre, lane);
                if (lane == 0) sh.ntop = m;
            }
        }
        __syncthreads();

        // the next round's condition
        const int ntop = sh.ntop, done = k == 0 ? 0 : a.used[c];
        const bool go = ntop > 1 && (a.times == 0 || done < a.times);
        if (!go) {
            if (tid == 0) {
                a.final_labels[cell] = ntop > 0 ? (int32_t)sh.top[0] : 0;
                a.rounds[cell] = done;
            }
            continue;
        }
        // gene set: union over ordered candidate pairs of the first min(len, gene_thre(n)) genes of the
        // pair's list (src/cusingler.cu:1141-1156), precomputed masks where they fit (launch_pair_masks)
        const int gthre = a.gene_thre[ntop], np = ntop * ntop, nw = a.nwords;
        for (int w = tid; w < nw; w += NT) bits[w] = 0u;
        __syncthreads();
        // A warp takes up to 32 pairs at a time, few enough that every warp gets some.  Each lane fetches
        // one pair's list range; then the warp walks the pairs together, lanes over the mask's words (or
        // over a list's genes), so that the loads of several pairs are in flight at once.
        const int ppw = min(32, (np + NW - 1) / NW);
        for (int base = warp * ppw; base < np; base += NW * ppw) {
            const int pr = base + lane;
            uint32_t pi = 0, pos = 0;
            int len = 0;
            if (lane < ppw && pr < np) {
                const int i = pr / ntop, j = pr - i * ntop;
                if (i != j) {
                    pi = (uint32_t)sh.top[i] * a.L + sh.top[j];
                    const uint2 r = __ldg(reinterpret_cast<const uint2*>(a.ft_idx) + pi);
                    pos = r.x;
                    len = (int)r.y;
                }
            }
            const bool cut = len > gthre, masked = cut ? a.cut_mask != nullptr : a.pair_mask != nullptr;
            const unsigned by_mask = __ballot_sync(FULL, masked && len > 0), is_cut = __ballot_sync(FULL, cut);
            const uint32_t* cut_rows = a.cut_mask + (size_t)(ntop - 2) * a.L * a.L * nw;
            for (int w0 = 0; by_mask && w0 < nw; w0 += 32) {
                uint32_t m = 0;
#pragma unroll 16
                for (int t = 0; t < ppw; ++t) {
                    const size_t p = __shfl_sync(FULL, pi, t);
                    if (((by_mask >> t) & 1u) && w0 + lane < nw)
                        m |= __ldg(((is_cut >> t) & 1u ? cut_rows : a.pair_mask) + p * nw + w0 + lane);
                }
                if (m) atomicOr(&bits[w0 + lane], m);
            }
            if (masked) len = 0;
            len = min(len, gthre);
            const int maxn = __reduce_max_sync(FULL, len);
            for (int e0 = 0; e0 < maxn; e0 += 32) {
#pragma unroll 16
                for (int t = 0; t < ppw; ++t) {
                    const uint32_t g0 = __shfl_sync(FULL, pos, t);
                    if (e0 + lane < __shfl_sync(FULL, len, t)) {
                        const uint32_t g = __ldg(a.ft_genes + g0 + e0 + lane);
                        atomicOr(&bits[g >> 5], 1u << (g & 31));
                    }
                }
            }
        }
        __syncthreads();
        int pc = 0;
        for (int w = tid; w < nw; w += NT) pc += __popc(bits[w]);
        pc = __reduce_add_sync(FULL, pc);
        if (lane == 0) sh.red[warp] = pc;
        __syncthreads();
        int nS = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) nS += sh.red[w];
        if (tid == 0) my_rounds++;
        if (nS < 20) {  // keep the first candidate (src/cusingler.cu:1158-1159)
            if (tid == 0) {
                a.final_labels[cell] = (int32_t)sh.top[0];
                a.rounds[cell] = done + 1;
            }
            continue;
        }
        // the query's e-values over S: |S| - k + (kept entries before the run's end) + (before its start)
        const size_t beg = (size_t)c * a.row_stride;
        const int len = a.row_len[c];
        const uint32_t one = 1u << a.shift;
        const int nwd = (len + 31) / 32;
#pragma unroll 4
        for (int w = warp; w < nwd; w += NW) {
            const int j = 32 * w + lane;
            const uint32_t g = j < len ? a.s_gene[beg + j] & GENE : 0u;
            const unsigned b = __ballot_sync(FULL, j < len && ((bits[g >> 5] >> (g & 31)) & 1u));
            if (lane == 0) in[w] = b;
        }
        for (int g = tid; g < a.eq_stride; g += NT) eq[g] = g < a.Wt && ((bits[g >> 5] >> (g & 31)) & 1u) ? one : 0u;
        for (int l = tid; l < a.L; l += NT) sh.is_cand[l] = 0;
        __syncthreads();
        if (warp == 0) {
            int m = 0;
            for (int base = 0; base < nwd; base += 32) {
                const int w = base + lane;
                const int p = w < nwd ? __popc(in[w]) : 0, incl = warp_incl_scan(p, lane);
                if (w < nwd) before[w] = (uint32_t)(m + incl - p);
                m += __shfl_sync(FULL, incl, 31);
            }
            if (lane == 0) {
                in[nwd] = 0u;
                before[nwd] = (uint32_t)m;
                sh.kq = m;
            }
        }
        for (int i = tid; i < ntop; i += NT) sh.is_cand[sh.top[i]] = 1;
        __syncthreads();
        const int kq = sh.kq;
        auto kept = [&](int x) {  // kept entries before position x
            return (int)before[x >> 5] + __popc(in[x >> 5] & ((1u << (x & 31)) - 1u));
        };
        long long sq = 0;
        for (int j = tid; j < len; j += NT) {
            if (!((in[j >> 5] >> (j & 31)) & 1u)) continue;
            const int e = nS - kq + kept(a.s_lo[beg + j]) + kept(a.s_hi[beg + j]);
            const uint32_t g = a.s_gene[beg + j];
            if (g & NAN_GENE) atomicOr(a.status, 2);  // a NaN inside the gene set
            eq[g & GENE] = one + (uint32_t)e;
            sq += (long long)(e - kq) * (e - kq);
        }
        sq = warp_sum_i64(sq);
        if (lane == 0) sh.red64[warp] = sq;
        __syncthreads();
        uint4* out = reinterpret_cast<uint4*>(a.eq + (size_t)c * a.eq_stride);
        for (int g = tid; g < a.eq_stride / 4; g += NT) out[g] = reinterpret_cast<const uint4*>(eq)[g];
        for (int i = tid; i < ntop; i += NT) gtop[i] = sh.top[i];
        if (tid == 0) {
            long long nq = (long long)(nS - kq) * kq * kq;
            for (int w = 0; w < NW; ++w) nq += sh.red64[w];
            a.par[c] = FtCell{nq > 0 ? 1.0 / sqrt((double)nq) : 0.0, (int64_t)nq, nS, kq};
            a.ntop[c] = ntop;
            a.used[c] = done + 1;
        }
        if (mode == STEP_LIST && tid == 0) a.act[(size_t)nxt * a.n_cells + atomicAdd(a.n_act + nxt, 1)] = c;
        if (mode == STEP_ORDER && warp == 0) {
            // sort key: the candidates among the 32 longest labels as a reflected Gray code, so that cells
            // whose candidates differ little are close
            const unsigned m = __ballot_sync(FULL, lane < a.L && sh.is_cand[a.lorder[min(lane, a.L - 1)]]);
            const uint32_t key = __brev(__ballot_sync(FULL, __popc(m & (0xffffffffu >> (31 - lane))) & 1));
            if (lane == 0) {
                a.un[atomicAdd(a.n_act + nxt, 1)] = ((unsigned long long)key << 32) | (uint32_t)c;
                if (bits_key) atomicAdd(a.key_count + (key >> (32 - bits_key)), 1);
            }
        }
        if (warp == NW - 1) {  // the candidates' score blocks
            uint32_t acc = 0;
            int quad = 0;
            if (mode == STEP_QUAD) {
                if (lane == 0) quad = atomicAdd(a.n_act + nxt, 1);
                quad = __shfl_sync(FULL, quad, 0);
            }
            for (int base = 0; base < ntop; base += 32) {
                const int i = base + lane;
                const int l = i < ntop ? sh.top[i] : 0;
                const int nb = i < ntop ? (int)(a.ctidx[2 * l + 1] + 31) / 32 : 0;
                const int incl = warp_incl_scan(nb, lane);
                if (i < ntop) {
                    a.ext_min[(size_t)c * a.L + i] = 0xffffffffu;
                    a.ext_max[(size_t)c * a.L + i] = 0u;
                    const uint32_t blk = blk0 + acc + (uint32_t)(incl - nb);
                    a.blk_of[(size_t)c * a.L + i] = blk;
                    if (mode == STEP_QUAD) {
                        const size_t at = (size_t)quad * a.L + i;
                        a.q_label[at] = make_int2(l, (int)acc + incl - nb);
                        a.q_entry[4 * at] = FtEntry{(uint32_t)(c * a.L + i), blk};
#pragma unroll
                        for (int t = 1; t < 4; ++t) a.q_entry[4 * at + t] = FtEntry{~0u, 0u};
                    }
                }
                acc += (uint32_t)__shfl_sync(FULL, incl, 31);
            }
            if (mode == STEP_QUAD && lane == 0) {
                a.act[(size_t)nxt * a.n_cells + quad] = c;
                a.quads[quad] = FtQuad{{c, c, c, c}, 1, ntop, (int)acc};
            }
            if (lane == 0) my_rows += (unsigned long long)acc * 32;
        }
    }
    if (tid == 0 && my_rounds) atomicAdd(a.stats, my_rounds);
    if (warp == NW - 1 && lane == 0 && my_rows) atomicAdd(a.stats + 1, my_rows);
}

// State of one row's pass for NC cells.
template <int NC, bool X64>
struct RowSums {
    using T = typename std::conditional<X64, uint64_t, uint32_t>::type;
    uint32_t P[NC], tot[NC], ka[NC], B3[NC];
    T X[NC];
};

// The table's words of one gene for NC cells.
template <int NC>
__device__ __forceinline__ void lookup(uint32_t addr, uint32_t (&v)[NC]) {
    if (NC == 1) {
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[0]) : "r"(addr));
    } else {
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1 % NC]), "=r"(v[2 % NC]), "=r"(v[3 % NC])
                     : "r"(addr));
    }
}

// One group of four entries: w0 = entries 0 | 1 << 16 (bit 15: the group ends a run), w1 = 2 | 3 << 16.
// m = {16 C, 2, -1} as run-time values: with them the addresses, z and acc are multiply-adds, which
// leaves the integer ALU (half rate, as the multiplier is) and the multiplier with about the same number
// of instructions.
template <int NC, bool X64>
__device__ __forceinline__ void scan_group(RowSums<NC, X64>& s, uint32_t w0, uint32_t w1, uint32_t tab, int sh,
                                           uint32_t low, int3 m) {
    uint32_t va[NC], vb[NC], vc[NC], vd[NC];
    lookup<NC>((w0 & 0x7fffu) * (uint32_t)m.x + tab, va);
    lookup<NC>((w0 >> 16) * (uint32_t)m.x + tab, vb);
    lookup<NC>((w1 & 0xffffu) * (uint32_t)m.x + tab, vc);
    lookup<NC>((w1 >> 16) * (uint32_t)m.x + tab, vd);
    const bool end = (w0 & 0x8000u) != 0;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        s.P[i] += va[i] + vb[i];
        s.P[i] += vc[i] + vd[i];
        const uint32_t t = end ? s.P[i] : s.tot[i];
        const uint32_t acc = s.tot[i] * (uint32_t)m.z + t;
        s.tot[i] = t;
        const uint32_t n = acc >> sh;
        const uint32_t z = (uint32_t)m.y * s.ka[i] + n;
        s.ka[i] += n;
        if (X64) s.X[i] += (uint64_t)z * (acc & low);
        else s.X[i] += z * acc;  // the count field's part is taken off at the end
        s.B3[i] += n * n * n;
    }
}

constexpr int PLAN_NW = 8;
constexpr int ITEMS_PER_CTA = 16;  // scan items per CTA that a round's quads are cut into
constexpr int FEW_QUADS = 512;     // up to this many quads the items are sized by the round's total work
constexpr int SPLIT_QUADS = 64;    // from this many quads on, a label that one cell alone needs goes to its work list

// The active cells in the order of their keys: by rank (few cells; one warp per cell counts the smaller
// keys), or by the keys' leading bits (start: exclusive scan of their counts, advanced here).
__global__ void __launch_bounds__(256) ft_rank_kernel(FtRounds a, int k) {
    const int n = a.n_act[(k & 1) ^ 1], lane = threadIdx.x & 31;
    int* act = a.act + (size_t)((k & 1) ^ 1) * a.n_cells;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const unsigned long long mine = a.un[i];
        int less = 0;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) less += a.un[j] < mine;
        less = __reduce_add_sync(FULL, less);
        if (lane == 0) act[less] = (int)(uint32_t)mine;
    }
}

__global__ void __launch_bounds__(256) ft_place_kernel(FtRounds a, int k, int bits_key, int32_t* start) {
    const int n = a.n_act[(k & 1) ^ 1];
    int* act = a.act + (size_t)((k & 1) ^ 1) * a.n_cells;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long u = a.un[i];
        act[atomicAdd(start + (uint32_t)(u >> (64 - bits_key)), 1)] = (int)(uint32_t)u;
    }
}

// The round's quads: the active cells in order, four at a time.  One warp per quad.
__global__ void __launch_bounds__(PLAN_NW * 32) ft_plan_kernel(FtRounds a, int k) {
    __shared__ uint16_t pos[PLAN_NW][4][256];  // position of each label in the four candidate lists
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cur = k & 1;
    const int n = a.n_act[cur ^ 1];
    const int n_quads = (n + 3) / 4, least = n_quads >= SPLIT_QUADS ? 2 : 1;
    for (int q = blockIdx.x * PLAN_NW + warp; q < n_quads; q += gridDim.x * PLAN_NW) {
        const int nq = min(4, n - 4 * q);
        const int c = lane < nq ? a.act[(size_t)(cur ^ 1) * a.n_cells + 4 * q + lane] : 0;
        for (int i = lane; i < 4 * 256; i += 32) (&pos[warp][0][0])[i] = 0xffffu;
        __syncwarp();
        const int m_c = lane < nq ? a.ntop[c] : 0, most = __reduce_max_sync(FULL, m_c);
        int cell[4], m[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            cell[t] = __shfl_sync(FULL, c, min(t, nq - 1));
            m[t] = __shfl_sync(FULL, m_c, t);
        }
        for (int i = lane; i < most; i += 32) {
            int l[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) l[t] = i < m[t] ? a.top[(size_t)cell[t] * a.L + i] : -1;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (l[t] >= 0) pos[warp][t][l[t]] = (uint16_t)i;
        }
        __syncwarp();
        int n_lab = 0, units = 0;
        for (int base = 0; base < a.L; base += 32) {
            const int l = base + lane;
            FtEntry e[4];
            int need = 0, last = 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const uint32_t i = l < a.L && t < nq ? pos[warp][t][l] : 0xffffu;
                e[t] = FtEntry{~0u, 0u};
                if (i != 0xffffu) {
                    const uint32_t cp = (uint32_t)cell[t] * a.L + i;
                    e[t] = FtEntry{cp, a.blk_of[cp]};
                    ++need;
                    last = t;
                }
            }
            const bool in = need >= least;
            const int nb = in ? (int)(a.ctidx[2 * l + 1] + 31) / 32 : 0;
            const unsigned mk = __ballot_sync(FULL, in);
            const int ps = warp_incl_scan(nb, lane);
            if (in) {
                const size_t at_q = (size_t)q * a.L + n_lab + __popc(mk & ((1u << lane) - 1u));
                a.q_label[at_q] = make_int2(l, units + ps - nb);
#pragma unroll
                for (int t = 0; t < 4; ++t) a.q_entry[at_q * 4 + t] = e[t];
            } else if (need) {
                FtEntry x = e[0];
#pragma unroll
                for (int t = 1; t < 4; ++t)
                    if (last == t) x = e[t];
                a.list[(size_t)l * a.n_cells + atomicAdd(a.n_list + cur * 256 + l, 1)] = x;
            }
            n_lab += __popc(mk);
            units += __shfl_sync(FULL, ps, 31);
        }
        if (lane == 0) a.quads[q] = FtQuad{{cell[0], cell[1], cell[2], cell[3]}, nq, n_lab, units};
        __syncwarp();
    }
}

// One work item of a round: four cells and a range of 32-row blocks ("units") of the labels they need.
struct ScanItem {
    FtCell par[4];
    FtEntry entry[4];  // work-list item: the cells' entries of the one label
    int cell[4];
    int quad;          // -1: work-list item
    int label;         // work-list item: its label
    int n_lab;         // labels (0: no item left)
    int u0, u1;
};

constexpr int SCAN_PF = 4;  // genes of the next table that a thread holds in registers

// Work items: the quads' labels, each quad cut into parts when a round has few quads; then the labels'
// work lists in order of length (lorder), four entries at a time, in parts of at most `bpp` blocks.
// Items are fetched two ahead while the current one is scanned, and a warp that has finished its blocks
// loads its share of the next table into registers before it waits for the others, so that between two
// items only the table's stores are left.
// NC = 1: every quad is one cell (rounds of a few cells).  Its table is the same memory with the cell's word
// in all four places, 4 C copies of 4 bytes, and a row's pass takes half the instructions.
template <int C, int NC, bool X64>
__global__ void __launch_bounds__(SCAN_NW * 32, 1) ft_scan_kernel(FtRounds a, int k) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ int pre[257];      // work-list items before each label (in lorder)
    __shared__ int2 labs[256];    // the current item's labels and the units before each
    __shared__ int qpre[FEW_QUADS + 1];  // few quads: items before each
    __shared__ int s_bpp, s_upp;
    __shared__ ScanItem items[3];  // ring: current, next, the one being fetched
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cur = k & 1, nxt = cur ^ 1;
    constexpr int NT = SCAN_NW * 32;
    if (blockIdx.x == 0) {  // the next round's counters
        for (int l = tid; l < 256; l += NT) a.n_list[nxt * 256 + l] = 0;
        if (tid == 0) {
            a.queue[nxt] = 0;
            a.n_act[cur] = 0;
        }
    }
    const int n_quads = (a.n_act[nxt] + NC - 1) / NC;
    if (n_quads == 0) return;
    // Many quads: the same number of parts for each.  Few: parts of `upp` units so that every CTA gets some.
    // Filling a table costs about as much as scanning one unit at full rate, and four warps (one per
    // scheduler) scan at close to full rate, so a part is not below four units; parts are 16 units (one per
    // warp) as soon as there are enough for every CTA.
    const int parts = max(1, ((int)gridDim.x * ITEMS_PER_CTA + n_quads - 1) / n_quads);
    const bool few = n_quads <= FEW_QUADS;
    // Fetches the next work item into `it`.  One warp.
    auto fetch = [&](ScanItem& it) {
        for (;;) {
            int item = 0;
            if (lane == 0) item = atomicAdd(a.queue + cur, 1);
            item = __shfl_sync(FULL, item, 0);
            const int n_quad_items = few ? qpre[n_quads] : n_quads * parts;
            if (item < n_quad_items) {
                int q, part, upp = s_upp;
                if (few) {
                    int lo = 0, hi = n_quads - 1;  // qpre[lo] <= item < qpre[lo + 1]
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (qpre[mid] <= item) lo = mid;
                        else hi = mid - 1;
                    }
                    q = lo;
                    part = item - qpre[lo];
                } else {
                    q = item / parts;
                    part = item - q * parts;
                }
                const FtQuad h = a.quads[q];
                if (!few) upp = max(SCAN_NW, (h.units + parts - 1) / parts);
                const int u0 = part * upp;
                if (u0 >= h.units) continue;  // a quad with fewer parts
                if (lane < 4) {
                    const int c = a.quads[q].cell[lane];
                    it.cell[lane] = c;
                    it.par[lane] = a.par[c];
                }
                if (lane == 0) {
                    it.quad = q;
                    it.n_lab = h.n_lab;
                    it.u0 = u0;
                    it.u1 = min(h.units, u0 + upp);
                }
                return;
            }
            item -= n_quad_items;
            if (item >= pre[a.L]) {
                if (lane == 0) it.n_lab = 0;
                return;
            }
            int lo = 0, hi = a.L - 1;  // pre[lo] <= item < pre[lo + 1]
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (pre[mid] <= item) lo = mid;
                else hi = mid - 1;
            }
            const int l = a.lorder[lo], nblk = (int)(a.ctidx[2 * l + 1] + 31) / 32;
            const int lparts = (nblk + s_bpp - 1) / s_bpp, at = item - pre[lo];
            const int q0 = at / lparts * 4, nq = min(4, a.n_list[cur * 256 + l] - q0);
            if (lane < 4) {
                const FtEntry e = a.list[(size_t)l * a.n_cells + q0 + min(lane, nq - 1)];
                const int c = (int)(e.cellp / a.L);
                it.entry[lane] = lane < nq ? e : FtEntry{~0u, 0u};
                it.cell[lane] = c;
                it.par[lane] = a.par[c];
            }
            if (lane == 0) {
                it.quad = -1;
                it.label = l;
                it.n_lab = 1;
                it.u0 = at % lparts * s_bpp;
                it.u1 = min(nblk, it.u0 + s_bpp);
            }
            return;
        }
    };
    if (warp == 0) {
        unsigned long long work = 0;  // (four entries, block) pairs of the work lists
        for (int i = lane; i < a.L; i += 32) {
            const int l = a.lorder[i];
            work += (unsigned long long)((a.n_list[cur * 256 + l] + 3) / 4) * ((a.ctidx[2 * l + 1] + 31) / 32);
        }
        for (int o = 16; o > 0; o >>= 1) work += __shfl_xor_sync(FULL, work, o);
        const int bpp = (int)min(1ull << 24, max((unsigned long long)SCAN_NW, work / gridDim.x + 1));
        int acc = 0;
        for (int base = 0; base < a.L; base += 32) {
            const int i = base + lane;
            int n = 0;
            if (i < a.L) {
                const int l = a.lorder[i];
                const int nb = (int)(a.ctidx[2 * l + 1] + 31) / 32;
                n = (a.n_list[cur * 256 + l] + 3) / 4 * ((nb + bpp - 1) / bpp);
            }
            const int incl = warp_incl_scan(n, lane);
            if (i < a.L) pre[i] = acc + incl - n;
            acc += __shfl_sync(FULL, incl, 31);
        }
        if (lane == 0) {
            pre[a.L] = acc;
            s_bpp = bpp;
        }
        if (few) {
            int total = 0;
            for (int q = lane; q < n_quads; q += 32) total += a.quads[q].units;
            total = __reduce_add_sync(FULL, total);
            const int grid = (int)gridDim.x;
            const int upp = total <= grid * SCAN_NW ? max(4, (total + grid - 1) / grid)
                                                    : max(SCAN_NW, total / (grid * ITEMS_PER_CTA));
            int at = 0;
            for (int base = 0; base < n_quads; base += 32) {
                const int q = base + lane;
                const int n = q < n_quads ? (a.quads[q].units + upp - 1) / upp : 0, incl = warp_incl_scan(n, lane);
                if (q < n_quads) qpre[q] = at + incl - n;
                at += __shfl_sync(FULL, incl, 31);
            }
            if (lane == 0) {
                qpre[n_quads] = at;
                s_upp = upp;
            }
        }
        __syncwarp();
        fetch(items[0]);
        fetch(items[1]);
    }
    __syncthreads();
    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(dyn) +
                         (NC == 1 ? (lane & (4 * C - 1)) * 4 : (lane & (C - 1)) * 16);
    const uint32_t low = (1u << a.shift) - 1u;
    const int3 mul = a.mul;
    // the table's words of gene g for an item's four cells
    auto load_gene = [&](const ScanItem& it, int g) {
        uint4 v;
        v.x = __ldg(a.eq + (size_t)it.cell[0] * a.eq_stride + g);
        v.y = __ldg(a.eq + (size_t)it.cell[1] * a.eq_stride + g);
        v.z = __ldg(a.eq + (size_t)it.cell[2] * a.eq_stride + g);
        v.w = __ldg(a.eq + (size_t)it.cell[3] * a.eq_stride + g);
        return v;
    };
    // C copies, written in rotated order so that a quarter-warp's stores fall into different bank groups
    auto store_gene = [&](int g, const uint4& v) {
        uint4* t = reinterpret_cast<uint4*>(dyn) + (size_t)g * C;
#pragma unroll
        for (int i = 0; i < C; ++i) t[(i + lane) & (C - 1)] = v;
    };
    for (int turn = 0; items[turn].n_lab != 0; turn = turn == 2 ? 0 : turn + 1) {
        const ScanItem& it = items[turn];
        // the item's table and labels, into registers while other warps still scan the item before
        uint4 pf[SCAN_PF];
#pragma unroll
        for (int u = 0; u < SCAN_PF; ++u)
            if (tid + u * NT <= a.Wt) pf[u] = load_gene(it, tid + u * NT);
        const int n_lab = it.n_lab, quad = it.quad, u1 = it.u1;
        int2 my_lab = make_int2(it.label, 0);
        if (quad >= 0 && tid < n_lab) my_lab = __ldg(a.q_label + (size_t)quad * a.L + tid);
        __syncthreads();  // every warp is done with the previous item
#pragma unroll
        for (int u = 0; u < SCAN_PF; ++u)
            if (tid + u * NT <= a.Wt) store_gene(tid + u * NT, pf[u]);
        for (int g = tid + SCAN_PF * NT; g <= a.Wt; g += NT) store_gene(g, load_gene(it, g));
        if (tid < n_lab) labs[tid] = my_lab;
        __syncthreads();
        // the item after next, in the slot of the one before (read by nobody since the first barrier)
        if (warp == SCAN_NW - 1) fetch(items[turn == 0 ? 2 : turn - 1]);
        // unit u is block u - labs[j].y of label labs[j].x
        int j = 0, blk = 0, v0 = 0, nv = 0;
        uint4 w = make_uint4(0u, 0u, 0u, 0u), w2 = w;
        auto open = [&](int u) {  // the unit's label, block and first row vectors
            while (j + 1 < n_lab && labs[j + 1].y <= u) ++j;
            const int2 lb = labs[j];
            blk = u - lb.y;
            const int32_t* vo = a.blk_voff + a.blk_base[lb.x] + blk;
            v0 = vo[0];
            nv = (vo[1] - v0) >> 5;
            if (nv > 0) w = __ldg(a.groups + v0 + lane);
            if (nv > 1) w2 = __ldg(a.groups + v0 + 32 + lane);
        };
        int u = it.u0 + warp;
        if (u < u1) open(u);
        while (u < u1) {
            const int uj = j, ub = blk;
            FtEntry my = {~0u, 0u};
            if (lane < 4) my = quad >= 0 ? a.q_entry[((size_t)quad * a.L + uj) * 4 + lane] : it.entry[lane];
            const uint4* p = a.groups + v0 + lane;
            RowSums<NC, X64> s = {};
            for (int v = 0; v < nv; ++v) {
                const uint4 wn = v + 2 < nv ? __ldg(p + 32 * (v + 2)) : w;  // two vectors ahead
                scan_group<NC, X64>(s, w.x, w.y, tab, a.shift, low, mul);
                scan_group<NC, X64>(s, w.z, w.w, tab, a.shift, low, mul);
                w = w2;
                w2 = wn;
            }
            u += SCAN_NW;
            const bool valid = ub * 32 + lane < (int)a.ctidx[2 * labs[uj].x + 1];
            if (u < u1) open(u);  // the next unit's first vectors, on their way during the last steps
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const uint32_t cellp = __shfl_sync(FULL, my.cellp, i), sblk = __shfl_sync(FULL, my.blk, i);
                if (cellp == ~0u) continue;  // the cell does not need this label
                const FtCell c = it.par[i];
                // the longest row is below 1,024 entries wherever words are packed, so kr, the squares and
                // 4 kr^3 fit 32 bits; |S| k_q does too
                const uint32_t kr = s.ka[i], k2 = kr * kr;
                const int nS = c.nS;
                const int64_t X = X64 ? (int64_t)s.X[i] : (int64_t)(uint32_t)((uint32_t)s.X[i] - (k2 << a.shift));
                const int64_t N = X + (int64_t)(nS - (int)kr) * (int)(s.tot[i] & low) - (int64_t)(nS * c.kq) * (int)kr;
                const uint32_t Z2 = (4u * k2 * kr - s.B3[i]) / 3u;
                const int cc = nS - 2 * (int)kr;
                const int64_t nr = (int64_t)Z2 + (int64_t)(int)k2 * (3 * nS - 5 * (int)kr) + (int64_t)(int)kr * (cc * cc);
                const bool nan = c.nq == 0 || nr == 0;
                const float v = nan ? __int_as_float(0x7fffffff)
                                    : (float)(((double)N * c.rq) * (1.0 / sqrt((double)nr)));
                if (valid) a.scores[(size_t)(sblk + ub) * 32 + lane] = v;
                const uint32_t key = nan ? NAN_KEY : ord_key(v);
                const uint32_t mn = __reduce_min_sync(FULL, valid ? key : 0xffffffffu);
                const uint32_t mx = __reduce_max_sync(FULL, valid ? key : 0u);
                if (lane == 0) {
                    atomicMin(a.ext_min + cellp, mn);
                    atomicMax(a.ext_max + cellp, mx);
                }
            }
        }
    }
}

// ---- FP32-order scan ------------------------------------------------------------------------------

// The reference's spearman_reduce over one row (src/cusingler.cu:803-856): 128 contiguous gene chunks of
// `step` genes, one FP32 multiply-add chain each, then the stride-doubling pairwise tree.  Lane t holds
// chunks 4 t .. 4 t + 3; the sum is in lane 0.
__device__ __forceinline__ float tree128(const float (&c)[4], int lane) {
    float v = __fadd_rn(__fadd_rn(c[0], c[1]), __fadd_rn(c[2], c[3]));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float w = __shfl_down_sync(FULL, v, o);
        if ((lane & (2 * o - 1)) == 0) v = __fadd_rn(v, w);
    }
    return v;
}

// Correlations of a round in the reference's FP32 order.  Work item: a cell and a part of its candidate
// rows; one warp per row.  The ranks over S come from the row's value-sorted entries, as in the exact scan
// (an entry's z is the kept entries before its run's end plus those before its start), so no row is sorted
// or bucketed again.  They are scattered into a dense row in shared memory laid out [gene in chunk][chunk],
// so that a lane reads its four chunks' next genes with one conflict-free 16-byte load.
// Bound: the shared-memory pipe (73 % of its wavefronts in the first round: dense rows, scatters, shuffles), with
// 68 % of the issue slots.  1,000 queries x 20,000 reference cells, 1,215 cell rounds of 13 candidates, 13.4e6
// rows: 1,014 ms with the host's lists of (candidate set, row) rankings; 21.8 ms with rows dealt to the warps one
// by one, each after the loads of its place, genes and runs in turn; 18.5 ms (1.4 ns a row) with consecutive
// rows, 32 places and a row's genes and runs read at once.
// dense_len: floats of a dense row (128 x the longest chunk).  dynamic shared memory: the query's dense
// row, one per warp, the slot of each pool gene (halfwords).
// NANS: some reference row holds a NaN, and the rows' genes may be marked.
template <bool NANS>
__global__ void __launch_bounds__(256) ft_scan32_kernel(FtRounds a, int k, int dense_len, int parts) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ int off[257];  // candidate rows before each label of the cell's list
    __shared__ uint8_t top[256];
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5, NT = blockDim.x;
    const int cur = k & 1, nxt = cur ^ 1;
    float* x = reinterpret_cast<float*>(dyn);
    float* y = x + (size_t)(1 + warp) * dense_len;
    uint16_t* slot = reinterpret_cast<uint16_t*>(x + (size_t)(1 + nwarp) * dense_len);
    int* pre = reinterpret_cast<int*>(x + dense_len);  // genes of S before each word; before the rows use y
    if (blockIdx.x == 0 && tid == 0) {  // the next round's counters
        a.queue[nxt] = 0;
        a.n_act[cur] = 0;
    }
    const int n = a.n_act[nxt];
    const uint32_t low = (1u << a.shift) - 1u;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(a.queue + cur, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= n * parts) return;
        const int c = a.act[(size_t)nxt * a.n_cells + item / parts], part = item % parts, ntop = a.ntop[c];
        for (int i = tid; i < ntop; i += NT) top[i] = a.top[(size_t)c * a.L + i];
        __syncthreads();
        if (warp == 0) {
            int acc = 0;
            for (int base = 0; base < ntop; base += 32) {
                const int i = base + lane, len = i < ntop ? (int)a.ctidx[2 * top[i] + 1] : 0;
                const int incl = warp_incl_scan(len, lane);
                if (i < ntop) off[i] = acc + incl - len;
                acc += __shfl_sync(FULL, incl, 31);
            }
            if (lane == 0) off[ntop] = acc;
        }
        __syncthreads();
        const int rows = off[ntop], per = max(2 * nwarp, (rows + parts - 1) / parts);
        const int r0 = part * per, r1 = min(rows, r0 + per);
        if (r0 >= rows) continue;  // a cell with fewer parts
        // S in ascending gene order: position i is gene i % step of chunk i / step
        const FtCell par = a.par[c];
        const int nS = par.nS, step = (nS + 127) / 128;
        const uint32_t* eq = a.eq + (size_t)c * a.eq_stride;
        for (int w = warp; w < a.nwords; w += nwarp) {
            const int g = 32 * w + lane;
            const unsigned m = __ballot_sync(FULL, g < a.Wt && eq[g] != 0u);
            if (lane == 0) pre[w] = __popc(m);
        }
        for (int i = tid; i < step * 128; i += NT) x[i] = 0.f;
        __syncthreads();
        if (warp == 0) {
            int acc = 0;
            for (int base = 0; base < a.nwords; base += 32) {
                const int w = base + lane, v = w < a.nwords ? pre[w] : 0, incl = warp_incl_scan(v, lane);
                if (w < a.nwords) pre[w] = acc + incl - v;
                acc += __shfl_sync(FULL, incl, 31);
            }
        }
        __syncthreads();
        for (int w = warp; w < a.nwords; w += nwarp) {
            const int g = 32 * w + lane;
            const uint32_t e = g < a.Wt ? eq[g] : 0u;
            const unsigned m = __ballot_sync(FULL, e != 0u);
            const int i = pre[w] + __popc(m & ((1u << lane) - 1u)), ch = i / step, at = (i - ch * step) * 128 + ch;
            if (g < a.Wt) slot[g] = e ? (uint16_t)at : (uint16_t)0xffff;
            if (e) x[at] = (float)((int)(e & low) - par.kq) * 0.5f;
        }
        __syncthreads();  // pre (the first warp's row) is free again
        const float4* x4 = reinterpret_cast<const float4*>(x);
        float4* y4 = reinterpret_cast<float4*>(y);
        float qn[4] = {0.f, 0.f, 0.f, 0.f};
        for (int o = 0; o < step; ++o) {
            const float4 v = x4[o * 32 + lane];
            qn[0] = fmaf(v.x, v.x, qn[0]);
            qn[1] = fmaf(v.y, v.y, qn[1]);
            qn[2] = fmaf(v.z, v.z, qn[2]);
            qn[3] = fmaf(v.w, v.w, qn[3]);
        }
        const float qf = tree128(qn, lane);
        // a warp takes consecutive rows: the place of 32 of them is read at once, one per lane, and a label's
        // extremes are written once
        const int each = (r1 - r0 + nwarp - 1) / nwarp, w0 = r0 + warp * each, w1 = min(r1, w0 + each);
        int lab = 0, lab_end = 0, my_beg = 0, my_len = 0;
        size_t out = 0;
        uint32_t kmin = 0xffffffffu, kmax = 0u;
        auto flush = [&](int l) {
            if (lane == 0) {
                atomicMin(a.ext_min + (size_t)c * a.L + l, kmin);
                atomicMax(a.ext_max + (size_t)c * a.L + l, kmax);
            }
            kmin = 0xffffffffu;
            kmax = 0u;
        };
        for (int r = w0; r < w1; ++r) {
            if (((r - w0) & 31) == 0) {
                const int ri = min(r + lane, w1 - 1);
                int lo = 0, hi = ntop - 1;  // off[lo] <= ri < off[lo + 1]
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (off[mid] <= ri) lo = mid;
                    else hi = mid - 1;
                }
                const uint32_t start = a.ctidx[2 * top[lo]];
                const uint32_t row = start + a.perm[start + ri - off[lo]];
                my_beg = a.ref_ptr[row];
                my_len = a.ref_ptr[row + 1] - my_beg;
                if (r == w0) {
                    lab = __shfl_sync(FULL, lo, 0);
                    lab_end = off[lab + 1];
                    out = (size_t)a.blk_of[(size_t)c * a.L + lab] * 32;
                }
            }
            if (r >= lab_end) {
                flush(lab);
                while (off[lab + 1] <= r) ++lab;
                lab_end = off[lab + 1];
                out = (size_t)a.blk_of[(size_t)c * a.L + lab] * 32;
            }
            const int beg = __shfl_sync(FULL, my_beg, (r - w0) & 31), len = __shfl_sync(FULL, my_len, (r - w0) & 31);
            const int nwd = (len + 31) / 32;
            constexpr uint32_t ref_gene = NANS ? GENE : 0xffffu;
            if (NANS) {  // a NaN inside the gene set is refused
                bool bad = false;
                for (int e = lane; e < len; e += 32) {
                    const uint32_t g = a.ref_gene[beg + e];
                    bad |= (g & NAN_GENE) && slot[g & GENE] != 0xffffu;
                }
                if (bad) atomicOr(a.status, 2);
            }
            // the row's entries inside S as bits: lane w holds entries 32 w .. ; the first HELD words' slots and
            // run bounds stay in registers, all their loads in flight together
            constexpr int HELD = 4;
            uint32_t in = 0, sl[HELD], lh[HELD];
#pragma unroll
            for (int w = 0; w < HELD; ++w) {
                const int e = 32 * w + lane;
                sl[w] = e < len ? a.ref_gene[beg + e] : 0xffffffffu;
                lh[w] = e < len ? a.ref_lo[beg + e] | (uint32_t)a.ref_hi[beg + e] << 16 : 0u;
            }
#pragma unroll
            for (int w = 0; w < HELD; ++w) {
                sl[w] = sl[w] != 0xffffffffu ? slot[sl[w] & ref_gene] : 0xffffu;
                const unsigned m = __ballot_sync(FULL, sl[w] != 0xffffu);
                if (lane == w) in = m;
            }
            for (int w = HELD; w < nwd; ++w) {
                const int e = 32 * w + lane;
                const bool hit = e < len && slot[a.ref_gene[beg + e] & ref_gene] != 0xffffu;
                const unsigned m = __ballot_sync(FULL, hit);
                if (lane == w) in = m;
            }
            const int p = __popc(in), before = warp_incl_scan(p, lane) - p;
            const int kr = __shfl_sync(FULL, before + p, 31);
            // every gene of S at rank d = -k_r, then the stored ones
            const float d0 = (float)(-kr) * 0.5f;
            for (int o = 0; o < step; ++o) {
                const int i = 4 * lane * step + o;
                y4[o * 32 + lane] = make_float4(i < nS ? d0 : 0.f, i + step < nS ? d0 : 0.f,
                                                i + 2 * step < nS ? d0 : 0.f, i + 3 * step < nS ? d0 : 0.f);
            }
            __syncwarp();
            auto place = [&](uint32_t at, int l0, int h0) {
                const int z = __shfl_sync(FULL, before, l0 >> 5) +
                              __popc(__shfl_sync(FULL, in, l0 >> 5) & ((1u << (l0 & 31)) - 1u)) +
                              __shfl_sync(FULL, before, h0 >> 5) +
                              __popc(__shfl_sync(FULL, in, h0 >> 5) & ((1u << (h0 & 31)) - 1u));
                if (at != 0xffffu) y[at] = (float)(nS - 2 * kr + z) * 0.5f;
            };
#pragma unroll
            for (int w = 0; w < HELD; ++w)
                if (w < nwd) place(sl[w], (int)(lh[w] & 0xffffu), (int)(lh[w] >> 16));
            for (int w = HELD; w < nwd; ++w) {
                const int e = 32 * w + lane;
                const bool hit = e < len;
                place(hit ? slot[a.ref_gene[beg + e] & ref_gene] : 0xffffu, hit ? a.ref_lo[beg + e] : 0,
                      hit ? a.ref_hi[beg + e] : 0);
            }
            __syncwarp();
            float d[4] = {0.f, 0.f, 0.f, 0.f}, rn[4] = {0.f, 0.f, 0.f, 0.f};
            for (int o = 0; o < step; ++o) {
                const float4 u = x4[o * 32 + lane], v = y4[o * 32 + lane];
                d[0] = fmaf(u.x, v.x, d[0]);
                d[1] = fmaf(u.y, v.y, d[1]);
                d[2] = fmaf(u.z, v.z, d[2]);
                d[3] = fmaf(u.w, v.w, d[3]);
                rn[0] = fmaf(v.x, v.x, rn[0]);
                rn[1] = fmaf(v.y, v.y, rn[1]);
                rn[2] = fmaf(v.z, v.z, rn[2]);
                rn[3] = fmaf(v.w, v.w, rn[3]);
            }
            const float s = tree128(d, lane), rf = tree128(rn, lane);
            const float div = sqrtf(qf * rf);
            const float v = div != 0.f ? s / div : __int_as_float(0x7fffffff);  // lane 0's counts
            if (lane == 0) a.scores[out + (r - off[lab])] = v;
            const uint32_t key = div != 0.f ? ord_key(v) : NAN_KEY;
            kmin = min(kmin, key);
            kmax = max(kmax, key);
            __syncwarp();
        }
        if (w0 < w1) flush(lab);
    }
}

int dense_len_of(int Wt) { return (Wt + 127) / 128 * 128; }

size_t scan32_smem(int Wt, int nwarp) {
    return sizeof(float) * (size_t)(1 + nwarp) * dense_len_of(Wt) + sizeof(uint16_t) * (((size_t)Wt + 7) & ~size_t(7));
}

size_t step_smem(const FtRounds& a) {
    return sizeof(uint32_t) * ((size_t)a.eq_stride + a.nwords) + sizeof(uint32_t) * 2 * ((size_t)a.Wt / 32 + 2);
}

size_t scan_smem(int Wt, int copies) { return (size_t)(Wt + 1) * 16 * copies; }

constexpr size_t kStepSmem = 128 * 1024;    // the widest pool (14,143 genes) takes 60 KB
constexpr size_t kScan32Smem = 200 * 1024;
constexpr size_t kScanSmem = 221 * 1024;  // with the kernel's static shared memory (6 KB), under 227 KB

template <int C>
void launch_scan_c(const FtRounds& a, int k, bool one, bool x64, cudaStream_t s) {
    const size_t smem = scan_smem(a.Wt, C);
    auto kern = one ? (x64 ? ft_scan_kernel<C, 1, true> : ft_scan_kernel<C, 1, false>)
                    : (x64 ? ft_scan_kernel<C, 4, true> : ft_scan_kernel<C, 4, false>);
    kern<<<device_sm_count(), SCAN_NW * 32, smem, s>>>(a, k);
}

template <int C>
void scan_attr() {
    allow_smem(ft_scan_kernel<C, 4, true>, kScanSmem);
    allow_smem(ft_scan_kernel<C, 4, false>, kScanSmem);
    allow_smem(ft_scan_kernel<C, 1, true>, kScanSmem);
    allow_smem(ft_scan_kernel<C, 1, false>, kScanSmem);
}

}  // namespace

int ft_scan_copies(int Wt) {
    for (int c = 8; c >= 1; c >>= 1)
        if (scan_smem(Wt, c) <= kScanSmem) return c;
    return 0;
}

void launch_row_runs(const float* data, const int32_t* idx, const int32_t* ptr, uint32_t n_rows, int longest,
                     uint16_t* sorted, int32_t* n_groups, cudaStream_t s) {
    if (!n_rows) return;
    int cap = 32;
    while (cap < longest) cap <<= 1;
    const int wpb = std::max(1, std::min(8, (int)(96 * 1024 / (cap * 8))));
    const size_t smem = (size_t)wpb * cap * 8;
    allow_smem(row_runs_kernel, 96 * 1024);
    const unsigned blocks = std::min<unsigned>((n_rows + wpb - 1) / wpb, device_sm_count() * 8);
    row_runs_kernel<<<blocks, 32 * wpb, smem, s>>>(data, idx, ptr, n_rows, cap, sorted, n_groups);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_row_groups(const uint16_t* sorted, const int32_t* ptr, const int32_t* slot_row, const int32_t* blk_voff,
                       uint32_t n_slots, uint32_t pad, uint4* groups, cudaStream_t s) {
    if (!n_slots) return;
    row_groups_kernel<<<(n_slots + 127) / 128, 128, 0, s>>>(sorted, ptr, slot_row, blk_voff, n_slots, pad, groups);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_pair_masks(const uint32_t* ft_genes, const uint32_t* ft_idx, int L, int nwords, const int32_t* gene_thre,
                       uint32_t* mask, uint32_t* cut_mask, cudaStream_t s) {
    SGR_CUDA(cudaMemsetAsync(mask, 0, (size_t)L * L * nwords * sizeof(uint32_t), s));
    const int blocks = std::max(1, std::min((L * L + 7) / 8, device_sm_count() * 8));
    pair_mask_kernel<<<blocks, 256, 0, s>>>(ft_genes, ft_idx, L * L, nwords, mask);
    SGR_LAUNCH_CHECK();
    count_launch();
    if (!cut_mask) return;
    cut_mask_kernel<<<blocks, 256, sizeof(uint32_t) * 8 * nwords, s>>>(ft_genes, ft_idx, L * L, L, nwords, gene_thre,
                                                                     cut_mask);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_ft_cells(int n, const int32_t* list, const int* n_dev, int L, const uint8_t* flags,
                     const uint32_t* ctidx, int32_t* cells, int64_t* blk_off, int32_t* final_labels, int32_t* rounds,
                     unsigned long long* counter, unsigned long long* cand, cudaStream_t s) {
    if (n <= 0) return;
    ft_cells_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, list, n_dev, L, flags, ctidx, cells, blk_off, final_labels, rounds,
                                                    counter, cand);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_ft_sort_rows(int n, const float* data, const int32_t* idx, const int32_t* ptr, int longest,
                         uint16_t* s_gene, uint16_t* s_lo, uint16_t* s_hi, int* any_nan, cudaStream_t s) {
    if (n <= 0) return;
    int cap = 32;
    while (cap < longest) cap <<= 1;
    const int wpb = std::max(1, std::min(8, (int)(96 * 1024 / (cap * 8))));
    const size_t smem = (size_t)wpb * cap * 8;
    allow_smem(ft_sort_rows_kernel, 96 * 1024);
    const int blocks = std::min((n + wpb - 1) / wpb, device_sm_count() * 16);
    ft_sort_rows_kernel<<<blocks, 32 * wpb, smem, s>>>(n, data, idx, ptr, cap, s_gene, s_lo, s_hi, any_nan);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_ft_rows(const int32_t* cells, int n, const float* data, const int32_t* indices, const int32_t* indptr,
                    uint32_t n_cols, const int32_t* map, int Wt, int row_stride, uint16_t* s_gene, uint16_t* s_lo,
                    uint16_t* s_hi, int32_t* row_len, int* longest, bool mark_nan, cudaStream_t s) {
    if (n <= 0) return;
    const size_t smem = (size_t)Wt * 16;
    allow_smem(ft_rows_kernel, kScanSmem);
    ft_rows_kernel<<<std::min(n, device_sm_count() * 16), ROWS_NT, smem, s>>>(
        cells, n, data, indices, indptr, n_cols, map, Wt, row_stride, s_gene, s_lo, s_hi, row_len, longest,
        mark_nan);
    SGR_LAUNCH_CHECK();
    count_launch();
}

int ft_step_grid(int n) { return std::max(1, std::min(n, device_sm_count() * STEP_CTAS)); }

void ft_rounds_setup(int copies) {
    allow_smem(ft_step_kernel<STEP_NW>, kStepSmem);
    allow_smem(ft_step_kernel<STEP_NW_FEW>, kStepSmem);
    if (copies == 8) scan_attr<8>();
    else if (copies == 4) scan_attr<4>();
    else if (copies == 2) scan_attr<2>();
    else scan_attr<1>();
}

// Step k, and the quads of round k (quads; the FP32-order scan needs none).  n: no more cells than this.
void launch_ft_step(const FtRounds& a, int k, int n, bool quads, int32_t* scan_scratch, cudaStream_t s) {
    const int mode = !quads ? STEP_LIST : n <= kFtDirectCells ? STEP_QUAD : STEP_ORDER;
    // Few cells are ordered by counting the smaller keys (4,096 cells: 4,096 warps of 128 steps); more by a
    // counting sort on a few more key bits than the cells are many, at most 20.
    int bits = 0;
    if (mode == STEP_ORDER && n > 4096) {
        bits = 8;
        while (bits < 20 && (1 << bits) < 16 * n) ++bits;
        SGR_CUDA(cudaMemsetAsync(a.key_count, 0, sizeof(int32_t) << bits, s));
    }
    // With few cells a cell's own latency decides: four times the warps for its gene set and its labels'
    // quantiles.  With many labels a few cells hold on to most of them and take ten times as long as the
    // others, so there the line lies higher (whole calls in ms with the line at 2 and at 16 cells per SM, families of
    // labels, 20,000 reference cells: 2.45 / 2.92 for 2,000 cells of 30 labels, 6.10 / 6.38 of 60, 17.9 / 16.8 of 90,
    // 55.1 / 52.9 of 120; 57.9 / 58.8 for 16,384 cells of 66, 77.2 / 76.4 of 90).
    if (n <= (a.L > 64 ? 16 : 2) * device_sm_count())
        ft_step_kernel<STEP_NW_FEW><<<std::max(std::min(n, 2 * device_sm_count()), 1), STEP_NW_FEW * 32, step_smem(a),
                                      s>>>(a, k, mode, bits);
    else
        ft_step_kernel<STEP_NW><<<ft_step_grid(n), STEP_NW * 32, step_smem(a), s>>>(a, k, mode, bits);
    SGR_LAUNCH_CHECK();
    count_launch();
    if (mode != STEP_ORDER) return;
    if (bits) {
        int32_t* start = a.key_count + ((size_t)1 << bits);
        launch_exclusive_scan(a.key_count, start, 1u << bits, scan_scratch, s);
        ft_place_kernel<<<std::min((n + 255) / 256, device_sm_count() * 8), 256, 0, s>>>(a, k, bits, start);
    } else {
        ft_rank_kernel<<<std::max(1, std::min((n + 7) / 8, device_sm_count() * 8)), 256, 0, s>>>(a, k);
    }
    SGR_LAUNCH_CHECK();
    const int blocks = std::max(1, std::min((n + 4 * PLAN_NW - 1) / (4 * PLAN_NW), device_sm_count() * 4));
    ft_plan_kernel<<<blocks, PLAN_NW * 32, 0, s>>>(a, k);
    SGR_LAUNCH_CHECK();
    count_launch(2);
}

int ft_scan32_warps(int Wt) {
    for (int w = 8; w >= 1; --w)
        if (scan32_smem(Wt, w) <= kScan32Smem) return w;
    return 0;
}

void launch_ft_scan32(const FtRounds& a, int k, int n, bool nans, cudaStream_t s) {
    const int warps = ft_scan32_warps(a.Wt);
    const size_t smem = scan32_smem(a.Wt, warps);
    auto kern = nans ? ft_scan32_kernel<true> : ft_scan32_kernel<false>;
    allow_smem(kern, kScan32Smem);
    int per_sm = 0;
    SGR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem));
    const int grid = device_sm_count() * std::max(1, per_sm);
    // about eight items per CTA, so that the last ones do not leave the GPU idle
    const int parts = std::max(1, (8 * grid + n - 1) / std::max(n, 1));
    kern<<<grid, 32 * warps, smem, s>>>(a, k, dense_len_of(a.Wt), parts);
    SGR_LAUNCH_CHECK();
    count_launch();
}

void launch_ft_scan(const FtRounds& a, int k, int n, int copies, bool x64, cudaStream_t s) {
    const bool one = n <= kFtDirectCells;
    if (copies == 8) launch_scan_c<8>(a, k, one, x64, s);
    else if (copies == 4) launch_scan_c<4>(a, k, one, x64, s);
    else if (copies == 2) launch_scan_c<2>(a, k, one, x64, s);
    else launch_scan_c<1>(a, k, one, x64, s);
    SGR_LAUNCH_CHECK();
    count_launch();
}

}  // namespace sgr
