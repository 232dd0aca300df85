// Device helpers shared by the kernels: ordered float keys, warp sorts and searches, and the
// per-label quantile of the reference's percentile() (src/cusingler.cu:947-978 of
// STOmics/cusingler) by radix selection, with libstdc++'s sort order for NaN-bearing lists.
#pragma once

#include <climits>
#include <cstdint>

#include "kernels.cuh"
#include "stl_order.h"

namespace sgr {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// Unsigned keys in the order of the floats, the NaNs beyond the infinities on their sign's side.  The mask is computed:
// setting the sign bit of a float in so many words (u | 0x80000000) may be compiled to -|f|, which gives the NaN
// 0x7fffffff back as it is, a key near that of +0.
__device__ __forceinline__ uint32_t ord_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}

__device__ __forceinline__ float key_float(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// -0 and +0 are one value (the reference keys its per-row value codes with std::set<float>).
__device__ __forceinline__ float canon_zero(float v) {
    uint32_t u = __float_as_uint(v);
    return (u << 1) == 0 ? 0.0f : v;
}

// d = 128*h + l with l in [-64, 63]; s = h + l (the Karatsuba limb).
// Int8 limbs of a doubled centred rank d, written as planes (p0, l, s), with d = m * p0 + s:
//   w = 0: d = 128 h + l, l in [-64, 63], p0 = h, s = h + l (m = 127);
//   w > 0: d = C h + l with C = w^2 + 1, l in [-C/2, C - 1 - C/2], p0 = w h, s = h + l (m = w).
// The second split lets the exact product use two accumulators: d d' = C (p0 p0' + s s') - (C-1) l l'.
// The host picks w so that every limb of |d| < G fits int8.
__device__ __forceinline__ void split_limbs(int d, int w, int& p0, int& l, int& s) {
    if (w == 0) {
        l = ((d + 64) & 127) - 64;
        p0 = (d - l) >> 7;
        s = p0 + l;
        return;
    }
    const int C = w * w + 1, hc = C >> 1;
    const int h = (d + hc + 4096 * C) / C - 4096;  // floor((d + hc) / C) for |d| < 4096 C
    l = d - C * h;
    s = h + l;
    p0 = w * h;
}


__device__ __forceinline__ int64_t warp_sum_i64(int64_t v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

__device__ __forceinline__ int lower_hi(const uint64_t* keys, int n, uint32_t hv) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if ((uint32_t)(keys[mid] >> 32) < hv) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ int upper_hi(const uint64_t* keys, int n, uint32_t hv) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if ((uint32_t)(keys[mid] >> 32) <= hv) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Ascending bitonic sort of n (power of two) keys in shared memory by one warp.
__device__ void warp_bitonic(uint64_t* keys, int n, int lane) {
    for (int size = 2; size <= n; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = lane; t < (n >> 1); t += 32) {
                int i = 2 * t - (t & (stride - 1));
                int j = i + stride;
                uint64_t a = keys[i], b = keys[j];
                bool up = (i & size) == 0;
                if ((a > b) == up) {
                    keys[i] = b;
                    keys[j] = a;
                }
            }
            __syncwarp();
        }
    }
}

__device__ __forceinline__ float interp(float p, float prev_index, float step, float a, float b) {
    // (p - prev_index) * (b - a) / step + a, each operation rounded once (src/cusingler.cu:975)
    return __fadd_rn(__fdiv_rn(__fmul_rn(__fsub_rn(p, prev_index), __fsub_rn(b, a)), step), a);
}

__device__ __forceinline__ int warp_incl_scan(int x, int lane) {
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Key of the j-th smallest (0-based) of v[0..n) by 4 passes of an 8-bit radix histogram.
// `common` high bits are shared by every key (from the list's minimum and maximum): the radix
// passes start below them.
__device__ uint32_t warp_select(const float* v, int n, int j, int* hist, int lane, uint32_t kmin = 0,
                                int common = 0) {
    uint32_t mask = common ? ~0u << (32 - common) : 0u;
    uint32_t prefix = kmin & mask;
    const int low = 32 - common;  // bits still to resolve
    int shift = low - 8;
    for (;; shift -= 8) {
        if (shift < 0) shift = 0;
        for (int b = lane; b < 256; b += 32) hist[b] = 0;
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            const uint32_t u = ord_key(v[i]);
            if ((u & mask) == prefix) atomicAdd(&hist[(u >> shift) & 255], 1);
        }
        __syncwarp();
        int c[8], s = 0;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            c[t] = hist[8 * lane + t];
            s += c[t];
        }
        const int incl = warp_incl_scan(s, lane), excl = incl - s;
        const unsigned own = __ballot_sync(FULL, excl <= j && j < incl);
        const int src = __ffs(own) - 1;
        int bin = 0, before = 0;
        if (lane == src) {
            int acc = excl;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                if (j < acc + c[t]) {
                    bin = 8 * lane + t;
                    before = acc;
                    break;
                }
                acc += c[t];
            }
        }
        bin = __shfl_sync(FULL, bin, src);
        before = __shfl_sync(FULL, before, src);
        j -= before;
        prefix |= (uint32_t)bin << shift;
        mask |= 0xffu << shift;
        __syncwarp();
        if (shift == 0) break;
    }
    return prefix;
}

__device__ __forceinline__ uint32_t warp_min_u32(uint32_t x) { return __reduce_min_sync(FULL, x); }
__device__ __forceinline__ uint32_t warp_max_u32(uint32_t x) { return __reduce_max_sync(FULL, x); }

// Keys of order statistics j and j+1 (0-based) of v[0..n) (no NaN, kmin < kmax) by one warp: a
// 256-bin histogram over a monotone linear map of [min, max] locates the bin holding statistic j;
// that bin's keys (at most 256) are compacted into `buf` (the histogram's memory, 16-byte aligned) and sorted.
// Returns false (nothing decided) when the bin is larger than 256 or the range is degenerate.
__device__ bool bucket_select(const float* v, int n, int j, int* hist, int lane, uint32_t kmin, uint32_t kmax,
                              uint32_t* ka, uint32_t* kb) {
    const float fmin = key_float(kmin), fmax = key_float(kmax);
    const float span = fmax - fmin;
    if (!(span > 1e-30f) || !(span < 1e30f)) return false;
    // The bin of x is round-to-nearest(255 * y) with y = (x - min) / span saturated to [0, 1], so that a value
    // outside [min, max] (extremes that do not match the list) still lands in a bin.  The second FMA's result
    // lies in [2^23, 2^23 + 255], where floats are the integers: bits = 0x4B000000 + bin.  The map from x to
    // those bits is monotone non-decreasing for any positive scale, which is all the selection needs (both
    // passes use the same map).
    constexpr int B0 = 0x4B000000;
    const float scale = __fdividef(1.0f, span);
    const float shift = -fmin * scale;
    auto bin_bits = [&](float x) {
        return __float_as_int(fmaf(__saturatef(fmaf(x, scale, shift)), 255.0f, 8388608.0f));
    };
    int4* h4 = reinterpret_cast<int4*>(hist);
    h4[lane] = make_int4(0, 0, 0, 0);
    h4[32 + lane] = make_int4(0, 0, 0, 0);
    __syncwarp();
    int i = lane;
    for (; i + 96 < n; i += 128) {  // four independent loads in flight per lane
        const float x0 = v[i], x1 = v[i + 32], x2 = v[i + 64], x3 = v[i + 96];
        atomicAdd(&hist[bin_bits(x0) - B0], 1);
        atomicAdd(&hist[bin_bits(x1) - B0], 1);
        atomicAdd(&hist[bin_bits(x2) - B0], 1);
        atomicAdd(&hist[bin_bits(x3) - B0], 1);
    }
    for (; i < n; i += 32) atomicAdd(&hist[bin_bits(v[i]) - B0], 1);
    __syncwarp();
    // Lane l holds bins 4 l .. 4 l + 3 of each half of the histogram (conflict-free 16-byte loads).  The half
    // with statistic j is known from the first half's total, and only that half's counts are scanned.
    const int4 ch[2] = {h4[lane], h4[32 + lane]};
    const int s0 = ch[0].x + ch[0].y + ch[0].z + ch[0].w, s1 = ch[1].x + ch[1].y + ch[1].z + ch[1].w;
    const int tot0 = __reduce_add_sync(FULL, s0);
    const bool upper = j >= tot0;
    const int4 c = upper ? ch[1] : ch[0];
    const int s = upper ? s1 : s0;
    const int incl = warp_incl_scan(s, lane) + (upper ? tot0 : 0), excl = incl - s;
    const unsigned own = __ballot_sync(FULL, excl <= j && j < incl);
    const int src = __ffs(own) - 1;
    const int e1 = excl + c.x, e2 = e1 + c.y, e3 = e2 + c.z;
    const bool p1 = j >= e1, p2 = j >= e2, p3 = j >= e3;
    int bin = (upper ? 128 : 0) + 4 * lane + (p1 ? 1 : 0) + (p2 ? 1 : 0) + (p3 ? 1 : 0);
    int before = p3 ? e3 : p2 ? e2 : p1 ? e1 : excl;
    int cnt = p3 ? c.w : p2 ? c.z : p1 ? c.y : c.x;
    bin = __shfl_sync(FULL, bin, src);
    before = __shfl_sync(FULL, before, src);
    cnt = __shfl_sync(FULL, cnt, src);
    if (cnt > 256) return false;
    // when statistic j is the last of its bin and j + 1 exists, statistic j + 1 is the smallest value
    // of the next non-empty bin: collect that bin too (the bins between are empty)
    int nb = -1, total = cnt;
    if (j + 1 >= before + cnt && j + 1 < n) {
        int cand = 256, ccand = 0;
        auto look = [&](int b, int count) {
            if (cand == 256 && b > bin && count > 0) {
                cand = b;
                ccand = count;
            }
        };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            look(128 * h + 4 * lane, ch[h].x);
            look(128 * h + 4 * lane + 1, ch[h].y);
            look(128 * h + 4 * lane + 2, ch[h].z);
            look(128 * h + 4 * lane + 3, ch[h].w);
        }
        nb = __reduce_min_sync(FULL, cand);
        const int cnb = __reduce_add_sync(FULL, cand == nb ? ccand : 0);
        if (cnt + cnb <= 256) total = cnt + cnb;
        else nb = -1;
    }
    __syncwarp();
    // Collect the values of bins bin..last (the bins between bin and nb are empty), compared on the map's
    // bits.  Raw float bits are stored and turned into order keys afterwards.
    const int last = nb >= 0 ? nb : bin;
    const unsigned lo = (unsigned)(B0 + bin), width = (unsigned)(last - bin);
    uint32_t* buf = reinterpret_cast<uint32_t*>(hist);
    int w = 0;
    const unsigned lt = (1u << lane) - 1u;
    int base = 0;
    for (; base + 128 <= n; base += 128) {  // four 32-value chunks per step
        float x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = v[base + 32 * t + lane];
        bool in[4];
        unsigned m[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            in[t] = (unsigned)bin_bits(x[t]) - lo <= width;
            m[t] = __ballot_sync(FULL, in[t]);
        }
        const int w1 = w + __popc(m[0]), w2 = w1 + __popc(m[1]), w3 = w2 + __popc(m[2]);
        if (in[0]) buf[w + __popc(m[0] & lt)] = __float_as_uint(x[0]);
        if (in[1]) buf[w1 + __popc(m[1] & lt)] = __float_as_uint(x[1]);
        if (in[2]) buf[w2 + __popc(m[2] & lt)] = __float_as_uint(x[2]);
        if (in[3]) buf[w3 + __popc(m[3] & lt)] = __float_as_uint(x[3]);
        w = w3 + __popc(m[3]);
    }
    for (; base < n; base += 32) {
        const int i0 = base + lane;
        const float x0 = i0 < n ? v[i0] : 0.f;
        const bool in0 = i0 < n && (unsigned)bin_bits(x0) - lo <= width;
        const unsigned m0 = __ballot_sync(FULL, in0);
        if (in0) buf[w + __popc(m0 & lt)] = __float_as_uint(x0);
        w += __popc(m0);
    }
    __syncwarp();
    const int r = j - before;  // statistic j is the r-th smallest collected key (r < cnt <= total)
    bool have_b = r + 1 < total;
    if (total <= 32) {
        // one key per lane; with le = the number of collected keys not above it, statistic r is the smallest
        // key with le > r, and r + 1 the smallest with le > r + 1
        const uint32_t key = lane < total ? ord_key(__uint_as_float(buf[lane])) : 0xffffffffu;
        int le = 0;
        for (int t = 0; t < total; ++t) le += __shfl_sync(FULL, key, t) <= key;
        *ka = __reduce_min_sync(FULL, lane < total && le > r ? key : 0xffffffffu);
        if (have_b) *kb = __reduce_min_sync(FULL, lane < total && le > r + 1 ? key : 0xffffffffu);
    } else {
        for (int i = lane; i < total; i += 32) buf[i] = ord_key(__uint_as_float(buf[i]));
        int np = 1;
        while (np < total) np <<= 1;
        for (int i = total + lane; i < np; i += 32) buf[i] = 0xffffffffu;
        __syncwarp();
        for (int size = 2; size <= np; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = lane; t < (np >> 1); t += 32) {
                    const int a = 2 * t - (t & (stride - 1)), b = a + stride;
                    const uint32_t x = buf[a], y = buf[b];
                    if ((x > y) == ((a & size) == 0)) {
                        buf[a] = y;
                        buf[b] = x;
                    }
                }
                __syncwarp();
            }
        *ka = buf[r];
        if (have_b) *kb = buf[r + 1];
    }
    if (!have_b) {  // statistic j + 1 lies beyond the collected bins: the smallest key above ka
        uint32_t nxt = 0xffffffffu;
        for (int i = lane; i < n; i += 32) {
            const uint32_t u = ord_key(v[i]);
            if (u > *ka) nxt = min(nxt, u);
        }
        *kb = __reduce_min_sync(FULL, nxt);
    }
    __syncwarp();
    return true;
}

// quantile_warp after its min / max / NaN pass: kmin, kmax are the warp-wide extreme order keys of
// the list and nan whether it holds a NaN (all lanes agree).  Lists holding NaN are sorted exactly as
// libstdc++ would, in `scratch` (n floats), by lane 0.
__device__ float quantile_warp_core(const float* v, const LabelQ& lq, float p, int* hist, float* scratch, int lane,
                                    int* status, uint32_t kmin, uint32_t kmax, bool nan) {
    const int n = lq.len;
    if (nan) {
        float r = 0.f;
        if (scratch == nullptr) {
            if (lane == 0) atomicOr(status, 8);
            return __int_as_float(0x7fffffff);
        }
        for (int i = lane; i < n; i += 32) scratch[i] = v[i];
        __syncwarp();
        if (lane == 0) {
            int oob = 0;
            stl::sort(scratch, n, &oob);
            if (oob) atomicOr(status, 4);
            if (lq.kind == 1) r = scratch[0];
            else if (lq.kind == 2) r = scratch[n - 1];
            else r = interp(p, lq.prev_index, lq.step, scratch[lq.k - 1], scratch[lq.k]);
        }
        __syncwarp();
        return __shfl_sync(FULL, r, 0);
    }
    if (lq.kind == 1) return key_float(kmin);
    if (lq.kind == 2) return key_float(kmax);
    if (kmin == kmax) return interp(p, lq.prev_index, lq.step, key_float(kmin), key_float(kmin));
    uint32_t ka, kb;
    if (bucket_select(v, n, lq.k - 1, hist, lane, kmin, kmax, &ka, &kb))
        return interp(p, lq.prev_index, lq.step, key_float(ka), key_float(kb));
    ka = warp_select(v, n, lq.k - 1, hist, lane);
    int le = 0;
    uint32_t nxt = 0xffffffffu;
    for (int i = lane; i < n; i += 32) {
        const uint32_t u = ord_key(v[i]);
        le += u <= ka;
        if (u > ka) nxt = min(nxt, u);
    }
    le = __reduce_add_sync(FULL, le);
    nxt = warp_min_u32(nxt);
    kb = le > lq.k ? ka : nxt;
    return interp(p, lq.prev_index, lq.step, key_float(ka), key_float(kb));
}

// The reference's percentile(v, n, p) (src/cusingler.cu:947-978) for one score list, by one warp.
__device__ float quantile_warp(const float* v, const LabelQ& lq, float p, int* hist, float* scratch, int lane,
                               int* status) {
    const int n = lq.len;
    if (lq.kind == 0) return v[0];
    bool nan = false;
    uint32_t mn0 = 0xffffffffu, mn1 = 0xffffffffu, mx0 = 0u, mx1 = 0u;
    int i = lane;
    for (; i + 32 < n; i += 64) {  // two independent chains per lane
        const float x0 = v[i], x1 = v[i + 32];
        nan |= (x0 != x0) | (x1 != x1);
        const uint32_t u0 = ord_key(x0), u1 = ord_key(x1);
        mn0 = min(mn0, u0);
        mx0 = max(mx0, u0);
        mn1 = min(mn1, u1);
        mx1 = max(mx1, u1);
    }
    if (i < n) {
        const float x = v[i];
        nan |= x != x;
        const uint32_t u = ord_key(x);
        mn0 = min(mn0, u);
        mx0 = max(mx0, u);
    }
    nan = __any_sync(FULL, nan);
    const uint32_t kmin = __reduce_min_sync(FULL, min(mn0, mn1));
    const uint32_t kmax = __reduce_max_sync(FULL, max(mx0, mx1));
    return quantile_warp_core(v, lq, p, hist, scratch, lane, status, kmin, kmax, nan);
}


}  // namespace
}  // namespace sgr
