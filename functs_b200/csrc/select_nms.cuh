// Block-level building blocks for "mask -> nonzero -> stable descending sort -> top-k -> greedy NMS".
//
// All of it is integer / exactly-rounded fp32 work: the selection orders 64-bit keys (score bits, inverted
// index), and the IoU test reproduces, operation by operation, what a scalar CPU loop over
//   inter / (area_i + area_j - inter) > thr
// computes in fp32 (every product, sum and quotient rounded on its own; no fused multiply-add).
#pragma once

#include "common.cuh"

namespace fb {

constexpr int kHistBits = 11;
constexpr int kHistBins = 1 << kHistBits;
constexpr int kBinListCap = 1024;  // keys of the boundary bin that are finished by a local sort

// ---- coarse score histogram shared by a candidate producer and the binned top-k ----------------------------
// Positive fp32 bit patterns are ordered like their values, so (bits - bits(thr)) >> shift is a monotone bucketing
// of the scores above thr; everything at or above the last bucket is clamped into it.
struct HistParams {
    uint32_t base;
    int shift;
};

inline HistParams hist_params_for(float thr) {
    HistParams h;
    uint32_t one_bits = 0x3F800000u;  // scores are products of probabilities: <= 1.0
    float t = thr > 0.0f ? thr : 0.0f;
    uint32_t b;
    static_assert(sizeof(float) == 4, "fp32");
    __builtin_memcpy(&b, &t, 4);
    h.base = b;
    uint32_t diff = one_bits > b ? one_bits - b : 1u;
    h.shift = 0;
    while (((diff - 1u) >> h.shift) > static_cast<uint32_t>(kHistBins - 1)) ++h.shift;
    return h;
}

#ifdef __CUDACC__
__device__ __forceinline__ int hist_digit(uint64_t key, uint32_t base, int shift) {
    uint32_t bits = static_cast<uint32_t>(key >> 32);
    uint32_t d = bits > base ? (bits - base) >> shift : 0u;
    return d > static_cast<uint32_t>(kHistBins - 1) ? kHistBins - 1 : static_cast<int>(d);
}
#endif

// ---- bitonic sort, descending, on `n` (power of two) 64-bit keys in shared memory -------------------
template <int NT>
__device__ __forceinline__ void bitonic_sort_desc(uint64_t* s, int n) {
    // one thread per compare-exchange pair: pair p of a (k, j) step is (i, i | j) with bit j of i clear
    const int pairs = n >> 1;
    for (int k = 2; k <= n; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int p = threadIdx.x; p < pairs; p += NT) {
                const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));
                const int ixj = i | j;
                const uint64_t a = s[i], b = s[ixj];
                const bool desc_seg = (i & k) == 0;
                if (desc_seg ? (a < b) : (a > b)) {
                    s[i] = b;
                    s[ixj] = a;
                }
            }
            __syncthreads();
        }
    }
}

__device__ __forceinline__ int next_pow2(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

template <int SELCAP>
struct SelectSmem {
    __align__(16) uint64_t sel[SELCAP];
    uint64_t binlist[kBinListCap];
    int hist[kHistBins];
    uint64_t red_min[32];
    uint64_t red_max[32];
    int red_cnt[32];
    // broadcast slots
    uint64_t kmin, kmax;
    int nvalid;
    int digit, above, inbin;
    int sel_cnt, bin_cnt;
};

// Adds 1 to hist[d] for every lane with valid != 0, one shared-memory atomic per distinct digit per warp.
__device__ __forceinline__ void warp_hist_add(int* hist, int d, bool valid) {
    int dd = valid ? d : -1;
    unsigned peers = __match_any_sync(kFullMask, dd);
    if (valid) {
        int leader = __ffs(peers) - 1;
        if ((threadIdx.x & 31) == leader) atomicAdd(&hist[d], __popc(peers));
    }
}

// Selects the `topk` largest non-zero keys among key(0..n-1) and leaves them sorted descending in sm.sel.
// Returns the number selected (min(#non-zero keys, topk)).  Keys must be distinct; key(i) == 0 means "absent".
// All NT threads of the block must call it; SELCAP is a power of two >= topk and NT a multiple of 32.
template <int NT, int SELCAP, int UNROLL, class KeyFn>
__device__ int block_select_topk(KeyFn key, int n, int topk, SelectSmem<SELCAP>& sm) {
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;

    // pass 0: count, min and max of the present keys
    uint64_t lmin = ~0ull, lmax = 0ull;
    int lcnt = 0;
    for (int base = 0; base < n; base += NT * UNROLL) {
        uint64_t k[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            int i = base + u * NT + tid;
            k[u] = (i < n) ? key(i) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            if (k[u] != 0ull) {
                lmin = k[u] < lmin ? k[u] : lmin;
                lmax = k[u] > lmax ? k[u] : lmax;
                ++lcnt;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        uint64_t omin = __shfl_xor_sync(kFullMask, lmin, o);
        uint64_t omax = __shfl_xor_sync(kFullMask, lmax, o);
        lcnt += __shfl_xor_sync(kFullMask, lcnt, o);
        lmin = omin < lmin ? omin : lmin;
        lmax = omax > lmax ? omax : lmax;
    }
    if (lane == 0) {
        sm.red_min[warp] = lmin;
        sm.red_max[warp] = lmax;
        sm.red_cnt[warp] = lcnt;
    }
    if (tid == 0) {
        sm.sel_cnt = 0;
        sm.bin_cnt = 0;
    }
    __syncthreads();
    if (warp == 0) {
        uint64_t a = lane < NW ? sm.red_min[lane] : ~0ull;
        uint64_t b = lane < NW ? sm.red_max[lane] : 0ull;
        int c = lane < NW ? sm.red_cnt[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            uint64_t oa = __shfl_xor_sync(kFullMask, a, o);
            uint64_t ob = __shfl_xor_sync(kFullMask, b, o);
            c += __shfl_xor_sync(kFullMask, c, o);
            a = oa < a ? oa : a;
            b = ob > b ? ob : b;
        }
        if (lane == 0) {
            sm.kmin = a;
            sm.kmax = b;
            sm.nvalid = c;
        }
    }
    __syncthreads();
    const int nvalid = sm.nvalid;
    const uint64_t kmin = sm.kmin, kmax = sm.kmax;
    if (nvalid == 0) return 0;

    int sort_n;
    int result;
    if (nvalid <= topk) {
        // everything is selected
        for (int base = 0; base < n; base += NT * UNROLL) {
            uint64_t k[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                int i = base + u * NT + tid;
                k[u] = (i < n) ? key(i) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (k[u] != 0ull) {
                    int pos = atomicAdd(&sm.sel_cnt, 1);
                    if (pos < SELCAP) sm.sel[pos] = k[u];
                }
            }
        }
        __syncthreads();
        result = nvalid;
    } else {
        // radix descent from the highest bit in which the keys differ
        uint64_t diff = kmin ^ kmax;  // != 0 because nvalid >= 2 distinct keys
        int hb = 63 - __clzll(static_cast<long long>(diff));
        uint64_t mask = (hb >= 63) ? 0ull : ~((1ull << (hb + 1)) - 1ull);
        uint64_t prefix = kmax & mask;
        int want = topk;
        while (true) {
            int shift = hb - kHistBits + 1;
            if (shift < 0) shift = 0;
            const int nb = hb - shift + 1;
            const int nbins = 1 << nb;
            for (int i = tid; i < nbins; i += NT) sm.hist[i] = 0;
            __syncthreads();
            for (int base = 0; base < n; base += NT * UNROLL) {
                uint64_t k[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    int i = base + u * NT + tid;
                    k[u] = (i < n) ? key(i) : 0ull;
                }
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    bool v = (k[u] != 0ull) && ((k[u] & mask) == prefix);
                    int d = static_cast<int>((k[u] >> shift) & static_cast<uint64_t>(nbins - 1));
                    warp_hist_add(sm.hist, d, v);
                }
            }
            __syncthreads();
            // warp 0 finds the largest digit d with (count of digits >= d) >= want
            if (warp == 0) {
                const int per = (nbins + 31) / 32;  // bins per lane, lane 31 holds the highest bins
                int lo = lane * per, hi = lo + per;
                if (hi > nbins) hi = nbins;
                int s = 0;
                for (int i = lo; i < hi; ++i) s += sm.hist[i];
                // suffix sum over lanes: suf = sum of s over lanes > lane
                int incl = s;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    int t = __shfl_down_sync(kFullMask, incl, o);
                    if (lane + o < 32) incl += t;
                }
                int suf = incl - s;  // strictly higher lanes
                bool mine = (suf < want) && (incl >= want);
                if (mine) {
                    int cum = suf;
                    int d = hi - 1;
                    for (; d >= lo; --d) {
                        int h = sm.hist[d];
                        if (cum + h >= want) break;
                        cum += h;
                    }
                    sm.digit = d;
                    sm.above = cum;
                    sm.inbin = sm.hist[d];
                }
            }
            __syncthreads();
            const int digit = sm.digit, above = sm.above, inbin = sm.inbin;
            want -= above;
            mask |= static_cast<uint64_t>(nbins - 1) << shift;
            prefix |= static_cast<uint64_t>(digit) << shift;
            hb = shift - 1;
            if (inbin == want || shift == 0 || inbin <= kBinListCap) break;
            __syncthreads();
        }
        // collect: strictly above the boundary bin -> sel; inside the bin -> binlist
        for (int base = 0; base < n; base += NT * UNROLL) {
            uint64_t k[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                int i = base + u * NT + tid;
                k[u] = (i < n) ? key(i) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (k[u] != 0ull) {
                    uint64_t km = k[u] & mask;
                    if (km > prefix) {
                        int pos = atomicAdd(&sm.sel_cnt, 1);
                        if (pos < SELCAP) sm.sel[pos] = k[u];
                    } else if (km == prefix) {
                        int pos = atomicAdd(&sm.bin_cnt, 1);
                        if (pos < kBinListCap) sm.binlist[pos] = k[u];
                    }
                }
            }
        }
        __syncthreads();
        int bc = sm.bin_cnt < kBinListCap ? sm.bin_cnt : kBinListCap;
        int bn = next_pow2(bc);
        for (int i = bc + tid; i < bn; i += NT) sm.binlist[i] = 0ull;
        __syncthreads();
        bitonic_sort_desc<NT>(sm.binlist, bn);
        const int have = sm.sel_cnt;  // == topk - want
        for (int i = tid; i < want && i < bc; i += NT) {
            if (have + i < SELCAP) sm.sel[have + i] = sm.binlist[i];
        }
        __syncthreads();
        result = topk;
    }
    sort_n = next_pow2(result);
    for (int i = result + tid; i < sort_n; i += NT) sm.sel[i] = 0ull;
    __syncthreads();
    bitonic_sort_desc<NT>(sm.sel, sort_n);
    return result;
}

// The exact generic selection as an out-of-line call: it is the rare way out of the binned selections below, and its
// code (three passes, two sorts) should not sit in the middle of their instruction stream.
template <int NT, int SELCAP, int UNROLL, class KeyFn>
__device__ __noinline__ int block_select_topk_outlined(KeyFn key, int n, int topk, SelectSmem<SELCAP>* sm) {
    return block_select_topk<NT, SELCAP, UNROLL>(key, n, topk, *sm);
}

// Same result as block_select_topk, but in two passes for keys whose scores lie above a known threshold: one pass
// fills the coarse score histogram (hist_digit), the second collects the keys above / inside the boundary bucket,
// and only the boundary bucket is sorted.  Falls back to block_select_topk when that bucket exceeds kBinListCap.
// KeyFn::kDenseScores marks a key function over a plain fp32 score array (members s, thr, vec4: the array may be read
// four at a time): the two passes then read the scores directly and build keys only for the elements they keep.
template <int NT, int SELCAP, int UNROLL, class KeyFn>
__device__ int block_select_topk_binned(KeyFn key, int n, int topk, uint32_t hist_base, int hist_shift,
                                        SelectSmem<SELCAP>& sm) {
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kHistBins; i += NT) sm.hist[i] = 0;
    if (tid == 0) {
        sm.sel_cnt = 0;
        sm.bin_cnt = 0;
        sm.digit = -1;
        sm.above = 0;
        sm.inbin = 0;
        sm.nvalid = 0;
    }
    __syncthreads();
    if constexpr (KeyFn::kDenseScores) {
        // fp32 scores, four per load: an element below the threshold costs a compare, nothing else
        const float thr = key.thr;
        auto add = [&](float v) {
            if (v > thr) atomicAdd(&sm.hist[hist_digit(static_cast<uint64_t>(__float_as_uint(v)) << 32, hist_base, hist_shift)], 1);
        };
        const int n4 = key.vec4 ? (n >> 2) : 0;
        const float4* s4 = reinterpret_cast<const float4*>(key.s);
        for (int c = tid; c < n4; c += NT) {
            const float4 q = s4[c];
            add(q.x);
            add(q.y);
            add(q.z);
            add(q.w);
        }
        for (int i = 4 * n4 + tid; i < n; i += NT) add(key.s[i]);
    } else {
        for (int base = 0; base < n; base += NT * UNROLL) {
            uint64_t k[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int i = base + u * NT + tid;
                k[u] = (i < n) ? key(i) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (k[u] != 0ull) atomicAdd(&sm.hist[hist_digit(k[u], hist_base, hist_shift)], 1);
            }
        }
    }
    __syncthreads();
    // boundary bucket: the largest digit d with (keys in buckets >= d) >= topk.  Every thread sums its share of the
    // buckets (higher thread = higher buckets), suffix sums over the block locate the thread that holds the boundary
    {
        static_assert(kHistBins % NT == 0, "the histogram must split evenly over the block");
        constexpr int per = kHistBins / NT;
        int h[per];
        int s = 0;
#pragma unroll
        for (int k = 0; k < per; ++k) {
            h[k] = sm.hist[tid * per + k];
            s += h[k];
        }
        int incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_down_sync(kFullMask, incl, o);
            if (lane + o < 32) incl += t;
        }
        if (lane == 0) sm.red_cnt[warp] = incl;
        __syncthreads();
        int higher = 0, total = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            const int c = sm.red_cnt[w];
            total += c;
            higher += (w > warp) ? c : 0;
        }
        incl += higher;
        const int suf = incl - s;
        if (tid == 0) sm.nvalid = total;
        // the counts are not needed again: every bucket now holds the number of keys in the buckets above it, which
        // is where its keys start in the final descending order
        {
            int above_k = suf;
#pragma unroll
            for (int k = per - 1; k >= 0; --k) {
                sm.hist[tid * per + k] = above_k;
                above_k += h[k];
            }
        }
        if (total > topk && suf < topk && incl >= topk) {
            int cum = suf, dsel = 0, hsel = 0, above = 0;
            bool found = false;
#pragma unroll
            for (int k = per - 1; k >= 0; --k) {  // incl >= topk: one of the buckets is the boundary
                if (!found) {
                    if (cum + h[k] >= topk) {
                        found = true;
                        dsel = k;
                        hsel = h[k];
                        above = cum;
                    } else {
                        cum += h[k];
                    }
                }
            }
            sm.digit = tid * per + dsel;
            sm.above = above;
            sm.inbin = hsel;
        }
    }
    __syncthreads();
    const int nvalid = sm.nvalid;
    if (nvalid == 0) return 0;
    const int dstar = sm.digit;  // -1: everything is selected
    if (sm.inbin > kBinListCap) {
        __syncthreads();
        return block_select_topk_outlined<NT, SELCAP, UNROLL>(key, n, topk, &sm);
    }
    auto place = [&](uint64_t k) {
        const int d = hist_digit(k, hist_base, hist_shift);
        if (d > dstar) {
            const int pos = atomicAdd(&sm.sel_cnt, 1);
            if (pos < SELCAP) sm.sel[pos] = k;
        } else if (d == dstar) {
            const int pos = atomicAdd(&sm.bin_cnt, 1);
            if (pos < kBinListCap) sm.binlist[pos] = k;
        }
    };
    if constexpr (KeyFn::kDenseScores) {
        // a score can only reach bucket dstar or above if its bits reach the bucket's first value: one integer
        // compare per element, the few that pass take the exact path
        const float thr = key.thr;
        const uint32_t lo_bits = dstar > 0 ? hist_base + (static_cast<uint32_t>(dstar) << hist_shift) : 0u;
        auto look = [&](float v, int i) {
            if (v > thr && __float_as_uint(v) >= lo_bits) place(make_key(v, static_cast<uint32_t>(i)));
        };
        const int n4 = key.vec4 ? (n >> 2) : 0;
        const float4* s4 = reinterpret_cast<const float4*>(key.s);
        for (int c = tid; c < n4; c += NT) {
            const float4 q = s4[c];
            look(q.x, 4 * c);
            look(q.y, 4 * c + 1);
            look(q.z, 4 * c + 2);
            look(q.w, 4 * c + 3);
        }
        for (int i = 4 * n4 + tid; i < n; i += NT) look(key.s[i], i);
    } else {
        for (int base = 0; base < n; base += NT * UNROLL) {
            uint64_t k[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int i = base + u * NT + tid;
                k[u] = (i < n) ? key(i) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                if (k[u] != 0ull) place(k[u]);
            }
        }
    }
    __syncthreads();
    const int result = nvalid < topk ? nvalid : topk;
    if (dstar >= 0) {
        const int bc = sm.bin_cnt;
        const int bn = next_pow2(bc);
        for (int i = bc + tid; i < bn; i += NT) sm.binlist[i] = 0ull;
        __syncthreads();
        bitonic_sort_desc<NT>(sm.binlist, bn);
        const int have = sm.sel_cnt;
        const int want = topk - have;
        for (int i = tid; i < want && i < bc; i += NT) {
            if (have + i < SELCAP) sm.sel[have + i] = sm.binlist[i];
        }
        __syncthreads();
    }
    // Final order.  The boundary bucket's share already sits sorted behind the `have` keys of the higher buckets.
    // Those are ordered by a counting sort: a key of bucket d goes to the run that starts at hist[d] (keys in higher
    // buckets), in arrival order; afterwards hist[d] is the run's end and hist[d + 1] its start, and every key
    // counts the larger keys of its own run (a run holds a key or two unless many scores are nearly equal).
    static_assert(SELCAP <= kBinListCap, "the boundary list doubles as the scatter target");
    {
        const int have = dstar >= 0 ? (sm.sel_cnt < SELCAP ? sm.sel_cnt : SELCAP) : result;
        uint64_t* tmp = sm.binlist;  // not needed any more
        __syncthreads();
        for (int i = tid; i < have; i += NT) {
            const uint64_t k = sm.sel[i];
            tmp[atomicAdd(&sm.hist[hist_digit(k, hist_base, hist_shift)], 1)] = k;
        }
        __syncthreads();
        for (int i = tid; i < have; i += NT) {
            const uint64_t mine = tmp[i];
            const int d = hist_digit(mine, hist_base, hist_shift);
            const int lo = d + 1 < kHistBins ? sm.hist[d + 1] : 0, hi = sm.hist[d];
            int rank = lo;
            for (int q = lo; q < hi; ++q) rank += (tmp[q] > mine) ? 1 : 0;
            sm.sel[rank] = mine;
        }
        __syncthreads();
    }
    return result;
}

// A plain fp32 score array as a key function (key = score above thr, index); kDenseScores lets the binned selection
// read the array four scores at a time when vec4 says it is 16-byte aligned.
struct DenseScores {
    static constexpr bool kDenseScores = true;
    const float* s;
    float thr;
    bool vec4;
    __device__ __forceinline__ uint64_t operator()(int i) const {
        const float v = s[i];
        return (v > thr) ? make_key(v, static_cast<uint32_t>(i)) : 0ull;
    }
};

// Keys that already sit in a list (shared memory): the non-dense form of the key functions above.
struct ListKeys {
    static constexpr bool kDenseScores = false;
    const uint64_t* k;
    __device__ __forceinline__ uint64_t operator()(int i) const { return k[i]; }
};

constexpr int kCandCap = 1024;  // candidate keys block_select_topk_sampled may collect before it gives up

// the two-pass selection over a whole score array, out of line (the sampled selection's rare way out)
template <int NT, int SELCAP>
__device__ __noinline__ int block_select_dense_outlined(const float* s, bool vec4, float thr, int n, int topk, uint32_t hist_base,
                                                        int hist_shift, SelectSmem<SELCAP>* sm) {
    return block_select_topk_binned<NT, SELCAP, 8>(DenseScores{s, thr, vec4}, n, topk, hist_base, hist_shift, *sm);
}

// The `want` largest of n keys, in order.  room: the next power of two.
template <int NT>
__device__ __noinline__ void block_sort_bucket(const uint64_t* keys, int n, uint64_t* room, int want, uint64_t* out) {
    const int n2 = next_pow2(n);
    for (int i = threadIdx.x; i < n2; i += NT) room[i] = i < n ? keys[i] : 0ull;
    __syncthreads();
    bitonic_sort_desc<NT>(room, n2);
    for (int i = threadIdx.x; i < want; i += NT) out[i] = room[i];
}

// Same result as block_select_topk_binned for 1 <= c <= kCandCap keys in shared memory (whose place it uses), by one counting sort: a
// key's bucket and its place among the bucket's arrivals come from one atomic, the buckets' places from a scan, and every key counts
// the larger ones of its own bucket, a key or two unless many scores are nearly equal.  Buckets behind the top-k are not looked
// at, and those that lie in it hold no more than topk keys; one that reaches beyond it is sorted where it holds many.
// sm.hist is zero.  The caller synchronises before it reads sm.sel or uses binlist, hist or the keys' place again.
template <int NT, int SELCAP>
__device__ __forceinline__ int block_select_topk_list(uint64_t* keys, int c, int topk, uint32_t hist_base, int hist_shift,
                                                      SelectSmem<SELCAP>& sm) {
    constexpr int kPer = kCandCap / NT, kBuckets = kHistBins / NT, kCrowd = 128;
    static_assert(kCandCap % NT == 0 && kBuckets % 4 == 0 && kCandCap <= kBinListCap, "whole keys and buckets per thread");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint64_t k[kPer];
    int d[kPer], arrival[kPer];
    if (tid == 0) sm.inbin = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        if (u * NT >= c) break;  // uniform
        if (u * NT + tid >= c) continue;
        k[u] = keys[u * NT + tid];
        d[u] = hist_digit(k[u], hist_base, hist_shift);
        arrival[u] = atomicAdd(&sm.hist[d[u]], 1);
    }
    __syncthreads();
    int4* mine = reinterpret_cast<int4*>(sm.hist) + tid * (kBuckets / 4);
    int h[kBuckets], sum = 0;
#pragma unroll
    for (int q = 0; q < kBuckets / 4; ++q) {
        const int4 v = mine[q];
        h[4 * q] = v.x; h[4 * q + 1] = v.y; h[4 * q + 2] = v.z; h[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < kBuckets; ++q) sum += h[q];
    int incl = sum;  // from the higher buckets down
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(kFullMask, incl, o);
        if (lane + o < 32) incl += v;
    }
    if (lane == 0) sm.red_cnt[warp] = incl;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) incl += w > warp ? sm.red_cnt[w] : 0;
    int start = incl - sum;
    if (sum > kCrowd && start < topk && incl > topk) {  // one thread at most
        int above = start;
#pragma unroll
        for (int q = kBuckets - 1; q >= 0; --q) {
            if (h[q] > kCrowd && above < topk && above + h[q] > topk) {
                sm.above = above;
                sm.inbin = h[q];
            }
            above += h[q];
        }
    }
#pragma unroll
    for (int q = kBuckets - 1; q >= 0; --q) {
        const int n = h[q];
        h[q] = start;
        start += n;
    }
#pragma unroll
    for (int q = 0; q < kBuckets / 4; ++q) mine[q] = make_int4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
    __syncthreads();
    uint64_t* sorted = sm.binlist;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        if (u * NT >= c) break;
        if (u * NT + tid >= c) continue;
        const int first = sm.hist[d[u]];
        sorted[first + arrival[u]] = k[u];
        arrival[u] = first;
    }
    __syncthreads();
    int upto = topk;  // keys of buckets that start here or later are not ranked below
    if (sm.inbin > 0) {
        upto = sm.above;
        block_sort_bucket<NT>(sorted + upto, sm.inbin, keys, topk - upto, sm.sel + upto);
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        if (u * NT >= c) break;
        if (u * NT + tid >= c || arrival[u] >= upto) continue;
        const int end = d[u] > 0 ? sm.hist[d[u] - 1] : c;
        int rank = arrival[u];
        if (end - rank > 1)
            for (int q = arrival[u]; q < end; ++q) rank += sorted[q] > k[u] ? 1 : 0;
        if (rank < topk) sm.sel[rank] = k[u];
    }
    return c < topk ? c : topk;
}

// Same result as block_select_topk_binned for a plain fp32 score array in GLOBAL memory (key = score above thr, index),
// reading the array once: a spread sample of the scores (one 16-byte chunk per thread) gives a score floor that should
// leave a few hundred candidates; one pass collects every key at or above the floor into `cand` (kCandCap keys of
// shared memory); the exact selection then runs on that list.  The floor is only a guess, the count decides: with fewer
// than topk candidates (while keys below the floor exist) or more than kCandCap, the two-pass selection over the whole
// array runs instead, so the result never depends on the sample.
// The pass is bound by issue, not by memory: twelve scores per lane cost one compare and one mask bit each, lanes without a
// hit (about half of them) stop there, and a lane with hits reserves its places with one shared-memory atomic and reads the
// few scores again (L1).  A warp prefix sum per 16-byte chunk instead took half as long again.
template <int NT, int SELCAP>
__device__ int block_select_topk_sampled(const float* __restrict__ s, float thr, int n, int topk, uint32_t hist_base,
                                         int hist_shift, SelectSmem<SELCAP>& sm, uint64_t* cand) {
    const int tid = threadIdx.x;
    // an array that starts off a 16-byte boundary has up to three scores in front of its first whole chunk
    const int head = min(n, static_cast<int>(((16u - static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s) & 15u)) & 15u) >> 2));
    const int n4 = (n - head) >> 2;
    const float4* s4 = reinterpret_cast<const float4*>(s + head);
    float floor_score = __uint_as_float(__float_as_uint(thr) + 1u);  // (thr > 0) "above thr" as a >=
    bool floored = false;
    if (n > kCandCap && n4 >= NT) {
        // a coarse histogram will do: NT buckets, one per thread
        constexpr int kCoarse = kHistBins / NT;
        static_assert(kHistBins % NT == 0, "whole buckets per thread");
        sm.hist[tid] = 0;
        __syncthreads();
        const float4 q = __ldg(s4 + static_cast<int>((static_cast<int64_t>(tid) * n4) / NT));
        auto add = [&](float v) {
            if (v > thr)
                atomicAdd(&sm.hist[hist_digit(static_cast<uint64_t>(__float_as_uint(v)) << 32, hist_base, hist_shift) / kCoarse], 1);
        };
        add(q.x);
        add(q.y);
        add(q.z);
        add(q.w);
        if (tid == 0) sm.digit = 0;
        __syncthreads();
        // rank in the sample that corresponds to 1.8 * topk in the whole array (the spread of a count of a few dozen
        // sample hits is about a sixth of it: falling short of topk takes three standard deviations)
        const int target = static_cast<int>((static_cast<int64_t>(topk) * (4 * NT) * 9) / (static_cast<int64_t>(n) * 5)) + 4;
        const int lane = tid & 31, warp = tid >> 5;
        const int mine = sm.hist[tid];
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_down_sync(kFullMask, incl, o);
            if (lane + o < 32) incl += t;
        }
        if (lane == 0) sm.red_cnt[warp] = incl;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) incl += (w > warp) ? sm.red_cnt[w] : 0;
        if (incl >= target && incl - mine < target) sm.digit = tid * kCoarse;
    }
    if (tid == 0) sm.bin_cnt = 0;
    for (int i = tid; i < kHistBins / 4; i += NT) reinterpret_cast<int4*>(sm.hist)[i] = make_int4(0, 0, 0, 0);  // for the selection
    __syncthreads();
    if (n > kCandCap && n4 >= NT && sm.digit > 0) {
        floor_score = __uint_as_float(hist_base + (static_cast<uint32_t>(sm.digit) << hist_shift));
        floored = true;
    }
    auto put = [&](float v, int i) {
        const int pos = atomicAdd(&sm.bin_cnt, 1);
        if (pos < kCandCap) cand[pos] = make_key(v, static_cast<uint32_t>(i));
    };
    constexpr int UN = 3;
    for (int c0 = tid; c0 < n4; c0 += NT * UN) {
        uint32_t hits = 0u;
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int c = c0 + u * NT;
            const float4 q = c < n4 ? __ldg(s4 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            hits |= (q.x >= floor_score ? 1u : 0u) << (4 * u);
            hits |= (q.y >= floor_score ? 2u : 0u) << (4 * u);
            hits |= (q.z >= floor_score ? 4u : 0u) << (4 * u);
            hits |= (q.w >= floor_score ? 8u : 0u) << (4 * u);
        }
        if (hits != 0u) {
            int pos = atomicAdd(&sm.bin_cnt, __popc(hits));
            while (hits != 0u) {
                const int k = __ffs(hits) - 1;
                hits &= hits - 1u;
                const int i = head + 4 * (c0 + (k >> 2) * NT) + (k & 3);
                if (pos < kCandCap) cand[pos] = make_key(__ldg(s + i), static_cast<uint32_t>(i));
                ++pos;
            }
        }
    }
    const int tail0 = head + 4 * n4;
    if (tid < head + n - tail0) {  // the scores in front of and behind the whole chunks: at most six
        const int i = tid < head ? tid : tail0 + tid - head;
        const float v = __ldg(s + i);
        if (v >= floor_score) put(v, i);
    }
    __syncthreads();
    const int c = sm.bin_cnt;
    if (c == 0 && !floored) return 0;
    if (c > kCandCap || (floored && c < topk)) {
        __syncthreads();  // (the selection resets the counter)
        return block_select_dense_outlined<NT, SELCAP>(s, head == 0, thr, n, topk, hist_base, hist_shift, &sm);
    }
    return block_select_topk_list<NT, SELCAP>(cand, c, topk, hist_base, hist_shift, sm);
}

// ---- IoU suppression test ------------------------------------------------------------------------
struct NmsBox {
    float x1, y1, x2, y2, area;
};

__device__ __forceinline__ NmsBox make_nms_box(float x1, float y1, float x2, float y2) {
    NmsBox b;
    b.x1 = x1;
    b.y1 = y1;
    b.x2 = x2;
    b.y2 = y2;
    b.area = __fmul_rn(__fsub_rn(x2, x1), __fsub_rn(y2, y1));
    return b;
}

// true iff fp32(inter / (area_i + area_j - inter)) > thr.  thr_lo / thr_hi bracket thr by a relative 1e-6:
// outside the bracket the comparison against thr * union decides without a division, inside it the
// correctly rounded quotient is formed, so the answer is always that of the division.
__device__ __forceinline__ bool iou_exceeds(const NmsBox& a, const NmsBox& b, float thr, float thr_lo, float thr_hi) {
    // x extent first: boxes of different classes sit in disjoint coordinate ranges, so most pairs end here
    float w = fmaxf(0.0f, __fsub_rn(fminf(a.x2, b.x2), fmaxf(a.x1, b.x1)));
    if (!(w > 0.0f)) return false;  // inter = w * h = 0: the quotient is 0 (or NaN): never above a positive threshold
    float h = fmaxf(0.0f, __fsub_rn(fminf(a.y2, b.y2), fmaxf(a.y1, b.y1)));
    float inter = __fmul_rn(w, h);
    if (!(inter > 0.0f)) return false;
    float uni = __fsub_rn(__fadd_rn(a.area, b.area), inter);
    if (uni > 0.0f && uni < 3.0e38f && inter < 3.0e38f) {
        if (inter > __fmul_rn(uni, thr_hi)) return true;
        if (inter < __fmul_rn(uni, thr_lo)) return false;
    }
    return __fdiv_rn(inter, uni) > thr;
}

// Finite coordinates and an area below 1e37: the guards of iou_exceeds are then implied by a positive intersection
// (inter <= min(area) and max(area) <= union <= 2e37).
__device__ __forceinline__ bool nms_box_is_tame(const NmsBox& b) {
    return fabsf(b.x1) < 1.0e18f && fabsf(b.y1) < 1.0e18f && fabsf(b.x2) < 1.0e18f && fabsf(b.y2) < 1.0e18f && b.area < 1.0e37f;
}
// Candidate pairs for the suppression test of up to 256 boxes, as bit sets: box j can only suppress or be suppressed by box i
// if their x ranges and their y ranges overlap and their areas are within a factor of thr of one another (IoU <= smaller /
// larger area).  Every one of the three is a range condition on a monotone cell number, so six tables of cumulative sets
// answer it: lo tables hold the boxes whose cell is <= c, hi tables those whose cell is >= c, and the candidates of box i are
// the AND of six look-ups per 32 boxes.  On SSD priors this leaves a few per cent of the pairs, where sorted windows along
// one axis left most of them.
constexpr int kCells = 32;  // one lane per cell in the cumulation
template <int WORDS>
struct PairCells {
    uint32_t t[6][WORDS][kCells];  // x1 <=, x2 >=, y1 <=, y2 >=, area <=, area >=
    float lo, hi;
    uint32_t ordered_lo, ordered_hi, area_base;
};
// an fp32 value as an unsigned number of the same order
__device__ __forceinline__ uint32_t ordered_bits(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }

// A box's cells in the six tables.  The windows along x and y are as narrow as the threshold makes them: the intersection is no wider
// than the overlap w of the x ranges and no higher than either box, so IoU <= w / (width of box i), and a box that reaches less than
// thr * width into box i suppresses nothing (580 -> 230 candidate pairs of 200 boxes on SSD priors).
struct PairWindow {
    int x1, x2, y1, y2, area_lo, area_hi;
    bool real;
};
// The boxes 32w .. 32w + 31 behind box t = threadIdx.x that box t might suppress.
template <int WORDS>
__device__ __forceinline__ uint32_t pair_word(const PairCells<WORDS>& pc, const PairWindow& m, int w) {
    const int t = threadIdx.x, lane = t & 31;
    uint32_t b = pc.t[0][w][m.x2] & pc.t[1][w][m.x1] & pc.t[2][w][m.y2] & pc.t[3][w][m.y1] & pc.t[4][w][m.area_hi] & pc.t[5][w][m.area_lo];
    if (w == t >> 5) b &= lane == 31 ? 0u : (0xffffffffu << (lane + 1));
    return m.real && w >= t >> 5 ? b : 0u;
}
// All 32 * WORDS threads; thread t owns box t (t < n; all boxes tame).  Fills the tables.
template <int WORDS>
__device__ __forceinline__ PairWindow pair_tables(const float4 me, float area, int n, float thr, PairCells<WORDS>& pc) {
    constexpr int NT = 32 * WORDS;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool real = t < n && me.z > me.x && me.w > me.y && area > 0.0f;  // others intersect nothing
    for (int i = t; i < 6 * WORDS * kCells; i += NT) (&pc.t[0][0][0])[i] = 0u;
    if (t == 0) {
        pc.ordered_lo = 0xffffffffu;
        pc.ordered_hi = 0u;
        pc.area_base = 0u;
    }
    __syncthreads();
    {
        const uint32_t l = __reduce_min_sync(kFullMask, real ? ordered_bits(fminf(me.x, me.y)) : 0xffffffffu);
        const uint32_t h = __reduce_max_sync(kFullMask, real ? ordered_bits(fmaxf(me.z, me.w)) : 0u);
        const uint32_t a = __reduce_max_sync(kFullMask, real ? __float_as_uint(area) >> 22 : 0u);
        if (lane == 0) {
            atomicMin(&pc.ordered_lo, l);
            atomicMax(&pc.ordered_hi, h);
            atomicMax(&pc.area_base, a);
        }
    }
    __syncthreads();
    const float lo = from_ordered_bits(pc.ordered_lo), hi = from_ordered_bits(pc.ordered_hi);
    const float scale = hi > lo ? __fdividef(static_cast<float>(kCells), hi - lo) : 0.0f;
    const int abase = static_cast<int>(pc.area_base) - (kCells - 1);  // the largest area sits in the last cell; two cells per octave
    // monotone in v whatever the rounding of `scale`: a subtraction, a product and a conversion, each monotone
    auto cell = [&](float v) { return min(max(__float2int_rd(__fmul_rn(__fsub_rn(v, lo), scale)), 0), kCells - 1); };
    auto area_cell = [&](float a) { return min(max(static_cast<int>(__float_as_uint(a) >> 22) - abase, 0), kCells - 1); };
    int cx1 = 0, cx2 = 0, cy1 = 0, cy2 = 0;
    if (real) {
        cx1 = cell(me.x);
        cy1 = cell(me.y);
        cx2 = cell(me.z);
        cy2 = cell(me.w);
        const int ca = area_cell(area);
        const uint32_t bit = 1u << lane;
        atomicOr(&pc.t[0][warp][cx1], bit);
        atomicOr(&pc.t[1][warp][cx2], bit);
        atomicOr(&pc.t[2][warp][cy1], bit);
        atomicOr(&pc.t[3][warp][cy2], bit);
        atomicOr(&pc.t[4][warp][ca], bit);
        atomicOr(&pc.t[5][warp][ca], bit);
    }
    __syncthreads();
    // cumulation: lane = cell; warp w takes word w of the six tables, the six scans side by side
    uint32_t v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = pc.t[k][warp][lane];
#pragma unroll
    for (int o = 1; o < kCells; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const uint32_t u = (k & 1) == 0 ? __shfl_up_sync(kFullMask, v[k], o) : __shfl_down_sync(kFullMask, v[k], o);
            if ((k & 1) == 0 ? lane >= o : lane + o < kCells) v[k] |= u;
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) pc.t[k][warp][lane] = v[k];
    __syncthreads();
    // the area window, a relative 1e-5 wider than the bound so that no rounding of areas or of the quotient matters
    const int a_hi = real ? area_cell(__fdividef(area, thr * (1.0f - 1.0e-5f)) * (1.0f + 1.0e-5f)) : 0;
    const int a_lo = real ? area_cell(area * (thr * (1.0f - 2.0e-5f))) : 0;
    int qx1 = 0, qx2 = 0, qy1 = 0, qy2 = 0;
    if (real) {
        // (a relative 1e-4 of the width and 4e-7 of the coordinates wider: roundings of widths, products, sums and of the quotient)
        const float reach = thr * (1.0f - 1.0e-4f);
        const float dx = fmaf(me.z - me.x, reach, -4.0e-7f * fmaxf(fabsf(me.x), fabsf(me.z)));
        const float dy = fmaf(me.w - me.y, reach, -4.0e-7f * fmaxf(fabsf(me.y), fabsf(me.w)));
        qx1 = cell(me.x + dx);
        qx2 = cell(me.z - dx);
        qy1 = cell(me.y + dy);
        qy2 = cell(me.w - dy);
    }
    return {qx1, qx2, qy1, qy2, a_lo, a_hi, real};
}

// Greedy NMS over up to 256 boxes by a list of the candidate pairs: every thread adds its own, all threads test them in turn
// (a thread that walks its own candidates waits for the one with the most: 12 300 cycles of 49 500 of an SSD class, of which 230
// candidates and 20 real pairs remain), and one warp resolves the few pairs that are left, in rounds without a block barrier; more than
// kHits are walked through in order (block_nms_walk).
// A box is certainly kept once every box that could suppress it is certainly removed, and certainly removed once a certainly kept
// box suppresses it; both sets only grow, every round settles at least the first undecided box, and the fixed point is the
// greedy result.  Returns false, the same for all threads, where a list does not fit; keep_words is then untouched.
struct PairLists {
    static constexpr int kPairs = 4096, kHits = 64;
    uint16_t* pairs;  // [kPairs] i << 8 | j, i < j
    uint16_t* hits;   // [kHits], on a 4-byte boundary
    uint32_t* rows;   // [NT * WORDS] may lie where `pc` does
    int* count;       // [2]: pairs, hits; zero, with a barrier since
    uint32_t* words;  // [2 * WORDS]
};
// Greedy NMS of more pairs than that: bit k of `mine` stands for the pair t + k * NT, which suppresses.  One round by all threads settles
// heaps around a best box each; the pairs that are still open become rows of bits, and one warp goes from one kept box that suppresses
// others to the next, some hundred cycles each.  (More rounds take the longer the more pairs there are and the longer their chains.
// Whole calls of 16 images x 80 classes of 200 boxes, us, rounds of one warp / of the block over rows / this: in a row with scores that
// fall along it, each box over the next 326 / 259 / 54, over the next five 412 / 128 / 58, those with random scores 77 / 73 / 58; 50 heaps of
// four boxes 33 / 34 / 32, without the round 39.  At 49 pairs in a row one warp takes 60, rows 79.)
template <int WORDS>
__device__ __noinline__ void block_nms_walk(const uint16_t* pairs, uint32_t mine, uint32_t* rows, uint32_t* suppressors, uint32_t* words, int n,
                                            uint32_t* keep_words) {
    constexpr int NT = 32 * WORDS;
    const int t = threadIdx.x, lane = t & 31;
    uint32_t *maybe = words, *settled = words + WORDS;  // boxes that others suppress, and those whose suppressor nobody suppresses
#pragma unroll
    for (int w = 0; w < WORDS; ++w) rows[w * NT + t] = 0u;
    if (t < 2 * WORDS) words[t] = 0u;
    else if (t < 3 * WORDS) suppressors[t - 2 * WORDS] = 0u;
    __syncthreads();
    auto has = [](const uint32_t* set, uint32_t b) { return ((set[b >> 5] >> (b & 31u)) & 1u) != 0u; };
    for (uint32_t left = mine; left != 0u; left &= left - 1u) {
        const uint32_t e = pairs[t + (__ffs(left) - 1) * NT];
        atomicOr(&maybe[(e >> 5) & 7u], 1u << (e & 31u));
    }
    __syncthreads();
    for (uint32_t left = mine; left != 0u; left &= left - 1u) {
        const uint32_t e = pairs[t + (__ffs(left) - 1) * NT];
        if (!has(maybe, e >> 8)) atomicOr(&settled[(e >> 5) & 7u], 1u << (e & 31u));
    }
    __syncthreads();
    for (; mine != 0u; mine &= mine - 1u) {
        const uint32_t e = pairs[t + (__ffs(mine) - 1) * NT];
        if (!has(maybe, e >> 8) || has(settled, e >> 8) || has(settled, e & 255u)) continue;
        atomicOr(&rows[(e >> 8) * WORDS + ((e >> 5) & 7u)], 1u << (e & 31u));
        atomicOr(&suppressors[e >> 13], 1u << ((e >> 8) & 31u));
    }
    __syncthreads();
    if (t >= 32) return;
    const int word = lane < WORDS ? lane : 0;
    uint32_t next = lane < WORDS ? suppressors[lane] : 0u, gone = settled[word];
    for (int left = n; left > 0; --left) {
        const unsigned any = __ballot_sync(kFullMask, next != 0u);
        if (any == 0u) break;
        const int from = __ffs(any) - 1, bit = __shfl_sync(kFullMask, __ffs(next) - 1, from);
        gone |= rows[(32 * from + bit) * WORDS + word];
        if (lane == from) next &= next - 1u;
        next &= ~gone;
    }
    if (lane < WORDS) {
        const uint32_t there = n >= 32 * lane + 32 ? 0xffffffffu : n > 32 * lane ? (1u << (n - 32 * lane)) - 1u : 0u;
        keep_words[lane] = there & ~gone;
    }
}
template <int WORDS>
__device__ __forceinline__ bool block_nms_pairs(const float4* sxy, const float* sarea, const PairCells<WORDS>& pc, const PairWindow& window,
                                                int n, float thr, float thr_lo, float thr_hi, const PairLists& pl, uint32_t* keep_words) {
    constexpr int NT = 32 * WORDS;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t bits[WORDS];
    int mine = 0;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        bits[w] = w >= warp && 32 * w < n ? pair_word(pc, window, w) : 0u;
        mine += __popc(bits[w]);
    }
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFullMask, upto, o);
        if (lane >= o) upto += u;
    }
    int at = 0;  // (an atomic per lane instead of this scan takes turns for every lane: 3000 cycles more)
    if (lane == 31 && upto > 0) at = atomicAdd(pl.count, upto);
    at = __shfl_sync(kFullMask, at, 31) + upto - mine;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        for (uint32_t left = bits[w]; left != 0u; left &= left - 1u) {
            if (at < PairLists::kPairs) pl.pairs[at] = static_cast<uint16_t>((t << 8) | (32 * w + __ffs(left) - 1));
            ++at;
        }
    }
    __syncthreads();
    const int pairs = pl.count[0];
    if (pairs > PairLists::kPairs) return false;
    constexpr int kAtOnce = 2;
    static_assert(PairLists::kPairs <= 32 * NT, "a bit for every pair of a thread");
    uint32_t suppress = 0u;
    for (int p0 = t, k = 0; p0 < pairs; p0 += kAtOnce * NT, k += kAtOnce) {
        uint32_t e[kAtOnce];
        float inter[kAtOnce], uni[kAtOnce];
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
            const int p = p0 + u * NT;
            e[u] = pl.pairs[p < pairs ? p : 0];
            const float4 a = sxy[e[u] >> 8], b = sxy[e[u] & 255u];
            const float w = fmaxf(0.0f, __fsub_rn(fminf(a.z, b.z), fmaxf(a.x, b.x)));
            const float h = fmaxf(0.0f, __fsub_rn(fminf(a.w, b.w), fmaxf(a.y, b.y)));
            inter[u] = __fmul_rn(w, h);
            uni[u] = __fsub_rn(__fadd_rn(sarea[e[u] >> 8], sarea[e[u] & 255u]), inter[u]);
        }
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
            // iou_exceeds for tame boxes: a positive intersection implies its guards
            if (p0 + u * NT >= pairs || !(inter[u] > 0.0f) || inter[u] < __fmul_rn(uni[u], thr_lo)) continue;
            if (inter[u] > __fmul_rn(uni[u], thr_hi) || __fdiv_rn(inter[u], uni[u]) > thr) {
                suppress |= 1u << (k + u);
                const int pos = atomicAdd(pl.count + 1, 1);
                if (pos < PairLists::kHits) pl.hits[pos] = static_cast<uint16_t>(e[u]);
            }
        }
    }
    __syncthreads();
    const int hits = pl.count[1];
    if (hits > PairLists::kHits) {
        block_nms_walk<WORDS>(pl.pairs, suppress, pl.rows, reinterpret_cast<uint32_t*>(pl.hits), pl.words, n, keep_words);
    } else if (warp == 0) {
        uint32_t* maybe = pl.words;          // boxes that a not-yet-removed box suppresses
        uint32_t* gone = pl.words + WORDS;   // boxes that a kept box suppresses
        if (lane < 2 * WORDS) pl.words[lane] = 0u;
        __syncwarp();
        auto has = [](const uint32_t* set, uint32_t b) { return ((*reinterpret_cast<const volatile uint32_t*>(set + (b >> 5)) >> (b & 31u)) & 1u) != 0u; };
        for (int round = 0; round <= n && hits > 0; ++round) {
            for (int h = lane; h < hits; h += 32) {
                const uint32_t e = pl.hits[h];
                if (!has(gone, e >> 8)) atomicOr(&maybe[(e >> 5) & 7u], 1u << (e & 31u));
            }
            __syncwarp();
            for (int h = lane; h < hits; h += 32) {
                const uint32_t e = pl.hits[h];
                // (a box that this loop has removed meanwhile is one of `maybe`)
                if (!has(gone, e >> 8) && !has(maybe, e >> 8)) atomicOr(&gone[(e >> 5) & 7u], 1u << (e & 31u));
            }
            __syncwarp();
            const uint32_t open = lane < WORDS ? maybe[lane] & ~gone[lane] : 0u;
            if (!__any_sync(kFullMask, open != 0u)) break;
            if (lane < WORDS) maybe[lane] = 0u;
            __syncwarp();
        }
        if (lane < WORDS) {
            const uint32_t there = n >= 32 * lane + 32 ? 0xffffffffu : n > 32 * lane ? (1u << (n - 32 * lane)) - 1u : 0u;
            keep_words[lane] = there & ~gone[lane];
        }
    }
    return true;
}

// The same by suppression rows (boxes that suppress many others): thread i owns row i (NT == 32 * WORDS, n <= NT), the whole block
// goes through the rounds.  or_words: 2 * WORDS words of shared memory.  keep_words[w] receives the keep bits.
template <int NT, int WORDS>
__device__ __forceinline__ void block_nms_resolve(const uint32_t (&row)[WORDS], int n, uint32_t* keep_words, uint32_t* or_words) {
    static_assert(NT == 32 * WORDS, "one thread per row, one warp per word");
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool valid = t < n;
    uint32_t any = 0u;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) any |= row[w];
    uint32_t* maybe = or_words;            // boxes that a not-yet-removed box suppresses
    uint32_t* gone = or_words + WORDS;     // boxes that a kept box suppresses
    bool kept = false, removed = false;
    for (int round = 0; round <= n; ++round) {
        if (t < 2 * WORDS) or_words[t] = 0u;
        __syncthreads();
        if (__any_sync(kFullMask, any != 0u && !removed)) {
#pragma unroll
            for (int w = 0; w < WORDS; ++w) {
                const uint32_t v = __reduce_or_sync(kFullMask, removed ? 0u : row[w]);
                if (lane == w && v != 0u) atomicOr(&maybe[w], v);
            }
        }
        __syncthreads();
        kept = valid && !removed && ((maybe[warp] >> lane) & 1u) == 0u;
        if (__any_sync(kFullMask, any != 0u && kept)) {
#pragma unroll
            for (int w = 0; w < WORDS; ++w) {
                const uint32_t v = __reduce_or_sync(kFullMask, kept ? row[w] : 0u);
                if (lane == w && v != 0u) atomicOr(&gone[w], v);
            }
        }
        __syncthreads();
        removed = valid && ((gone[warp] >> lane) & 1u) != 0u;
        if (__syncthreads_or((valid && !kept && !removed) ? 1 : 0) == 0) break;
    }
    const uint32_t kw = __ballot_sync(kFullMask, kept);
    if (lane == 0) keep_words[warp] = kw;
}

}  // namespace fb
