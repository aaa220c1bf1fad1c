// C2, second half: one CTA per image turns the candidate list into detections: top-k in "score descending, index ascending"
// order (functs/benchmark/ai_model/yolov3/yolov3_bbox.py:128-134), class-wise greedy NMS through the coordinate offsets of
// :144-146 and :177, and the compacted outputs.
//
// What bounds it: a chain of short dependent phases on some 2000 keys and 1000 boxes, i.e. latency.  One CTA keeps all of it in
// shared memory; with the work in one launch there is no second kernel to start, no ticket and no round trip through global
// memory between the phases (two kernels of up to sixteen CTAs per image took 22 + 24 us for 64 images and 22 + 16 for one).
//   select     counting sort on 2048 score buckets that start at the image's floor (a bucket holds a key or two) + rank
//              inside the bucket;
//   boxes      decoded here for the selected candidates only, from the logits (four scattered loads each), so that nobody
//              has to write and read all boxes;
//   pairs      boxes are laid out by class; a box looks at its own class and at the classes within reach of the offsets
//              (boxes with negative coordinates reach into the next class), skipping a class whose smallest corner lies
//              behind its own largest one.  What overlaps enough goes into a list of (suppressor, suppressed) pairs;
//   greedy     parallel rounds over the pair list: a box is kept once every box that could suppress it is removed.
// Slow exact ways for the rare inputs: the floor was too high (fewer than topk candidates in the list: the image's scores are
// formed again without one), more candidates than fit (two-pass selection from global memory), a crowded score bucket (bitonic
// sort), more pairs than fit (bit matrix in global memory, walked row by row).
#include "yolo.cuh"

namespace fb {

constexpr int kPostThreads = 1024;
constexpr int kPostKeys = 4096;    // candidates the shared-memory selection takes
constexpr int kPostTop = 1024;     // largest topk
constexpr int kPostPairs = 8192;
constexpr int kPostCrowded = 64;   // keys of one score bucket beyond which ranks are not counted
constexpr int kPostWords = kPostTop / 32;

struct RescanSlot {
    float so;  // objectness score
    int slot;  // of the level
};

struct PostSmem {
    union {
        uint64_t keys[kPostKeys];
        RescanSlot rescan[kPostKeys];
        struct {
            float4 xy[kPostTop];       // NMS-space corners, by position (class order)
            float area[kPostTop];
            uint16_t rank[kPostTop];   // position -> place in the sorted top-k
            uint8_t label[kPostTop];
        } box;
        float rows_out[kPostTop * 5];      // the kept rows on their way out
    };
    union {
        uint64_t sorted[kPostKeys];
        uint32_t pairs[kPostPairs];    // suppressor << 16 | suppressed (places in the top-k)
        uint32_t rows[32][kPostWords]; // staging of the dense matrix
        SelectSmem<kPostTop> generic;
    };
    int hist[kHistBins];
    uint64_t sel[kPostTop];
    uint8_t removed[kPostTop], blocked[kPostTop], kept[kPostTop];
    int cls_start[kYoloClasses + 1], cls_cursor[kYoloClasses];
    uint32_t cls_min_x[kYoloClasses], cls_min_y[kYoloClasses];  // smallest corners of a class, as ordered bits
    int warp_sum[32];
    uint32_t words[kPostWords];
    uint32_t hi, lo;  // extreme coordinates, as ordered bits
    int npairs;
    int live, found;  // post_rescan
};
static_assert(sizeof(PostSmem) < 100 * 1024, "two CTAs per SM");

// 2048 buckets of the scores from `bar` to 1
__device__ __forceinline__ void post_buckets(float bar, uint32_t& base, int& shift) {
    base = __float_as_uint(bar);
    const uint32_t span = 0x3F800000u > base ? 0x3F800000u - base : 1u;  // scores are products of probabilities: <= 1
    shift = max(0, 21 - __clz(static_cast<int>(span - 1u)));            // (span - 1) >> shift < 2048
}

// The image's candidates once more, without a floor.  Latency bounds it (one CTA, 3.6 MB at 416 x 416): so the boxes that can yield
// any are listed first, 4096 slots at a time, and a thread then takes sixteen classes of one of them, loaded together.  (A thread
// per box, one class after another: some 200 us.)
constexpr int kRescanClasses = 16;
__device__ __noinline__ void post_rescan(const YoloLevels& L, const YoloPostArgs& A, int img, PostSmem* smp) {
    PostSmem& sm = *smp;
    const int t = threadIdx.x, lane = t & 31;
    if (t == 0) sm.found = 0;
    for (int lvl = 0; lvl < 3; ++lvl) {
        const int plane = L.plane[lvl];
        const float* img_map = L.map[lvl] + static_cast<int64_t>(img) * 3 * kYoloAttrib * plane;
        for (int s0 = 0; s0 < 3 * plane; s0 += kPostKeys) {
            __syncthreads();  // the list of the slots before is done with
            if (t == 0) sm.live = 0;
            __syncthreads();
            float so[kPostKeys / kPostThreads];
#pragma unroll
            for (int q = 0; q < kPostKeys / kPostThreads; ++q) {
                const int slot = s0 + q * kPostThreads + t;
                int anchor, pos;
                yolo_slot(plane, min(slot, 3 * plane - 1), anchor, pos);
                so[q] = slot < 3 * plane ? __ldg(img_map + (anchor * kYoloAttrib + 4) * plane + pos) : -INFINITY;
            }
#pragma unroll
            for (int q = 0; q < kPostKeys / kPostThreads; ++q) {
                so[q] = sigmoid_f32(so[q]);
                const bool alive = so[q] > A.thr;
                const unsigned m = __ballot_sync(kFullMask, alive);
                int at = 0;
                if (lane == 0 && m != 0u) at = atomicAdd(&sm.live, __popc(m));
                at = __shfl_sync(kFullMask, at, 0) + __popc(m & ((1u << lane) - 1u));
                if (alive) sm.rescan[at] = RescanSlot{so[q], s0 + q * kPostThreads + t};
            }
            __syncthreads();
            const int n = sm.live, items = n * (kYoloClasses / kRescanClasses);
            for (int i = t; i < items; i += kPostThreads) {  // neighbouring threads: neighbouring slots
                const int group = i / n;
                const RescanSlot o = sm.rescan[i - group * n];
                int anchor, pos;
                yolo_slot(plane, o.slot, anchor, pos);
                const float* src = img_map + (anchor * kYoloAttrib + 5 + group * kRescanClasses) * plane + pos;
                float v[kRescanClasses];
#pragma unroll
                for (int u = 0; u < kRescanClasses; ++u) v[u] = __ldg(src + u * plane);
                const float cut = logit_cut(o.so, A.thr);
                const uint32_t flat0 = static_cast<uint32_t>(L.box_begin[lvl] + pos * 3 + anchor) * kYoloClasses + group * kRescanClasses;
#pragma unroll
                for (int u = 0; u < kRescanClasses; ++u) {
                    if (!(v[u] > cut)) continue;
                    const float s = __fmul_rn(o.so, sigmoid_f32(v[u]));
                    if (!(s > A.thr)) continue;
                    const int64_t at = atomicAdd(&sm.found, 1);
                    if (at < A.capacity) A.keys[img * A.capacity + at] = make_key(s, flat0 + static_cast<uint32_t>(u));
                    else if (A.status != nullptr) atomicOr(A.status, FB_STATUS_CAND_OVERFLOW);
                }
            }
        }
    }
    __syncthreads();
    if (t == 0) A.counts[img] = sm.found;
}

struct GlobalKeysView {
    static constexpr bool kDenseScores = false;
    const uint64_t* p;
    __device__ __forceinline__ uint64_t operator()(int i) const { return __ldcg(p + i); }
};
// more keys than the shared-memory selection takes: two passes over the list (a third way stands behind a crowded bucket)
__device__ __noinline__ void post_select_many(const uint64_t* keys, int n, int topk, float bar, PostSmem* sm) {
    uint32_t base;
    int shift;
    post_buckets(bar, base, shift);
    const int m = block_select_topk_binned<kPostThreads, kPostTop, 8>(GlobalKeysView{keys}, n, topk, base, shift, sm->generic);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < m) sm->sel[threadIdx.x] = sm->generic.sel[threadIdx.x];
    __syncthreads();
}

// sel[0 .. min(n, topk)) = the largest keys, sorted; n <= kPostKeys
__device__ __forceinline__ void post_select(const uint64_t* __restrict__ keys, int n, int topk, float bar, PostSmem& sm) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t base;
    int shift;
    post_buckets(bar, base, shift);
    constexpr int kPer = kPostKeys / kPostThreads;
    uint64_t k[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) k[q] = q * kPostThreads + t < n ? __ldcg(keys + q * kPostThreads + t) : 0ull;
    sm.hist[t] = 0;
    sm.hist[t + kPostThreads] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q)
        if (k[q] != 0ull) atomicAdd(&sm.hist[hist_digit(k[q], base, shift)], 1);
    __syncthreads();
    // hist[d] becomes the place where bucket d starts: the number of keys in higher buckets
    const int h0 = sm.hist[2 * t], h1 = sm.hist[2 * t + 1];
    int incl = h0 + h1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(kFullMask, incl, o);
        if (lane + o < 32) incl += v;
    }
    if (lane == 0) sm.warp_sum[warp] = incl;
    __syncthreads();
    int higher = lane > warp ? sm.warp_sum[lane] : 0;
    higher = __reduce_add_sync(kFullMask, higher);
    const int above = incl - (h0 + h1) + higher;
    sm.hist[2 * t + 1] = above;
    sm.hist[2 * t] = above + h1;
    const bool crowded = above < topk && (h0 > kPostCrowded || h1 > kPostCrowded);
    if (__syncthreads_or(crowded ? 1 : 0) != 0) {
        const int sn = next_pow2(n);
#pragma unroll
        for (int q = 0; q < kPer; ++q)
            if (q * kPostThreads + t < sn) sm.keys[q * kPostThreads + t] = k[q];
        __syncthreads();
        bitonic_sort_desc<kPostThreads>(sm.keys, sn);
        if (t < min(n, topk)) sm.sel[t] = sm.keys[t];
        __syncthreads();
        return;
    }
    int start[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        start[q] = topk;
        if (q * kPostThreads >= n) break;  // uniform
        if (k[q] == 0ull) continue;
        const int d = hist_digit(k[q], base, shift);
        const int at = atomicAdd(&sm.hist[d], 1);
        sm.sorted[at] = k[q];
        start[q] = at;
    }
    __syncthreads();
    // now hist[d] is where bucket d ends and hist[d + 1] where it starts; a key counts the larger keys of its bucket
    int end[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        if (q * kPostThreads >= n) break;
        end[q] = 0;
        if (start[q] >= topk + kPostCrowded) continue;  // (a bucket that starts below topk holds no more)
        const int d = hist_digit(k[q], base, shift);
        start[q] = d + 1 < kHistBins ? sm.hist[d + 1] : 0;
        end[q] = sm.hist[d];
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        if (q * kPostThreads >= n) break;
        if (k[q] == 0ull || start[q] >= topk) continue;
        int r = start[q];
        if (end[q] - r > 1)
            for (int j = start[q]; j < end[q]; ++j) r += sm.sorted[j] > k[q] ? 1 : 0;
        if (r < topk) sm.sel[r] = k[q];
    }
    __syncthreads();
}

// Calls pair(i, j), i < j places in the top-k, for every pair of boxes that overlap by more than the threshold, once.
template <class F>
__device__ __forceinline__ void post_pairs(const PostSmem& sm, int m, int reach, float thr, float thr_lo, float thr_hi, F pair) {
    const int p = threadIdx.x;
    if (p >= m) return;
    const float4 me = sm.box.xy[p];
    const NmsBox bi{me.x, me.y, me.z, me.w, sm.box.area[p]};
    const int label = sm.box.label[p], rank = sm.box.rank[p];
    const uint32_t end_x = ordered_bits(me.z), end_y = ordered_bits(me.w);
    // four tests at a time without branches: a pair can only exceed the threshold if its intersection reaches union * thr_lo (or a
    // guard of iou_exceeds may be involved: wild values, which compare as "maybe").  (Only the overlaps in x and in y against the
    // box's own extent: shorter, but what passes walks through the exact test lane by lane, 5300 cycles instead of 4200.)
    auto test4 = [&](const int (&at)[4], const bool (&valid)[4]) {
        bool maybe[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4 c = sm.box.xy[at[u]];
            const float w = __fsub_rn(fminf(me.z, c.z), fmaxf(me.x, c.x)), h = __fsub_rn(fminf(me.w, c.w), fmaxf(me.y, c.y));
            const float inter = __fmul_rn(w, h), uni = __fsub_rn(__fadd_rn(bi.area, sm.box.area[at[u]]), inter);
            maybe[u] = valid[u] && w > 0.0f && h > 0.0f && !(inter < __fmul_rn(uni, thr_lo));
        }
        if (!(maybe[0] || maybe[1] || maybe[2] || maybe[3])) return;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (!maybe[u]) continue;
            const float4 c = sm.box.xy[at[u]];
            const NmsBox bj{c.x, c.y, c.z, c.w, sm.box.area[at[u]]};
            if (iou_exceeds(bi, bj, thr, thr_lo, thr_hi)) {
                const int other = sm.box.rank[at[u]];
                pair(min(rank, other), max(rank, other));
            }
        }
    };
    // the box's own class in a circle, half way round: every box has the same number of partners, and a warp does not wait for the
    // first box of the largest class
    {
        const int s = sm.cls_start[label], n = sm.cls_start[label + 1] - s, i = p - s;
        const int partners = (n - 1) / 2 + ((n & 1) == 0 && i < n / 2 ? 1 : 0);
        for (int k = 1; k <= partners; k += 4) {
            int at[4];
            bool valid[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                valid[u] = k + u <= partners;
                const int j = i + (valid[u] ? k + u : k);
                at[u] = s + (j >= n ? j - n : j);
            }
            test4(at, valid);
        }
    }
    for (int b = label + 1; b <= min(label + reach, kYoloClasses - 1); ++b) {
        if (end_x <= sm.cls_min_x[b] || end_y <= sm.cls_min_y[b]) continue;
        const int q1 = sm.cls_start[b + 1];
        for (int q = sm.cls_start[b]; q < q1; q += 4) {
            int at[4];
            bool valid[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                valid[u] = q + u < q1;
                at[u] = min(q + u, q1 - 1);
            }
            test4(at, valid);
        }
    }
}

// Greedy NMS when the pair list overflowed: the bit matrix in global memory, rows walked in order, 32 staged at a time.
__device__ __noinline__ void post_dense(PostSmem* smp, uint32_t* mask, int m, int reach, float thr, float thr_lo, float thr_hi) {
    PostSmem& sm = *smp;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < m * kPostWords; i += kPostThreads) mask[i] = 0u;
    __threadfence_block();
    __syncthreads();
    post_pairs(sm, m, reach, thr, thr_lo, thr_hi, [&](int i, int j) { atomicOr(mask + i * kPostWords + (j >> 5), 1u << (j & 31)); });
    __threadfence();
    uint32_t gone = 0u;  // warp 0, lane w: removed bits of the boxes 32w .. 32w + 31
    for (int r0 = 0; r0 < m; r0 += 32) {
        __syncthreads();
        sm.rows[warp][lane] = r0 + warp < m ? __ldcg(mask + (r0 + warp) * kPostWords + lane) : 0u;
        __syncthreads();
        if (warp == 0) {
            for (int r = 0; r < 32; ++r) {
                const uint32_t word = __shfl_sync(kFullMask, gone, r0 >> 5);
                if (!((word >> r) & 1u)) gone |= sm.rows[r][lane];
            }
        }
    }
    if (warp == 0) sm.words[lane] = gone;
    __syncthreads();
    sm.removed[t] = (sm.words[warp] >> lane) & 1u;
    __syncthreads();
}

__global__ void __launch_bounds__(kPostThreads, 1)
yolo_post_kernel(const __grid_constant__ YoloLevels L, const __grid_constant__ YoloPostArgs A, float thr_lo, float thr_hi) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PostSmem& sm = *reinterpret_cast<PostSmem*>(smem_raw);
    const int img = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    sm.removed[t] = 0;
    sm.blocked[t] = 0;
    if (t < kYoloClasses) {
        sm.cls_cursor[t] = 0;
        sm.cls_min_x[t] = 0xffffffffu;
        sm.cls_min_y[t] = 0xffffffffu;
    }
    if (t == 0) {
        sm.hi = 0u;
        sm.lo = 0xffffffffu;
        sm.npairs = 0;
    }
    pdl_wait();  // the candidates

    // ---- top-k ----
    float floor = __ldcg(A.floor + img);
    int64_t n64 = *reinterpret_cast<volatile int32_t*>(A.counts + img);
    const bool short_list = floor > 0.0f && n64 < A.topk;
    if (short_list) {
        post_rescan(L, A, img, &sm);
        floor = 0.0f;
        n64 = sm.found;
    }
    const int n = static_cast<int>(n64 < 0 ? 0 : (n64 > A.capacity ? A.capacity : n64));
    const uint64_t* keys = A.keys + img * A.capacity;
    const float4* boxes = A.boxes != nullptr ? reinterpret_cast<const float4*>(A.boxes) + static_cast<int64_t>(img) * L.num_boxes : nullptr;
    if (n <= kPostKeys) post_select(keys, n, A.topk, fmaxf(A.thr, floor), sm);
    else post_select_many(keys, n, A.topk, fmaxf(A.thr, floor), &sm);
    if (t == 0 && (short_list || n > kPostKeys)) A.fallback[img] = 1;
    const int m = min(n, A.topk);

    // ---- boxes of the selected candidates ----
    uint64_t key = 0ull;
    uint32_t flat = 0u;
    int label = 0;
    float4 bx = make_float4(0.f, 0.f, 0.f, 0.f);
    float top = -INFINITY, bottom = INFINITY;
    if (t < m) {
        key = sm.sel[t];
        flat = key_index(key);
        const int box = static_cast<int>(flat / kYoloClasses);
        label = static_cast<int>(flat) - box * kYoloClasses;
        if (boxes != nullptr) {
            bx = __ldcg(boxes + box);
        } else {
            const int lvl = box >= L.box_begin[2] ? 2 : (box >= L.box_begin[1] ? 1 : 0);
            const int plane = L.plane[lvl], local = box - L.box_begin[lvl];
            const int pos = local / 3, anchor = local - pos * 3;
            const float* src = L.map[lvl] + (static_cast<int64_t>(img) * 3 + anchor) * kYoloAttrib * plane + pos;
            bx = yolo_box(L, lvl, anchor, pos, __ldg(src), __ldg(src + plane), __ldg(src + 2 * plane), __ldg(src + 3 * plane));
        }
        top = fmaxf(top, fmaxf(fmaxf(bx.x, bx.y), fmaxf(bx.z, bx.w)));
        bottom = fminf(bottom, fminf(fminf(bx.x, bx.y), fminf(bx.z, bx.w)));
        atomicAdd(&sm.cls_cursor[label], 1);
    }
    {
        const uint32_t h = __reduce_max_sync(kFullMask, ordered_bits(top)), l = __reduce_min_sync(kFullMask, ordered_bits(bottom));
        if (lane == 0) {
            atomicMax(&sm.hi, h);
            atomicMin(&sm.lo, l);
        }
    }
    __syncthreads();
    const float hi = from_ordered_bits(sm.hi), lo = from_ordered_bits(sm.lo);
    const float scale = __fadd_rn(hi, 1.0f);
    // With class offsets, class c occupies the coordinates [c * M + lo, c * M + hi] (M = hi + 1), so boxes whose labels differ
    // by more than floor((hi - lo) / M) + 1 cannot intersect (one class more than exact: the fp32 rounding of the shifts).
    int reach = kYoloClasses;
    if (scale > 0.0f) {
        const float r = floorf((hi - lo) / scale) + 1.0f;
        if (r < static_cast<float>(kYoloClasses)) reach = static_cast<int>(r);
    }
    if (warp == 0) {  // class starts: an exclusive prefix over 80 counts, three per lane
        int c[3], s = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            c[q] = 3 * lane + q < kYoloClasses ? sm.cls_cursor[3 * lane + q] : 0;
            s += c[q];
        }
        int incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += v;
        }
        int run = incl - s;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (3 * lane + q < kYoloClasses) {
                sm.cls_start[3 * lane + q] = run;
                sm.cls_cursor[3 * lane + q] = run;
            }
            run += c[q];
        }
        if (lane == 31) sm.cls_start[kYoloClasses] = incl;
    }
    __syncthreads();
    if (t < m) {
        const float off = __fmul_rn(static_cast<float>(label), scale);
        const NmsBox b = make_nms_box(__fadd_rn(bx.x, off), __fadd_rn(bx.y, off), __fadd_rn(bx.z, off), __fadd_rn(bx.w, off));
        const int p = atomicAdd(&sm.cls_cursor[label], 1);
        sm.box.xy[p] = make_float4(b.x1, b.y1, b.x2, b.y2);
        sm.box.area[p] = b.area;
        sm.box.rank[p] = static_cast<uint16_t>(t);
        sm.box.label[p] = static_cast<uint8_t>(label);
        atomicMin(&sm.cls_min_x[label], ordered_bits(b.x1));
        atomicMin(&sm.cls_min_y[label], ordered_bits(b.y1));
    }
    __syncthreads();

    // ---- greedy NMS ----
    post_pairs(sm, m, reach, A.iou_thr, thr_lo, thr_hi, [&](int i, int j) {
        const int at = atomicAdd(&sm.npairs, 1);
        if (at < kPostPairs) sm.pairs[at] = static_cast<uint32_t>(i) << 16 | static_cast<uint32_t>(j);
    });
    __syncthreads();
    const int np = sm.npairs;
    if (np > kPostPairs) {
        post_dense(&sm, A.mask + static_cast<int64_t>(img) * kPostTop * kPostWords, m, reach, A.iou_thr, thr_lo, thr_hi);
    } else if (np > 0) {
        for (int round = 0; round <= m; ++round) {  // (blocked: zero)
            for (int i = t; i < np; i += kPostThreads) {
                const uint32_t pr = sm.pairs[i];
                if (sm.removed[pr >> 16] == 0) sm.blocked[pr & 0xffffu] = 1;
            }
            __syncthreads();
            const bool kept = t < m && sm.removed[t] == 0 && sm.blocked[t] == 0;
            sm.kept[t] = kept ? 1 : 0;
            sm.blocked[t] = 0;
            __syncthreads();
            for (int i = t; i < np; i += kPostThreads) {
                const uint32_t pr = sm.pairs[i];
                if (sm.kept[pr >> 16] != 0) sm.removed[pr & 0xffffu] = 1;
            }
            __syncthreads();
            if (__syncthreads_or(t < m && !kept && sm.removed[t] == 0 ? 1 : 0) == 0) break;
        }
    }

    // ---- outputs ----
    const bool kept = t < m && sm.removed[t] == 0;
    const unsigned word = __ballot_sync(kFullMask, kept);
    if (lane == 0) sm.warp_sum[warp] = __popc(word);
    __syncthreads();
    const int mine = sm.warp_sum[lane];
    const int before = __reduce_add_sync(kFullMask, lane < warp ? mine : 0), total = __reduce_add_sync(kFullMask, mine);
    const int64_t obase = static_cast<int64_t>(img) * A.topk;
    int4* records = reinterpret_cast<int4*>(A.records);
    if (kept) {
        const int64_t row = obase + before + __popc(word & ((1u << lane) - 1u));
        float* d = sm.rows_out + (row - obase) * 5;  // (stored below, whole lines at a time)
        d[0] = bx.x;
        d[1] = bx.y;
        d[2] = bx.z;
        d[3] = bx.w;
        d[4] = key_score(key);
        A.labels[row] = label;
        if (A.flat_ids != nullptr) A.flat_ids[row] = static_cast<int64_t>(flat);
        if (records != nullptr) {  // the 32-byte record of the multi-GPU gather (layout of pack_detections_kernel)
            records[2 * row] = make_int4(__float_as_int(bx.x), __float_as_int(bx.y), __float_as_int(bx.z), __float_as_int(bx.w));
            records[2 * row + 1] = make_int4(__float_as_int(key_score(key)), label, static_cast<int>(flat), 1);
        }
    }
    for (int i = total + t; i < A.topk; i += kPostThreads) {  // padded rows are deterministic
        const int64_t row = obase + i;
        A.labels[row] = -1;
        if (A.flat_ids != nullptr) A.flat_ids[row] = -1;
        if (records != nullptr) {
            records[2 * row] = make_int4(0, 0, 0, 0);
            records[2 * row + 1] = make_int4(0, -1, -1, 0);
        }
    }
    __syncthreads();
    for (int i = t; i < 5 * A.topk; i += kPostThreads) A.dets[obase * 5 + i] = i < 5 * total ? sm.rows_out[i] : 0.0f;
    if (A.host_counts != nullptr) __syncthreads();  // a host that watches the count finds the rows complete
    if (t == 0) {
        A.out_counts[img] = total;
        if (A.host_counts != nullptr) {
            __threadfence_system();
            *reinterpret_cast<volatile int32_t*>(A.host_counts + img) = total;
        }
    }
}

int64_t yolo_post_mask_bytes(int batch) { return static_cast<int64_t>(batch) * kPostTop * kPostWords * 4; }

int check_yolo_post(int batch, const YoloPostArgs& a) {
    FB_REQUIRE(a.dets && a.labels && a.out_counts && a.keys && a.counts, "yolo_postprocess: null pointer");
    FB_REQUIRE(batch > 0 && a.topk > 0 && a.topk <= kPostTop, "yolo_postprocess: bad sizes (topk must be in [1, %d])", kPostTop);
    FB_REQUIRE(a.thr > 0.0f, "yolo_postprocess: the score threshold must be positive");
    FB_REQUIRE(a.iou_thr > 0.0f && a.iou_thr < 1.0f, "yolo_postprocess: iou threshold must be in (0, 1)");
    FB_REQUIRE(a.records == nullptr || (reinterpret_cast<uintptr_t>(a.records) & 15) == 0, "yolo_postprocess: records must be 16-byte aligned");
    return FB_OK;
}

int launch_yolo_post(const YoloLevels& L, int batch, const YoloPostArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(PostSmem);
    FB_TRY(check_cuda(cudaFuncSetAttribute(yolo_post_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                      "yolo_post attr"));
    const float thr_lo = a.iou_thr * (1.0f - 1.0e-6f), thr_hi = a.iou_thr * (1.0f + 1.0e-6f);
    return launch_after(yolo_post_kernel, dim3(static_cast<unsigned>(batch)), dim3(kPostThreads), smem, st, true, "yolo_post_kernel", L, a, thr_lo,
                      thr_hi);
}

}  // namespace fb
