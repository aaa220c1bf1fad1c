// C2, first half: a score floor per image from a sample of its boxes, then one pass over the logits that leaves the boxes'
// candidates (yolo.cuh says what the group computes; kernels_yolo_post.cu is the second half).
//
// What bounds it: reading the 80 class planes and the objectness plane of every level (81 of the 85 channels; the box channels
// are only read for callers that want every box).  Everything else is kept off that stream:
//   - the score floor.  The program keeps the topk best candidates of an image, but with logits near N(0, 1) one score in
//     thirteen passes the threshold: 65 000 per image.  yolo_floor_kernel takes the scores of one box in sixteen (32
//     neighbouring slots of every 512, one 128-byte line per plane) and picks the score that about 2 * topk candidates
//     should reach.  The floor is a guess: whoever uses the list has to see that it holds at least topk candidates, and
//     takes the exact way otherwise (yolo_post_kernel does).
//   - with the floor known before the first class logit is read, a box whose objectness lies below it is never walked, and
//     a class logit costs a compare against its box's cut.  Hits (about two in a hundred of those) are queued in shared
//     memory and evaluated exactly, together, at the end of the tile.
// Before, the floor was found while the kernel ran, from a histogram in global memory that every candidate incremented: the
// first wave of CTAs had none, and 12 000 candidates per image reached the selection.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <utility>

#include "yolo.cuh"

namespace fb {

namespace cg = cooperative_groups;

// ---- score floor ------------------------------------------------------------------------------------------------------
constexpr int kFloorCtas = 8;        // one cluster per image
constexpr int kFloorThreads = 384;   // 8 x 3 runs of 32 slots, four warps each (21 runs at 13 / 26 / 52)
constexpr int kFloorShift = 9;       // one run of 32 slots per 512: a whole 128-byte line per plane, because that is what DRAM is read
                                     // in (runs of eight slots, four times as many, moved 58 MB instead of 15: 26 us for 64 images)
constexpr int kFloorAll = 5;         // every run
constexpr int kFloorSpread = 128;    // sampled boxes that can yield candidates, below which the floor aims at three times the top-k
                                     // instead of twice.  A few clusters of boxes are met by the sample or missed: a floor that
                                     // comes out too high costs a second look at the image by one CTA (some 50 us), one too low
                                     // a longer selection (some 10).  Always three times: 64 images at N(0, 1) 76.6 us (71.4)
constexpr int kFloorBins = 256;      // score buckets (a guess needs no finer ones; one thread each)
constexpr int kFloorMinSample = 256; // sampled boxes below which a guess is not worth the risk: such a pyramid (below some 3000 boxes)
                                     // is sampled whole, in some 90 runs, four per warp.  Without any floor one CTA had to select from
                                     // all candidates: 6 / 12 / 24 cells 66 us, at a threshold of 0.05 302 us

struct YoloFloorArgs {
    YoloLevels L;
    float thr;
    uint32_t hist_base;
    int hist_shift;
    int topk;
    int sample;  // 0: no floor (every candidate above the threshold is wanted)
    float* floor;
    int32_t* counts;
    int32_t* fallback;
};

// Also clears the image's counters.  The scores of the sample may be approximate: they only pick a bucket.
// SHIFT: log2 of the slots that one run is taken from.
template <int SHIFT>
__global__ void __cluster_dims__(kFloorCtas, 1, 1) __launch_bounds__(kFloorThreads, 4)
yolo_floor_kernel(const YoloFloorArgs A) {
    __shared__ int hist[kFloorBins];    // this CTA's scores
    __shared__ int merged[kFloorBins];  // rank 0: the cluster's
    __shared__ int s_valid, s_alive, s_bucket;
    __shared__ int s_warp[kFloorBins / 32];
    pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank());
    const int img = blockIdx.x / kFloorCtas;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (A.sample) {
        if (t < kFloorBins) {
            hist[t] = 0;
            merged[t] = 0;
        }
        if (t == 0) {
            s_valid = 0;
            s_alive = 0;
            s_bucket = 0;
        }
        __syncthreads();
        auto cleared = cluster.barrier_arrive();  // (waited for before anybody adds to rank 0's words)
        const YoloLevels& L = A.L;
        int nvalid = 0, nalive = 0;
        const int quarter = warp & 3;  // twenty of the eighty classes
        for (int block = rank * (kFloorThreads / 128) + (warp >> 2);; block += kFloorCtas * (kFloorThreads / 128)) {
            int lvl = 0, local = block;  // level and number of the 512-slot block inside it
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                const int nb = (3 * L.plane[l] + (1 << SHIFT) - 1) >> SHIFT;
                if (lvl == l && local >= nb) {
                    local -= nb;
                    ++lvl;
                }
            }
            if (lvl > 2) break;  // warp-uniform
            const int plane = L.plane[lvl], s0 = local << SHIFT;
            const int runs = max(1, min(1 << SHIFT, 3 * plane - s0) >> 5);
            const int slot = s0 + 32 * ((block * 5 + img * 3) % runs) + lane;
            const bool valid = slot < 3 * plane;
            int anchor, pos;
            yolo_slot(plane, valid ? slot : s0, anchor, pos);
            const float* src = L.map[lvl] + (static_cast<int64_t>(img) * 3 + anchor) * kYoloAttrib * plane + pos;
            const float tobj = __ldg(src + 4 * plane);
            const float* csrc = src + (5 + quarter * (kYoloClasses / 4)) * plane;
            float v[kYoloClasses / 4];
#pragma unroll
            for (int u = 0; u < kYoloClasses / 4; ++u) v[u] = __ldg(csrc + u * plane);
            const float so = __fdividef(1.0f, 1.0f + __expf(-tobj));
            const bool alive = valid && so > A.thr;
            const float cut = alive ? logit_cut(so, A.thr) : INFINITY;
#pragma unroll
            for (int u = 0; u < kYoloClasses / 4; ++u) {
                if (v[u] > cut) {
                    const float s = so * __fdividef(1.0f, 1.0f + __expf(-v[u]));
                    if (s > A.thr)
                        atomicAdd(&hist[hist_digit(static_cast<uint64_t>(__float_as_uint(s)) << 32, A.hist_base, A.hist_shift) /
                                        (kHistBins / kFloorBins)], 1);
                }
            }
            if (quarter == 0) {
                nvalid += __popc(__ballot_sync(kFullMask, valid));
                nalive += __popc(__ballot_sync(kFullMask, alive));
            }
        }
        __syncthreads();
        cluster.barrier_wait(std::move(cleared));
        if (lane == 0 && nvalid > 0) {
            atomicAdd(cluster.map_shared_rank(&s_valid, 0), nvalid);
            atomicAdd(cluster.map_shared_rank(&s_alive, 0), nalive);
        }
        if (t < kFloorBins && hist[t] != 0) atomicAdd(cluster.map_shared_rank(merged, 0) + t, hist[t]);
        cluster.sync();
        if (rank != 0) return;
        // the largest bucket d with (sampled candidates in buckets >= d) >= target
        const int total_valid = s_valid;
        const int aim = s_alive < kFloorSpread ? 3 : 2;
        const int target = static_cast<int>(static_cast<int64_t>(aim) * A.topk * total_valid / L.num_boxes) + 8;
        const int mine = t < kFloorBins ? merged[t] : 0;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_down_sync(kFullMask, incl, o);
            if (lane + o < 32) incl += x;
        }
        if (t < kFloorBins && lane == 0) s_warp[warp] = incl;
        __syncthreads();
        if (t < kFloorBins) {
            for (int w = warp + 1; w < kFloorBins / 32; ++w) incl += s_warp[w];
            if (incl >= target && incl - mine < target) s_bucket = t * (kHistBins / kFloorBins);
        }
        __syncthreads();
        if (t == 0) {
            const int d = total_valid >= kFloorMinSample || total_valid == L.num_boxes ? s_bucket : 0;
            A.floor[img] = d > 0 ? __uint_as_float(A.hist_base + (static_cast<uint32_t>(d) << A.hist_shift)) : 0.0f;
            A.counts[img] = 0;
            A.fallback[img] = 0;
        }
    } else if (rank == 0 && t == 0) {
        A.floor[img] = 0.0f;
        A.counts[img] = 0;
        A.fallback[img] = 0;
    }
}

// ---- decode -----------------------------------------------------------------------------------------------------------
constexpr int kDecThreads = 128;
constexpr int kDecWarps = kDecThreads / 32;
constexpr int kDecClasses = kYoloClasses / kDecWarps;  // classes per warp
constexpr int kDecStep = 10;                           // of which loaded at a time
constexpr int kDenseRow = kYoloClasses + 4;  // floats per slot of the dense form's staging: an odd number of 16-byte chunks, so that
                                             // eight neighbouring slots store to different banks

struct YoloDecodeArgs {
    YoloLevels L;
    float thr;
    const float* floor;  // [batch] or null
    float* boxes;        // [batch, N, 4] or null
    float* obj_out;      // dense form only, each may be null
    float* cls_out;
    uint64_t* keys;
    int32_t* counts;
    int64_t capacity;
    int32_t* status;
    int32_t* hist;       // [batch, kHistBins] or null
    uint32_t hist_base;
    int hist_shift;
};

struct __align__(16) YoloLive {  // a slot that can yield candidates
    float so;      // objectness score
    float cut;     // class logits at or below this cannot reach the bar
    int off;       // first class logit, from the start of the image's level
    uint32_t box;  // box index inside the image
};
struct __align__(8) YoloHit {
    float v;        // class logit (dense form: the finished score)
    uint32_t meta;  // live slot << 7 | class
};

// Slots [first, first + count) of a level of an image.
struct YoloTile {
    int img, lvl, s0;
};
__device__ __forceinline__ YoloTile yolo_tile(const YoloLevels& L, int index, int slots) {
    YoloTile T;
    int per_image = 0, begin[3];
#pragma unroll
    for (int l = 0; l < 3; ++l) {
        begin[l] = per_image;
        per_image += (3 * L.plane[l] + slots - 1) / slots;
    }
    T.img = index / per_image;
    const int tile = index - T.img * per_image;
    T.lvl = tile >= begin[2] ? 2 : (tile >= begin[1] ? 1 : 0);
    T.s0 = (tile - (T.lvl == 2 ? begin[2] : (T.lvl == 1 ? begin[1] : 0))) * slots;
    return T;
}

// Whole warps: appends the keys of the lanes with `pass` to the image's list.
__device__ __forceinline__ void yolo_append(const YoloDecodeArgs& A, int img, bool pass, float s, uint32_t flat) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(kFullMask, pass);
    if (m == 0u) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(A.counts + img, __popc(m));
    base = __shfl_sync(kFullMask, base, 0);
    if (pass) {
        const int64_t at = static_cast<int64_t>(base) + __popc(m & ((1u << lane) - 1u));
        if (at < A.capacity) A.keys[img * A.capacity + at] = make_key(s, flat);
        else if (A.status != nullptr) atomicOr(A.status, FB_STATUS_CAND_OVERFLOW);
        if (A.hist != nullptr)
            atomicAdd(A.hist + static_cast<int64_t>(img) * kHistBins +
                          hist_digit(static_cast<uint64_t>(__float_as_uint(s)) << 32, A.hist_base, A.hist_shift), 1);
    }
}

// The queued hits of a tile, evaluated together.
template <bool DENSE>
__device__ __forceinline__ void yolo_eval_queue(const YoloDecodeArgs& A, const YoloLive* live, const YoloHit* queue, int img, int n, float bar) {
    for (int i0 = 0; i0 < n; i0 += kDecThreads) {
        const int i = i0 + static_cast<int>(threadIdx.x);
        bool pass = i < n;
        float s = 0.0f;
        uint32_t flat = 0u;
        if (pass) {
            const YoloHit h = queue[i];
            const YoloLive o = live[h.meta >> 7];
            s = DENSE ? h.v : __fmul_rn(o.so, sigmoid_f32(h.v));
            flat = o.box * kYoloClasses + (h.meta & 127u);
            pass = s > A.thr && s >= bar;
        }
        yolo_append(A, img, pass, s, flat);
    }
}

// The same for a long queue: a warp evaluates its share first and makes room for all of it with one atomic (one for 32 hits
// each waits for the one before).  The evaluated scores go back to the queue.
template <bool DENSE>
__device__ __forceinline__ void yolo_eval_many(const YoloDecodeArgs& A, const YoloLive* live, YoloHit* queue, int img, int n, float bar) {
    constexpr uint32_t kNone = 0xffffffffu;
    const int t = threadIdx.x, lane = t & 31;
    int found = 0;
    for (int i0 = 0; i0 < n; i0 += kDecThreads) {
        const int i = i0 + t;
        bool pass = false;
        if (i < n) {
            const YoloHit h = queue[i];
            const YoloLive o = live[h.meta >> 7];
            const float s = DENSE ? h.v : __fmul_rn(o.so, sigmoid_f32(h.v));
            pass = s > A.thr && s >= bar;
            queue[i] = YoloHit{s, pass ? o.box * kYoloClasses + (h.meta & 127u) : kNone};  // (flat indices are below 2^32 - 1)
        }
        found += __popc(__ballot_sync(kFullMask, pass));
    }
    if (found == 0) return;
    int64_t at = 0;
    if (lane == 0) at = atomicAdd(A.counts + img, found);
    at = __shfl_sync(kFullMask, at, 0);
    for (int i0 = 0; i0 < n; i0 += kDecThreads) {
        const int i = i0 + t;
        const YoloHit h = i < n ? queue[i] : YoloHit{0.0f, kNone};
        const unsigned m = __ballot_sync(kFullMask, h.meta != kNone);
        if (h.meta != kNone) {
            const int64_t k = at + __popc(m & ((1u << lane) - 1u));
            if (k < A.capacity) A.keys[img * A.capacity + k] = make_key(h.v, h.meta);
            else if (A.status != nullptr) atomicOr(A.status, FB_STATUS_CAND_OVERFLOW);
            if (A.hist != nullptr)
                atomicAdd(A.hist + static_cast<int64_t>(img) * kHistBins +
                              hist_digit(static_cast<uint64_t>(__float_as_uint(h.v)) << 32, A.hist_base, A.hist_shift), 1);
        }
        at += __popc(m);
    }
}

// All candidates of a tile, for callers without a floor and for tiles whose hits did not fit the queue: in rounds of 32 live slots
// and STEP classes per warp; the queue is evaluated whenever another round might not fit (ROOM: its entries).  DENSE: the class
// scores come from s_cls.  (One live slot per thread through all its classes with an append for every class took 375 us for 32
// images at N(0, 1), seven candidates in a hundred: 320 global atomics a tile, most of them for a hit or two.)
template <int STEP>
constexpr int kRoundHits = 32 * STEP * kDecWarps;
template <bool DENSE, int STEP, int ROOM>
__device__ __noinline__ void yolo_collect_all(const YoloDecodeArgs* A, int lvl, int img, const YoloLive* live, int n, float bar,
                                              YoloHit* queue, int* counter) {
    extern __shared__ __align__(16) float s_cls[];  // [128][kDenseRow]
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int plane = A->L.plane[lvl];
    const float* img_map = A->L.map[lvl] + static_cast<int64_t>(img) * 3 * kYoloAttrib * plane;
    __syncthreads();  // whoever filled the queue before has seen how far
    if (t == 0) *counter = 0;
    __syncthreads();
    constexpr int kSteps = kDecClasses / STEP;
    static_assert(kDecClasses % STEP == 0, "whole steps");
    const int rounds = (n + 31) / 32 * kSteps;
    float v[STEP], cut = 0.0f;
    uint32_t first = 0u;  // of this lane's values: live slot << 7 | class
    auto load = [&](int round) {
        const int i = round / kSteps * 32 + lane, k0 = warp * kDecClasses + round % kSteps * STEP;
        const bool on = i < n;
        YoloLive o{0.0f, INFINITY, 0, 0u};
        if (on) o = live[i];
        cut = o.cut;
        first = static_cast<uint32_t>(i << 7 | k0);
#pragma unroll
        for (int u = 0; u < STEP; ++u) {
            if (DENSE) v[u] = on ? __fmul_rn(o.so, s_cls[i * kDenseRow + k0 + u]) : 0.0f;
            else v[u] = on ? __ldg(img_map + o.off + (k0 + u) * plane) : -INFINITY;
        }
    };
    load(0);
#pragma unroll 1
    for (int round = 0; round < rounds; ++round) {
        uint32_t hits = 0u;
#pragma unroll
        for (int u = 0; u < STEP; ++u) hits |= (DENSE ? v[u] > A->thr && v[u] >= bar : v[u] > cut) ? 1u << u : 0u;
        int at = 0;
        if (hits != 0u) {
            at = atomicAdd(counter, __popc(hits));
#pragma unroll
            for (int u = 0; u < STEP; ++u)
                if ((hits >> u) & 1u) queue[at++] = YoloHit{v[u], first + static_cast<uint32_t>(u)};
        }
        const bool last = round + 1 == rounds;
        if (!last) load(round + 1);  // on its way while these hits are evaluated
        if (__syncthreads_or(last || at > ROOM - kRoundHits<STEP> ? 1 : 0) == 0) continue;
        yolo_eval_many<DENSE>(*A, live, queue, img, *counter, bar);
        __syncthreads();
        if (t == 0) *counter = 0;
        __syncthreads();
    }
}

// One CTA per tile of 128 * E slots.  First the objectness of its slots, E per thread; the slots that clear the bar (one in seven
// at N(0, 1), a few per cent behind a trained head) are listed in shared memory; then lane k of every warp takes live slot k
// through the warp's twenty class planes.  The planes are streamed from DRAM almost whole either way (a 128-byte line rarely
// holds no live slot), so what the list saves is instructions: forms in which every lane kept four neighbouring slots, dead
// ones included, executed 17 to 22 million warp instructions for 64 images and took 42 to 53 us whatever the loads looked
// like (registers, ten planes at a time; asynchronous copies, fifteen at a time, next tile prefetched).
// E = 2 to 4 fill the lanes (35 to 70 live slots); E = 1 makes more CTAs where there are few tiles (launch_yolo_decode).
// ALL: no floor, every candidate above the threshold is wanted (yolo_collect_all from the start, with a longer queue; in the other
// form that queue would take the L1 cache its loads need: 64 images 76.0 us instead of 71.2).
template <int E, bool BOXES, bool ALL>
__global__ void __launch_bounds__(kDecThreads, 8)
yolo_decode_kernel(const __grid_constant__ YoloDecodeArgs A) {
    constexpr int kSlots = kDecThreads * E;
    constexpr int kQueue = ALL ? kRoundHits<kDecStep> * 3 / 2 : kRoundHits<kDecStep>;  // hits: some 1.5 per live slot with a floor
    static_assert(kQueue >= 2 * kSlots, "room for the usual hits of a tile");
    __shared__ YoloLive live[kSlots];
    __shared__ YoloHit queue[kQueue];
    __shared__ int s_live, s_queued;
    pdl_launch_dependents();
    const YoloLevels& L = A.L;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const YoloTile T = yolo_tile(L, blockIdx.x, kSlots);
    const int plane = L.plane[T.lvl], nslots = 3 * plane;
    const float* __restrict__ img_map = L.map[T.lvl] + static_cast<int64_t>(T.img) * 3 * kYoloAttrib * plane;
    float so[E];
    int off[E];
    uint32_t box[E];
    bool valid[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int slot = T.s0 + e * kDecThreads + t;
        valid[e] = slot < nslots;
        int anchor, pos;
        yolo_slot(plane, valid[e] ? slot : T.s0, anchor, pos);
        off[e] = anchor * kYoloAttrib * plane + pos;
        box[e] = static_cast<uint32_t>(L.box_begin[T.lvl] + pos * 3 + anchor);
        so[e] = __ldg(img_map + off[e] + 4 * plane);
    }
    if (t == 0) {
        s_live = 0;
        s_queued = 0;
    }
    if (BOXES) {
#pragma unroll 1
        for (int e = 0; e < E; ++e) {
            const int slot = T.s0 + e * kDecThreads + t;
            if (slot >= nslots) continue;
            int anchor, pos;
            yolo_slot(plane, slot, anchor, pos);
            const float* src = img_map + anchor * kYoloAttrib * plane + pos;
            reinterpret_cast<float4*>(A.boxes)[static_cast<int64_t>(T.img) * L.num_boxes + L.box_begin[T.lvl] + pos * 3 + anchor] =
                yolo_box(L, T.lvl, anchor, pos, __ldg(src), __ldg(src + plane), __ldg(src + 2 * plane), __ldg(src + 3 * plane));
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) so[e] = sigmoid_f32(so[e]);
    pdl_wait();  // the floor, and the counters that the floor kernel cleared
    const float bar = fmaxf(A.thr, A.floor != nullptr ? __ldcg(A.floor + T.img) : 0.0f);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) {
        // a score is so * sigmoid(v) <= so: the box can only yield candidates if so itself clears both bars
        const bool alive = valid[e] && so[e] > A.thr && so[e] >= bar;
        const unsigned m = __ballot_sync(kFullMask, alive);
        int base = 0;
        if (lane == 0 && m != 0u) base = atomicAdd(&s_live, __popc(m));
        base = __shfl_sync(kFullMask, base, 0);
        if (alive) live[base + __popc(m & ((1u << lane) - 1u))] = YoloLive{so[e], logit_cut(so[e], bar), off[e] + 5 * plane, box[e]};
    }
    __syncthreads();
    const int n = s_live;
    if (n == 0) return;
    bool all = ALL;
    if (!ALL) {
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < n;
            YoloLive o{0.0f, INFINITY, 0, 0u};
            if (on) o = live[i];
            const float* p = img_map + o.off + warp * kDecClasses * plane;
#pragma unroll 1
            for (int k0 = 0; k0 < kDecClasses; k0 += kDecStep) {
                float v[kDecStep];
#pragma unroll
                for (int u = 0; u < kDecStep; ++u) v[u] = on ? __ldg(p + (k0 + u) * plane) : -INFINITY;
                uint32_t hits = 0u;
#pragma unroll
                for (int u = 0; u < kDecStep; ++u) hits |= v[u] > o.cut ? 1u << u : 0u;
                if (hits != 0u) {
                    int at = atomicAdd(&s_queued, __popc(hits));
#pragma unroll
                    for (int u = 0; u < kDecStep; ++u) {
                        if ((hits >> u) & 1u) {
                            if (at < kQueue) queue[at] = YoloHit{v[u], static_cast<uint32_t>(i << 7 | (warp * kDecClasses + k0 + u))};
                            ++at;
                        }
                    }
                }
            }
        }
        __syncthreads();
        all = s_queued > kQueue;
    }
    if (all) yolo_collect_all<false, kDecStep, kQueue>(&A, T.lvl, T.img, live, n, bar, queue, &s_queued);
    else yolo_eval_queue<false>(A, live, queue, T.img, s_queued, bar);
}

// The dense form, one CTA per tile of 128 slots: the objectness and class scores are outputs too; every score is formed, staged
// in shared memory and written as whole 320-byte rows (written straight from the threads, every store instruction touched 32
// rows: 145 us for 8 images of 608 x 608 against 19 us of traffic).
// The exact sigmoid of every logit bounds it (some twenty instructions each), so everything else goes four classes at a time, with
// reciprocals that the compiler can interleave; and the class loop stays a loop: unrolled, a warp passes once through 30 KB of
// instructions and waits for most of them to arrive (49 us for 8 images of 608 x 608; 36 as it is).
// ALL: no floor (790 hits in a tile at N(0, 1)).
template <bool ALL>
__global__ void __launch_bounds__(kDecThreads, 4)
yolo_decode_dense_kernel(const __grid_constant__ YoloDecodeArgs A) {
    __shared__ YoloLive live[kDecThreads];  // every slot of the tile; so = 0: it cannot yield candidates
    constexpr int kStep = ALL ? 10 : 4, kQueue = kRoundHits<kStep>;
    __shared__ YoloHit queue[kQueue];
    __shared__ int s_queued;
    extern __shared__ __align__(16) float s_cls[];  // [128][kDenseRow]
    pdl_launch_dependents();
    const YoloLevels& L = A.L;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const YoloTile T = yolo_tile(L, blockIdx.x, kDecThreads);
    const int plane = L.plane[T.lvl], nslots = 3 * plane;
    const float* __restrict__ img_map = L.map[T.lvl] + static_cast<int64_t>(T.img) * 3 * kYoloAttrib * plane;
    const bool valid = T.s0 + t < nslots;
    int anchor, pos;
    yolo_slot(plane, valid ? T.s0 + t : T.s0, anchor, pos);
    const float* src = img_map + anchor * kYoloAttrib * plane + pos;
    const uint32_t box = static_cast<uint32_t>(L.box_begin[T.lvl] + pos * 3 + anchor);
    const int64_t gbox = static_cast<int64_t>(T.img) * L.num_boxes + box;
    const float so = sigmoid_f32(__ldg(src + 4 * plane));
    if (valid) {
        if (A.boxes != nullptr)
            reinterpret_cast<float4*>(A.boxes)[gbox] =
                yolo_box(L, T.lvl, anchor, pos, __ldg(src), __ldg(src + plane), __ldg(src + 2 * plane), __ldg(src + 3 * plane));
        if (A.obj_out != nullptr) A.obj_out[gbox] = so;
    }
    if (t == 0) s_queued = 0;
    live[t] = YoloLive{valid && so > A.thr ? so : 0.0f, 0.0f, static_cast<int>(src - img_map) + 5 * plane, box};
    __syncthreads();
    const float* p4[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) p4[e] = img_map + live[32 * e + lane].off + warp * kDecClasses * plane;
    // a step's 16 logits are on their way while the step before is worked on, the first ones while the floor is waited for
    float next[4][4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) next[e][u] = __ldg(p4[e] + (k0 + u) * plane);
    };
    fetch(0);
    pdl_wait();
    const float bar = fmaxf(A.thr, A.floor != nullptr ? __ldcg(A.floor + T.img) : 0.0f);
    float cut4[4];  // class scores below this cannot bring the product to the bar
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float so_e = live[32 * e + lane].so;
        cut4[e] = so_e > 0.0f && so_e >= bar ? __fdividef(bar, so_e) * (1.0f - 1.0e-5f) : INFINITY;
    }
#pragma unroll 1
    for (int k0 = 0; k0 < kDecClasses; k0 += 4) {
        float v[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int u = 0; u < 4; ++u) v[e][u] = next[e][u];
        if (k0 + 4 < kDecClasses) fetch(k0 + 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int slot = 32 * e + lane;
            sigmoid_f32_n(v[e]);
            *reinterpret_cast<float4*>(s_cls + slot * kDenseRow + warp * kDecClasses + k0) = make_float4(v[e][0], v[e][1], v[e][2], v[e][3]);
            if (fmaxf(fmaxf(v[e][0], v[e][1]), fmaxf(v[e][2], v[e][3])) >= cut4[e]) {
                const float so_e = live[slot].so;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float s = __fmul_rn(so_e, v[e][u]);
                    if (s > A.thr && s >= bar) {
                        const int at = atomicAdd(&s_queued, 1);
                        if (at < kQueue) queue[at] = YoloHit{s, static_cast<uint32_t>(slot << 7 | (warp * kDecClasses + k0 + u))};
                    }
                }
            }
        }
    }
    __syncthreads();
    if (A.cls_out != nullptr) {
        constexpr int kQuads = kYoloClasses / 4;
        const int total = min(kDecThreads, nslots - T.s0) * kQuads;
        float* img_out = A.cls_out + static_cast<int64_t>(T.img) * L.num_boxes * kYoloClasses;
        if ((reinterpret_cast<uintptr_t>(img_out) & 15) == 0) {
            float4* out = reinterpret_cast<float4*>(img_out);
            int slot = t / kQuads, c = t - slot * kQuads;
            for (int i = t; i < total; i += kDecThreads) {
                out[static_cast<int64_t>(live[slot].box) * kQuads + c] = *reinterpret_cast<const float4*>(s_cls + slot * kDenseRow + 4 * c);
                slot += kDecThreads / kQuads;
                c += kDecThreads % kQuads;
                if (c >= kQuads) {
                    c -= kQuads;
                    ++slot;
                }
            }
        } else {  // a caller's array off a 16-byte boundary
            for (int i = t; i < 4 * total; i += kDecThreads) {
                const int slot = i / kYoloClasses, c = i - slot * kYoloClasses;
                img_out[static_cast<int64_t>(live[slot].box) * kYoloClasses + c] = s_cls[slot * kDenseRow + c];
            }
        }
    }
    if (s_queued > kQueue) yolo_collect_all<true, kStep, kQueue>(&A, T.lvl, T.img, live, kDecThreads, bar, queue, &s_queued);
    else if (s_queued > kDecThreads) yolo_eval_many<true>(A, live, queue, T.img, s_queued, bar);
    else yolo_eval_queue<true>(A, live, queue, T.img, s_queued, bar);
}

// Development switch (functs_b200_debug_set "yolo_prune"): 0 keeps every candidate above the score threshold.
static std::atomic<int> g_yolo_prune{1};
void yolo_set_prune(int on) { g_yolo_prune.store(on ? 1 : 0, std::memory_order_relaxed); }

static const float kAnchors[3][3][2] = {{{116, 90}, {156, 198}, {373, 326}},
                                        {{30, 61}, {62, 45}, {59, 119}},
                                        {{10, 13}, {16, 30}, {33, 23}}};  // yolov3_bbox.py:191-193
static const float kStrides[3] = {32.f, 16.f, 8.f};

static int yolo_levels(const float* map0, const float* map1, const float* map2, int batch, int s0, int s1, int s2, YoloLevels& L) {
    FB_REQUIRE(map0 && map1 && map2, "yolo_decode: null pointer");
    FB_REQUIRE(batch > 0 && s0 > 0 && s1 > 0 && s2 > 0 && s0 <= 1024 && s1 <= 1024 && s2 <= 1024, "yolo_decode: bad sizes");
    const int S[3] = {s0, s1, s2};
    const float* maps[3] = {map0, map1, map2};
    int tiles = 0;
    int64_t boxes = 0;
    for (int l = 0; l < 3; ++l) {
        L.map[l] = maps[l];
        L.size[l] = S[l];
        L.plane[l] = S[l] * S[l];
        tiles += (3 * L.plane[l] + kDecThreads - 1) / kDecThreads;
        L.box_begin[l] = static_cast<int>(boxes);
        boxes += 3 * L.plane[l];
        L.stride[l] = kStrides[l];
        for (int a = 0; a < 3; ++a) {
            L.anchor_w[l][a] = kAnchors[l][a][0];
            L.anchor_h[l][a] = kAnchors[l][a][1];
        }
    }
    FB_REQUIRE(boxes * kYoloClasses < (1ll << 32), "yolo_decode: flat index exceeds 32 bits");
    FB_REQUIRE(static_cast<int64_t>(tiles) * batch < (1ll << 31), "yolo_decode: too many tiles");
    L.num_boxes = static_cast<int>(boxes);
    return FB_OK;
}

// A run per 512 slots, or all runs if that leaves too small a sample.
static int yolo_floor_shift(const YoloLevels& L) {
    int sampled = 0;
    for (int l = 0; l < 3; ++l)
        for (int left = 3 * L.plane[l]; left > 0 && sampled < kFloorMinSample; left -= 1 << kFloorShift) sampled += std::min(left, 32);
    return sampled >= kFloorMinSample ? kFloorShift : kFloorAll;
}

// pdl: the launch may overlap the end of the kernel before it (the floor kernel)
static int launch_yolo_decode(const YoloDecodeArgs& a, int batch, bool pdl, cudaStream_t st) {
    FB_REQUIRE(a.keys && a.counts, "yolo_decode: null pointer");
    FB_REQUIRE(a.capacity > 0, "yolo_decode: bad sizes");
    FB_REQUIRE(a.thr > 0.0f, "yolo_decode: score threshold must be positive (keys require positive scores)");
    FB_REQUIRE((reinterpret_cast<uintptr_t>(a.boxes) & 15) == 0, "yolo_decode: boxes must be 16-byte aligned");
    auto tiles = [&](int slots) {
        int n = 0;
        for (int l = 0; l < 3; ++l) n += (3 * a.L.plane[l] + slots - 1) / slots;
        return n * batch;
    };
    if (a.obj_out != nullptr || a.cls_out != nullptr) {
        const size_t smem = sizeof(float) * kDecThreads * kDenseRow;
        auto kernel = a.floor == nullptr ? yolo_decode_dense_kernel<true> : yolo_decode_dense_kernel<false>;
        FB_TRY(check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                          "yolo_decode attr"));
        return launch_after(kernel, dim3(static_cast<unsigned>(tiles(kDecThreads))), dim3(kDecThreads), smem, st, pdl,
                            "yolo_decode_dense_kernel", a);
    }
    auto run = [&](auto kernel, int n) {
        return launch_after(kernel, dim3(static_cast<unsigned>(n)), dim3(kDecThreads), 0, st, pdl, "yolo_decode_kernel", a);
    };
    // larger tiles once tiles of four slots per thread make four CTAs per SM
    const int large = tiles(4 * kDecThreads), one = tiles(kDecThreads);
    const bool is_large = large >= 4 * kNumSMs;
    if (a.floor == nullptr || a.boxes != nullptr) {
        const int n = is_large ? large : one;
        if (a.floor == nullptr) return is_large ? run(yolo_decode_kernel<4, true, true>, n) : run(yolo_decode_kernel<1, true, true>, n);
        return is_large ? run(yolo_decode_kernel<4, true, false>, n) : run(yolo_decode_kernel<1, true, false>, n);
    }
    // Few tiles: one slot per thread, even in a second wave: a tile of two whose slots are all live takes twice as long, and the others end
    // before it.  Whole call, us, one / two slots: 16 images of 416 x 416 at random 28.6 / 29.5, with few live boxes 25.3 / 24.0, of live
    // boxes only 37.7 / 41.8, with 160 live slots in one run 68 / 86; 8 of 608 x 608 30.5 / 29.2, 26.9 / 24.9, 39.7 / 41.9, 99 / 119.
    // Otherwise two, or three if only then all run at once (eight CTAs per SM): small tiles end together, and a few that are left for a
    // second wave wait for the first.  One / two / three / four slots: 32 images of 416 x 416 42 / 42 / 41 / 43, 64 63.5 / 65 / 67 / 70, 64
    // with few live boxes 46.5 / 43 / 43 / 43; 30 of 608 x 608 62 / 62 / 65 / 67.
    if (!is_large) return run(yolo_decode_kernel<1, false, false>, one);
    constexpr int kWave = 8 * kNumSMs;
    const int two = tiles(2 * kDecThreads), three = tiles(3 * kDecThreads);
    if (two > kWave && three <= kWave) return run(yolo_decode_kernel<3, false, false>, three);
    return run(yolo_decode_kernel<2, false, false>, two);
}

static inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// Scratch of the one-call post-process: [candidate counts][fallback flags][floors][keys][dense suppression matrix].
struct YoloScratch {
    int64_t counts_off, fallback_off, floor_off, keys_off, mask_off, total;
};

static YoloScratch yolo_scratch_layout(int batch, int64_t capacity) {
    YoloScratch S;
    const int64_t words = align_up(static_cast<int64_t>(batch) * 4, 256);
    S.counts_off = 0;
    S.fallback_off = words;
    S.floor_off = 2 * words;
    S.keys_off = 3 * words;
    S.mask_off = align_up(S.keys_off + static_cast<int64_t>(batch) * capacity * 8, 256);
    S.total = align_up(S.mask_off + yolo_post_mask_bytes(batch), 256);
    return S;
}

}  // namespace fb

extern "C" {

int functs_b200_yolo_decode(const float* map0, const float* map1, const float* map2, int32_t batch, int32_t s0,
                            int32_t s1, int32_t s2, float score_thr, float* boxes, float* obj_out, float* cls_out,
                            uint64_t* cand_keys, int32_t* cand_counts, int64_t capacity, int32_t* hist,
                            int32_t* status, void* stream) {
    using namespace fb;
    cudaStream_t st = as_stream(stream);
    YoloDecodeArgs a{};
    FB_REQUIRE(boxes != nullptr && cand_counts != nullptr, "yolo_decode: null pointer");
    FB_TRY(yolo_levels(map0, map1, map2, batch, s0, s1, s2, a.L));
    const HistParams hp = hist_params_for(score_thr);
    a.thr = score_thr;
    a.boxes = boxes;
    a.obj_out = obj_out;
    a.cls_out = cls_out;
    a.keys = cand_keys;
    a.counts = cand_counts;
    a.capacity = capacity;
    a.status = status;
    a.hist = hist;
    a.hist_base = hp.base;
    a.hist_shift = hp.shift;
    FB_TRY(check_cuda(cudaMemsetAsync(cand_counts, 0, sizeof(int32_t) * batch, st), "memset cand_counts"));
    if (hist != nullptr) FB_TRY(check_cuda(cudaMemsetAsync(hist, 0, sizeof(int32_t) * batch * kHistBins, st), "memset hist"));
    return launch_yolo_decode(a, batch, false, st);
}

int64_t functs_b200_yolo_scratch_bytes(int32_t batch, int32_t s0, int32_t s1, int32_t s2, int64_t capacity,
                                       int32_t topk) {
    (void)s0;
    (void)s1;
    (void)s2;
    if (batch <= 0 || capacity <= 0 || topk <= 0) return 0;
    return fb::yolo_scratch_layout(batch, capacity).total;
}

int functs_b200_yolo_postprocess(const float* map0, const float* map1, const float* map2, int32_t batch, int32_t s0,
                                 int32_t s1, int32_t s2, float score_thr, int32_t topk, float iou_thr,
                                 int64_t capacity, float* boxes, float* dets, int64_t* labels, int64_t* flat_ids,
                                 int32_t* out_counts, int32_t* status, void* scratch, void* stream) {
    return functs_b200_yolo_postprocess_dense(map0, map1, map2, batch, s0, s1, s2, score_thr, topk, iou_thr, capacity,
                                              boxes, nullptr, nullptr, dets, labels, flat_ids, out_counts, nullptr,
                                              status, scratch, stream);
}

int functs_b200_yolo_postprocess_dense(const float* map0, const float* map1, const float* map2, int32_t batch,
                                       int32_t s0, int32_t s1, int32_t s2, float score_thr, int32_t topk,
                                       float iou_thr, int64_t capacity, float* boxes, float* obj_out, float* cls_out,
                                       float* dets, int64_t* labels, int64_t* flat_ids, int32_t* out_counts,
                                       int32_t* records, int32_t* status, void* scratch, void* stream) {
    FB_REQUIRE(boxes != nullptr && flat_ids != nullptr, "yolo_postprocess: null pointer");
    return functs_b200_yolo_detect(map0, map1, map2, batch, s0, s1, s2, score_thr, topk, iou_thr, capacity, boxes, obj_out,
                                   cls_out, dets, labels, flat_ids, out_counts, records, nullptr, status, scratch, stream);
}

int functs_b200_yolo_detect(const float* map0, const float* map1, const float* map2, int32_t batch, int32_t s0, int32_t s1,
                            int32_t s2, float score_thr, int32_t topk, float iou_thr, int64_t capacity, float* boxes,
                            float* obj_out, float* cls_out, float* dets, int64_t* labels, int64_t* flat_ids,
                            int32_t* out_counts, int32_t* records, int32_t* host_counts, int32_t* status, void* scratch,
                            void* stream) {
    using namespace fb;
    FB_REQUIRE(scratch != nullptr && (reinterpret_cast<uintptr_t>(scratch) & 255) == 0,
               "yolo_postprocess: scratch must be non-null and 256-byte aligned");
    FB_REQUIRE(batch > 0 && batch <= 65535 && capacity > 0 && capacity < (1ll << 31), "yolo_postprocess: bad sizes");
    cudaStream_t st = as_stream(stream);
    const YoloScratch S = yolo_scratch_layout(batch, capacity);
    unsigned char* base = static_cast<unsigned char*>(scratch);
    YoloDecodeArgs d{};
    FB_TRY(yolo_levels(map0, map1, map2, batch, s0, s1, s2, d.L));
    const HistParams hp = hist_params_for(score_thr);
    YoloFloorArgs f{};
    f.L = d.L;
    f.thr = score_thr;
    f.hist_base = hp.base;
    f.hist_shift = hp.shift;
    f.topk = topk;
    f.sample = g_yolo_prune.load(std::memory_order_relaxed);
    f.floor = reinterpret_cast<float*>(base + S.floor_off);
    f.counts = reinterpret_cast<int32_t*>(base + S.counts_off);
    f.fallback = reinterpret_cast<int32_t*>(base + S.fallback_off);
    YoloPostArgs p{};
    p.keys = reinterpret_cast<uint64_t*>(base + S.keys_off);
    p.counts = f.counts;
    p.fallback = f.fallback;
    p.floor = f.floor;
    p.capacity = capacity;
    p.boxes = boxes;
    p.mask = reinterpret_cast<uint32_t*>(base + S.mask_off);
    p.thr = score_thr;
    p.iou_thr = iou_thr;
    p.topk = topk;
    p.dets = dets;
    p.labels = labels;
    p.flat_ids = flat_ids;
    p.out_counts = out_counts;
    p.host_counts = host_counts;
    p.records = records;
    p.status = status;
    FB_TRY(check_yolo_post(batch, p));  // before anything is launched
    record_stage_event(0, st);
    auto floor_kernel = yolo_floor_shift(d.L) == kFloorShift ? yolo_floor_kernel<kFloorShift> : yolo_floor_kernel<kFloorAll>;
    floor_kernel<<<static_cast<unsigned>(batch) * kFloorCtas, kFloorThreads, 0, st>>>(f);
    count_launch();
    FB_TRY(check_launch("yolo_floor_kernel"));
    record_stage_event(1, st);
    d.thr = score_thr;
    d.floor = f.floor;
    d.boxes = boxes;
    d.obj_out = obj_out;
    d.cls_out = cls_out;
    d.keys = reinterpret_cast<uint64_t*>(base + S.keys_off);
    d.counts = f.counts;
    d.capacity = capacity;
    d.status = status;
    FB_TRY(launch_yolo_decode(d, batch, true, st));
    record_stage_event(2, st);
    const int rc = launch_yolo_post(d.L, batch, p, st);
    record_stage_event(3, st);
    return rc;
}

}  // extern "C"
