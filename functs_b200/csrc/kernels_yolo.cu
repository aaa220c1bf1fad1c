// C2, first half: a score floor per image from a sample of its boxes, then one pass over the logits that leaves the boxes'
// candidates (yolo.cuh says what the group computes; kernels_yolo_post.cu is the second half).
//
// What bounds it: reading the 80 class planes and the objectness plane of every level (81 of the 85 channels; the box channels
// are only read for callers that want every box).  Everything else is kept off that stream:
//   - the score floor.  The program keeps the topk best candidates of an image, but with logits near N(0, 1) one score in
//     thirteen passes the threshold: 65 000 per image.  yolo_floor_kernel takes the scores of one box in sixteen (eight
//     neighbouring slots of every tile, one 32-byte sector per plane) and picks the score that about 2 * topk candidates
//     should reach.  The floor is a guess: whoever uses the list has to see that it holds at least topk candidates, and
//     takes the exact way otherwise (yolo_post_kernel does).
//   - with the floor known before the first class logit is read, a box whose objectness lies below it is never walked, and
//     a class logit costs a compare against its box's cut.  Hits (about two in a thousand) are queued in shared memory and
//     evaluated exactly, together, at the end of the tile.
// Before, the floor was found while the kernel ran, from a histogram in global memory that every candidate incremented: the
// first wave of CTAs had none, and 12 000 candidates per image reached the selection.
#include <cooperative_groups.h>

#include <atomic>

#include "yolo.cuh"

namespace fb {

namespace cg = cooperative_groups;

// ---- score floor ------------------------------------------------------------------------------------------------------
constexpr int kFloorCtas = 8;        // one cluster per image
constexpr int kFloorThreads = 384;   // 8 x 12 warps: one tile per warp up to 96 tiles (84 at 13 / 26 / 52)
constexpr int kFloorMinSample = 256; // sampled boxes below which a floor is not worth the risk (small pyramids)

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
__global__ void __cluster_dims__(kFloorCtas, 1, 1) __launch_bounds__(kFloorThreads)
yolo_floor_kernel(const YoloFloorArgs A) {
    __shared__ __align__(16) int hist[kHistBins];
    __shared__ int s_valid, s_bucket;
    __shared__ int s_warp[8];
    pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank());
    const int img = blockIdx.x / kFloorCtas;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (A.sample) {
        if (rank == 0) {
            for (int i = t; i < kHistBins; i += kFloorThreads) hist[i] = 0;
            if (t == 0) {
                s_valid = 0;
                s_bucket = 0;
            }
        }
        cluster.sync();
        int* hist0 = cluster.map_shared_rank(hist, 0);
        int* valid0 = cluster.map_shared_rank(&s_valid, 0);
        const YoloLevels& L = A.L;
        int nvalid = 0;
        for (int tile = rank * (kFloorThreads / 32) + warp; tile < L.tile_begin[3]; tile += kFloorCtas * (kFloorThreads / 32)) {
            const int lvl = tile >= L.tile_begin[2] ? 2 : (tile >= L.tile_begin[1] ? 1 : 0);
            const int plane = L.plane[lvl];
            const int s0 = (tile - L.tile_begin[lvl]) * kYoloTile;
            const int groups = max(1, min(kYoloTile, 3 * plane - s0) >> 3);
            const int slot = s0 + 8 * ((tile * 5 + img * 3) % groups) + (lane & 7);
            const bool valid = slot < 3 * plane;
            int anchor, pos;
            yolo_slot(plane, valid ? slot : s0, anchor, pos);
            const float* src = L.map[lvl] + (static_cast<int64_t>(img) * 3 + anchor) * kYoloAttrib * plane + pos;
            const float tobj = __ldg(src + 4 * plane);
            const float* csrc = src + (5 + (lane >> 3)) * plane;
            float v[kYoloClasses / 4];
#pragma unroll
            for (int u = 0; u < kYoloClasses / 4; ++u) v[u] = __ldg(csrc + u * 4 * plane);
            const float so = __fdividef(1.0f, 1.0f + __expf(-tobj));
            const bool alive = valid && so > A.thr;
            const float cut = alive ? logit_cut(so, A.thr) : INFINITY;
#pragma unroll
            for (int u = 0; u < kYoloClasses / 4; ++u) {
                if (v[u] > cut) {
                    const float s = so * __fdividef(1.0f, 1.0f + __expf(-v[u]));
                    if (s > A.thr)
                        atomicAdd(hist0 + hist_digit(static_cast<uint64_t>(__float_as_uint(s)) << 32, A.hist_base, A.hist_shift), 1);
                }
            }
            nvalid += __popc(__ballot_sync(kFullMask, valid)) >> 2;  // four lanes per box
        }
        if (lane == 0 && nvalid > 0) atomicAdd(valid0, nvalid);
        cluster.sync();
        if (rank != 0) return;
        // the largest bucket d with (sampled candidates in buckets >= d) >= target
        const int total_valid = s_valid;
        const int target = static_cast<int>(2ll * A.topk * total_valid / L.num_boxes) + 8;
        int h[8], mine = 0, incl = 0;
        if (t < 256) {
            const int4 a = reinterpret_cast<const int4*>(hist)[2 * t], b = reinterpret_cast<const int4*>(hist)[2 * t + 1];
            h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
            h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
#pragma unroll
            for (int k = 0; k < 8; ++k) mine += h[k];
            incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_down_sync(kFullMask, incl, o);
                if (lane + o < 32) incl += x;
            }
            if (lane == 0) s_warp[warp] = incl;
        }
        __syncthreads();
        if (t < 256) {
            for (int w = warp + 1; w < 8; ++w) incl += s_warp[w];
            if (incl >= target && incl - mine < target) {
                int cum = incl - mine, d = 7;
#pragma unroll
                for (int k = 7; k >= 0; --k) {
                    if (cum < target) {
                        cum += h[k];
                        d = k;
                    }
                }
                s_bucket = 8 * t + d;
            }
        }
        __syncthreads();
        if (t == 0) {
            const int d = total_valid >= kFloorMinSample ? s_bucket : 0;
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
constexpr int kDecQueue = 512;                    // queued hits of a tile (a floored tile has some twenty); more are evaluated on the spot
constexpr int kDecWarps = kYoloTile / 32;
constexpr int kDecClasses = kYoloClasses / kDecWarps;  // classes per warp
constexpr int kDecStep = 10;                      // class planes of a warp in flight: 5 KB

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

struct __align__(8) YoloHit {
    float v;        // class logit (dense form: the finished score)
    uint32_t meta;  // slot << 7 | class
};

struct YoloTileSmem {
    float cut[kYoloTile];     // class logits at or below this cannot reach the bar; +inf: the slot is dead
    float so[kYoloTile];      // objectness score
    uint32_t box[kYoloTile];  // box index inside the image
    YoloHit queue[kDecQueue];
    int queued;
};

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
// One lane on its own (the queue is full).
__device__ __noinline__ void yolo_append_one(const YoloDecodeArgs* A, int img, float s, uint32_t flat) {
    const int64_t at = atomicAdd(A->counts + img, 1);
    if (at < A->capacity) A->keys[img * A->capacity + at] = make_key(s, flat);
    else if (A->status != nullptr) atomicOr(A->status, FB_STATUS_CAND_OVERFLOW);
    if (A->hist != nullptr)
        atomicAdd(A->hist + static_cast<int64_t>(img) * kHistBins +
                      hist_digit(static_cast<uint64_t>(__float_as_uint(s)) << 32, A->hist_base, A->hist_shift), 1);
}

// The slot of lane `lane`, element e of a tile: four neighbours per lane where the planes are 16-byte aligned (a group of four
// then lies inside one anchor), else a warp-wide run per element.
template <bool VEC>
__device__ __forceinline__ int tile_slot(int lane, int e) {
    return VEC ? 4 * lane + e : 32 * e + lane;
}

// Warp `warp` of a tile walks its twenty class planes: four slots per lane, ten planes in flight.
template <bool VEC>
__device__ __forceinline__ void yolo_walk(const YoloDecodeArgs& A, YoloTileSmem& sm, const float* __restrict__ img_map, int plane, int s0,
                                          int nslots, int img, float bar) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float cut[4];
    int off[4];
    if (VEC) {
        const float4 c = reinterpret_cast<const float4*>(sm.cut)[lane];
        cut[0] = c.x; cut[1] = c.y; cut[2] = c.z; cut[3] = c.w;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (!VEC) cut[e] = sm.cut[32 * e + lane];
        int anchor, pos;
        yolo_slot(plane, min(s0 + tile_slot<VEC>(lane, e), nslots - 1), anchor, pos);
        off[e] = (anchor * kYoloAttrib + 5 + warp * kDecClasses) * plane + pos;
    }
    const bool on = cut[0] < INFINITY || cut[1] < INFINITY || cut[2] < INFINITY || cut[3] < INFINITY;
#pragma unroll 1
    for (int k0 = 0; k0 < kDecClasses; k0 += kDecStep) {
        uint32_t hits[2] = {0u, 0u};
        if (on) {
            float4 v[kDecStep];
            if (VEC) {
                const float* p = img_map + off[0] + k0 * plane;
#pragma unroll
                for (int u = 0; u < kDecStep; ++u) v[u] = __ldg(reinterpret_cast<const float4*>(p + u * plane));
            } else {
#pragma unroll
                for (int u = 0; u < kDecStep; ++u) {
                    const float* p = img_map + (k0 + u) * plane;
                    v[u] = make_float4(__ldg(p + off[0]), __ldg(p + off[1]), __ldg(p + off[2]), __ldg(p + off[3]));
                }
            }
#pragma unroll
            for (int u = 0; u < kDecStep; ++u) {
                const int sh = 4 * (u % 5);
                uint32_t& h = hits[u / 5];
                h |= v[u].x > cut[0] ? 1u << sh : 0u;
                h |= v[u].y > cut[1] ? 2u << sh : 0u;
                h |= v[u].z > cut[2] ? 4u << sh : 0u;
                h |= v[u].w > cut[3] ? 8u << sh : 0u;
            }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t h = hits[half];
            if (h == 0u) continue;
            int at = atomicAdd(&sm.queued, __popc(h));
            while (h != 0u) {
                const int k = __ffs(h) - 1;
                h &= h - 1u;
                const int e = k & 3, c = k0 + 5 * half + (k >> 2);
                const int o = e == 0 ? off[0] : (e == 1 ? off[1] : (e == 2 ? off[2] : off[3]));
                const float v = __ldg(img_map + o + c * plane);  // (read again: a hit's register cannot be named at run time)
                const int slot = tile_slot<VEC>(lane, e), cls = warp * kDecClasses + c;
                if (at < kDecQueue) {
                    sm.queue[at].v = v;
                    sm.queue[at].meta = static_cast<uint32_t>(slot << 7 | cls);
                } else {
                    const float s = __fmul_rn(sm.so[slot], sigmoid_f32(v));
                    if (s > A.thr && s >= bar) yolo_append_one(&A, img, s, sm.box[slot] * kYoloClasses + static_cast<uint32_t>(cls));
                }
                ++at;
            }
        }
    }
}

constexpr int kDenseRow = kYoloClasses + 1;  // odd: a warp that stores one class of 32 slots hits 32 banks

// grid = batch * tiles per image.  DENSE: the objectness and class scores are outputs too; every score is formed, staged in
// shared memory and written as whole 320-byte rows (written straight from the threads, every store instruction touched 32
// rows: 145 us for 8 images of 608 x 608 against 19 us of traffic).
template <bool DENSE>
__global__ void __launch_bounds__(kYoloTile, DENSE ? 5 : 7)
yolo_decode_kernel(const __grid_constant__ YoloDecodeArgs A) {
    __shared__ YoloTileSmem sm;
    extern __shared__ float s_cls[];  // DENSE: [kYoloTile][kDenseRow]
    pdl_launch_dependents();
    const YoloLevels& L = A.L;
    const int img = blockIdx.x / L.tile_begin[3], tile = blockIdx.x - img * L.tile_begin[3], t = threadIdx.x;
    const int lvl = tile >= L.tile_begin[2] ? 2 : (tile >= L.tile_begin[1] ? 1 : 0);
    const int plane = L.plane[lvl], nslots = 3 * plane;
    const int s0 = (tile - L.tile_begin[lvl]) * kYoloTile;
    const float* __restrict__ img_map = L.map[lvl] + static_cast<int64_t>(img) * 3 * kYoloAttrib * plane;

    // one slot per thread: objectness, cut, and the box where it is wanted
    const bool valid = s0 + t < nslots;
    int anchor, pos;
    yolo_slot(plane, valid ? s0 + t : s0, anchor, pos);
    const float* src = img_map + anchor * kYoloAttrib * plane + pos;
    const float tobj = __ldg(src + 4 * plane);
    const uint32_t box = static_cast<uint32_t>(L.box_begin[lvl] + pos * 3 + anchor);
    const int64_t gbox = static_cast<int64_t>(img) * L.num_boxes + box;
    if (A.boxes != nullptr && valid) {
        reinterpret_cast<float4*>(A.boxes)[gbox] =
            yolo_box(L, lvl, anchor, pos, __ldg(src), __ldg(src + plane), __ldg(src + 2 * plane), __ldg(src + 3 * plane));
    }
    const float so = sigmoid_f32(tobj);
    sm.so[t] = so;
    sm.box[t] = box;
    if (t == 0) sm.queued = 0;
    if (DENSE && valid && A.obj_out != nullptr) A.obj_out[gbox] = so;
    pdl_wait();  // the floor, and the counters that the floor kernel cleared
    const float bar = fmaxf(A.thr, A.floor != nullptr ? __ldcg(A.floor + img) : 0.0f);
    // a score is so * sigmoid(v) <= so: the box can only yield candidates if so itself clears both bars
    const bool alive = valid && so > A.thr && so >= bar;
    if (!DENSE) {
        sm.cut[t] = alive ? logit_cut(so, bar) : INFINITY;
        if (__syncthreads_or(alive ? 1 : 0) == 0) return;
        if (L.vec4[lvl]) yolo_walk<true>(A, sm, img_map, plane, s0, nslots, img, bar);
        else yolo_walk<false>(A, sm, img_map, plane, s0, nslots, img, bar);
    } else {
        sm.cut[t] = alive ? 0.0f : INFINITY;  // only tells the dead slots
        __syncthreads();
        const int lane = t & 31, warp = t >> 5;
        int off[4];
        float so4[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int a, p;
            yolo_slot(plane, min(s0 + 32 * e + lane, nslots - 1), a, p);
            off[e] = (a * kYoloAttrib + 5 + warp * kDecClasses) * plane + p;
            so4[e] = sm.cut[32 * e + lane] < INFINITY ? sm.so[32 * e + lane] : 0.0f;
        }
#pragma unroll 1
        for (int k0 = 0; k0 < kDecClasses; k0 += 5) {
            float v[5][4];
#pragma unroll
            for (int u = 0; u < 5; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) v[u][e] = __ldg(img_map + off[e] + (k0 + u) * plane);
#pragma unroll
            for (int u = 0; u < 5; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int slot = 32 * e + lane, cls = warp * kDecClasses + k0 + u;
                    const float c = sigmoid_f32(v[u][e]);
                    s_cls[slot * kDenseRow + cls] = c;
                    const float s = __fmul_rn(so4[e], c);
                    if (s > A.thr && s >= bar) {
                        const int at = atomicAdd(&sm.queued, 1);
                        if (at < kDecQueue) {
                            sm.queue[at].v = s;
                            sm.queue[at].meta = static_cast<uint32_t>(slot << 7 | cls);
                        } else {
                            yolo_append_one(&A, img, s, sm.box[slot] * kYoloClasses + static_cast<uint32_t>(cls));
                        }
                    }
                }
        }
    }
    __syncthreads();
    if (DENSE && A.cls_out != nullptr) {
        const int total = min(kYoloTile, nslots - s0) * kYoloClasses;
        float* out = A.cls_out + static_cast<int64_t>(img) * L.num_boxes * kYoloClasses;
        int slot = t / kYoloClasses, c = t - slot * kYoloClasses;
        for (int i = t; i < total; i += kYoloTile) {
            out[static_cast<int64_t>(sm.box[slot]) * kYoloClasses + c] = s_cls[slot * kDenseRow + c];
            slot += kYoloTile / kYoloClasses;
            c += kYoloTile % kYoloClasses;
            if (c >= kYoloClasses) {
                c -= kYoloClasses;
                ++slot;
            }
        }
    }
    // the queued hits, evaluated together
    const int n = min(sm.queued, kDecQueue);
    for (int i0 = 0; i0 < n; i0 += kYoloTile) {
        const int i = i0 + t;
        bool pass = i < n;
        float s = 0.0f;
        uint32_t flat = 0u;
        if (pass) {
            const YoloHit h = sm.queue[i];
            const uint32_t slot = h.meta >> 7;
            s = DENSE ? h.v : __fmul_rn(sm.so[slot], sigmoid_f32(h.v));
            flat = sm.box[slot] * kYoloClasses + (h.meta & 127u);
            pass = s > A.thr && s >= bar;
        }
        yolo_append(A, img, pass, s, flat);
    }
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
        L.tile_begin[l] = tiles;
        tiles += (3 * L.plane[l] + kYoloTile - 1) / kYoloTile;
        L.box_begin[l] = static_cast<int>(boxes);
        boxes += 3 * L.plane[l];
        L.vec4[l] = (L.plane[l] % 4 == 0 && (reinterpret_cast<uintptr_t>(maps[l]) & 15) == 0) ? 1 : 0;
        L.stride[l] = kStrides[l];
        for (int a = 0; a < 3; ++a) {
            L.anchor_w[l][a] = kAnchors[l][a][0];
            L.anchor_h[l][a] = kAnchors[l][a][1];
        }
    }
    FB_REQUIRE(boxes * kYoloClasses < (1ll << 32), "yolo_decode: flat index exceeds 32 bits");
    FB_REQUIRE(static_cast<int64_t>(tiles) * batch < (1ll << 31), "yolo_decode: too many tiles");
    L.tile_begin[3] = tiles;
    L.num_boxes = static_cast<int>(boxes);
    return FB_OK;
}

// pdl: the launch may overlap the end of the kernel before it (the floor kernel)
static int launch_yolo_decode(const YoloDecodeArgs& a, int batch, bool pdl, cudaStream_t st) {
    FB_REQUIRE(a.keys && a.counts, "yolo_decode: null pointer");
    FB_REQUIRE(a.capacity > 0, "yolo_decode: bad sizes");
    FB_REQUIRE(a.thr > 0.0f, "yolo_decode: score threshold must be positive (keys require positive scores)");
    FB_REQUIRE((reinterpret_cast<uintptr_t>(a.boxes) & 15) == 0, "yolo_decode: boxes must be 16-byte aligned");
    const dim3 grid(static_cast<unsigned>(a.L.tile_begin[3]) * static_cast<unsigned>(batch));
    const bool dense = a.obj_out != nullptr || a.cls_out != nullptr;
    const size_t smem = dense ? sizeof(float) * kYoloTile * kDenseRow : 0;
    if (pdl) {
        return dense ? launch_pdl(yolo_decode_kernel<true>, grid, dim3(kYoloTile), smem, st, "yolo_decode_kernel", a)
                     : launch_pdl(yolo_decode_kernel<false>, grid, dim3(kYoloTile), smem, st, "yolo_decode_kernel", a);
    }
    if (dense) yolo_decode_kernel<true><<<grid, kYoloTile, smem, st>>>(a);
    else yolo_decode_kernel<false><<<grid, kYoloTile, smem, st>>>(a);
    count_launch();
    return check_launch("yolo_decode_kernel");
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
    yolo_floor_kernel<<<static_cast<unsigned>(batch) * kFloorCtas, kFloorThreads, 0, st>>>(f);
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
