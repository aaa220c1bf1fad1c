// C3: SSD-style post-process in two launches.
//
// Group 1 (ssd_softmax_decode_kernel): softmax over every confidence row with the background column dropped
// (functs/benchmark/ai_model/ssd/ssd_bbox.py:268) fused with the box decode and its strided in-place clamp
// (ssd_bbox.py:121-154).  A CTA stages a tile of conf rows in shared memory with one bulk (TMA) copy when the
// tile is 16-byte aligned; one thread reduces a row (row stride 81 words: conflict-free), or two threads a long one: the first hands
// the sum of its columns over in s_inv, the second goes on adding in column order and leaves the reciprocal there.  The scores are
// written class-major so that group 2 reads contiguous runs.
//
// Group 2 (ssd_class_nms_kernel): the loop over classes (ssd_bbox.py:163-172 + :212 per class) with every
// (image, class) iteration mapped onto one CTA: mask > thr, top-k by (score desc, prior asc), gather boxes,
// greedy NMS, write the kept rows and their count.
#include <algorithm>

#include "select_nms.cuh"

namespace fb {

constexpr int kSsdTile = 128;     // priors per CTA in group 1
// Conf columns from which two threads share a row.  One / two threads, us per launch: 21 columns, 48 images of 8732 priors 14.8 / 20.9,
// of 24 564 priors 39.5 / 52; 61 columns, 48 of 8732 39.4 / 41.3; 81 columns 50.6 / 49.6, 91 58.7 / 56.8.
constexpr int kSsdTwoParts = 70;
constexpr int kSsdMaxRow = 96;    // maximum conf columns (C + 1) supported by the register/smem layout

// dynamic smem: [tile rows * ncol floats][8-byte mbarrier]
// PARTS = 2: two threads per row, in two groups of four warps: the first columns and the last ones (fewer: the second group also decodes
// the box and finishes the sum, which runs in column order whoever adds).  A tile of 81 columns takes 41 KB of shared memory, so that
// one thread per row leaves five warps per scheduler; shorter rows leave room for more CTAs (launch_ssd_softmax_decode).
template <int PARTS>
__global__ void __launch_bounds__(PARTS * kSsdTile)
ssd_softmax_decode_kernel(const float* __restrict__ loc, const float* __restrict__ conf, const float* __restrict__ priors,
                          int num_priors, int num_classes, float clamp_max, float* __restrict__ boxes,
                          float* __restrict__ scores_cm, int use_bulk, int32_t* __restrict__ clear, int num_clear) {
    constexpr int kThreads = PARTS * kSsdTile;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ float s_max[PARTS][kSsdTile];
    __shared__ __align__(16) float s_inv[kSsdTile];  // first the sum over the first columns
    // the words the class kernel of a ragged call counts in (none otherwise): cleared here, so that no memset runs
    for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * kThreads + threadIdx.x; i < num_clear; i += gridDim.x * gridDim.y * kThreads)
        clear[i] = 0;
    const int ncol = num_classes + 1;
    float* tile = reinterpret_cast<float*>(smem_raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + ((static_cast<size_t>(kSsdTile) * ncol * 4 + 15) / 16) * 16);
    const int img = blockIdx.y;
    const int p0 = blockIdx.x * kSsdTile;
    const int rows = min(kSsdTile, num_priors - p0);
    const int r = threadIdx.x % kSsdTile, part = threadIdx.x / kSsdTile;
    const float* gsrc = conf + (static_cast<int64_t>(img) * num_priors + p0) * ncol;
    const int nfl = rows * ncol;
    bool staged = false;
    if (use_bulk) {
        if (threadIdx.x == 0) {
            mbar_init(bar, 1);
            fence_barrier_init();
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            mbar_arrive_expect_tx(bar, static_cast<uint32_t>(nfl) * 4u);
            bulk_copy_g2s(tile, gsrc, static_cast<uint32_t>(nfl) * 4u, bar);
        }
        // one warp polls, the others sleep at the barrier; if the wait ran out (never observed), fall through to the plain loads
        // below after the copy engine had its chance
        staged = threadIdx.x >= 32 || mbar_wait_bounded(bar, 0, 200000u);
        staged = __syncthreads_and(staged ? 1 : 0) != 0;
    }
    if (!staged) {
        for (int i = threadIdx.x; i < nfl; i += kThreads) tile[i] = __ldg(gsrc + i);
        __syncthreads();
    }

    const int p = p0 + r;
    const int split = PARTS == 1 ? ncol : ncol * 3 / 5, first = part == 0 ? 0 : split, last = part == 0 ? split : ncol;  // this thread's columns
    constexpr int kAtOnce = 8;  // columns: loads and exponentials side by side
    const int whole = first + (last - first) / kAtOnce * kAtOnce;
    const bool live = r < rows;
    float* row = tile + r * ncol;
    float mx = -INFINITY;  // (a row of nothing but NaN: exp(NaN) below)
    if (live) {
        for (int c = first; c < whole; c += kAtOnce) {
            float v[kAtOnce];
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) v[u] = row[c + u];
            mx = fmaxf(mx, fmaxf(fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])), fmaxf(fmaxf(v[4], v[5]), fmaxf(v[6], v[7]))));
        }
        for (int c = whole; c < last; ++c) mx = fmaxf(mx, row[c]);
        if (PARTS == 2) s_max[part][r] = mx;
    }
    if (PARTS == 2) __syncthreads();
    float sum = 0.0f;
    if (live) {
        if (PARTS == 2) mx = fmaxf(s_max[0][r], s_max[PARTS - 1][r]);
        for (int c = first; c < whole; c += kAtOnce) {
            float e[kAtOnce];
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) e[u] = expf(__fsub_rn(row[c + u], mx));
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
                row[c + u] = e[u];
                if (part == 0) sum = __fadd_rn(sum, e[u]);
            }
        }
        for (int c = whole; c < last; ++c) {
            const float e = expf(__fsub_rn(row[c], mx));
            row[c] = e;
            if (part == 0) sum = __fadd_rn(sum, e);
        }
        if (PARTS == 2 && part == 0) s_inv[r] = sum;
    }
    if (live && part == PARTS - 1) {
        // decode (centre/size priors, variances 0.1 / 0.2), then clamp x to [0, max], y to [0, max]
        const float4 pr = __ldg(reinterpret_cast<const float4*>(priors) + p);
        const float4 d = __ldg(reinterpret_cast<const float4*>(loc) + static_cast<int64_t>(img) * num_priors + p);
        const float gx = __fadd_rn(pr.x, __fmul_rn(pr.z, __fmul_rn(d.x, 0.1f)));
        const float gy = __fadd_rn(pr.y, __fmul_rn(pr.w, __fmul_rn(d.y, 0.1f)));
        const float gw = __fmul_rn(pr.z, expf(__fmul_rn(d.z, 0.2f)));
        const float gh = __fmul_rn(pr.w, expf(__fmul_rn(d.w, 0.2f)));
        const float hw = __fmul_rn(gw, 0.5f), hh = __fmul_rn(gh, 0.5f);
        float4 o;
        o.x = min_nan(max_nan(__fsub_rn(gx, hw), 0.0f), clamp_max);
        o.y = min_nan(max_nan(__fsub_rn(gy, hh), 0.0f), clamp_max);
        o.z = min_nan(max_nan(__fadd_rn(gx, hw), 0.0f), clamp_max);
        o.w = min_nan(max_nan(__fadd_rn(gy, hh), 0.0f), clamp_max);
        reinterpret_cast<float4*>(boxes)[static_cast<int64_t>(img) * num_priors + p] = o;
    }
    if (PARTS == 2) __syncthreads();
    if (PARTS == 2 && live && part == 1) {
        sum = s_inv[r];
        int c = split;
        for (; c + 4 <= ncol; c += 4) {
            const float e0 = row[c], e1 = row[c + 1], e2 = row[c + 2], e3 = row[c + 3];
            sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, e0), e1), e2), e3);
        }
        for (; c < ncol; ++c) sum = __fadd_rn(sum, row[c]);
        s_inv[r] = __fdiv_rn(1.0f, sum);
    }
    if (PARTS == 2) __syncthreads();
    // class-major store: for a fixed class consecutive threads write consecutive priors
    if (live) {
        const float inv = PARTS == 2 ? s_inv[r] : __fdiv_rn(1.0f, sum);
        float* dst = scores_cm + static_cast<int64_t>(img) * num_classes * num_priors + p;
#pragma unroll 4
        for (int c = part; c < num_classes; c += PARTS) dst[static_cast<int64_t>(c) * num_priors] = __fmul_rn(row[c], inv);
    }
}

// ---- group 2 ------------------------------------------------------------------------------------------------
constexpr int kSsdNmsThreads = 256;
constexpr int kSsdNmsMinBlocks = 6;  // CTAs per SM the register allocation aims at (27 KB of shared memory each)
constexpr int kSsdSelCap = 256;
constexpr int kSsdWords = kSsdSelCap / 32;

constexpr size_t kSsdSelBytes = (sizeof(SelectSmem<kSsdSelCap>) + 127) / 128 * 128;

// Ragged output (RAGGED = true): the kept rows of an image's classes follow one another in class order from row
// img * num_classes * topk on, instead of every class owning topk padded rows.  A CTA publishes its own count first and
// then reads the counts of the classes before its own, all at once (one word per lane); work is handed out by a ticket, so
// those classes belong to CTAs that are already running and wait for nobody before they publish.  The padded form left
// the compaction to some thirty ATen launches and three synchronisations per image: 8.9 ms for 64 images against 0.35.
struct SsdRagged {
    int32_t* words;        // [batch * num_classes] kept count + 1 (0 = not known yet), then the ticket; zero at launch
    unsigned long long* done;  // [batch] classes that have written their rows << 32 | rows; zero at launch
    int64_t* labels;       // like prior_ids
    int32_t* img_counts;   // [batch] rows of every image (may be pinned host memory): written when they are all in place
    int32_t* status;       // optional; plain store (may be pinned host memory)
    int batch;
};
constexpr unsigned long long kSsdWaitCycles = 2000000000ull;  // ~1 s

// NMS by suppression rows, thread t = row t: of the candidates in the tables (tame boxes), or of every box behind the row.  Out of line:
// its code should not sit in the middle of the class kernel's instruction stream.
__device__ __noinline__ void ssd_nms_rows(const float4* sxy, const float* sarea, int n, const PairCells<kSsdWords>* pc, const PairWindow window,
                                          float iou_thr, float thr_lo, float thr_hi, uint32_t* keep_words, uint32_t* or_words) {
    const int t = threadIdx.x;
    uint32_t row[kSsdWords];
    const float4 me = t < n ? sxy[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    const NmsBox bi{me.x, me.y, me.z, me.w, t < n ? sarea[t] : 0.0f};
#pragma unroll
    for (int w = 0; w < kSsdWords; ++w) {
        const int first = max(t + 1 - 32 * w, 0), last = min(n - 32 * w, 32);  // the boxes behind the row: bits first .. last - 1
        uint32_t left = t >= n || first >= last ? 0u : (0xffffffffu << first) & (0xffffffffu >> (32 - last));
        if (pc != nullptr) left &= pair_word(*pc, window, w);
        row[w] = 0u;
        for (; left != 0u; left &= left - 1u) {
            const int b = __ffs(left) - 1;
            const float4 cj = sxy[32 * w + b];
            if (iou_exceeds(bi, NmsBox{cj.x, cj.y, cj.z, cj.w, sarea[32 * w + b]}, iou_thr, thr_lo, thr_hi)) row[w] |= 1u << b;
        }
    }
    __syncthreads();
    block_nms_resolve<kSsdNmsThreads, kSsdWords>(row, n, keep_words, or_words);
}

// dynamic smem: [SelectSmem<256>][kCandCap candidate keys]; after the selection the NMS boxes live in the selection's boundary
// list and the pair tables in the candidate list, which are not needed any more.  The class's scores (one contiguous
// run of the class-major array) are read from global memory once: a sampled score floor, one collection pass, and the
// exact selection on the few hundred candidates (block_select_topk_sampled).
template <bool RAGGED>
__global__ void __launch_bounds__(kSsdNmsThreads, kSsdNmsMinBlocks)
ssd_class_nms_kernel(const float* __restrict__ boxes, const float* __restrict__ scores_cm, int num_priors, int num_classes,
                     float score_thr, uint32_t hist_base, int hist_shift, int topk, float iou_thr, float thr_lo,
                     float thr_hi, float* __restrict__ dets, int64_t* __restrict__ prior_ids,
                     int32_t* __restrict__ out_counts, const SsdRagged rag) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SelectSmem<kSsdSelCap>& sm = *reinterpret_cast<SelectSmem<kSsdSelCap>*>(smem_raw);
    static_assert(sizeof(PairCells<kSsdWords>) <= sizeof(uint64_t) * kCandCap, "the pair tables reuse the candidate list");
    // selected boxes as corners (one 16-byte shared load) + area, in the boundary list of the finished selection
    static_assert(sizeof(float4) * kSsdSelCap + sizeof(float) * kSsdSelCap <= sizeof(sm.binlist) &&
                      offsetof(SelectSmem<kSsdSelCap>, binlist) % 16 == 0,
                  "the corner / area arrays must fit (and be 16-byte aligned in) the boundary list");
    float4* sxy = reinterpret_cast<float4*>(sm.binlist);
    float* sarea = reinterpret_cast<float*>(sxy + kSsdSelCap);
    uint64_t* cand = reinterpret_cast<uint64_t*>(smem_raw + kSsdSelBytes);
    __shared__ uint32_t keep_words[kSsdWords];
    __shared__ int word_prefix[kSsdWords + 1];
    __shared__ uint32_t or_words[2 * kSsdWords];
    __shared__ int pair_count[2];

    const int t = threadIdx.x;
    int cls = blockIdx.x, img = blockIdx.y;
    if (RAGGED) {
        __shared__ int s_ticket;
        if (t == 0) s_ticket = atomicAdd(rag.words + static_cast<int64_t>(rag.batch) * num_classes, 1);
        __syncthreads();
        img = s_ticket / num_classes;
        cls = s_ticket - img * num_classes;
    }
    const float* src = scores_cm + (static_cast<int64_t>(img) * num_classes + cls) * num_priors;
    const int n = block_select_topk_sampled<kSsdNmsThreads, kSsdSelCap>(src, score_thr, num_priors, topk, hist_base, hist_shift, sm, cand);
    __syncthreads();  // behind the selection's last stores and reads, as it asks

    const float* bimg = boxes + static_cast<int64_t>(img) * num_priors * 4;
    float4 mybox = make_float4(0.f, 0.f, 0.f, 0.f);
    uint64_t mykey = 0ull;
    float myarea = 0.0f;
    bool tame_box = true;
    if (t < n) {
        mykey = sm.sel[t];
        mybox = __ldg(reinterpret_cast<const float4*>(bimg) + key_index(mykey));
        const NmsBox nb = make_nms_box(mybox.x, mybox.y, mybox.z, mybox.w);
        tame_box = nms_box_is_tame(nb);
        myarea = nb.area;
        sxy[t] = mybox;
        sarea[t] = myarea;
    }
    if (t < 2) pair_count[t] = 0;
    const bool tame = __syncthreads_and(tame_box ? 1 : 0) != 0;  // also the barrier behind the box stores

    // Tame boxes only test the pairs that PairCells leaves (200 x 200 all-pairs votes took 45 % of this kernel's time); lists with
    // a wild box, or with more pairs than fit, form suppression rows.
    const int lane = t & 31, warp = t >> 5;
    PairCells<kSsdWords>& pc = *reinterpret_cast<PairCells<kSsdWords>*>(cand);
    PairWindow window = {};
    bool done = false;
    if (tame) {
        // (the histogram of the selection and the rest of its boundary list are free)
        static_assert(sizeof(uint16_t) * PairLists::kPairs <= sizeof(sm.hist) &&
                          (sizeof(float4) + sizeof(float)) * kSsdSelCap + sizeof(uint16_t) * PairLists::kHits <= sizeof(sm.binlist) &&
                          sizeof(uint32_t) * kSsdNmsThreads * kSsdWords <= sizeof(uint64_t) * kCandCap,
                      "the pair lists reuse the selection's memory");
        const PairLists pl{reinterpret_cast<uint16_t*>(sm.hist), reinterpret_cast<uint16_t*>(sarea + kSsdSelCap), reinterpret_cast<uint32_t*>(cand),
                           pair_count, or_words};
        window = pair_tables<kSsdWords>(mybox, myarea, n, iou_thr, pc);
        done = block_nms_pairs<kSsdWords>(sxy, sarea, pc, window, n, iou_thr, thr_lo, thr_hi, pl, keep_words);
    }
    if (!done) ssd_nms_rows(sxy, sarea, n, tame ? &pc : nullptr, window, iou_thr, thr_lo, thr_hi, keep_words, or_words);
    __syncthreads();
    if (t == 0) {
        int acc = 0;
        for (int w = 0; w < kSsdWords; ++w) {
            word_prefix[w] = acc;
            acc += __popc(keep_words[w]);
        }
        word_prefix[kSsdWords] = acc;
        if (RAGGED) atomicExch(rag.words + static_cast<int64_t>(img) * num_classes + cls, acc + 1);
        else out_counts[img * num_classes + cls] = acc;
    }
    if (RAGGED) {
        __shared__ int s_before;
        if (warp == 0) {
            const volatile int32_t* words = rag.words + static_cast<int64_t>(img) * num_classes;
            int before = 0;
            const unsigned long long start = clock64();
            for (int c = lane; c < cls; c += 32) {
                int v;
                while ((v = words[c]) == 0) {
                    if (clock64() - start > kSsdWaitCycles) {
                        if (rag.status != nullptr) *reinterpret_cast<volatile int32_t*>(rag.status) = FB_STATUS_WAIT_TIMEOUT;
                        __threadfence_system();  // before this image's count
                        break;
                    }
                }
                before += v > 0 ? v - 1 : 0;
            }
            before = __reduce_add_sync(kFullMask, before);
            if (lane == 0) s_before = before;
        }
        __syncthreads();
        const int64_t obase = static_cast<int64_t>(img) * num_classes * topk + s_before;
        if (t < n) {
            const uint32_t kw = keep_words[t >> 5];
            const int b = t & 31;
            if ((kw >> b) & 1u) {
                const int64_t row = obase + word_prefix[t >> 5] + __popc(kw & ((1u << b) - 1u));
                float* d = dets + row * 5;
                d[0] = mybox.x;
                d[1] = mybox.y;
                d[2] = mybox.z;
                d[3] = mybox.w;
                d[4] = key_score(mykey);
                rag.labels[row] = cls;
                prior_ids[row] = static_cast<int64_t>(key_index(mykey));
            }
        }
        __syncthreads();
        if (t == 0) {
            // the class that finishes last publishes the image: a host that watches the count finds the rows complete
            __threadfence();
            const unsigned long long mine = (1ull << 32) + static_cast<unsigned>(word_prefix[kSsdWords]);
            const unsigned long long all = atomicAdd(rag.done + img, mine) + mine;
            if (static_cast<int>(all >> 32) == num_classes) {
                __threadfence_system();
                *reinterpret_cast<volatile int32_t*>(rag.img_counts + img) = static_cast<int32_t>(all);
            }
        }
        return;
    }
    __syncthreads();
    const int64_t obase = (static_cast<int64_t>(img) * num_classes + cls) * topk;
    if (t < n) {
        const uint32_t kw = keep_words[t >> 5];
        const int b = t & 31;
        if ((kw >> b) & 1u) {
            const int rank = word_prefix[t >> 5] + __popc(kw & ((1u << b) - 1u));
            float* d = dets + (obase + rank) * 5;
            d[0] = mybox.x;
            d[1] = mybox.y;
            d[2] = mybox.z;
            d[3] = mybox.w;
            d[4] = key_score(mykey);
            prior_ids[obase + rank] = static_cast<int64_t>(key_index(mykey));
        }
    }
    const int kept = word_prefix[kSsdWords];
    for (int i = kept + t; i < topk; i += kSsdNmsThreads) {
        float* d = dets + (obase + i) * 5;
        d[0] = d[1] = d[2] = d[3] = d[4] = 0.0f;
        prior_ids[obase + i] = -1;
    }
}

// Rows [b * stride, b * stride + counts[b]) of every image b, moved together: grid = (images).
constexpr int kPackThreads = 256;
__global__ void __launch_bounds__(kPackThreads)
ragged_pack_kernel(const float* __restrict__ dets, const int64_t* __restrict__ labels, const int64_t* __restrict__ ids,
                   const int32_t* __restrict__ counts, int64_t stride, float* __restrict__ out_dets,
                   int64_t* __restrict__ out_labels, int64_t* __restrict__ out_ids) {
    __shared__ int64_t part[kPackThreads / 32];
    const int b = blockIdx.x, t = threadIdx.x;
    int64_t before = 0;
    for (int i = t; i < b; i += kPackThreads) before += counts[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(kFullMask, before, o);
    if ((t & 31) == 0) part[t >> 5] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < kPackThreads / 32; ++w) before += part[w];
    const int n = counts[b];
    const int64_t src = b * stride;
    for (int i = t; i < 5 * n; i += kPackThreads) out_dets[before * 5 + i] = dets[src * 5 + i];
    for (int i = t; i < n; i += kPackThreads) {
        out_labels[before + i] = labels[src + i];
        if (out_ids != nullptr) out_ids[before + i] = ids[src + i];
    }
}

// Every part's rows into arrays of its own: grid = (256 rows, parts).  Latency bounds it, so a thread's words are on their way
// together.
struct RaggedParts {
    functs_b200_ragged_part part[FB_RAGGED_MAX_PARTS];
};
__global__ void __launch_bounds__(kPackThreads)
ragged_split_kernel(const float* __restrict__ dets, const int64_t* __restrict__ labels, const __grid_constant__ RaggedParts P) {
    const functs_b200_ragged_part& G = P.part[blockIdx.y];
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * kPackThreads;
    if (r0 >= G.rows) return;
    const int t = threadIdx.x, rows = static_cast<int>(min(G.rows - r0, static_cast<int64_t>(kPackThreads)));
    const float* src = dets + 5 * (G.first + r0);
    float* dst = G.dets + 5 * r0;
    float v[5];
#pragma unroll
    for (int u = 0; u < 5; ++u) v[u] = t + u * kPackThreads < 5 * rows ? __ldg(src + t + u * kPackThreads) : 0.0f;
    const int64_t label = t < rows ? __ldg(reinterpret_cast<const long long*>(labels) + G.first + r0 + t) : 0;
#pragma unroll
    for (int u = 0; u < 5; ++u)
        if (t + u * kPackThreads < 5 * rows) dst[t + u * kPackThreads] = v[u];
    if (t < rows) G.labels[r0 + t] = label;
}

static int launch_ssd_softmax_decode(const float* loc, const float* conf, const float* priors, int batch, int num_priors,
                                     int num_classes, float clamp_max, float* boxes, float* scores_cm, int32_t* clear,
                                     int num_clear, cudaStream_t st) {
    FB_REQUIRE(loc && conf && priors && boxes && scores_cm, "ssd_softmax_decode: null pointer");
    FB_REQUIRE(batch > 0 && batch <= 65535 && num_priors > 0 && num_classes > 0 && num_classes + 1 <= kSsdMaxRow,
               "ssd_softmax_decode: bad sizes (classes + 1 must be <= %d)", kSsdMaxRow);
    FB_REQUIRE(((reinterpret_cast<uintptr_t>(loc) | reinterpret_cast<uintptr_t>(priors) | reinterpret_cast<uintptr_t>(boxes)) & 15) == 0,
               "ssd_softmax_decode: loc, priors and boxes must be 16-byte aligned");
    const int ncol = num_classes + 1;
    // the bulk copy needs every tile start and length to be a multiple of 16 bytes
    const bool aligned = (reinterpret_cast<uintptr_t>(conf) & 15) == 0 && ((static_cast<int64_t>(num_priors) * ncol) % 4 == 0) &&
                         ((static_cast<int64_t>(kSsdTile) * ncol) % 4 == 0) &&
                         ((static_cast<int64_t>(num_priors % kSsdTile) * ncol) % 4 == 0);
    const size_t smem = ((static_cast<size_t>(kSsdTile) * ncol * 4 + 15) / 16) * 16 + 16;
    auto run = [&](auto kernel, int threads) {
        FB_TRY(check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                          "ssd_softmax_decode attr"));
        const dim3 grid((num_priors + kSsdTile - 1) / kSsdTile, batch);
        kernel<<<grid, threads, smem, st>>>(loc, conf, priors, num_priors, num_classes, clamp_max, boxes, scores_cm, aligned ? 1 : 0, clear,
                                            num_clear);
        return FB_OK;
    };
    FB_TRY(ncol >= kSsdTwoParts ? run(ssd_softmax_decode_kernel<2>, 2 * kSsdTile) : run(ssd_softmax_decode_kernel<1>, kSsdTile));
    count_launch();
    return check_launch("ssd_softmax_decode_kernel");
}

// rag != nullptr: ragged output
static int launch_ssd_class_nms(const float* boxes, const float* scores_cm, int batch, int num_priors, int num_classes,
                                float score_thr, int topk, float iou_thr, float* dets, int64_t* prior_ids, int32_t* out_counts,
                                const SsdRagged* rag, cudaStream_t st) {
    FB_REQUIRE(boxes && scores_cm && dets && prior_ids && (out_counts || rag), "ssd_class_nms: null pointer");
    FB_REQUIRE(batch > 0 && batch <= 65535 && num_priors > 0 && num_classes > 0, "ssd_class_nms: bad sizes");
    FB_REQUIRE(topk > 0 && topk <= kSsdSelCap, "ssd_class_nms: topk must be in [1, %d]", kSsdSelCap);
    FB_REQUIRE(score_thr > 0.0f, "ssd_class_nms: score threshold must be positive");
    FB_REQUIRE(iou_thr > 0.0f && iou_thr < 1.0f, "ssd_class_nms: iou threshold must be in (0, 1)");
    FB_REQUIRE(((reinterpret_cast<uintptr_t>(boxes) | reinterpret_cast<uintptr_t>(scores_cm)) & 15) == 0,
               "ssd_class_nms: boxes and scores must be 16-byte aligned");
    const size_t smem = kSsdSelBytes + sizeof(uint64_t) * kCandCap;
    auto kfn = rag != nullptr ? ssd_class_nms_kernel<true> : ssd_class_nms_kernel<false>;
    FB_TRY(check_cuda(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                      "ssd_class_nms attr"));
    const float thr_lo = iou_thr * (1.0f - 1.0e-6f), thr_hi = iou_thr * (1.0f + 1.0e-6f);
    dim3 grid(num_classes, batch);
    const HistParams hp = hist_params_for(score_thr);
    kfn<<<grid, kSsdNmsThreads, smem, st>>>(boxes, scores_cm, num_priors, num_classes, score_thr, hp.base, hp.shift, topk, iou_thr,
                                            thr_lo, thr_hi, dets, prior_ids, out_counts, rag != nullptr ? *rag : SsdRagged{});
    count_launch();
    return check_launch("ssd_class_nms_kernel");
}

}  // namespace fb

extern "C" {

int functs_b200_ssd_softmax_decode(const float* loc, const float* conf, const float* priors, int32_t batch,
                                   int32_t num_priors, int32_t num_classes, float clamp_max, float* boxes,
                                   float* scores_cm, void* stream) {
    return fb::launch_ssd_softmax_decode(loc, conf, priors, batch, num_priors, num_classes, clamp_max, boxes, scores_cm, nullptr, 0,
                                         fb::as_stream(stream));
}

int functs_b200_ssd_class_nms(const float* boxes, const float* scores_cm, int32_t batch, int32_t num_priors,
                              int32_t num_classes, float score_thr, int32_t topk, float iou_thr, float* dets,
                              int64_t* prior_ids, int32_t* out_counts, void* stream) {
    return fb::launch_ssd_class_nms(boxes, scores_cm, batch, num_priors, num_classes, score_thr, topk, iou_thr, dets, prior_ids,
                                    out_counts, nullptr, fb::as_stream(stream));
}

int64_t functs_b200_ssd_scratch_bytes(int32_t batch, int32_t num_classes) {
    if (batch <= 0 || num_classes <= 0) return 0;
    return static_cast<int64_t>(batch) * 8 + (static_cast<int64_t>(batch) * num_classes + 1) * 4;
}

int functs_b200_ssd_postprocess(const float* loc, const float* conf, const float* priors, int32_t batch, int32_t num_priors,
                                int32_t num_classes, float clamp_max, float score_thr, int32_t topk, float iou_thr, float* boxes,
                                float* scores_cm, float* dets, int64_t* labels, int64_t* prior_ids, int32_t* img_counts,
                                int32_t* status, void* scratch, void* stream) {
    using namespace fb;
    FB_REQUIRE(labels && img_counts && scratch, "ssd_postprocess: null pointer");
    const int64_t words = static_cast<int64_t>(batch) * num_classes;
    FB_REQUIRE(batch > 0 && num_classes > 0 && words < (1ll << 30), "ssd_postprocess: bad sizes");
    FB_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 7) == 0, "ssd_postprocess: scratch must be 8-byte aligned");
    int32_t* sync = static_cast<int32_t*>(scratch);
    SsdRagged rag{sync + 2 * batch, static_cast<unsigned long long*>(scratch), labels, img_counts, status, batch};
    FB_TRY(launch_ssd_softmax_decode(loc, conf, priors, batch, num_priors, num_classes, clamp_max, boxes, scores_cm, sync,
                                     2 * batch + static_cast<int>(words) + 1, as_stream(stream)));
    return launch_ssd_class_nms(boxes, scores_cm, batch, num_priors, num_classes, score_thr, topk, iou_thr, dets, prior_ids, nullptr,
                                &rag, as_stream(stream));
}

int functs_b200_ragged_pack(const float* dets, const int64_t* labels, const int64_t* ids, const int32_t* counts, int32_t groups,
                            int64_t stride, float* out_dets, int64_t* out_labels, int64_t* out_ids, void* stream) {
    using namespace fb;
    FB_REQUIRE(dets && labels && counts && out_dets && out_labels && (out_ids == nullptr || ids != nullptr), "ragged_pack: null pointer");
    FB_REQUIRE(groups > 0 && stride > 0, "ragged_pack: bad sizes");
    ragged_pack_kernel<<<static_cast<unsigned>(groups), kPackThreads, 0, as_stream(stream)>>>(dets, labels, ids, counts, stride, out_dets,
                                                                                           out_labels, out_ids);
    count_launch();
    return check_launch("ragged_pack_kernel");
}

int functs_b200_ragged_split(const float* dets, const int64_t* labels, const functs_b200_ragged_part* parts, int32_t count, void* stream) {
    using namespace fb;
    FB_REQUIRE(dets && labels && parts, "ragged_split: null pointer");
    FB_REQUIRE(count > 0 && count <= FB_RAGGED_MAX_PARTS, "ragged_split: between 1 and %d parts", FB_RAGGED_MAX_PARTS);
    RaggedParts p{};
    int64_t most = 0;
    for (int k = 0; k < count; ++k) {
        FB_REQUIRE(parts[k].first >= 0 && parts[k].rows >= 0 && (parts[k].rows == 0 || (parts[k].dets && parts[k].labels)),
                   "ragged_split: bad part %d", k);
        p.part[k] = parts[k];
        most = std::max(most, parts[k].rows);
    }
    FB_REQUIRE(most <= (1ll << 30), "ragged_split: bad sizes");
    const int64_t chunks = std::max<int64_t>(1, (most + kPackThreads - 1) / kPackThreads);
    ragged_split_kernel<<<dim3(static_cast<unsigned>(chunks), static_cast<unsigned>(count)), kPackThreads, 0, as_stream(stream)>>>(dets, labels, p);
    count_launch();
    return check_launch("ragged_split_kernel");
}

}  // extern "C"
