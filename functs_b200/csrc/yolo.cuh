// C2: what the kernels of the YOLOv3-style post-process share (kernels_yolo.cu: score floor and decode, kernels_yolo_post.cu:
// selection and NMS).
//
// The decode group is "permute -> reshape -> sigmoid on the xy / objectness / class slices (slice + sigmoid + slice_rev) -> xy
// grid offset -> exp * anchor -> corner form -> objectness * class score -> score mask" of
// functs/benchmark/ai_model/yolov3/yolov3_bbox.py:209-220 and :122-127.
#pragma once

#include "select_nms.cuh"

namespace fb {

constexpr int kYoloClasses = 80;
constexpr int kYoloAttrib = 85;

struct YoloLevels {
    const float* map[3];  // [batch, 255, S, S]
    int size[3];          // S
    int plane[3];         // S * S
    int box_begin[3];     // first box index of every level inside an image
    float stride[3];
    float anchor_w[3][3];
    float anchor_h[3][3];
    int num_boxes;
};

#ifdef __CUDACC__

// Slot s of a level: anchor-major, then position; box order is position-major, then anchor.
__device__ __forceinline__ void yolo_slot(int plane, int slot, int& anchor, int& pos) {
    anchor = (slot >= plane ? 1 : 0) + (slot >= 2 * plane ? 1 : 0);
    pos = slot - anchor * plane;
}

// Box of one slot from its four logits: every operation rounded on its own, in the program's order.
__device__ __forceinline__ float4 yolo_box(const YoloLevels& L, int lvl, int anchor, int pos, float t0, float t1, float t2, float t3) {
    const int gy = pos / L.size[lvl], gx = pos - gy * L.size[lvl];
    const float stride = L.stride[lvl];
    const float aw = anchor == 0 ? L.anchor_w[lvl][0] : (anchor == 1 ? L.anchor_w[lvl][1] : L.anchor_w[lvl][2]);
    const float ah = anchor == 0 ? L.anchor_h[lvl][0] : (anchor == 1 ? L.anchor_h[lvl][1] : L.anchor_h[lvl][2]);
    const float cx = __fmul_rn(__fadd_rn(sigmoid_f32(t0), static_cast<float>(gx)), stride);
    const float cy = __fmul_rn(__fadd_rn(sigmoid_f32(t1), static_cast<float>(gy)), stride);
    const float hw = __fmul_rn(__fmul_rn(expf(t2), aw), 0.5f);
    const float hh = __fmul_rn(__fmul_rn(expf(t3), ah), 0.5f);
    return make_float4(__fsub_rn(cx, hw), __fsub_rn(cy, hh), __fadd_rn(cx, hw), __fadd_rn(cy, hh));
}

// v > cut is necessary for so * sigmoid(v) to reach `bar` (> 0).  The cut sits a relative 1e-5 below the exact bound
// (hundreds of fp32 ulps: rounding of the sigmoid and of the product) and another 0.02 lower in the logit domain, so it
// never loses a candidate; the 0.02 also covers the fast division and logarithm used here (a few ulps).
__device__ __forceinline__ float logit_cut(float so, float bar) {
    const float q = __fdividef(bar, so) * (1.0f - 1.0e-5f);
    if (!(q < 1.0f)) return INFINITY;
    return __logf(__fdividef(q, 1.0f - q)) - 0.02f;
}

#endif  // __CUDACC__

// kernels_yolo_post.cu
struct YoloPostArgs {
    uint64_t* keys;           // [batch, capacity] candidates, unordered
    int32_t* counts;          // [batch] candidates
    int32_t* fallback;        // [batch] 1: the image took one of the slow exact paths (observability only)
    const float* floor;       // [batch] every candidate of the image that scores at least this is in `keys` (0: all above thr)
    int64_t capacity;
    const float* boxes;       // [batch, num_boxes, 4] decoded boxes, or null: from the logits
    uint32_t* mask;           // [batch, 1024, 32] room for the dense suppression matrix (crowded images only)
    float thr, iou_thr;
    int topk;
    float* dets;
    int64_t* labels;
    int64_t* flat_ids;
    int32_t* out_counts;
    int32_t* host_counts;     // optional: the counts once more, in memory the host can read
    int32_t* records;         // optional 32-byte gather records
    int32_t* status;          // optional
};
int check_yolo_post(int batch, const YoloPostArgs& a);  // argument errors, nothing launched
int launch_yolo_post(const YoloLevels& L, int batch, const YoloPostArgs& a, cudaStream_t st);
int64_t yolo_post_mask_bytes(int batch);

}  // namespace fb
