// Whole detection calls on the host side (detect.cpp): allocation, launch, the one wait for the counts, and the ragged
// per-image lists, shared by the region operators and by the Python modules.
#pragma once

#include <ATen/ATen.h>

#include <functional>
#include <vector>

namespace functs_b200 {

struct Detections {  // one image
    at::Tensor dets, labels, ids;
};

using EmitImage = std::function<void(Detections&&)>;  // called once per image, in order

// What an image's lists are.  Views share the batch's memory: for callers that take a batch's lists apart at once.  Own lists
// are tensors with a storage of their own, filled by one more launch: for callers that may keep some and drop others.
enum class Lists { kViews, kOwn };  // kViews: with ids; kOwn: Detections::ids stays undefined

struct SsdResult {
    at::Tensor boxes, scores_cm;  // [B, P, 4], [B, C, P]
};
SsdResult ssdDetect(const at::Tensor& loc, const at::Tensor& conf, const at::Tensor& priors, double clamp_max, double score_thr,
                    int64_t topk, double iou_thr, Lists lists, const EmitImage& emit);

struct YoloResult {
    at::Tensor boxes, obj, cls;  // [B, N, 4], [B, N], [B, N, 80]; dense = true only
};
YoloResult yoloDetect(const std::vector<at::Tensor>& maps, double score_thr, int64_t topk, double iou_thr, bool dense, Lists lists,
                      const EmitImage& emit);

}  // namespace functs_b200
