#include "detect.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../../include/functs_b200.h"

namespace functs_b200 {

namespace {

void checkRc(int rc, const char* what) { TORCH_CHECK(rc == FB_OK, "functs_b200 ", what, ": ", functs_b200_last_error()); }

// `sizes` elements of base's storage from element `offset` on, contiguous.  A batch of 64 images is 128 to 192 such views:
// made as a bare TensorImpl each costs a tenth of a select + narrow through the dispatcher (64 images: 0.3 ms).
at::Tensor viewAt(const at::Tensor& base, int64_t offset, at::IntArrayRef sizes) {
    auto impl = c10::make_intrusive<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
    impl->set_storage_offset(base.storage_offset() + offset);
    impl->set_sizes_contiguous(sizes);
    return at::Tensor(std::move(impl));
}

// Host words that the kernels write themselves (pinned memory is mapped into the device's address space): waiting for the
// stream is all a caller has to do, there is no copy and one wait.
at::Tensor pinnedWords(int64_t n) { return at::empty({n}, at::TensorOptions().dtype(at::kInt).pinned_memory(true)); }

void raiseOnStatus(int bits, const char* what) {
    TORCH_CHECK(bits == 0, "functs_b200 ", what, ": device status ", bits,
                (bits & FB_STATUS_CAND_OVERFLOW) ? " (a candidate list overflowed)" : "",
                (bits & FB_STATUS_WAIT_TIMEOUT) ? " (a bounded device-side wait ran out)" : "",
                (bits & FB_STATUS_INDEX_RANGE) ? " (an index was out of range)" : "");
}

// A ragged result is written into room for the largest possible one.  Results that fill less than a quarter of a large
// room are moved to memory of their own size (one launch, nothing waits for it), so that a caller who keeps them does not
// keep the room.
constexpr int64_t kKeepRoomBytes = 4 << 20;

}  // namespace

SsdResult ssdDetect(const at::Tensor& loc, const at::Tensor& conf, const at::Tensor& priors, double clamp_max, double score_thr,
                    int64_t topk, double iou_thr, bool want_ids) {
    TORCH_CHECK(loc.dim() == 3 && loc.size(2) == 4 && conf.dim() == 3 && conf.size(0) == loc.size(0) && conf.size(1) == loc.size(1) &&
                    conf.size(2) >= 2 && priors.dim() == 2 && priors.size(0) == loc.size(1) && priors.size(1) == 4,
                "ssd: loc [B, P, 4] / conf [B, P, C+1] do not fit the prior table");
    c10::cuda::CUDAGuard guard(loc.device());
    const int64_t B = loc.size(0), P = loc.size(1), C = conf.size(2) - 1, rows = B * C * topk;
    const auto f32 = loc.options();
    SsdResult r;
    r.boxes = at::empty({B, P, 4}, f32);
    r.scores_cm = at::empty({B, C, P}, f32);
    at::Tensor dets = at::empty({rows, 5}, f32), labels = at::empty({rows}, f32.dtype(at::kLong)), ids = at::empty({rows}, f32.dtype(at::kLong));
    at::Tensor scratch = at::empty({functs_b200_ssd_scratch_bytes(static_cast<int32_t>(B), static_cast<int32_t>(C))}, f32.dtype(at::kByte));
    at::Tensor host = pinnedWords(B + 1);
    int32_t* words = host.data_ptr<int32_t>();
    words[B] = 0;
    const auto stream = at::cuda::getCurrentCUDAStream();
    checkRc(functs_b200_ssd_postprocess(loc.data_ptr<float>(), conf.data_ptr<float>(), priors.data_ptr<float>(), static_cast<int32_t>(B),
                                        static_cast<int32_t>(P), static_cast<int32_t>(C), static_cast<float>(clamp_max),
                                        static_cast<float>(score_thr), static_cast<int32_t>(topk), static_cast<float>(iou_thr),
                                        r.boxes.data_ptr<float>(), r.scores_cm.data_ptr<float>(), dets.data_ptr<float>(),
                                        labels.data_ptr<int64_t>(), ids.data_ptr<int64_t>(), words, words + B, scratch.data_ptr(),
                                        stream.stream()),
            "ssd post-process");
    C10_CUDA_CHECK(cudaStreamSynchronize(stream.stream()));
    raiseOnStatus(words[B], "ssd post-process");
    int64_t total = 0, stride = C * topk;
    for (int64_t b = 0; b < B; ++b) total += words[b];
    const bool packed = rows * 28 > kKeepRoomBytes && total * 4 < rows;
    if (packed) {
        at::Tensor d = at::empty({total, 5}, f32), l = at::empty({total}, labels.options());
        at::Tensor i = want_ids ? at::empty({total}, ids.options()) : at::Tensor();
        if (total > 0) {
            // (`host` goes back to its pool before the kernel runs: copy_ tells the pool when the copy is done)
            at::Tensor dev_counts = at::empty({B}, f32.dtype(at::kInt));
            dev_counts.copy_(host.narrow(0, 0, B), /*non_blocking=*/true);
            checkRc(functs_b200_ragged_pack(dets.data_ptr<float>(), labels.data_ptr<int64_t>(), ids.data_ptr<int64_t>(),
                                            dev_counts.data_ptr<int32_t>(), static_cast<int32_t>(B), stride, d.data_ptr<float>(),
                                            l.data_ptr<int64_t>(), want_ids ? i.data_ptr<int64_t>() : nullptr, stream.stream()),
                    "ragged pack");
        }
        dets = d;
        labels = l;
        ids = i;
    }
    r.images.reserve(static_cast<size_t>(B));
    int64_t at_row = 0;
    for (int64_t b = 0; b < B; ++b) {
        const int64_t n = words[b], row = packed ? at_row : b * stride;
        r.images.push_back({viewAt(dets, row * 5, {n, 5}), viewAt(labels, row, {n}), want_ids ? viewAt(ids, row, {n}) : at::Tensor()});
        at_row += n;
    }
    return r;
}

YoloResult yoloDetect(const std::vector<at::Tensor>& maps, double score_thr, int64_t topk, double iou_thr, bool dense, bool want_ids) {
    TORCH_CHECK(maps.size() == 3, "yolov3: expected three prediction maps");
    int64_t S[3], N = 0;
    const int64_t B = maps[0].size(0);
    for (int l = 0; l < 3; ++l) {
        TORCH_CHECK(maps[l].dim() == 4 && maps[l].size(0) == B && maps[l].size(1) == 255 && maps[l].size(2) == maps[l].size(3),
                    "yolov3: expected three [B, 255, S, S] maps");
        S[l] = maps[l].size(2);
        N += 3 * S[l] * S[l];
    }
    c10::cuda::CUDAGuard guard(maps[0].device());
    const int64_t capacity = N * 80;
    const auto f32 = maps[0].options();
    const auto i64 = f32.dtype(at::kLong);
    YoloResult r;
    if (dense) {
        r.boxes = at::empty({B, N, 4}, f32);
        r.obj = at::empty({B, N}, f32);
        r.cls = at::empty({B, N, 80}, f32);
    }
    at::Tensor dets = at::empty({B, topk, 5}, f32), labels = at::empty({B, topk}, i64);
    at::Tensor ids = want_ids ? at::empty({B, topk}, i64) : at::Tensor();
    const int64_t bytes = functs_b200_yolo_scratch_bytes(static_cast<int32_t>(B), static_cast<int32_t>(S[0]), static_cast<int32_t>(S[1]),
                                                         static_cast<int32_t>(S[2]), capacity, static_cast<int32_t>(topk));
    at::Tensor scratch = at::empty({bytes + B * 4}, f32.dtype(at::kByte));  // and the device's copy of the counts
    int32_t* counts = reinterpret_cast<int32_t*>(static_cast<char*>(scratch.data_ptr()) + bytes);
    at::Tensor host = pinnedWords(B + 1);
    int32_t* words = host.data_ptr<int32_t>();
    words[B] = 0;
    const auto stream = at::cuda::getCurrentCUDAStream();
    checkRc(functs_b200_yolo_detect(maps[0].data_ptr<float>(), maps[1].data_ptr<float>(), maps[2].data_ptr<float>(),
                                    static_cast<int32_t>(B), static_cast<int32_t>(S[0]), static_cast<int32_t>(S[1]),
                                    static_cast<int32_t>(S[2]), static_cast<float>(score_thr), static_cast<int32_t>(topk),
                                    static_cast<float>(iou_thr), capacity, dense ? r.boxes.data_ptr<float>() : nullptr,
                                    dense ? r.obj.data_ptr<float>() : nullptr, dense ? r.cls.data_ptr<float>() : nullptr,
                                    dets.data_ptr<float>(), labels.data_ptr<int64_t>(), want_ids ? ids.data_ptr<int64_t>() : nullptr,
                                    counts, nullptr, words, words + B, scratch.data_ptr(), stream.stream()),
            "yolov3 post-process");
    C10_CUDA_CHECK(cudaStreamSynchronize(stream.stream()));
    raiseOnStatus(words[B], "yolov3 post-process");
    r.images.reserve(static_cast<size_t>(B));
    for (int64_t b = 0; b < B; ++b) {
        const int64_t n = words[b];
        r.images.push_back({viewAt(dets, b * topk * 5, {n, 5}), viewAt(labels, b * topk, {n}),
                            want_ids ? viewAt(ids, b * topk, {n}) : at::Tensor()});
    }
    return r;
}

}  // namespace functs_b200
