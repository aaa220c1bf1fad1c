#include "detect.h"

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>

#include <chrono>
#include <limits>

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

void raiseOnStatus(int bits, const char* what) {
    TORCH_CHECK(bits == 0, "functs_b200 ", what, ": device status ", bits,
                (bits & FB_STATUS_CAND_OVERFLOW) ? " (a candidate list overflowed)" : "",
                (bits & FB_STATUS_WAIT_TIMEOUT) ? " (a bounded device-side wait ran out)" : "",
                (bits & FB_STATUS_INDEX_RANGE) ? " (an index was out of range)" : "");
}

// Host words that the kernels write themselves (pinned memory is mapped into the device's address space): one per image, its
// count, written after its rows, and the status word.  The host watches the counts instead of waiting for the stream: no
// copy, no wake-up (about 6 us), and the lists of an image are made while the kernel works on later ones.  The kernels write
// the status word before the count of the image it concerns, so the host loads the count with acquire order and the status
// behind it.  The words return to their pool only when all of them have been written, or the stream is idle.
class HostCounts {
public:
    HostCounts(int64_t n, cudaStream_t stream)
        : host_(at::empty({n + 1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true))), words_(host_.data_ptr<int32_t>()), n_(n), stream_(stream) {
        for (int64_t i = 0; i < n; ++i) words_[i] = kPending;
        words_[n] = 0;
    }
    ~HostCounts() {
        if (launched && seen_ < n_) (void)cudaStreamSynchronize(stream_);  // leaving through an exception
    }
    int32_t* counts() { return words_; }  // for the kernels
    int32_t* status() { return words_ + n_; }
    const at::Tensor& tensor() const { return host_; }
    // the next image's count, images in order; raises if a kernel reported a problem up to there
    int64_t next(const char* what) {
        const auto start = std::chrono::steady_clock::now();
        int32_t count = load(seen_);
        for (unsigned spin = 1; count == kPending; ++spin, count = load(seen_)) {
            cpuRelax();
            if (spin % 1024 != 0) continue;
            cudaError_t e = cudaStreamQuery(stream_);
            if (e == cudaErrorNotReady && std::chrono::steady_clock::now() - start > std::chrono::milliseconds(5)) e = cudaStreamSynchronize(stream_);
            if (e == cudaErrorNotReady) continue;
            C10_CUDA_CHECK(e);
            TORCH_CHECK(load(seen_) != kPending, "functs_b200: the kernels ended without a count");
        }
        ++seen_;
        raiseOnStatus(load(n_), what);
        return count;
    }
    bool launched = false;

private:
    static constexpr int32_t kPending = std::numeric_limits<int32_t>::min();
    int32_t load(int64_t i) const { return __atomic_load_n(words_ + i, __ATOMIC_ACQUIRE); }
    static void cpuRelax() {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }
    at::Tensor host_;
    int32_t* words_;
    int64_t n_, seen_ = 0;
    cudaStream_t stream_;
};

// A ragged result is written into room for the largest possible one.  Views of a large room of which less than a quarter is
// filled are made of memory of their own total size instead (one launch, nothing waits for it), so that a caller who keeps
// them does not keep the room.
constexpr int64_t kKeepRoomBytes = 4 << 20;

// The first n rows of a list of its own, which then has a storage of that size (the memory behind it stays what it is).
void cutTo(Detections& d, int64_t n) {
    d.dets.unsafeGetTensorImpl()->set_sizes_contiguous({n, 5});
    d.labels.unsafeGetTensorImpl()->set_sizes_contiguous({n});
    for (const at::Tensor* t : {&d.dets, &d.labels}) t->storage().unsafeGetStorageImpl()->set_nbytes(static_cast<size_t>(t->numel() * t->element_size()));
}

// Lists with storages of their own, their rows copied by a launch behind the kernel that makes them, for 64 images at a time.  Two
// allocations for an image cost about as much as all the rest of it on the host, so they belong where the host has to wait
// anyway: an image's, of its size, when its count is known, while the kernel works on later ones; or, where all counts come at
// once and the largest list is small, all of them beforehand, cut to size later (reserve).  64 images of SSD take 320 us
// against 285 with views of the room, 64 of YOLO 161 (220 without the reserve) against 127, one of YOLO the same 45.
class OwnLists {
public:
    OwnLists(const at::Tensor& dets, const at::Tensor& labels, cudaStream_t stream) : dets_(dets), labels_(labels), stream_(stream) {}
    void reserve(int64_t lists, int64_t rows) {
        for (int64_t i = 0; i < lists; ++i) ready_.push_back(make(rows));
    }
    Detections take(int64_t first, int64_t n) {
        Detections d;
        if (taken_ < ready_.size()) {
            d = std::move(ready_[taken_++]);
            cutTo(d, n);
        } else {
            d = make(n);
        }
        if (n > 0) {
            parts_[count_++] = {first, n, d.dets.data_ptr<float>(), d.labels.data_ptr<int64_t>()};
            if (count_ == FB_RAGGED_MAX_PARTS) flush();
        }
        return d;
    }
    void flush() {
        if (count_ == 0) return;
        checkRc(functs_b200_ragged_split(dets_.data_ptr<float>(), labels_.data_ptr<int64_t>(), parts_, count_, stream_), "ragged split");
        count_ = 0;
    }

private:
    Detections make(int64_t rows) const {  // (at::empty without the dispatcher)
        return {at::detail::empty_cuda({rows, 5}, at::kFloat, dets_.device(), c10::nullopt),
                at::detail::empty_cuda({rows}, at::kLong, dets_.device(), c10::nullopt), at::Tensor()};
    }
    const at::Tensor &dets_, &labels_;
    cudaStream_t stream_;
    std::vector<Detections> ready_;
    size_t taken_ = 0;
    functs_b200_ragged_part parts_[FB_RAGGED_MAX_PARTS];
    int32_t count_ = 0;
};

}  // namespace

SsdResult ssdDetect(const at::Tensor& loc, const at::Tensor& conf, const at::Tensor& priors, double clamp_max, double score_thr,
                    int64_t topk, double iou_thr, Lists lists, const EmitImage& emit) {
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
    const auto stream = at::cuda::getCurrentCUDAStream();
    HostCounts host(B, stream.stream());
    host.launched = true;
    checkRc(functs_b200_ssd_postprocess(loc.data_ptr<float>(), conf.data_ptr<float>(), priors.data_ptr<float>(), static_cast<int32_t>(B),
                                        static_cast<int32_t>(P), static_cast<int32_t>(C), static_cast<float>(clamp_max),
                                        static_cast<float>(score_thr), static_cast<int32_t>(topk), static_cast<float>(iou_thr),
                                        r.boxes.data_ptr<float>(), r.scores_cm.data_ptr<float>(), dets.data_ptr<float>(),
                                        labels.data_ptr<int64_t>(), ids.data_ptr<int64_t>(), host.counts(), host.status(), scratch.data_ptr(),
                                        stream.stream()),
            "ssd post-process");
    const int64_t stride = C * topk;
    if (lists == Lists::kOwn) {
        OwnLists own(dets, labels, stream.stream());
        for (int64_t b = 0; b < B; ++b) {
            const int64_t n = host.next("ssd post-process");
            if (B == 1 && 2 * n >= rows) {  // the room is one list, and not much larger
                Detections d{std::move(dets), std::move(labels), at::Tensor()};
                cutTo(d, n);
                emit(std::move(d));
                return r;
            }
            emit(own.take(b * stride, n));
        }
        own.flush();
        return r;
    }
    const bool may_pack = rows * 36 > kKeepRoomBytes;
    std::vector<int64_t> counts(static_cast<size_t>(B));
    int64_t total = 0, emitted = 0;
    auto emitUpTo = [&](int64_t end, bool packed) {
        for (int64_t row = 0; emitted < end; ++emitted) {
            const int64_t n = counts[static_cast<size_t>(emitted)], at_row = packed ? row : emitted * stride;
            emit({viewAt(dets, at_row * 5, {n, 5}), viewAt(labels, at_row, {n}), viewAt(ids, at_row, {n})});
            row += n;
        }
    };
    for (int64_t b = 0; b < B; ++b) {
        total += counts[static_cast<size_t>(b)] = host.next("ssd post-process");
        // (once a quarter of the room is filled the results stay where they are)
        if (!may_pack || total * 4 >= rows) emitUpTo(b + 1, false);
    }
    if (may_pack && total * 4 < rows) {
        at::Tensor d = at::empty({total, 5}, f32), l = at::empty({total}, labels.options()), i = at::empty({total}, ids.options());
        if (total > 0) {
            // (`host` goes back to its pool before the kernel runs: copy_ tells the pool when the copy is done)
            at::Tensor dev_counts = at::empty({B}, f32.dtype(at::kInt));
            dev_counts.copy_(host.tensor().narrow(0, 0, B), /*non_blocking=*/true);
            checkRc(functs_b200_ragged_pack(dets.data_ptr<float>(), labels.data_ptr<int64_t>(), ids.data_ptr<int64_t>(),
                                            dev_counts.data_ptr<int32_t>(), static_cast<int32_t>(B), stride, d.data_ptr<float>(),
                                            l.data_ptr<int64_t>(), i.data_ptr<int64_t>(), stream.stream()),
                    "ragged pack");
        }
        dets = d;
        labels = l;
        ids = i;
        emitUpTo(B, true);
    }
    return r;
}

YoloResult yoloDetect(const std::vector<at::Tensor>& maps, double score_thr, int64_t topk, double iou_thr, bool dense, Lists lists,
                      const EmitImage& emit) {
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
    at::Tensor dets = at::empty({B * topk, 5}, f32), labels = at::empty({B * topk}, i64);
    at::Tensor ids = lists == Lists::kViews ? at::empty({B, topk}, i64) : at::Tensor();
    const int64_t bytes = functs_b200_yolo_scratch_bytes(static_cast<int32_t>(B), static_cast<int32_t>(S[0]), static_cast<int32_t>(S[1]),
                                                         static_cast<int32_t>(S[2]), capacity, static_cast<int32_t>(topk));
    at::Tensor scratch = at::empty({bytes + B * 4}, f32.dtype(at::kByte));  // and the device's copy of the counts
    int32_t* counts = reinterpret_cast<int32_t*>(static_cast<char*>(scratch.data_ptr()) + bytes);
    const auto stream = at::cuda::getCurrentCUDAStream();
    HostCounts host(B, stream.stream());
    host.launched = true;
    checkRc(functs_b200_yolo_detect(maps[0].data_ptr<float>(), maps[1].data_ptr<float>(), maps[2].data_ptr<float>(),
                                    static_cast<int32_t>(B), static_cast<int32_t>(S[0]), static_cast<int32_t>(S[1]),
                                    static_cast<int32_t>(S[2]), static_cast<float>(score_thr), static_cast<int32_t>(topk),
                                    static_cast<float>(iou_thr), capacity, dense ? r.boxes.data_ptr<float>() : nullptr,
                                    dense ? r.obj.data_ptr<float>() : nullptr, dense ? r.cls.data_ptr<float>() : nullptr,
                                    dets.data_ptr<float>(), labels.data_ptr<int64_t>(), ids.defined() ? ids.data_ptr<int64_t>() : nullptr,
                                    counts, nullptr, host.counts(), host.status(), scratch.data_ptr(), stream.stream()),
            "yolov3 post-process");
    OwnLists own(dets, labels, stream.stream());
    if (lists == Lists::kOwn) {
        if (B == 1) {  // the room is one list
            Detections d{dets, labels, at::Tensor()};
            cutTo(d, host.next("yolov3 post-process"));
            emit(std::move(d));
            return r;
        }
        own.reserve(B, topk);
    }
    for (int64_t b = 0; b < B; ++b) {
        const int64_t n = host.next("yolov3 post-process");
        if (lists == Lists::kOwn) emit(own.take(b * topk, n));
        else emit({viewAt(dets, b * topk * 5, {n, 5}), viewAt(labels, b * topk, {n}), viewAt(ids, b * topk, {n})});
    }
    own.flush();
    return r;
}

}  // namespace functs_b200
