"""The calls that users of this package make, as cases for a timing harness.

Five post-processing programs (row assignment in a loop, YOLOv3-style and SSD-style detection, an imperative LSTM, YOLACT
mask assembly) and the two single-group programs, called the way a program would call them: through the modules of
``functs_b200.workloads`` or through a TorchScript program built with ``functs_b200.jit.build``.

listed()         named cases, from the smallest call to the largest
draw(rng)        one more case of the same ranges
prepare(case, seed), run(state), work(case), tolerance(case)
"""
import functools
import math

import numpy as np
import torch

from functs_b200 import jit, patterns, simpleops, workloads

DEVICE = "cuda"
YOLO_CHANNELS = 255
YOLO_TOPK = 1000
SSD_TOPK = 200


def listed():
    return [
        # the smallest call: an imperative loop over the rows of a small matrix, one launch, latency is everything
        {"name": "rows 64x1024", "kind": "rows", "rows": 64, "cols": 1024},
        # box decoding with strided slices on an ordinary number of proposals: one small fusion group
        {"name": "offset2bbox 3000x4", "kind": "offset2bbox", "boxes": 3000, "classes": 1},
        # image normalisation with a channel swap, full-size image: one large fusion group
        {"name": "normalize 800x1333", "kind": "normalize", "height": 800, "width": 1333},
        # one image of a video stream through the detection module: latency
        {"name": "yolo 416 b1 call", "kind": "yolo", "via": "call", "batch": 1, "cell": 13, "sparse": False},
        # offline batch, detections stay on the device in padded form for the next stage
        {"name": "yolo 416 b64 padded", "kind": "yolo", "via": "padded", "batch": 64, "cell": 13, "sparse": False},
        # larger images, a trained head's few confident boxes, and the decoded scores wanted as well (user's own program)
        {"name": "yolo 608 b8 dense graph", "kind": "yolo", "via": "dense", "batch": 8, "cell": 19, "sparse": True},
        # one image through the user's own SSD program
        {"name": "ssd 300 b1 graph", "kind": "ssd", "via": "graph", "batch": 1, "image": 300, "classes": 80, "sparse": False},
        # offline batch through the SSD module, ragged per-image lists
        {"name": "ssd 300 b64 call", "kind": "ssd", "via": "call", "batch": 64, "image": 300, "classes": 80, "sparse": False},
        # one short sequence, small cell, odd length: streaming inference
        {"name": "lstm t25 b1 h256", "kind": "lstm", "via": "call", "steps": 25, "batch": 1, "inputs": 256, "hidden": 256},
        # the training-size sequence batch
        {"name": "lstm t64 b64 h512", "kind": "lstm", "via": "call", "steps": 64, "batch": 64, "inputs": 512, "hidden": 512},
        # one image, few detections, the mask logits wanted as well (user's own program)
        {"name": "yolact b1 logits graph", "kind": "yolact", "via": "logits", "batch": 1, "size": 138, "dets": 15},
        # offline batch with the full hundred detections per image
        {"name": "yolact b64 call", "kind": "yolact", "via": "call", "batch": 64, "size": 138, "dets": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("rows", "offset2bbox", "normalize", "yolo", "yolo", "ssd", "ssd", "lstm", "yolact", "yolact"))
    if kind == "rows":
        rows = _log(rng, 8, 4096)
        return {"kind": kind, "rows": rows, "cols": _log(rng, 64, 4096)}
    if kind == "offset2bbox":  # class-agnostic deltas, or one set of deltas per class
        classes = rng.choice((1, 1, 1, 20, 80))
        return {"kind": kind, "boxes": _log(rng, 100, 200000 // classes), "classes": classes}
    if kind == "normalize":
        return {"kind": kind, "height": _log(rng, 96, 1440), "width": _log(rng, 96, 1920)}
    if kind == "yolo":  # images of 320 to 608 pixels; the batch of the largest ones is bounded by the listed work
        cell = rng.randint(10, 19)
        via = rng.choice(("call", "padded", "graph", "dense"))
        most = 64 * 13 * 13 // (cell * cell) if via != "dense" else 16
        return {"kind": kind, "via": via, "batch": _log(rng, 1, min(64, most)), "cell": cell, "sparse": rng.random() < 0.5}
    if kind == "ssd":
        image = rng.randint(200, 512)
        classes = rng.choice((20, 80, rng.randint(5, 90)))
        most = 64 * 8732 * 81 // (_num_priors(image) * (classes + 1))
        return {"kind": kind, "via": rng.choice(("call", "graph")), "batch": _log(rng, 1, min(64, max(1, most))),
                "image": image, "classes": classes, "sparse": rng.random() < 0.5}
    if kind == "lstm":
        return {"kind": kind, "via": rng.choice(("call", "device")), "steps": _log(rng, 4, 64), "batch": _log(rng, 1, 64),
                "inputs": rng.choice((128, 256, 512, 16 * rng.randint(4, 32))), "hidden": rng.choice((256, 512))}
    via, size, dets = rng.choice(("call", "graph", "logits")), 2 * rng.randint(40, 80), _log(rng, 4, 200)
    most = 64 * 138 * 138 * (128 + 100) // (size * size * (128 + dets * (5 if via == "logits" else 1)))
    return {"kind": kind, "via": via, "batch": _log(rng, 1, min(64, most)), "size": size, "dets": dets}


# ---- programs and handles ------------------------------------------------------------------------------------------------


def rows_program(a: torch.Tensor, b: torch.Tensor, n: int):
    a = a.clone()
    b = b.clone()
    for i in range(n):
        b[i] = b[i] + 1
    return b


def _ssd_features(image):
    feats = [-(-image // 8)]
    while feats[-1] > 1:
        f = feats[-1]
        feats.append(-(-f // 2) if f > 5 else f - 2 if f > 2 else 1)
    return feats


def _ssd_shapes(level, levels):
    return 6 if 0 < level < max(2, levels - 2) else 4


def _num_priors(image):
    feats = _ssd_features(image)
    return sum(f * f * _ssd_shapes(k, len(feats)) for k, f in enumerate(feats))


def _ssd_priors(image):
    """The usual grid: 4 or 6 boxes per cell of feature maps that halve from image / 8 down to 1; 8732 at 300 pixels."""
    feats = _ssd_features(image)
    out = []
    for k, f in enumerate(feats):
        step = image / f
        small = image * (0.07 if k == 0 else 0.15 + 0.75 * (k - 1) / max(1, len(feats) - 1))
        large = image * (0.15 + 0.75 * k / max(1, len(feats) - 1))
        sizes = [(small, small), (math.sqrt(small * large),) * 2]
        for r in (2.0, 3.0)[:(_ssd_shapes(k, len(feats)) - 2) // 2]:
            q = math.sqrt(r)
            sizes += [(small * q, small / q), (small / q, small * q)]
        for i in range(f):
            for j in range(f):
                out += [((j + 0.5) * step, (i + 0.5) * step, w, h) for w, h in sizes]
    return torch.tensor(out, dtype=torch.float64).to(torch.float32)


# A program builds its modules and graphs once and feeds them one input after another.
@functools.lru_cache(maxsize=12)
def _handle(kind, via, *config):
    if kind == "rows":
        return jit.build(rows_program)
    if kind == "offset2bbox":
        return jit.build(simpleops.offset2bbox)
    if kind == "normalize":
        return jit.build(simpleops.normalize)
    if kind == "yolo":
        sizes = config
        if via == "graph":
            return jit.build(patterns.YOLOV3Det(sizes))
        if via == "dense":
            return jit.build(patterns.YOLOV3Post(sizes))
        return workloads.YOLOV3BBox(sizes, device=DEVICE)
    if kind == "ssd":
        priors = _ssd_priors(config[0])
        if via == "graph":
            return jit.build(patterns.SSDPost(priors, clamp_max=float(config[0])))
        return workloads.SSDBBox(priors, clamp_max=float(config[0]), device=DEVICE)
    if via == "graph":
        return jit.build(patterns.YolactMasksOnly())
    if via == "logits":
        return jit.build(patterns.YolactMasks())
    return workloads.YolactBBoxMask(device=DEVICE)


def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEVICE)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=DEVICE)

    kind, via = case["kind"], case.get("via", "graph")
    if kind == "rows":
        shape = (case["rows"], case["cols"])
        return {"kind": kind, "fn": _handle(kind, via), "args": (randn(*shape), randn(*shape), case["rows"])}
    if kind == "offset2bbox":
        xy, wh = rand(case["boxes"], 2) * 800, rand(case["boxes"], 2) * 200 + 1
        boxes = torch.cat([xy, xy + wh], dim=1)
        return {"kind": kind, "fn": _handle(kind, via), "args": (boxes, randn(case["boxes"], 4 * case["classes"]))}
    if kind == "normalize":
        return {"kind": kind, "fn": _handle(kind, via), "args": (rand(case["height"], case["width"], 3), 0.45, 4.4)}
    if kind == "yolo":
        sizes = tuple(case["cell"] * f for f in (1, 2, 4))
        maps = [randn(case["batch"], YOLO_CHANNELS, s, s) for s in sizes]
        if case["sparse"]:  # a trained head: most boxes hold nothing, and the classes that are absent score low
            for m in maps:
                heads = m.view(m.size(0), 3, YOLO_CHANNELS // 3, -1)
                heads[:, :, 4:].mul_(2.0)
                heads[:, :, 4].sub_(4.0)
                heads[:, :, 5:].sub_(2.0)
        return {"kind": kind, "via": via, "fn": _handle(kind, via, *sizes), "maps": maps,
                "buffers": _collect_into(case["batch"] * YOLO_TOPK) if via != "padded" else None}
    if kind == "ssd":
        priors = _num_priors(case["image"])
        loc, conf = randn(case["batch"], priors, 4), randn(case["batch"], priors, case["classes"] + 1)
        if case["sparse"]:  # a trained head: nearly every prior is background
            conf.mul_(2.0)
            conf[..., -1].add_(9.0)
        return {"kind": kind, "via": via, "fn": _handle(kind, via, case["image"]), "args": (loc, conf),
                "buffers": _collect_into(case["batch"] * case["classes"] * SSD_TOPK)}
    if kind == "lstm":
        i, h = case["inputs"], case["hidden"]
        bound = 1.0 / math.sqrt(h)
        w = [(rand(*shape) * 2 - 1) * bound for shape in ((4, i, h), (4, h, h), (4, 1, h), (4, 1, h))]
        return {"kind": kind, "via": via, "fn": workloads.LSTM(*w, device=DEVICE), "x": randn(case["steps"], case["batch"], i)}
    b, s, n = case["batch"], case["size"], case["dets"]
    corners = torch.sort(rand(b, n, 2, 2), dim=2).values.reshape(b, n, 4) * float(s)  # (x1, y1, x2, y2)
    return {"kind": kind, "fn": _handle(kind, via), "args": (randn(b, s, s, 32), torch.tanh(randn(b, n, 32)), corners)}


def _collect_into(rows):
    """The buffers in which a program collects the ragged detections of a batch: boxes with scores, labels and, where the
    program returns them, box numbers.  Rows past the end stay zero."""
    return [torch.zeros(rows, 5, device=DEVICE)] + [torch.zeros(rows, dtype=torch.int64, device=DEVICE) for _ in range(2)]


def _collected(lists, buffers):
    """Per-image tuples of ragged tensors, one image after another, and the number of detections of every image."""
    counts = np.array([t[0].size(0) for t in lists])
    total = int(counts.sum())
    for field, buffer in zip(zip(*lists), buffers):
        torch.cat(field, out=buffer[:total])
    return buffers[:len(lists[0])] + [counts]


def run(state):
    kind, via, fn = state["kind"], state.get("via"), state["fn"]
    if kind == "yolo":
        if via == "padded":
            return fn.forward_padded(state["maps"])
        if via == "dense":
            boxes, obj, cls, results = fn(state["maps"])
            return [boxes, obj, cls] + _collected(results, state["buffers"])
        return _collected(fn(state["maps"]), state["buffers"])
    if kind == "ssd":
        if via == "graph":
            boxes, scores, results = fn(*state["args"])
            return [boxes, scores] + _collected(results, state["buffers"])
        return _collected(fn(*state["args"]), state["buffers"])
    if kind == "lstm":
        return fn.forward_device(state["x"]) if via == "device" else fn(state["x"])
    return fn(*state["args"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------


def work(case):
    kind, via = case["kind"], case.get("via")
    if kind == "rows":
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n, "flops": n}
    if kind == "offset2bbox":
        n = case["boxes"] * case["classes"]
        return {"bytes": 16 * case["boxes"] + 32 * n, "flops": 20 * n + 6 * case["boxes"]}
    if kind == "normalize":
        n = case["height"] * case["width"] * 3
        return {"bytes": 8 * n, "flops": 2 * n}
    b = case["batch"]
    if kind == "yolo":
        boxes = b * 3 * sum((case["cell"] * f) ** 2 for f in (1, 2, 4))
        out = b * YOLO_TOPK * (36 if via == "padded" else 28) + (boxes * (4 + 1 + 80) * 4 if via == "dense" else 0)
        return {"bytes": boxes * 85 * 4 + out, "flops": boxes * 85 * 4}
    if kind == "ssd":
        p, c = _num_priors(case["image"]), case["classes"]
        out = b * c * 50 * 28 + (b * p * (4 + c) * 4 if via == "graph" else 0)
        return {"bytes": b * p * (c + 1 + 4) * 4 + p * 16 + out, "flops": b * p * (c + 1) * 4}
    if kind == "lstm":
        t, i, h = case["steps"], case["inputs"], case["hidden"]
        return {"bytes": 4 * (t * b * i + 4 * h * (i + h + 2) + 2 * t * b * h), "flops": 2 * t * b * 4 * h * (i + h)}
    hw, n = case["size"] ** 2, case["dets"]
    logits = via == "logits"
    # without the logits only the pixels inside a box need their dot product: a ninth of the image for random corners
    return {"bytes": b * (hw * 32 * 4 + n * 36 * 4 + n * hw * (5 if logits else 1)),
            "flops": 2 * 32 * b * n * hw / (1 if logits else 9)}


def tolerance(case):
    if case["kind"] in ("rows", "normalize", "offset2bbox"):
        return "exact"  # every step rounds on its own, in the program's order
    if case["kind"] == "lstm":
        return {"rel": 1e-5}  # sums of fp32 products in another order
    if case["kind"] == "yolact":
        return {"rel": 1e-5, "differ": 1e-5}  # a pixel whose logit lies on the threshold to the last bit
    return {"rel": 1e-5, "differ": 1e-4}  # a tie between candidates that are equal to the last bit
