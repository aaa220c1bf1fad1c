"""GPU parity for C5 (YOLACT-style mask assembly) and C4 (imperative LSTM) against the TorchScript CPU oracle."""
import pytest
import torch

from oracle import workloads as W
from tests.util import close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb(cuda_device):
    import functs_b200
    return functs_b200


def yolact_case(fb, proto, coef, boxes):
    masks, logits = fb.ops.yolact_masks(proto.cuda(), coef.cuda(), boxes.cuda(), with_logits=True)
    masks_fast = fb.ops.yolact_masks(proto.cuda(), coef.cuda(), boxes.cuda())
    assert torch.equal(masks, masks_fast)  # the value-check variant and the product variant agree bit for bit
    masks, logits = masks.cpu(), logits.cpu().permute(0, 2, 3, 1)  # [B,H,W,N]
    oracle = torch.jit.script(W.YolactMasks())
    ndiff = 0
    for s in range(0, proto.size(0), 16):  # the comparison runs in slices of 16 images to bound host memory
        e = min(s + 16, proto.size(0))
        ndiff += yolact_compare(oracle, proto[s:e], coef[s:e], boxes[s:e], masks[s:e], logits[s:e])
    print(f"mask bytes differing from the oracle inside the 1e-5 boundary band: {ndiff} of {masks.numel()}")
    return ndiff


def yolact_compare(oracle, proto, coef, boxes, masks, logits):
    want_masks, want_logits = oracle(proto, coef, boxes)
    # a dot product is accurate relative to the sum of the magnitudes of its terms
    mag = torch.einsum("bhwk,bnk->bhwn", proto.abs(), coef.abs())
    close(logits, want_logits, rtol=1e-5, scale=mag, what="mask logits")
    # thresholded masks: identical except where the fp64 logit is within 1e-5 of zero (the sigmoid > 0.5 boundary)
    diff = masks != want_masks
    ndiff = int(diff.sum())
    if ndiff:
        l64 = torch.einsum("bhwk,bnk->bnhw", proto.double(), coef.double())
        assert bool((l64[diff].abs() < 1e-5).all()), "mask mismatch away from the threshold boundary"
    return ndiff


def test_yolact_config_shapes(fb):
    proto, coef, boxes = W.make_yolact_inputs(2)
    yolact_case(fb, proto, coef, boxes)


def test_yolact_full_batch_against_oracle(fb):
    """B = 64 (the configured maximum): 122 M mask bytes against the oracle's own run."""
    proto, coef, boxes = W.make_yolact_inputs(64)
    yolact_case(fb, proto, coef, boxes)


def test_yolact_small_and_degenerate_boxes(fb):
    proto, coef, boxes = W.make_yolact_inputs(2, size=20, num_det=7)
    boxes[0, 0] = torch.tensor([5.0, 5.0, 5.0, 5.0])          # empty box -> still padded by 1
    boxes[0, 1] = torch.tensor([-4.0, -4.0, 30.0, 30.0])      # outside the image on every side
    boxes[0, 2] = torch.tensor([15.0, 3.0, 2.0, 12.0])        # x1 > x2
    boxes[1, 0] = torch.tensor([0.0, 0.0, 0.0, 20.0])
    yolact_case(fb, proto, coef, boxes)


def test_yolact_crop_golden(fb):
    """Crop rule against the fixture written by the reference's crop(): with all-ones coefficients on a one-hot
    prototype the logit is large and positive everywhere, so the mask is exactly the crop region."""
    import os
    f = torch.load(os.path.join(os.path.dirname(__file__), "golden", "yolact_crop.pt"))
    h, w, n = f["masks"].shape
    proto = torch.zeros(1, h, w, 32)
    proto[..., 0] = 10.0
    coef = torch.zeros(1, n, 32)
    coef[..., 0] = 1.0
    masks = fb.ops.yolact_masks(proto.cuda(), coef.cuda(), f["boxes"][None].cuda())
    want = (f["out"] > 0).permute(2, 0, 1).to(torch.uint8)
    assert torch.equal(masks[0].cpu(), want)


def test_yolact_full_batch_properties(fb):
    """B = 64: shard invariance and crop containment instead of an oracle run."""
    proto, coef, boxes = [t.cuda() for t in W.make_yolact_inputs(64)]
    full = fb.ops.yolact_masks(proto, coef, boxes)
    part = fb.ops.yolact_masks(proto[40:44].contiguous(), coef[40:44].contiguous(), boxes[40:44].contiguous())
    assert torch.equal(full[40:44], part)
    bounds = torch.stack([W.crop_bounds(b.cpu(), 138, 138) for b in boxes[:4]])  # [4,N,4]
    xs = torch.arange(138)
    inside = ((xs[None, None, None, :] >= bounds[:, :, 0, None, None]) & (xs[None, None, None, :] < bounds[:, :, 1, None, None]) &
              (xs[None, None, :, None] >= bounds[:, :, 2, None, None]) & (xs[None, None, :, None] < bounds[:, :, 3, None, None]))
    assert not bool((full[:4].cpu().bool() & ~inside).any())
    assert set(full.unique().tolist()) <= {0, 1}


# ---- LSTM ----------------------------------------------------------------------------------------------


def lstm_case(fb, seq, batch, hidden, mode):
    """Bar for fp32 values: 1e-5 relative.  h = o * tanh(c) lies in (-1, 1) and passes through zero, so a value is
    measured against max(|want|, 1): 1 is the bound of the gate activations every h and c is formed from.  No absolute
    term.  On top of that the device result is compared with the fp64 evaluation of the same program: the fp32 CUDA-core
    path (mode 1) must be as close to it as the fp32 CPU oracle itself is (factor 2); the tensor-core paths (modes 0, 2, 3)
    splits every fp32 operand into two TF32 numbers, which carry 22 of the 24 mantissa bits, so its products are about
    four times less accurate than fp32 products: factor 10, and always below 1e-5."""
    x, w_ih, w_hh, b_ih, b_hh = W.make_lstm_inputs(seq, batch, hidden)
    want_hs, want_cs = torch.jit.script(W.LSTMSeq(w_ih, w_hh, b_ih, b_hh))(x)
    mod = fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)
    hs, cs = mod(x, mode=mode)
    assert mod.kernels_last_call == fb.workloads.LSTM.expected_launches(seq, batch, hidden, mode)
    o64 = W.LSTMSeq(w_ih.double(), w_hh.double(), b_ih.double(), b_hh.double())
    hs64, cs64 = o64(x.double())
    for name, got, want, truth in (("hs", hs, want_hs, hs64), ("cs", cs, want_cs, cs64)):
        e_or = float((want.double() - truth).abs().max())
        e_gpu = float((got.cpu().double() - truth).abs().max())
        print(f"T={seq} B={batch} H={hidden} mode={mode} {name}: max |v - v64| oracle {e_or:.2e}, gpu {e_gpu:.2e}")
        assert e_gpu <= (2.0 if mode == 1 else 10.0) * e_or + 1e-7 and e_gpu < 1e-5, (name, e_gpu, e_or)
        close(got.cpu(), want, rtol=1e-5, atol=0.0, scale=1.0, what=name)


def test_lstm_tensor_core_projection_matches_cuda_cores(fb):
    """Runs first among the LSTM tests: the tcgen05 (3xTF32) input projection against the fp32 CUDA-core projection on
    a small shape.  Agreement to 1e-5 is the evidence that the shared-memory descriptor strides describe the pre-tiled
    operand layout."""
    x, w_ih, w_hh, b_ih, b_hh = W.make_lstm_inputs(2, 64, 512)
    mod = fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)
    ref_hs, _ = mod(x, mode=1)
    ref_hs = ref_hs.clone()
    hs, _ = mod(x, mode=0)
    err = float((hs - ref_hs).abs().max())
    print(f"tcgen05 projection vs CUDA-core projection, max |dh|: {err:.3e}")
    assert err < 1e-5


@pytest.mark.parametrize("mode", [1, 0, 2, 3])
def test_lstm_config_shapes(fb, mode):
    lstm_case(fb, 64, 64, 512, mode)


def test_lstm_tensor_core_recurrence_small(fb):
    """The tcgen05 recurrence (mode 2) on other lengths and on H = 256; a batch other than 64 takes the CUDA-core
    recurrence under the same mode."""
    lstm_case(fb, 1, 64, 512, 2)
    lstm_case(fb, 2, 64, 512, 2)
    lstm_case(fb, 9, 64, 256, 2)
    lstm_case(fb, 3, 33, 512, 2)


@pytest.mark.parametrize("seq,batch,hidden", [(3, 5, 256), (1, 64, 512), (7, 33, 512), (5, 8, 256)])
def test_lstm_ragged(fb, seq, batch, hidden):
    lstm_case(fb, seq, batch, hidden, 1)
    lstm_case(fb, seq, batch, hidden, 0)


def test_lstm_cell_golden(fb):
    """One step against the fixture written by the reference's LSTMCell.forward needs H in {256, 512}; the fixture
    is H=32, so embed it: zero-pad weights to H=256 (extra units stay decoupled) and compare the first 32 units."""
    import os
    f = torch.load(os.path.join(os.path.dirname(__file__), "golden", "lstm_cell.pt"))
    hid, big = 32, 256
    bat = f["x"].size(0)
    w_ih = torch.zeros(4, big, big)
    w_hh = torch.zeros(4, big, big)
    b_ih = torch.zeros(4, 1, big)
    b_hh = torch.zeros(4, 1, big)
    w_ih[:, :hid, :hid] = f["w_ih"]
    w_hh[:, :hid, :hid] = f["w_hh"]
    b_ih[..., :hid] = f["b_ih"]
    b_hh[..., :hid] = f["b_hh"]
    # the fixture starts from non-zero (h0, c0); the kernel starts from zero, so check the zero-state step of the
    # same cell with the oracle, which the CPU test pins to the fixture
    x = torch.zeros(1, bat, big)
    x[0, :, :hid] = f["x"]
    want_h, want_c = W.lstm_cell(x[0], torch.zeros(bat, big), torch.zeros(bat, big), w_ih, w_hh, b_ih, b_hh)
    hs, cs = fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)(x, mode=1)
    close(hs[0].cpu(), want_h, rtol=1e-5, atol=1e-6, what="h1")
    close(cs[0].cpu(), want_c, rtol=1e-5, atol=1e-6, what="c1")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("seq,batch,inputs,hidden", [
    (2, 64, 512, 512),    # one whole row tile
    (3, 5, 63, 256),      # rows and depth that fill no tile
    (40, 33, 512, 512),   # operands split by a launch of their own
])
def test_lstm_inputs_that_are_not_finite(fb, seq, batch, inputs, hidden, mode):
    """NaN of every sign and payload, infinities and the largest float pass through the projection as they do in the oracle:
    NaN rows become NaN, the others saturate their gates.  The bound for finite values is test_gpu_ragged's, on fp64."""
    g = torch.Generator().manual_seed(seq)
    bound = hidden ** -0.5
    w = [(torch.rand(*s, generator=g) * 2 - 1) * bound for s in ((4, inputs, hidden), (4, hidden, hidden), (4, 1, hidden), (4, 1, hidden))]
    x = torch.randn(seq, batch, inputs, generator=g)
    x[..., 3] *= 0.1  # (times the weight below: large, but no second infinity)
    odd = torch.tensor([0x7fffffff, -1, 0x7fc00000, 0x7f800000, -0x800000], dtype=torch.int32).view(torch.float32)
    x[0, torch.arange(5), torch.tensor([0, 31, 40, 62, 7])] = odd
    x[-1, 3, 1] = torch.finfo(torch.float32).max
    x[-1, 4, 61] = -torch.finfo(torch.float32).max
    w[0][2, 3, 7] = torch.finfo(torch.float32).max
    hs64, cs64 = W.LSTMSeq(*[t.double() for t in w])(x.double())
    assert bool(hs64[:, :3].isnan().all()) and bool(hs64[:, 3:].isfinite().all())
    for got, want in zip(fb.workloads.LSTM(*w)(x, mode=mode), (hs64, cs64)):
        got = got.cpu().double()
        assert torch.equal(got.isnan(), want.isnan())
        assert float((got - want)[:, 3:].abs().max()) < 3e-6


@pytest.mark.parametrize("seq,batch,inputs,hidden", [
    (1, 1, 1, 256), (17, 1, 128, 256), (56, 7, 129, 256), (16, 7, 300, 256), (32, 14, 512, 256), (15, 9, 385, 256),  # one launch
    (57, 1, 256, 256), (33, 14, 100, 256), (9, 1, 256, 512),          # a projection in front of the steps
    (1, 15, 64, 256), (1, 3, 64, 512), (1, 71, 100, 512),             # a single step: the gates alone
    (3, 15, 64, 256), (4, 29, 64, 512), (2, 50, 64, 256), (9, 63, 64, 512),  # halves of two to five rows, some of them empty
])
def test_lstm_recurrence_shapes(fb, seq, batch, inputs, hidden):
    """Every form of the recurrence at its edges against fp64: rows and steps that fill no cluster, half or buffer.  Bound: the gates
    are sums of K + H products of magnitudes that sum to a few units, so fp32 (or three TF32 products) leaves some 1e-6."""
    g = torch.Generator().manual_seed(seq * 100 + batch)
    bound = hidden ** -0.5
    w = [(torch.rand(*s, generator=g) * 2 - 1) * bound for s in ((4, inputs, hidden), (4, hidden, hidden), (4, 1, hidden), (4, 1, hidden))]
    x = torch.randn(seq, batch, inputs, generator=g)
    want = W.LSTMSeq(*[t.double() for t in w])(x.double())
    mod = fb.workloads.LSTM(*w)
    got = mod(x)
    assert mod.kernels_last_call == fb.workloads.LSTM.expected_launches(seq, batch, hidden, 0, inputs)
    for a, b in zip(got, want):
        assert float((a.cpu().double() - b).abs().max()) < 3e-6


@pytest.mark.parametrize("seq,batch,hidden,mode", [
    (2, 1, 256, 0), (25, 1, 256, 0), (25, 14, 256, 0), (25, 2, 256, 3), (40, 9, 512, 3),    # warps that multiply and apply gates
    (3, 15, 256, 0), (40, 50, 256, 0), (40, 20, 512, 0), (64, 64, 512, 0),                  # warps that only do one of the two
])
def test_lstm_waits_that_run_out(fb, seq, batch, hidden, mode):
    """With the exchange between the CTAs dropped every wait runs out: the kernel goes through its steps all the same, reports it and
    leaves the context usable.  (A warp that runs ahead of the gate warps then would leave them at a barrier for ever.)"""
    x, w_ih, w_hh, b_ih, b_hh = W.make_lstm_inputs(seq, batch, hidden)
    mod = fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)
    want = [t.clone() for t in mod(x, mode=mode)]
    lib = fb._lib.lib
    fb._lib.check(lib.functs_b200_debug_set(b"lstm_drop_exchange", 1), "debug_set")
    try:
        with pytest.raises(fb.FunctsB200Error, match="wait ran out"):
            mod(x, mode=mode)
    finally:
        fb._lib.check(lib.functs_b200_debug_set(b"lstm_drop_exchange", 0), "debug_set")
    mod._status.zero_()
    for got, ref in zip(mod(x, mode=mode), want):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("seq,batch,inputs,hidden", [(3, 5, 63, 256), (2, 6, 130, 256), (3, 8, 80, 256)])
def test_lstm_projection_of_ragged_depth_with_inputs_that_are_not_finite(fb, seq, batch, inputs, hidden):
    """Depths that fill no k-tile in the tensor-core projection, which mode 0 leaves to the one launch at these sizes."""
    test_lstm_inputs_that_are_not_finite(fb, seq, batch, inputs, hidden, 3)


@pytest.mark.parametrize("seq,batch,inputs,hidden,mode", [
    (2, 1, 256, 256, 3), (3, 8, 80, 256, 3), (5, 14, 500, 256, 3),  # one and two rows per cluster behind a projection
    (2, 150, 64, 256, 0), (3, 90, 64, 512, 0),                      # more clusters than run at once
])
def test_lstm_projection_and_steps(fb, seq, batch, inputs, hidden, mode):
    """Against fp64, bound as in test_lstm_recurrence_shapes."""
    g = torch.Generator().manual_seed(seq * 100 + batch)
    bound = hidden ** -0.5
    w = [(torch.rand(*s, generator=g) * 2 - 1) * bound for s in ((4, inputs, hidden), (4, hidden, hidden), (4, 1, hidden), (4, 1, hidden))]
    x = torch.randn(seq, batch, inputs, generator=g)
    want = W.LSTMSeq(*[t.double() for t in w])(x.double())
    mod = fb.workloads.LSTM(*w)
    got = mod(x, mode=mode)
    assert mod.kernels_last_call == 2
    for a, b in zip(got, want):
        assert float((a.cpu().double() - b).abs().max()) < 3e-6


def test_lstm_rejects_unsupported_hidden(fb):
    x, w_ih, w_hh, b_ih, b_hh = W.make_lstm_inputs(2, 2, 64)
    with pytest.raises(fb.FunctsB200Error):
        fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)(x)


@pytest.mark.parametrize("batch,height,width,dets,thr", [
    (1, 1, 2, 1, 0.5), (3, 5, 6, 33, 0.5), (2, 69, 70, 100, 0.3), (1, 138, 138, 16, 0.9), (5, 37, 130, 256, 0.5),
    (70, 33, 34, 129, 0.001), (2, 64, 64, 32, 0.9995),
])
def test_yolact_masks_on_the_tensor_cores(fb, batch, height, width, dets, thr):
    """Against the variant that forms every logit in fp32, byte for byte: planes that start off a word, tiles of many rows, one
    to 256 detections, logits at and around the threshold, and values that are not finite."""
    g = torch.Generator().manual_seed(batch + dets)
    proto = torch.randn(batch, height, width, 32, generator=g)
    coef = torch.tanh(torch.randn(batch, dets, 32, generator=g))
    xy = torch.rand(batch, dets, 4, generator=g) * torch.tensor([width, height, width, height], dtype=torch.float32)
    coef[:, ::5] *= 1e-5
    proto[:, ::3, :, 7] = float("inf")
    proto[:, -1, ::4] = float("nan")
    proto[:, 0, 1::2] = 0.0
    if batch == 3:
        coef[1, 0, 3] = float("nan")
    args = (proto.cuda(), coef.cuda(), xy.cuda(), thr)
    masks, _ = fb.ops.yolact_masks(*args, with_logits=True)
    assert torch.equal(fb.ops.yolact_masks(*args), masks)


@pytest.mark.parametrize("far", [3e9, 2147483648.0, float("inf")])
@pytest.mark.parametrize("height,width", [(1, 138), (33, 10)])
def test_yolact_boxes_outside_the_integers(fb, height, width, far):
    """Crops of boxes whose coordinates no 32-bit integer holds: empty on the far sides, everything where the box spans the image;
    the same from both mask kernels."""
    proto = torch.ones(1, height, width, 32, device="cuda")
    coef = torch.ones(1, 6, 32, device="cuda")
    h, w = float(height), float(width)
    boxes = torch.tensor([[[-far, 0, -far, h], [far, 0, far, h], [-far, 0, far, h], [0, -far, w, -far], [0, far, w, far],
                           [-far, -far, far, far]]], device="cuda")
    masks, _ = fb.ops.yolact_masks(proto, coef, boxes, with_logits=True)
    assert masks.flatten(2).sum(2).tolist() == [[n * height * width for n in (0, 0, 1, 0, 0, 1)]]
    assert torch.equal(fb.ops.yolact_masks(proto, coef, boxes), masks)


def test_yolact_rejects_shapes_that_do_not_fit(fb):
    """Sizes come from proto and coef: anything else that the kernel would read or write beside them is refused on the host."""
    mod = fb.workloads.YolactBBoxMask()
    proto, coef, boxes = [t.cuda() for t in W.make_yolact_inputs(2, size=20, num_det=7)]
    want = mod(proto, coef, boxes).clone()
    bad = [(proto, coef[:1], boxes), (proto, coef, boxes[:1]), (proto, coef, boxes[:, :6]), (proto, coef[..., :31], boxes),
           (proto, coef, boxes[..., :3]), (proto[..., :31], coef, boxes), (proto[0], coef, boxes)]
    for args in bad:
        with pytest.raises(ValueError):
            mod(*args)
        with pytest.raises(ValueError):
            fb.ops.yolact_masks(*args)
    with pytest.raises(ValueError):
        fb.ops.yolact_masks(proto, coef, boxes, out=torch.empty(2, 7, 20, 18, dtype=torch.uint8, device="cuda"))
    with pytest.raises(TypeError):
        mod(proto.double(), coef, boxes)
    assert torch.equal(mod(proto, coef, boxes), want)


def test_lstm_rejects_buffers_that_do_not_fit(fb):
    x, w_ih, w_hh, b_ih, b_hh = W.make_lstm_inputs(2, 3, 256)
    mod = fb.workloads.LSTM(w_ih, w_hh, b_ih, b_hh)
    # an input of another depth is refused, and the buffers allocated for it do not serve the next call
    with pytest.raises(ValueError):
        mod(x[..., :8])
    hs, cs = mod(x)
    want = W.LSTMSeq(w_ih, w_hh, b_ih, b_hh)(x)
    close(hs.cpu(), want[0], rtol=1e-5, scale=1.0, what="hs")
    native = fb.workloads._native()._lstm_forward
    ok = [x.cuda(), mod.w_ih, mod.w_hh, mod.b_ih, mod.b_hh, hs, cs, mod._scratch, mod._status, 0, True]
    assert native(*ok) == 0
    for at, other in [(0, x[0].cuda()), (1, mod.w_ih.transpose(1, 2)), (1, mod.w_ih.double()), (2, mod.w_hh[:3]), (3, mod.b_ih[:, :255]),
                      (5, hs[:1]), (6, cs[..., :255]), (7, mod._scratch[:-256]), (8, torch.zeros(1, dtype=torch.int32)),
                      (8, torch.zeros(1, dtype=torch.int32, device="cuda")), (1, mod.w_ih.cpu())]:
        args = list(ok)
        args[at] = other
        with pytest.raises(ValueError):
            native(*args)
