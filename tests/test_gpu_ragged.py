"""Ragged results written by the kernels themselves: SSDBBox.__call__ against forward_padded + unpad, and the packed form
that large, sparse results take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,priors,classes,topk,background", [
    (1, 8732, 80, 200, 0.0),      # one image
    (3, 333, 1, 50, 0.0),         # one class: nobody before it
    (2, 700, 95, 200, 0.0),       # the most classes a row may have, three rounds of lanes in the look-back
    (5, 257, 33, 256, 8.0),       # one class more than a warp, many empty lists
    (16, 900, 80, 200, 7.0),      # large room, a third of it filled
    (16, 900, 80, 200, 40.0),     # no row at all
])
def test_ssd_call_equals_padded_and_unpadded(cuda_device, batch, priors, classes, topk, background):
    import functs_b200 as fb
    g = torch.Generator().manual_seed(priors + classes)
    pri = torch.cat([torch.rand(priors, 2, generator=g) * 300, torch.rand(priors, 2, generator=g) * 80 + 4], dim=1)
    loc = torch.randn(batch, priors, 4, generator=g).cuda()
    conf = torch.randn(batch, priors, classes + 1, generator=g) * 2
    conf[..., -1] += background
    conf = conf.cuda()
    mod = fb.workloads.SSDBBox(pri, topk=topk)
    got = mod(loc, conf)
    assert mod.kernels_last_call in (2, 3)
    _, dets, ids, counts = mod.forward_padded(loc, conf)
    want = mod.unpad(dets, ids, counts)
    assert len(got) == batch
    for (d, l), (wd, wl, _) in zip(got, want):
        assert d.is_contiguous() and torch.equal(d, wd) and torch.equal(l, wl)
    again = mod(loc, conf)  # the first call's results are not overwritten
    for (d, l), (d2, l2) in zip(got, again):
        assert torch.equal(d, d2) and torch.equal(l, l2)
        assert d.numel() == 0 or d.data_ptr() != d2.data_ptr()


@pytest.mark.parametrize("background,packed", [(0.0, False), (12.0, True), (40.0, True)])
def test_ssd_program_keeps_or_packs_its_room(cuda_device, background, packed):
    """The lists of a built program are views: of the room they were written into, or, where that is large and less than a quarter
    filled, of memory of their own total size."""
    import functs_b200 as fb
    from functs_b200 import jit, patterns
    batch, priors, classes = 16, 900, 80
    g = torch.Generator().manual_seed(1)
    pri = torch.cat([torch.rand(priors, 2, generator=g) * 300, torch.rand(priors, 2, generator=g) * 80 + 4], dim=1)
    loc = torch.randn(batch, priors, 4, generator=g).cuda()
    conf = torch.randn(batch, priors, classes + 1, generator=g) * 2
    conf[..., -1] += background
    conf = conf.cuda()
    _, _, res = jit.build(patterns.SSDPost(pri))(loc, conf)
    mod = fb.workloads.SSDBBox(pri)
    _, dets, ids, counts = mod.forward_padded(loc, conf)
    total = int(counts.sum())
    assert (total * 4 < batch * classes * 200) == packed
    for (d, l, i), (wd, wl, wi) in zip(res, mod.unpad(dets, ids, counts)):
        assert torch.equal(d, wd) and torch.equal(l, wl) and torch.equal(i, wi)
        assert d.untyped_storage().nbytes() == 20 * (total if packed else batch * classes * 200)


@pytest.mark.parametrize("batch", [1, 65])  # 65: a second launch of the splitting kernel
def test_lists_of_the_modules_own_their_storage(cuda_device, batch):
    """A list that is kept (or saved) keeps its own rows and nothing else, as a copy does."""
    import functs_b200 as fb
    g = torch.Generator().manual_seed(batch)
    maps = [torch.randn(batch, 255, s, s, generator=g).cuda() for s in (4, 8, 16)]
    maps[0][batch // 2, 4::85] = maps[1][batch // 2, 4::85] = maps[2][batch // 2, 4::85] = -20.0  # an image without detections
    pri = torch.cat([torch.rand(900, 2, generator=g) * 300, torch.rand(900, 2, generator=g) * 80 + 4], dim=1)
    loc, conf = torch.randn(batch, 900, 4, generator=g).cuda(), (torch.randn(batch, 900, 21, generator=g) * 2).cuda()
    yolo, ssd = fb.workloads.YOLOV3BBox(sizes=(4, 8, 16)), fb.workloads.SSDBBox(pri)
    got = yolo(maps) + ssd(loc, conf)
    dets, labels, _, counts = yolo.forward_padded(maps)
    want = [(dets[b, :n], labels[b, :n]) for b, n in enumerate(counts.tolist())]
    want += [(d, l) for d, l, _ in ssd.unpad(*ssd.forward_padded(loc, conf)[1:])]
    assert len(got) == len(want) == 2 * batch
    for pair, expected in zip(got, want):
        for t, w in zip(pair, expected):
            assert torch.equal(t, w) and t.untyped_storage().nbytes() == t.numel() * t.element_size()
            assert not t._is_view() and torch.cat([t, t]).size(0) == 2 * t.size(0)
    grown = [t.clone() for t in got[0]]
    for t in got[0]:
        t.resize_(2000, *t.shape[1:])  # (past what lies behind the storage)
    assert all(torch.equal(t[:len(w)], w) for t, w in zip(got[0], grown)) and got[0][0].untyped_storage().nbytes() == 40000
    assert len({t.untyped_storage().data_ptr() for pair in got for t in pair if t.numel()}) == sum(t.numel() > 0 for pair in got for t in pair)


@pytest.mark.parametrize("seq,batch,inputs,hidden", [
    (2, 1, 256, 256), (3, 7, 96, 512),     # one row per cluster, the last batch of that form; K not a power of two
    (3, 8, 80, 256), (2, 14, 512, 512),    # two rows, K not a multiple of the k-tile
    (2, 15, 63, 256), (3, 28, 512, 512),   # four rows; K not a multiple of four
    (2, 42, 256, 512), (2, 56, 128, 256), (3, 61, 512, 512),  # six, eight, ten rows, ragged last cluster
    (1, 150, 64, 256),                     # more clusters than run at once
    (40, 33, 512, 512),                    # operands split by a launch of their own, ragged rows
])
def test_lstm_rows_per_cluster_and_ragged_projection(cuda_device, seq, batch, inputs, hidden):
    import functs_b200 as fb
    from oracle import workloads as W
    g = torch.Generator().manual_seed(seq * 1000 + batch)
    bound = hidden ** -0.5
    w = [(torch.rand(*s, generator=g) * 2 - 1) * bound for s in ((4, inputs, hidden), (4, hidden, hidden), (4, 1, hidden), (4, 1, hidden))]
    x = torch.randn(seq, batch, inputs, generator=g)
    hs64, cs64 = W.LSTMSeq(*[t.double() for t in w])(x.double())
    hs, cs = fb.workloads.LSTM(*w)(x)
    assert float((hs.cpu().double() - hs64).abs().max()) < 3e-6
    assert float((cs.cpu().double() - cs64).abs().max()) < 3e-6
