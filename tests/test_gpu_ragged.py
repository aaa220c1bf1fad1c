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
    (16, 900, 80, 200, 7.0),      # large room, few rows: packed
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
