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
