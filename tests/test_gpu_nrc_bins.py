"""The fused network encodes as ct_nrc_encode does, bit for bit, in the
one-blob bins below the smallest normal number too: weights that scale them up
bring them to the output."""
import math

import pytest


@pytest.mark.gpu
def test_fused_network_keeps_subnormal_bins():
    import torch
    from cube_tracing import nrc
    cache = nrc.NrcCache((0.0, 0.0, 0.0), (256.0, 128.0, 256.0))
    # rgb = the direction's first bin: 2^100, then 2^30, along the first unit
    # of every layer, all else 0
    w, at = cache.weights.zero_(), 0
    for i, (rows, cols) in enumerate([(64, 256)] + [(64, 64)] * 4 + [(16, 64)]):
        m = w[at:at + rows * cols].view(rows, cols)
        m[0, 96 if i == 0 else 0] = 2.0 ** 100 if i == 0 else (2.0 ** 30 if i == 5 else 1.0)
        at += rows * cols
    # azimuths 32u from 11.5 to 15.5: bins 2^-87 to 2^-162
    n = 1001
    q = nrc.random_queries(n, seed=2)
    a = (torch.linspace(11.5, 15.5, n, device="cuda", dtype=torch.float64) / 32.0 - 0.5) * (2.0 * math.pi)
    q[:, 3], q[:, 4], q[:, 5] = torch.cos(a).float(), 0.0, torch.sin(a).float()
    enc = cache.encode_device(q)
    bins = enc[:, 96].double()
    below = (bins > 0) & (bins < 2.0 ** -126)
    assert int(below.sum()) > 50
    want, got = cache.infer_encoded(enc), cache.infer(q)
    # one product a layer, so the value itself
    assert torch.equal(want[:, 0].double(), bins * 2.0 ** 130)
    assert torch.equal(got, want)
