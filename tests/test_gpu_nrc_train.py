"""The radiance cache's training kernels against the torch expressions they
stand for, bit for bit: the single-precision encoding (ct_nrc_encode_f32)
against encode(), and train_step with the loss and its gradient in one kernel
(ct_nrc_loss) against the same step written in torch."""
import pytest

from cube_tracing import nrc

BOX = ((0.0, -3.0, 0.5), (256.0, 128.0, 250.7))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 257, 5000])
def test_encoding_matches_torch(n):
    import torch
    cache = nrc.NrcCache(*BOX, seed=1)
    q = nrc.random_queries(n, seed=n, bbox_min=BOX[0], bbox_extent=BOX[1])
    # outside the box, axis directions, zero vectors, infinities and NaN
    for i, v in enumerate((1e9, -1e9, float("inf"), float("nan"))):
        q[i::37, :3] = v
    q[5::41, 3:9] = torch.randint(-1, 2, q[5::41, 3:9].shape, device="cuda").float()
    want, got = nrc.encode(q, *BOX), cache._encode_fp32(q)
    same = (want.view(torch.int32) == got.view(torch.int32)) | (want.isnan() & got.isnan())
    assert bool(same.all())


def torch_step(self, queries, targets, weights):
    pred = self.mlp(nrc.encode(queries, self.bbox_min, self.bbox_extent))[:, :3]
    rel = ((pred - targets) ** 2) / (pred.detach() ** 2 + 1e-2)
    loss = (rel * weights[:, None]).sum() / (3.0 * weights.sum()).clamp(min=1.0)
    self.opt.zero_grad()
    loss.backward()
    self.opt.step()
    self.export()
    return loss.detach()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 63, 4096])
def test_train_step_matches_torch(n):
    import torch
    a, b = nrc.NrcCache(*BOX, seed=4), nrc.NrcCache(*BOX, seed=4)
    for k in range(3):
        q = nrc.random_queries(n, seed=k, bbox_min=BOX[0], bbox_extent=BOX[1])
        g = torch.Generator("cuda").manual_seed(k)
        t = torch.rand((n, 3), generator=g, device="cuda") * 5.0
        w = (torch.rand(n, generator=g, device="cuda") > 0.4).float() * (k != 1)  # step 1: no row counts
        assert torch.equal(a.train_step(q, t, weights=w), torch_step(b, q, t, w))
        for x, y in zip(a.mlp.weights, b.mlp.weights):
            assert torch.equal(x, y)
        assert torch.equal(a.weights, b.weights)
