"""The radiance cache made and used with gradients off, as a program that only
renders with it does, and training steps whose inputs the library's kernels do
not take."""
import itertools
import types

import pytest
import torch

from cube_tracing import nrc

BOX = ((0.0, -3.0, 0.5), (256.0, 128.0, 250.7))


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode, torch.enable_grad])
def test_autograd_starts_in_any_mode(mode):
    with mode():
        nrc._start_autograd("cpu")
        assert torch.is_inference_mode_enabled() == (mode is torch.inference_mode)
        assert torch.is_grad_enabled() == (mode is torch.enable_grad)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_cache_without_gradients(mode):
    q = nrc.random_queries(300, seed=1, bbox_min=BOX[0], bbox_extent=BOX[1])
    want = nrc.NrcCache(*BOX, seed=3).infer(q)
    with mode():
        assert torch.equal(nrc.NrcCache(*BOX, seed=3).infer(q), want)


def row(device="cuda:0", dtype=torch.float32, requires_grad=False):
    return types.SimpleNamespace(device=torch.device(device), dtype=dtype, requires_grad=requires_grad)


@pytest.fixture
def current_device(monkeypatch):
    """Makes device 0 current, on a machine without one too."""
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)


def test_kernels_take_rows_of_the_caches_device_alone(current_device):
    here = torch.device("cuda:0")
    assert nrc._kernel_rows(here, [row(), row(), row()])
    others = [row("cuda:1"), row("cpu"), row("meta"), row(dtype=torch.float64), row(requires_grad=True)]
    for odd, at in itertools.product(others, range(3)):
        rows = [row(), row(), row()]
        rows[at] = odd
        assert not nrc._kernel_rows(here, rows)
    # the kernels are launched on the current device: a cache on another one,
    # whose rows lie there too, trains by the torch expressions
    assert not nrc._kernel_rows(torch.device("cuda:1"), [row("cuda:1")] * 3)
    assert not nrc._kernel_rows(torch.device("cpu"), [row("cpu")] * 3)


def test_one_target_for_all_rows(current_device):
    """A number, or a tensor that broadcasts, as every row's target."""
    q = nrc.random_queries(9, seed=2, device="cpu", bbox_min=BOX[0], bbox_extent=BOX[1])
    full = torch.full((9, 3), 0.75)
    losses = [nrc.NrcCache(*BOX, device="cpu", seed=1).train_step(q, t) for t in (full, 0.75, full[:1], full[0, 0])]
    assert all(torch.equal(v, losses[0]) for v in losses)
    assert not nrc._kernel_rows(torch.device("cuda:0"), [row(), 0.75])


@pytest.mark.gpu
@pytest.mark.parametrize("extent", [(-256.0, 128.0, 250.0), (256.0, float("inf"), 250.0), (1e39, 128.0, 250.0)])
@pytest.mark.parametrize("weighted", [True, False])
def test_training_in_a_box_the_library_refuses(extent, weighted):
    """Mirrored and unbounded boxes train by the torch expressions, on the GPU
    as on the CPU."""
    caches = [nrc.NrcCache(BOX[0], extent, device=d, seed=5) for d in ("cuda", "cpu")]
    assert not caches[0]._box_in_range() and nrc.NrcCache(*BOX, device="cpu")._box_in_range()
    q = nrc.random_queries(65, seed=3, bbox_min=BOX[0], bbox_extent=BOX[1])
    rows = [q, torch.rand((65, 3), device="cuda")] + ([torch.ones(65, device="cuda")] if weighted else [])
    gpu, cpu = [c.train_step(*[t.to(c.weights.device) for t in rows]) for c in caches]
    # the networks differ by the order of fp32 sums of 256 and 64 products
    assert torch.isfinite(gpu) and abs(float(gpu) - float(cpu)) <= 1e-3 * float(cpu)


@pytest.mark.gpu
def test_gradient_of_a_transposed_output():
    """A network whose output's storage is column by column: the loss kernel's
    gradient is the torch expressions'."""
    from test_gpu_nrc_train import torch_step
    q = nrc.random_queries(65, seed=3, bbox_min=BOX[0], bbox_extent=BOX[1])
    t, w = torch.rand((65, 3), device="cuda") * 5.0, torch.ones(65, device="cuda")
    grads = []
    for step in (nrc.NrcCache.train_step, torch_step):
        cache = nrc.NrcCache(*BOX, seed=6)
        forward = cache.mlp.forward
        cache.mlp.forward = lambda enc: forward(enc).t().contiguous().t()
        assert cache.mlp(torch.zeros((65, nrc.IN), device="cuda")).stride() == (1, 65)
        step(cache, q, t, w)
        grads.append([p.grad for p in cache.mlp.weights])
    # sums of up to 256 fp32 products a layer, in another order
    for a, b in zip(*grads):
        assert bool((a - b).abs().max() <= 1e-4 * b.abs().max()) and bool(b.abs().max() > 0)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 257])
def test_unweighted_step_matches_torch(n):
    """Without weights the encoding is the kernel's and the loss torch's: bit
    for bit the step written in torch."""
    a, b = nrc.NrcCache(*BOX, seed=4), nrc.NrcCache(*BOX, seed=4)
    for k in range(3):
        q = nrc.random_queries(n, seed=k, bbox_min=BOX[0], bbox_extent=BOX[1])
        t = torch.rand((n, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(k)) * 5.0
        pred = b.mlp(nrc.encode(q, b.bbox_min, b.bbox_extent))[:, :3]
        loss = (((pred - t) ** 2) / (pred.detach() ** 2 + 1e-2)).mean()
        b.opt.zero_grad()
        loss.backward()
        b.opt.step()
        b.export()
        assert torch.equal(a.train_step(q, t), loss.detach())
        for x, y in zip(a.mlp.weights, b.mlp.weights):
            assert torch.equal(x, y)
        assert torch.equal(a.weights, b.weights)
