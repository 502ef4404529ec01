"""The radiance cache made and used with gradients off, as a program that only
renders with it does, and training steps whose inputs the library's kernels do
not take."""
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
