"""Parity of the CUDA path with the oracle's committed frames (tests/golden,
which the oracle reproduces byte for byte): the bar of test_gpu_parity.py
where the oracle library cannot be built."""
import os

import numpy as np
import pytest

from cases import CASES, PT_CASES, build_case, frame_keys
from cube_tracing import layouts as L

HERE = os.path.dirname(os.path.abspath(__file__))


def golden_problems(name, renderer, cams):
    """Renders the case's frames and lists where they leave the fixture."""
    from test_gpu_parity import compare_frame, gpu_frame
    keys = frame_keys(name)
    problems = []
    with np.load(os.path.join(HERE, "golden", f"{name}.npz")) as golden:
        for f, (iv, ip) in enumerate(cams):
            got = gpu_frame(renderer, renderer.render(iv, ip), keys)
            want = {k: L.view_buffer(k, golden[f"f{f}_{k}"].reshape(-1)) for k in keys}
            want["image"] = golden[f"f{f}_image"]
            problems += compare_frame(f"{name} frame {f}", renderer.W, got, want)
    return problems


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES + PT_CASES)
def test_gpu_matches_golden(name):
    from cube_tracing.frame import Renderer
    sc, W, H, cams, kw = build_case(name)
    gpu = Renderer(sc, W, H, **kw)
    problems = golden_problems(name, gpu, cams)
    assert gpu.device_error() == (0, 0, 0)
    assert not problems, "\n".join(problems)
