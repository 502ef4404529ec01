"""ReSTIR PT's two ways to run its paths, one thread per path (views that
render alone, up to 2^17 pixels) and wavefront rounds (larger frames, views
side by side), against each other: the same view rendered alone and in a
batch of two, byte for byte, at the sizes on either side of the line, at the
smallest frame, and with paths longer than the wavefront's rounds."""
import numpy as np
import pytest

KEYS = ("di", "previous_reservoir", "output_path_reservoir", "temporal_path_reservoir", "indirect_color")


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,depth,hybrid", [(512, 256, 4, 0), (513, 256, 4, 2), (1, 1, 3, 0), (33, 17, 12, 2),
                                                      (120, 90, 12, 0)])
def test_alone_matches_side_by_side(width, height, depth, hybrid):
    import torch
    from cases import build_case
    from cube_tracing import views
    from cube_tracing.frame import Renderer
    sc, _, _, _, _ = build_case("room16_deep_pt")
    view = {"scene": 0, "width": width, "height": height, "eye": np.array([7.5, 8.5, 3.5]),
            "target": np.array([8.0, 6.0, 14.0]), "step": np.array([0.05, 0.0, 0.0])}
    kw = {"indirect": True, "max_depth": depth, "params": {"pt_shift_mapping": hybrid}}
    mv = views.MultiViewRenderer([sc], [view, dict(view)], **kw)
    mv.set_schedule(lanes=2)
    alone = Renderer(sc, width, height, **kw)
    for f in range(3):
        cam = views.view_cameras(view, f)
        image = alone.render(*cam)
        mv.render([cam, cam], graph=False)
        for r in mv.r:
            assert torch.equal(r.images[f % 2], image)
            for key in KEYS:
                assert torch.equal(r.buf[key], alone.buf[key]), key
    assert alone.device_error() == (0, 0, 0)
