"""ReSTIR PT's two ways to run its paths, one thread per path (views that
render alone, up to 2^17 pixels) and wavefront rounds (larger frames, views
side by side), against each other: the same view rendered alone and in a
batch of two, byte for byte, at the sizes on either side of the line, at the
smallest frame, and with paths longer than the wavefront's rounds.
Below it, the path tracer's samples over a warp's lanes against one sample at
a time."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [2, 3, 5, 7, 8, 11, 17, 25, 32, 33, 70])
@pytest.mark.parametrize("rect", [None, (3, 2, 34, 9)])
def test_samples_over_lanes(spp, rect):
    """A pixel's samples over neighbouring lanes: the image of spp samples is,
    bit for bit, the float32 sum in sample order of the images of one sample
    (one lane per pixel) with seeds seed, seed + 1, ..., and its gradients are
    the sum of theirs to the rounding of a float32 sum of as many terms."""
    import torch

    from cube_tracing import adjoint
    a = adjoint.adjoint_scene(edge=32, occupancy=0.25, emissive_fraction=0.05, width=37, height=13)
    alb = torch.from_numpy(a.albedo_target).cuda()
    em = torch.from_numpy(a.emission_target).cuda()
    depth, seed = 3, 11
    r = adjoint.AdjointRenderer(a, spp=spp, max_depth=depth, seed=seed, miss_radiance=0.25)
    got = r.forward(alb, em, rect=rect)
    d_img = torch.rand((13, 37, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(4)) + 0.5
    got_a, got_e = r.backward(alb, em, d_img, rect=rect)
    total = torch.zeros_like(got)
    want_a, want_e = torch.zeros_like(got_a, dtype=torch.float64), torch.zeros_like(got_e, dtype=torch.float64)
    inv = torch.tensor(1.0, device="cuda") / float(spp)
    for s in range(spp):
        r.seed = seed + s
        total += r.forward(alb, em, rect=rect, spp=1)
        ga, ge = r.backward(alb, em, d_img * inv, rect=rect, spp=1)
        want_a += ga.double()
        want_e += ge.double()
    r.close()
    assert torch.equal(got, total * inv) and bool((got > 0).any())
    # all terms are >= 0: the relative error of a sum of n of them is at most
    # n 2^-24, on either side
    n = 37 * 13 * spp * depth
    for g, w in ((got_a, want_a), (got_e, want_e)):
        assert bool(((g.double() - w).abs() <= 2 * n * 2.0 ** -24 * w).all()) and bool((w > 0).any())
