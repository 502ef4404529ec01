"""The gradients of samples spread over a warp's lanes, voxel by voxel: against
one sample at a time, summed in 64 bits, within the rounding of a float32 sum of
as many terms as that voxel has, so that a term left out or added twice shows."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [3, 5, 8, 32, 70])
def test_gradients_per_voxel(spp):
    import torch
    from cube_tracing import adjoint
    a = adjoint.adjoint_scene(edge=24, occupancy=0.25, emissive_fraction=0.05, width=37, height=13)
    n = a.albedo_target.shape[0]
    a.emitter_index = np.arange(n, dtype=np.int32)  # every voxel emits, into a row of its own
    a.emission_target = np.ones((n, 3), np.float32)
    depth, seed = 3, 11
    r = adjoint.AdjointRenderer(a, spp=spp, max_depth=depth, seed=seed, miss_radiance=0.25)
    g = torch.Generator("cuda").manual_seed(4)
    alb = torch.rand((n, 3), generator=g, device="cuda") * 0.8 + 0.1
    em = torch.rand((n, 3), generator=g, device="cuda") * 9.0 + 1.0
    d_img = torch.rand((13, 37, 3), generator=g, device="cuda") + 0.5
    # vertices per voxel: the emission's gradient where every factor is 1
    ones = torch.ones_like(alb)
    terms = torch.round(r.backward(ones, ones, torch.full_like(d_img, float(spp)))[1][:, 0]).double()
    assert spp < float(terms.max()) < 2 ** 24
    got = r.backward(alb, em, d_img)
    want = [torch.zeros((n, 3), dtype=torch.float64, device="cuda") for _ in range(2)]
    inv = torch.tensor(1.0, device="cuda") / float(spp)
    single = torch.zeros_like(terms)
    for s in range(spp):
        r.seed = seed + s
        single += torch.round(r.backward(ones, ones, torch.ones_like(d_img), spp=1)[1][:, 0]).double()
        for w, v in zip(want, r.backward(alb, em, d_img * inv, spp=1)):
            w += v.double()
    r.close()
    assert torch.equal(single, terms)  # the same vertices
    # all terms are >= 0.  Either side sums `terms` of them in float32; a term
    # is the product of at most depth + 3 factors and sums of as many, each
    # rounded in the same order on both sides except for the pixel's factor
    # (d_img * inv against d_img / spp): two roundings more
    for g_, w in zip(got, want):
        assert bool(((g_.double() - w).abs() <= (2 * terms[:, None] + 4) * 2.0 ** -24 * w).all())
        assert bool((w > 0).any())
