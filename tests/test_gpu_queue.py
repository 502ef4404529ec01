"""The light-sample queue of paths finished by one thread each, filled past its
capacity: a closed, wholly Lambertian room lit by a point light, one spatial
neighbour (3 queued rays per pixel) and paths of up to 12 bounces.  The rays
that find no room are walked in place; the walker behind must neither read nor
answer past the queue's end."""
import ctypes

import numpy as np
import pytest

from cube_tracing import layouts as L
from cube_tracing import native, scenes

W, H, DEPTH = 40, 30, 12
PARAMS = {"min_num_of_neighbors": 1, "max_num_of_neighbors": 1}
# a ray's record read as an answer slot may name a byte this far behind the
# answers: a point light's primitive id, CT_MAX_PRIMITIVES
TAIL = L.MAX_PRIMITIVES + (16 << 20)
KEYS = ("di", "previous_reservoir", "output_path_reservoir", "temporal_path_reservoir", "indirect_color")


def room(edge=12):
    g = np.arange(edge)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    wall = (x == 0) | (y == 0) | (z == 0) | (x == edge - 1) | (y == edge - 1) | (z == edge - 1)
    coords = np.argwhere(wall)[:, ::-1].astype(np.int32)
    emits = np.zeros(len(coords), bool)
    emits[0] = True
    sc = scenes._build(coords, emits, np.full((1, 3), 0.7, np.float32), np.zeros(len(coords), np.uint32),
                       np.ones((1, 3), np.float32), 1.0, (edge,) * 3, "lambertian_room", {})
    pl = np.zeros(1, L.LIGHT)
    pl["position"] = (edge * 0.5, edge * 0.6, edge * 0.5)
    pl["emissive"] = (30.0,) * 3
    pl["instance_id"], pl["primitive_id"], pl["type"] = L.MAX_INSTANCES, L.MAX_PRIMITIVES, L.LIGHT_POINT
    sc.point_lights = pl
    sc.light_config["point_light_count"] = 1
    return sc


def renderer(sc, **kw):
    """A renderer whose scratch is followed by TAIL bytes of a pattern."""
    import torch
    from cube_tracing.frame import Renderer
    r = Renderer(sc, W, H, params=dict(PARAMS), max_depth=DEPTH, **kw)
    need = ctypes.c_uint64()
    native.check("ct_workspace_size", native.lib().ct_workspace_size(W, H, ctypes.byref(r.params), ctypes.byref(need)))
    r.workspace = torch.full((need.value + 256 + TAIL,), 0x5A, dtype=torch.uint8, device="cuda")
    r.params.workspace_address = (r.workspace.data_ptr() + 255) // 256 * 256
    r.tail = r.workspace[r.params.workspace_address - r.workspace.data_ptr() + need.value:]
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("count_rays", [True, False])
def test_full_light_sample_queue(count_rays):
    import torch
    from cube_tracing import views
    sc = room()
    view = {"scene": 0, "width": W, "height": H, "eye": np.array([4.5, 5.5, 2.5]), "target": np.array([7.0, 5.0, 9.0]),
            "step": np.array([0.05, 0.0, 0.0])}
    alone = renderer(sc, indirect=True, count_rays=count_rays)
    # the same frames in wavefront rounds
    mv = views.MultiViewRenderer([sc], [view, dict(view)], indirect=True, max_depth=DEPTH, params=dict(PARAMS))
    mv.set_schedule(lanes=2)
    for f in range(3):
        cam = views.view_cameras(view, f)
        image = alone.render(*cam)
        mv.render([cam, cam], graph=False)
        if count_rays and f == 0:
            direct = renderer(sc, count_rays=True)
            direct.render(*cam)
            # path reuse traces at most 3 rays per pixel itself
            asked = alone.ray_counts()["shadow"] - direct.ray_counts()["shadow"] - 3 * W * H
            assert asked > 3 * W * H, asked  # more than the queue holds
        for r in mv.r:
            assert torch.equal(r.images[f % 2], image)
            for key in KEYS:
                assert torch.equal(r.buf[key], alone.buf[key]), key
    assert bool((alone.tail == 0x5A).all())
    assert alone.device_error() == (0, 0, 0)
