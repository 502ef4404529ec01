"""Ray batches on either side of what the GPU holds at once, against the same
rays asked in small batches (which the walk tests check against brute force),
byte for byte: ct_trace_closest changes kernels there and ct_trace_visibility
starts to refill its lanes.  And a scene split into instances against the
whole."""
import numpy as np
import pytest

import rays
from cube_tracing import layouts as L
from cube_tracing import scenes
from test_gpu_traversal import gpu_queries

SMALL = 4096


def in_parts(accel, q, closest):
    return np.concatenate([gpu_queries(accel, q[i:i + SMALL], closest) for i in range(0, len(q), SMALL)])


def resident(closest):
    """Rays of a batch that gives every resident warp 32 (256 threads a block,
    3 or 4 blocks an SM)."""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * (3 if closest else 4) * 256


@pytest.mark.gpu
@pytest.mark.parametrize("closest", [True, False])
@pytest.mark.parametrize("instances", [1, 3])
def test_large_batches_match_small_ones(closest, instances):
    import cases
    from cube_tracing.frame import SceneBuffers
    sc = scenes.random_grid_scene(40, 0.2, seed=3)
    if instances > 1:
        sc = cases.split_into_instances(sc, [12, 25], [cases.rotation((0, 1, 0), a) for a in (0.0, 0.2, -0.3)],
                                        [(0, 0, 0), (1.5, 0, 0.25), (3.0, -1.0, 0)])
    sb = SceneBuffers(sc)
    full = resident(closest)
    n_max = 2 * full + 77
    make = [rays.camera_rays, rays.random_segments, rays.degenerate_rays] if closest else \
        [rays.shadow_rays, rays.random_segments, rays.degenerate_rays]
    q = np.concatenate([f(sc, n_max // 3 + 1, seed=i) for i, f in enumerate(make)])
    q = q[np.random.default_rng(1).permutation(len(q))][:n_max]
    want = in_parts(sb.accel, q, closest)
    hit = want["instance_id"] < L.MAX_INSTANCES if closest else want != 0
    assert 0.05 < hit.mean() < 0.95
    for n in (full - 1, full, full + 1, full + 33, n_max):
        assert np.array_equal(gpu_queries(sb.accel, q[:n], closest), want[:n]), n


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 257, 5000, 130001])
def test_instances_match_the_whole_scene(n):
    """The same voxels as one instance and as four untransformed ones."""
    import cases
    from cube_tracing.frame import SceneBuffers
    sc = scenes.random_grid_scene(32, 0.25, seed=8)
    parts = cases.split_into_instances(scenes.random_grid_scene(32, 0.25, seed=8), [8, 9, 20],
                                       [np.eye(3, dtype=np.float32)] * 4, [(0, 0, 0)] * 4)
    # the whole scene in the parts' primitive order
    sc.aabbs, sc.primitives = parts.aabbs, parts.primitives
    whole, split = SceneBuffers(sc), SceneBuffers(parts)
    first = parts.instances["first_primitive_index"]
    q = np.concatenate([f(sc, n // 2 + 1, seed=n) for f in (rays.random_segments, rays.degenerate_rays)])[:n]
    a, b = gpu_queries(whole.accel, q, True), gpu_queries(split.accel, q, True)
    hit = a["instance_id"] == 0
    assert np.array_equal(b["instance_id"] < 4, hit) and np.array_equal(a["t"], b["t"])
    assert np.array_equal(first[b["instance_id"][hit]] + b["primitive_id"][hit], a["primitive_id"][hit])
    # half of the rays with a target voxel
    target = np.random.default_rng(n).integers(0, sc.voxel_count, n)
    inst = np.searchsorted(first, target, side="right") - 1
    qa, qb = q.copy(), q.copy()
    for r, i, p in ((qa, 0, target), (qb, inst, target - first[inst])):
        r["flags"] = (np.arange(n) % 2) * L.QUERY_CHECK_TARGET
        r["target_instance"], r["target_primitive"] = i, p
    assert np.array_equal(gpu_queries(whole.accel, qa, False), gpu_queries(split.accel, qb, False))


@pytest.mark.gpu
@pytest.mark.parametrize("extent", [1.0, 0.3])
def test_build_from_unaligned_boxes(extent):
    """AABBs that are 4 but not 8 bytes aligned: the same structure."""
    import torch
    from cube_tracing.frame import Accel
    sc = scenes.random_grid_scene(24, 0.2, seed=5, voxel_extent=extent)
    raw = torch.from_numpy(np.ascontiguousarray(sc.aabbs).view(np.uint8).reshape(-1).copy()).cuda()
    inst = torch.from_numpy(sc.instances.view(np.uint8).reshape(-1).copy()).cuda()
    moved = torch.zeros(raw.numel() + 4, dtype=torch.uint8, device="cuda")
    moved[4:] = raw
    assert raw.data_ptr() % 8 == 0 and moved[4:].data_ptr() % 8 == 4
    a, b = (Accel(inst, 1, t, sc.voxel_count, extent) for t in (raw, moved[4:]))
    ia, ib = a.info(), b.info()
    for f, _ in ia._fields_:
        va, vb = getattr(ia, f), getattr(ib, f)
        assert (list(va) == list(vb)) if hasattr(va, "__len__") else va == vb, f
    for octant in range(8):
        assert np.array_equal(a.field(0, octant)[0], b.field(0, octant)[0])
    q = rays.random_segments(sc, 3000, seed=2)
    assert np.array_equal(gpu_queries(a, q, True), gpu_queries(b, q, True))
