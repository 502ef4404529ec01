"""A frame whose launch the driver refuses (more walker blocks than a grid may
have) is reported by that call alone: the next calls of the library succeed,
and so does the frame itself once the parameter is back in range."""
import pytest


@pytest.mark.gpu
def test_refused_launch_is_reported_once():
    import torch
    from cases import build_case
    from cube_tracing import layouts as L
    from cube_tracing import native
    from cube_tracing.frame import Accel, Renderer
    sc, W, H, cams, _ = build_case("room16_deep_pt")
    r = Renderer(sc, W, H, indirect=True)
    want = Renderer(sc, W, H, indirect=True).render(*cams[0])
    q = torch.zeros((64, L.RAY_QUERY.itemsize // 4), device="cuda")
    q[:, 0:3], q[:, 3], q[:, 6] = 7.5, 100.0, 1.0
    out = torch.zeros((64, 4), dtype=torch.int32, device="cuda")
    lib, s = native.lib(), torch.cuda.current_stream().cuda_stream

    def closest():
        return lib.ct_trace_closest(r.sb.accel.handle, q.data_ptr(), 64, out.data_ptr(), s)

    def visibility():
        return lib.ct_trace_visibility(r.sb.accel.handle, q.data_ptr(), 64, out.data_ptr(), s)

    def build():
        Accel(r.sb.instances, r.sb.n_instances, r.sb.aabbs, r.sb.n_primitives, sc.voxel_extent).free()
        return native.CT_OK

    for call in (closest, visibility, build):  # each as the first after a refusal
        r.params.walker_blocks = 0xFFFFFFFF
        with pytest.raises(native.CtError, match="CT_ERR_CUDA"):
            r.render(*cams[0])
        r.params.walker_blocks = 0
        assert call() == native.CT_OK
    assert torch.equal(r.render(*cams[0]), want)
    torch.cuda.synchronize()
