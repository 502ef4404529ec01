"""Structures freed while other work goes on: the free waits for work in flight
on any stream, and leaves the captures of other threads (and relaxed ones of
its own) alone, as cudaFree does.  Builds and frees from several threads and
streams share one pool of device memory."""
import threading

import pytest


def scene_buffers(edge=16, seed=1):
    from cube_tracing import scenes
    from cube_tracing.frame import SceneBuffers
    sc = scenes.random_grid_scene(edge, 0.3, seed=seed)
    return sc, SceneBuffers(sc)


def build(sc, sb):
    from cube_tracing.frame import Accel
    return Accel(sb.instances, sb.n_instances, sb.aabbs, sb.n_primitives, sc.voxel_extent)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,thread", [("thread_local", True), ("relaxed", True), ("relaxed", False)])
def test_free_leaves_captures_alone(mode, thread):
    import torch
    sc, sb = scene_buffers()
    acc = build(sc, sb)
    x = torch.arange(1024.0, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        g.capture_begin(capture_error_mode=mode)
        y.copy_(x * 2)
        if thread:
            t = threading.Thread(target=acc.free)
            t.start()
            t.join()
        else:
            acc.free()
        y.add_(1.0)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2 * x + 1)


@pytest.mark.gpu
def test_free_waits_for_work_on_any_stream():
    import torch
    sc, sb = scene_buffers()
    acc = build(sc, sb)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(50_000_000)  # some 25 ms
        done.record()
    assert not done.query()
    acc.free()
    assert done.query()
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_release_memory():
    """The pool's unused memory goes back to the driver; live structures stay."""
    import gc

    import torch
    from cube_tracing import native
    gc.collect()
    sc, sb = scene_buffers(edge=96)  # a cell field of over 4 MB, brick tables of 30
    release = native.lib().ct_release_memory

    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    assert release() == native.CT_OK
    before = free_bytes()
    accs = [build(sc, sb) for _ in range(4)]
    held = before - free_bytes()
    assert held >= 4 * 8 << 20
    field = [a.field(0, 3)[0] for a in accs[:1]]
    for a in accs[1:]:
        a.free()
    assert release() == native.CT_OK
    assert before - free_bytes() <= held // 2  # three of four
    assert (accs[0].field(0, 3)[0] == field[0]).all()
    accs[0].free()
    assert release() == native.CT_OK
    assert abs(before - free_bytes()) <= 4 << 20
    build(sc, sb).free()
