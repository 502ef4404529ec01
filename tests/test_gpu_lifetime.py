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

    warm = build(sc, sb)  # torch's own memory for what the test reads
    warm.field(0, 3)
    warm.free()
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


@pytest.mark.gpu
def test_builds_and_frees_on_several_threads_and_streams():
    """Every structure a thread builds, between other threads' builds and
    frees, has the field of the one built alone."""
    import numpy as np
    import torch
    work = [scene_buffers(edge=e, seed=e) for e in (24, 40, 56, 33)]
    want = [build(*w).field(0, 5)[0] for w in work]
    failures = []

    def run(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                kept = []
                for k in range(12):
                    j = (i + k) % len(work)
                    kept.append((build(*work[j]), j))
                    if k % 3 == i % 3:
                        acc, j = kept.pop(0)
                        if not np.array_equal(acc.field(0, 5)[0], want[j]):
                            failures.append((i, k, j))
                        acc.free()
                for acc, j in kept:
                    if not np.array_equal(acc.field(0, 5)[0], want[j]):
                        failures.append((i, "end", j))
                    acc.free()
        except Exception as e:  # noqa: BLE001
            failures.append(repr(e))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
