"""INSTANCE ranges of primitives that do not lie in the AABB table.  On the
CPU: the rule the structure build reads them by (cube-tracing_b200/csrc/
ct_range.h) against 64-bit sums, with counts and firsts up to 2^32 - 1, and the
strided loop over its result.  On the GPU: ct_build_accel refuses tables a few
entries too long, before and after builds that it accepts."""
import os
import subprocess

import numpy as np
import pytest

from cube_tracing import layouts as L
from cube_tracing import native, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include "ct_range.h"
int main() {
  const uint32_t v[] = {0u, 1u, 2u, 255u, 256u, 1000u, (1u << 27) - 1u, 1u << 27, 0x7FFFFFFFu, 0x80000000u,
                        0xFFFFFFFFu - (1u << 27), 0xFFFFFF00u, 0xFFFFFFFEu, 0xFFFFFFFFu};
  const uint32_t n_max = 1u << 27;  // CT_MAX_PRIMITIVES
  for (uint32_t n : v) {
    if (n > n_max) continue;
    for (uint32_t first : v)
      for (uint32_t count : v) {
        const bool outside = (uint64_t)first + count > n;
        const uint32_t in = ct_range_inside(first, count, n);
        if (ct_range_outside(first, count, n) != outside) return printf("outside %u %u %u\n", first, count, n);
        if (outside ? in > count : in != count) return printf("inside %u %u %u\n", first, count, n);
        if (in && (uint64_t)first + in > n) return printf("past the end %u %u %u\n", first, count, n);
        // the kernels' loop from its last thread, with the largest stride
        const uint32_t stride = 1u << 24;
        uint32_t turns = 0;
        for (uint32_t k = stride - 1u; k < in; k += stride)
          if (++turns > n_max / stride) return printf("endless %u %u %u\n", first, count, n);
      }
  }
  return 0;
}
"""


def test_range_rule(tmp_path):
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "cube-tracing_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_build_refuses_ranges_outside_the_table():
    import torch
    from cube_tracing.frame import Accel
    sc = scenes.random_grid_scene(8, 0.5, seed=2)
    n = sc.voxel_count
    aabbs = torch.from_numpy(sc.aabbs.view(np.uint8).reshape(-1).copy()).cuda()

    def build(ranges):
        inst = np.repeat(sc.instances, len(ranges))
        for i, (first, count) in enumerate(ranges):
            inst["first_primitive_index"][i], inst["primitive_count"][i] = first, count
        return Accel(torch.from_numpy(inst.view(np.uint8).reshape(-1).copy()).cuda(), len(ranges), aabbs, n,
                     sc.voxel_extent)

    for ranges in ([(0, n)], [(0, n - 3), (n - 3, 3)], [(n, 0), (0, n)]):
        build(ranges).free()
        for bad in ((0, n + 1), (n - 2, 3), (n, 1), (n + 1, 0), (n + 5, 7)):
            for where in (0, len(ranges)):
                with pytest.raises(native.CtError, match="CT_ERR_INVALID_ARG"):
                    build(ranges[:where] + [bad] + ranges[where:])
    a = build([(0, n)])
    assert a.info().voxel_count == n
    a.free()
