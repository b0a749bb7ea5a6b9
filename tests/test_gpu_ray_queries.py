"""Explicit closest-hit queries by ray count: one ray, warps of partial shares,
both sides of where a warp's share grows, many; alternating small and large
calls on one context, whose buffers come from the scratch that builds use too.

Ids and distances equal the oracle's bit for bit."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0, 8], ids=["quads", "wide"])
def test_any_count_of_rays_equals_the_oracle(rtg_lib, oracle_lib, width):
    import torch
    from rti_gb300 import Engine
    warps = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    t = scenes.trench_discs(domain=1.2, width=0.4, depth=1.0)
    s = oracle_lib.Scene(t.xyzr, t.normals)
    rng = np.random.default_rng(0)
    lo, hi = np.array(t.box_lo), np.array(t.box_hi)
    n = 32 * warps + 5
    rays = np.concatenate([lo + (hi - lo) * rng.random((n, 3)), rng.normal(size=(n, 3))], 1).astype(np.float32)
    rays[::7, 3:5] = 0.0  # axis-parallel
    pc, tc = s.closest_hit(rays)
    with Engine(0) as e:
        e.set_node_width(width)
        e.upload_discs(t.points, t.normals, t.radii)
        for k in (1, n, 31, 33, warps, warps + 1, 5 * warps - 3, 2, 32 * warps, n):
            pg, tg = e.trace_rays(rays[:k])
            assert np.array_equal(pg, pc[:k]) and np.array_equal(tg.view(np.uint32), tc[:k].view(np.uint32)), k
            if k == 33:  # a build in between takes the scratch
                e.update_discs(t.points, t.normals, t.radii)
        assert len(e.trace_rays(rays[:0])[0]) == 0
