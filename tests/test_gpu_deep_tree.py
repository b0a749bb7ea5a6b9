"""A surface whose clustered tree is so deep and so full of inner siblings that its
four-box nodes would need more than the 256 entries of the largest traversal stack:
nodes of two boxes take their place, in every kind of launch.

Cubes of eight small triangles around the origin, each 1.617 times as large as the
one before, from 3e-7 to 4e15: in the clustered tree every cube opens to three inner
nodes beside the chain of all smaller ones (270 entries at a height of 201).  Three
triangles far away put all others into few cells of the leaf order, where they keep
the order of their ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUBES, FAR = 106, 5e18


def _surface():
    rng = np.random.default_rng(1)
    v = []
    for i in range(CUBES):
        s = 3e-7 * (4e15 / 3e-7) ** (i / CUBES)
        for c in np.array([(x, y, z) for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)]):
            at = c * s * rng.uniform(0.98, 1.0, 3)
            v += [at + rng.uniform(-0.02, 0.02, 3) * s for _ in range(3)]
    v += [[FAR, FAR, FAR], [FAR * 1.01, FAR, FAR], [FAR, FAR * 1.01, FAR]]
    v = np.array(v, np.float32)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


def _rays(v, i, m):
    """Rays from around a triangle's cube through a point of the triangle."""
    rng = np.random.default_rng(2)
    k = rng.integers(0, len(i) - 1, m)
    k[:64] = np.arange(64)  # the innermost cubes
    t = v[i[k]].astype(np.float64)
    at = t.mean(1)
    o = at + rng.normal(size=(m, 3)) * np.abs(at).max(1, keepdims=True) * 10.0 ** rng.uniform(-2, 1, (m, 1))
    d = at - o
    return np.concatenate([o, d / np.linalg.norm(d, axis=1)[:, None]], 1).astype(np.float32)


@pytest.mark.parametrize("width", [2, 8], ids=["four-box", "eight-wide"])
def test_hits_equal_the_oracle(rtg_lib, oracle_lib, width):
    from rti_gb300 import Engine
    from rti_gb300 import _lib as L
    v, i = _surface()
    rays = _rays(v, i, 4000)
    pc, tc = oracle_lib.Scene(None, None, v, i).closest_hit(rays, 0.0)
    assert len(np.unique(pc)) > 400
    with Engine(0) as e:
        e.set_tree_builder(L.RTG_TREE_PLOC)
        e.set_node_width(width)
        e.upload_triangles(v, i)
        assert e.tree_depth > 128  # the clustered tree, not the radix tree in its place
        pg, tg = e.trace_rays(rays, 0.0)
        assert np.array_equal(pg, pc) and np.array_equal(tg.view(np.uint32), tc.view(np.uint32))
        e.update_vertices(v)
        pg, tg = e.trace_rays(rays, 0.0)
        assert np.array_equal(pg, pc) and np.array_equal(tg.view(np.uint32), tc.view(np.uint32))


def test_nodes_hold_two_boxes(rtg_lib):
    """A query for an innermost triangle visits a node a level (223 to 230 of them); of
    nodes of four boxes it would visit 106 to 109."""
    from rti_gb300 import Engine, RtgError
    from rti_gb300 import _lib as L
    v, i = _surface()
    rays = _rays(v, i, 64)
    with Engine(0) as e:
        e.set_tree_builder(L.RTG_TREE_PLOC)
        e.upload_triangles(v, i)
        for limit, reached in ((e.tree_depth - 10, True), (2 * e.tree_depth, False)):
            e.set_visit_limit(limit)
            for k in (0, 5, 20):
                if reached:
                    with pytest.raises(RtgError):
                        e.trace_rays(rays[k:k + 1], 0.0)
                else:
                    assert e.trace_rays(rays[k:k + 1], 0.0)[0][0] == k


def test_traces_do_not_outgrow_their_stacks(rtg_lib):
    """Paths among the cubes up to size 2, in every schedule and stack: no errors, and
    the counts of the radix tree."""
    from rti_gb300 import Engine
    from rti_gb300 import _lib as L
    v, i = _surface()
    box = ((-2.0, -2.0, -2.0), (2.0, 2.0, 2.0))
    out = []
    with Engine(0) as e:
        for builder in (L.RTG_TREE_KARRAS, L.RTG_TREE_PLOC):
            e.set_tree_builder(builder)
            e.upload_triangles(v, i)
            e.configure(box=box, sticking=0.1, x_bound=1, y_bound=1, max_segments=100, reset=True)
            for kw in ({}, {"scheduling": L.RTG_SCHED_PLAIN}, {"scheduling": L.RTG_SCHED_WAVEFRONT},
                       {"stack_memory": L.RTG_STACK_SHARED}, {"threads_per_block": 64}, {"stack_depth": 32}):
                e.set_launch_config(**kw)
                e.trace(200_000, 7)
                t = e.tally()
                assert t.errors == 0 and t.hitc > 100
                out.append((e.hit_counts(), t.segments))
            e.set_launch_config()
    for c in out[1:]:
        assert np.array_equal(c[0], out[0][0]) and c[1] == out[0][1]
