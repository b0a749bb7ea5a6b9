"""The four-box nodes that closest hits visit (QuadNode): trees of few
primitives (one to a little over two full levels, so that every fill of a node
occurs), chains and stacks of equal boxes, rays that start on flat faces, and
the near clip at tnear.

A box may be met without a hit in it, never missed with one: explicit rays give
the oracle's primitive ids and distances bit for bit (the oracle has a tree of
its own, binary and in float boxes without margins of this kind)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _discs(rng, n, kind):
    if kind == "flat":  # one plane, axis-parallel: boxes without thickness but for their padding
        p = np.stack([rng.uniform(0, 1, n), rng.uniform(0, 1, n), np.full(n, -0.5)], 1)
        nrm = np.tile([0.0, 0.0, 1.0], (n, 1))
    elif kind == "far":  # far from the origin: coordinates large against the boxes
        p = rng.uniform(0, 1, (n, 3)) + [700.0, -300.0, 50.0]
        nrm = rng.normal(size=(n, 3))
    elif kind == "same":  # every box the same
        p = np.tile([[0.5, 0.5, 0.5]], (n, 1))
        nrm = np.tile([0.6, 0.0, 0.8], (n, 1))
    else:
        p = rng.uniform(0, 1, (n, 3))
        nrm = rng.normal(size=(n, 3))
    nrm = nrm / np.linalg.norm(nrm, axis=1)[:, None]
    r = rng.uniform(0.05, 0.3, n)
    return p.astype(np.float32), nrm.astype(np.float32), r.astype(np.float32)


def _rays(rng, p, nrm, n):
    """A third from around the scene, a third on the primitives' planes (leaving
    along their normals' side), a third axis-parallel from the same points."""
    k = rng.integers(0, len(p), n)
    o = p[k] + rng.normal(scale=0.05, size=(n, 3))
    c, d = p.mean(0), rng.normal(size=(n, 3))
    o[: n // 3] = c + rng.normal(scale=2.0, size=(n // 3, 3))
    d[: n // 3] = c - o[: n // 3] + rng.normal(scale=0.5, size=(n // 3, 3))
    on = slice(n // 3, 2 * n // 3)
    o[on] -= ((o[on] - p[k[on]]) * nrm[k[on]]).sum(1)[:, None] * nrm[k[on]]
    ax = np.arange(2 * n // 3, n)
    d[ax] = np.eye(3)[rng.integers(0, 3, len(ax))] * rng.choice([-1.0, 1.0], (len(ax), 1))
    d /= np.linalg.norm(d, axis=1)[:, None]
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("builder", [0, 1], ids=["radix", "ploc"])
@pytest.mark.parametrize("kind", ["random", "flat", "far", "same"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 17, 65, 700])
def test_closest_hits_equal_the_oracle(eng, oracle_lib, n, kind, builder):
    rng = np.random.default_rng(100 * n + builder)
    p, nrm, r = _discs(rng, n, kind)
    rays = _rays(rng, p, nrm, 3000)
    s = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm)
    eng.set_tree_builder(builder)
    try:
        eng.upload_discs(p, nrm, r)
        for tnear in (0.0, 1e-4, 0.25):
            pc, tc = s.closest_hit(rays, tnear)
            pg, tg = eng.trace_rays(rays, tnear)
            assert np.array_equal(pg, pc), tnear
            assert np.array_equal(tg.view(np.uint32), tc.view(np.uint32)), tnear
            assert n < 3 or (pc >= 0).any()
    finally:
        eng.set_tree_builder(0)


def test_refit_makes_the_nodes_again(eng, oracle_lib):
    """After a refit the nodes hold the moved boxes and another choice of opened
    children: the same hits as a new upload."""
    rng = np.random.default_rng(5)
    p, nrm, r = _discs(rng, 900, "random")
    eng.upload_discs(p, nrm, r)
    q = (p * [1.0, 0.2, 3.0] + rng.normal(scale=0.05, size=p.shape)).astype(np.float32)
    eng.update_discs(q, nrm, r)
    rays = _rays(rng, q, nrm, 6000)
    pc, tc = oracle_lib.Scene(np.concatenate([q, r[:, None]], 1), nrm).closest_hit(rays)
    pg, tg = eng.trace_rays(rays)
    assert np.array_equal(pg, pc) and np.array_equal(tg.view(np.uint32), tc.view(np.uint32))
