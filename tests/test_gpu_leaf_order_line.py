"""Primitives whose centres differ along one axis only are still put in order
along it, so that a query visits few nodes instead of most of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("builder", [0, 1], ids=["radix", "ploc"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_few_visits(eng, axis, builder):
    n = 4096
    rng = np.random.default_rng(axis)
    at = 0.1 * rng.permutation(n)
    p, nrm, rays = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros((n, 6))
    p[:, axis], nrm[:, (axis + 1) % 3] = at, 1.0  # discs across the rays, 0.1 apart
    rays[:, axis], rays[:, (axis + 1) % 3], rays[:, 3 + (axis + 1) % 3] = at, -1.0, 1.0
    eng.set_tree_builder(builder)
    eng.upload_discs(p.astype(np.float32), nrm.astype(np.float32), np.full(n, 0.03, np.float32))
    eng.set_visit_limit(64)  # 12 levels of two; a random order takes about a thousand visits
    try:
        prim, t = eng.trace_rays(rays.astype(np.float32))
    finally:
        eng.set_visit_limit(0)
        eng.set_tree_builder(0)
    assert np.array_equal(prim, np.arange(n)) and np.all(t == 1.0)
