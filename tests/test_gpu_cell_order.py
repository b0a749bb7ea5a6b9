"""The order of the leaves (Morton codes whose bits go to the axis along which
the cell is longest): surfaces without extent along one axis, two, or all three,
flat, deep and wide ones, far from the origin, and few and many primitives per
cell, in both trees.

The order decides how many boxes a query visits, never which hit is closest:
ids and distances equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXTENTS = {"cube": (1, 1, 1), "sheet": (1, 1, 0.01), "plane": (1, 1, 0), "wall": (0, 1, 1), "deep": (1, 1, 30),
           "strip": (50, 1, 0.2), "line": (0, 3, 0), "point": (0, 0, 0), "tower": (0, 0, 5)}


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("builder", [0, 1], ids=["radix", "ploc"])
@pytest.mark.parametrize("shape", list(EXTENTS))
@pytest.mark.parametrize("n,shift", [(3, 0.0), (900, 200.0), (6000, 0.0)])
def test_hits_equal_the_oracle(eng, oracle_lib, n, shift, shape, builder):
    rng = np.random.default_rng(n)
    ext = np.array(EXTENTS[shape], np.float64)
    p = (ext * rng.random((n, 3)) + shift).astype(np.float32)
    nrm = rng.normal(size=(n, 3))
    nrm = (nrm / np.linalg.norm(nrm, axis=1)[:, None]).astype(np.float32)
    r = rng.uniform(0.02, 0.2, n).astype(np.float32)
    k = rng.integers(0, n, 4000)
    o = p[k] + rng.normal(scale=0.5, size=(4000, 3))
    rays = np.concatenate([o, p[rng.permutation(k)] + rng.normal(scale=0.05, size=(4000, 3)) - o], 1).astype(np.float32)
    rays[:, 3:] /= np.linalg.norm(rays[:, 3:], axis=1)[:, None]
    eng.set_tree_builder(builder)
    try:
        eng.upload_discs(p, nrm, r)
    finally:
        eng.set_tree_builder(0)
    pg, tg = eng.trace_rays(rays)
    pc, tc = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm).closest_hit(rays)
    assert np.array_equal(pg, pc) and np.array_equal(tg.view(np.uint32), tc.view(np.uint32))
    assert (pc >= 0).any()
