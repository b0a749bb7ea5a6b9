"""The kept basis of every normal: all three choices of the second vector and
their ties, axis-parallel and negated normals, zeros of either sign, discs and
triangles and both together, and bases made again when the surface moves.

A direction that differs in one bit changes the path, so the equality of counts
and tallies with the oracle, which builds the basis at every hit, needs no
tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECIAL = [[0, 0, 1], [0, 0, -1], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [-0.0, 0.0, 1.0], [1, 1, 1], [-1, -1, -1],
           [1, 1, 0], [1, -1, 0], [0, 1, 1], [1, 0, 1], [1, 1, -2], [-2, 1, 1], [1, -2, 1], [1e-7, 0, 1], [0, 1e-20, 1]]


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _discs(rng, n):
    nrm = rng.normal(size=(n, 3))
    nrm[: len(SPECIAL)] = SPECIAL
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    return rng.random((n, 3)).astype(np.float32), nrm.astype(np.float32), \
        rng.uniform(0.05, 0.2, n).astype(np.float32)


def _tris(rng, n):
    v = (rng.random((n, 1, 3)) + rng.normal(scale=0.1, size=(n, 3, 3))).astype(np.float32)
    v[0::5, :, 2] = v[0::5, :1, 2]  # normals along z, x, y
    v[1::5, :, 0] = v[1::5, :1, 0]
    v[2::5, :, 1] = v[2::5, :1, 1]
    return v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("kind", ["discs", "triangles", "both"])
@pytest.mark.parametrize("moved", [False, True], ids=["built", "moved"])
def test_paths_equal_the_oracle(eng, oracle_lib, kind, moved):
    if kind == "both" and moved:
        pytest.skip("a mixed surface is uploaded anew")
    rng = np.random.default_rng(10)
    lo, hi = (-0.5, -0.5, -0.5), (1.5, 1.5, 1.5)
    p, nrm, r = _discs(rng, 400)
    v, idx = _tris(rng, 300)
    if kind == "discs":
        eng.upload_discs(p, nrm, r)
        if moved:
            p, nrm, r = _discs(rng, 400)
            eng.update_discs(p, nrm, r)
        s = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm)
        s.neighbors()
    elif kind == "triangles":
        eng.upload_triangles(v, idx)
        if moved:
            v = _tris(rng, 300)[0]
            eng.update_vertices(v)
        s = oracle_lib.Scene(tri_vertices=v, tri_indices=idx)
    else:
        eng.upload_mixed(p, nrm, r, v, idx)
        s = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm, tri_vertices=v, tri_indices=idx)
        s.neighbors()
    eng.configure(box=(lo, hi), sticking=0.1, x_bound=1, y_bound=1, reset=True)
    eng.trace(50000, 6)
    c = s.trace(oracle_lib.make_config(lo, hi, sticking=0.1, seed=6), 0, 50000)
    t = eng.tally()
    assert np.array_equal(eng.hit_counts(), c.counts) and c.hitc > 20000
    assert (t.hitc, t.nonhitc, t.total, t.segments, t.nb_deposits, t.errors) == (
        c.hitc, c.nonhitc, c.total, c.segments, c.nb_deposits, 0)
