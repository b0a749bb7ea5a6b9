"""The window's one walk over the four-box nodes: stacks of front-face discs in
a window, from one to well over the eight hits that the walk keeps (more are
walked again), closed by nothing, by a back-face disc or by a triangle above, between
and below them, in trees of one to a few levels and under either node width.

Counts and tallies are whole numbers and equal the oracle's, which compares
every disc with the ray; sums within 1e-9 (order of additions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine, _lib as L
    e = Engine(0)
    e.set_deposit_mode(L.RTG_DEPOSIT_WINDOW, 5.0)
    yield e
    e.close()


@pytest.mark.parametrize("wide", [0, 8], ids=["quads", "wide"])
@pytest.mark.parametrize("closer", ["none", "disc", "triangle"])
@pytest.mark.parametrize("layers", [1, 2, 7, 8, 9, 16, 33])
def test_stacked_layers_equal_the_oracle(eng, oracle_lib, layers, closer, wide):
    rng = np.random.default_rng(layers)
    z = np.repeat(-0.02 * np.arange(layers), 4)  # four tilted discs of a layer cover the box's quarters
    xy = np.tile([[-0.25, -0.25], [0.25, -0.25], [0.25, 0.25], [-0.25, 0.25]], (layers, 1))
    p = np.concatenate([xy, z[:, None]], 1)
    nrm = np.tile([0.0, 0.0, 1.0], (len(p), 1)) + rng.normal(scale=0.02, size=(len(p), 3))
    r = np.full(len(p), 0.4)
    zc = -0.02 * (layers // 2) - 0.01
    if closer == "disc":
        p, nrm, r = np.vstack([p, [[0, 0, zc]]]), np.vstack([nrm, [[0, 0, -1.0]]]), np.append(r, 0.3)
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    p, nrm, r = p.astype(np.float32), nrm.astype(np.float32), r.astype(np.float32)
    v = np.float32([[-0.3, -0.3, zc], [0.3, -0.3, zc], [0.0, 0.4, zc]])
    idx = np.uint32([[0, 1, 2]])
    tri = dict(tri_vertices=v, tri_indices=idx) if closer == "triangle" else {}
    lo, hi = np.float32([-0.5, -0.5, -1.0]), np.float32([0.5, 0.5, 0.5])
    eng.set_node_width(wide)
    try:
        if tri:
            eng.upload_mixed(p, nrm, r, v, idx)
        else:
            eng.upload_discs(p, nrm, r)
        eng.configure(box=(lo, hi), sticking=0.2, x_bound=1, y_bound=1, reset=True)
        eng.trace(20000, 4)
    finally:
        eng.set_node_width(0)
    s = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm, **tri)
    c = s.trace(oracle_lib.make_config(lo, hi, sticking=0.2, seed=4, window=1, window_factor=5.0), 0, 20000)
    t = eng.tally()
    assert np.array_equal(eng.hit_counts(), c.counts)
    assert (t.hitc, t.nonhitc, t.total, t.segments, t.nb_deposits, t.errors) == (
        c.hitc, c.nonhitc, c.total, c.segments, c.nb_deposits, 0)
    for a, b in zip(eng.accumulators(), (c.s1, c.s2, c.s3, c.s4)):
        np.testing.assert_allclose(a, b, rtol=1e-9, atol=0)
    if closer == "none":
        assert c.total >= min(layers, 30) * c.hitc * 0.5  # the window holds the layers
