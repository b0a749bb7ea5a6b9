"""The surface build's kernels at the sizes where they change: the one-block
sort and the two tile widths of the long one, tile and warp remainders, rows of
neighbours beyond the thread's buffer, and the scratch buffer that a context
keeps between builds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _soup(n, seed):
    """n small triangles, scattered: Morton keys of all kinds, some of them equal."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (n, 1, 3))
    c[n // 2:] = np.round(c[n // 2:] * 8) / 8  # half of them share a few cells
    v = (c + rng.normal(scale=0.02, size=(n, 3, 3))).astype(np.float32).reshape(-1, 3)
    return v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


@pytest.mark.parametrize("builder", [0, 1], ids=["radix", "ploc"])
@pytest.mark.parametrize("n", [31, 33, 1023, 4095, 4096, 4097, 5120, 5121, 262144, 262145, 266241])
def test_sorted_trees_give_the_oracle_hits(eng, oracle_lib, n, builder):
    if builder and n > 262145:
        pytest.skip("one long size is enough for the clustering")
    v, t = _soup(n, n)
    rng = np.random.default_rng(n + 1)
    d = rng.normal(size=(4000, 3))
    rays = np.concatenate([rng.uniform(-0.1, 1.1, (4000, 3)), d / np.linalg.norm(d, axis=1)[:, None]], 1)
    rays = rays.astype(np.float32)
    eng.set_tree_builder(builder)
    try:
        eng.upload_triangles(v, t)
        pg, tg = eng.trace_rays(rays)
    finally:
        eng.set_tree_builder(0)
    pc, tc = oracle_lib.Scene(tri_vertices=v, tri_indices=t).closest_hit(rays)
    assert np.array_equal(pg, pc) and np.array_equal(tg.view(np.uint32), tc.view(np.uint32))


def _pairs(p, r):
    """Rows of overlapping discs by the float32 predicate, every pair tested."""
    rows = []
    for i in range(len(p)):
        a = p[i] - p
        dist = np.sqrt(a[:, 0] * a[:, 0] + a[:, 1] * a[:, 1] + a[:, 2] * a[:, 2])
        hit = dist < r[i] + r
        hit[i] = False
        rows.append(np.flatnonzero(hit))
    return rows


@pytest.mark.parametrize("n,spread,radius", [(2, 1.0, 0.5), (40, 0.0, 0.2), (129, 1.0, 0.3), (3000, 1.0, 0.03),
                                              (3000, 3000.0, 4.0), (2500, 1.0, 0.14)])
def test_neighbor_rows(eng, n, spread, radius):
    """Few, coincident, dense (rows beyond 32), and far-spread discs of unequal radii."""
    rng = np.random.default_rng(n)
    p = rng.uniform(0, 1, (n, 3)).astype(np.float32) * np.float32([spread, spread, 0.3 * spread])
    r = (radius * rng.uniform(0.3, 1.0, n)).astype(np.float32)
    eng.upload_discs(p, np.tile(np.float32([0, 0, 1]), (n, 1)), r)
    rp, cols = eng.neighbors()
    rows = _pairs(p, r)
    assert np.array_equal(np.diff(rp), [len(x) for x in rows])
    assert np.array_equal(cols, np.concatenate(rows))
    assert n != 2500 or max(len(x) for x in rows) > 32


def test_scratch_is_kept_and_outgrown(rtg_lib):
    """Surfaces of changing size through one context (the last beyond the scratch
    that is kept), with refits between, trace as they do in a context of their own."""
    from rti_gb300 import Engine, scenes

    def run(e, s):
        e.upload_discs(s.points, s.normals, s.radii)
        e.configure(box=(s.box_lo, s.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
        e.trace(20000, 3)
        a = e.hit_counts()
        e.update_discs(s.points + np.float32(0.002) * s.normals, s.normals, s.radii)
        e.trace(20000, 4)
        return a, e.hit_counts(), e.mc_estimates(), e.neighbors()[1]

    with Engine(0) as kept:
        for n in (40, 300, 16, 640, 64):
            s = scenes.rough_discs(n=n, seed=n)
            got = run(kept, s)
            with Engine(0) as fresh:
                want = run(fresh, s)
            for a, b in zip(got, want):
                assert np.array_equal(a, b) if a.dtype != np.float32 else np.allclose(a, b, rtol=1e-6)


def test_moved_vertices_are_checked_on_the_device(eng):
    from rti_gb300 import RtgError
    v, t = _soup(700, 1)
    eng.upload_triangles(v, t)
    box = eng.box()
    w = v * np.float32(1.5) + np.float32([1, 2, 3])
    eng.update_vertices(w)
    lo, hi = eng.box()
    assert np.array_equal(lo, w.min(0)) and np.array_equal(hi, w.max(0)) and not np.array_equal(lo, box[0])
    bad = w.copy()
    bad[1234, 1] = np.inf
    with pytest.raises(RtgError, match="not finite"):
        eng.update_vertices(bad)
    assert np.array_equal(eng.box()[0], w.min(0))
