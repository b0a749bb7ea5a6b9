"""Moved vertices.  Of a surface of discs and triangles the discs stay, so their
neighbour lists are kept as they are, and the surface traces as a new upload of it.
Few vertices are checked by the host and many on the device: either refuses what
is not finite and leaves the surface as it was."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu


def _mixed():
    t = scenes.trench_discs(domain=1.2, width=0.4, depth=1.0)
    lo, hi = np.array(t.box_lo), np.array(t.box_hi)
    v = lo + np.array([[0.1, 0.1, 0.9], [0.9, 0.1, 0.9], [0.1, 0.9, 0.9], [0.4, 0.1, 0.5], [0.6, 0.1, 0.5], [0.5, 0.6, 0.6]]) * (hi - lo)
    v = v.astype(np.float32)
    return t, v, np.array([[0, 1, 2], [3, 4, 5]], np.uint32)


def _upload(e, t, v, i):
    e.upload_mixed(t.points, t.normals, t.radii, v, i)
    e.configure(box=(t.box_lo, t.box_hi), x_bound=1, y_bound=1, sticking=0.1, reset=True)


def test_neighbour_lists_are_not_built_again(rtg_lib):
    from rti_gb300 import Engine, RtgError
    t, v, i = _mixed()
    said = []
    for k in range(60):
        with Engine(0) as e:
            _upload(e, t, v, i)
            e.inject_alloc_failure(k)
            try:
                e.update_vertices(v + np.float32(0.01))
            except RtgError as err:
                said.append(str(err))
            else:
                break
    assert 0 < len(said) < 60
    assert not [s for s in said if "grid" in s or "neighbour" in s], said


def test_traces_as_a_new_upload(rtg_lib):
    from rti_gb300 import Engine
    t, v, i = _mixed()
    moved = v + np.float32([0.02, 0.01, 0.05])
    with Engine(0) as e, Engine(0) as f:
        _upload(e, t, v, i)
        e.trace(20000, 1)
        before = e.neighbors()
        e.update_vertices(moved)
        _upload(f, t, moved, i)
        for g in (e, f):
            g.trace(20000, 1)
        assert np.array_equal(e.hit_counts(), f.hit_counts()) and e.hit_counts()[-2:].sum() > 0
        np.testing.assert_allclose(e.mc_estimates(), f.mc_estimates(), rtol=1e-6)
        for a, b, c in zip(before, e.neighbors(), f.neighbors()):
            assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("nv", [3, 4095, 4096, 4097])
def test_checked_on_the_host_or_the_device(rtg_lib, nv):
    from rti_gb300 import Engine, RtgError
    rng = np.random.default_rng(nv)
    v = rng.uniform(-1, 1, (nv, 3)).astype(np.float32)
    i = (np.arange(3 * ((nv + 2) // 3)) % nv).astype(np.uint32).reshape(-1, 3)
    moved = (v * np.float32(1.5) + np.float32([3, -2, 1])).astype(np.float32)
    rays = np.concatenate([rng.uniform(-1, 1, (500, 3)) + [3, -2, 4], np.tile([0, 0, -1.0], (500, 1))], 1).astype(np.float32)
    with Engine(0) as e, Engine(0) as f:
        e.upload_triangles(v, i)
        box = np.array(e.box())
        for bad in (np.nan, np.inf, -np.inf):
            for at in (0, nv - 1):
                w = moved.copy()
                w[at, at % 3] = bad
                with pytest.raises(RtgError):
                    e.update_vertices(w)
        assert np.array_equal(np.array(e.box()), box)
        e.update_vertices(moved)
        f.upload_triangles(moved, i)
        assert np.array_equal(np.array(e.box()), np.array(f.box()))
        (pe, te), (pf, tf) = e.trace_rays(rays), f.trace_rays(rays)
        assert np.array_equal(pe, pf) and np.array_equal(te, tf) and (nv == 3 or (pe >= 0).any())
