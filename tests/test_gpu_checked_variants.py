"""The checked build (every index read from device data is verified before use) in
the kernels that its first test does not run: stacks in shared memory and of 256
entries, the plain schedule, other block sizes, small launches of partial warps and
ordered launches.  No violation, and the hit counts of the production library."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu


def _run_all(L):
    from rti_gb300 import Engine
    out = {}
    t = scenes.trench_discs(domain=0.9, width=0.3, depth=1.0)
    h = scenes.hole_triangles(n_theta=64, n_wall=20, n_top=6, n_bottom=4, depth=4.0)
    with Engine(0) as e:
        for surface in ("discs", "triangles"):
            if surface == "discs":
                e.upload_discs(t.points, t.normals, t.radii)
                e.configure(box=(t.box_lo, t.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
            else:
                e.upload_triangles(h.vertices, h.indices)
                e.configure(box=(h.box_lo, h.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
            for name, n, kw in (("shared", 100_000, {"stack_memory": L.RTG_STACK_SHARED}),
                                ("256", 100_000, {"stack_depth": 256}),
                                ("plain", 100_000, {"scheduling": L.RTG_SCHED_PLAIN}),
                                ("64 threads", 100_000, {"threads_per_block": 64, "packet": 8}),
                                ("256 threads", 100_000, {"threads_per_block": 256, "packet": 32}),
                                ("small", 1024, {}), ("ordered", (1 << 21) + 77, {})):
                e.set_launch_config(**kw)
                e.trace(n, 5)
                out[surface, name] = (e.hit_counts(), e.tally().errors)
            e.set_launch_config()
            ds, dn, _ = e.adjoint(np.ones(e.num_primitives), (1 << 21) + 77, seed=2)
            out[surface, "ordered adjoint"] = (np.array([ds, dn]), 0)
            rng = np.random.default_rng(0)
            lo, hi = [np.array(x) for x in e.box()]
            d = rng.normal(size=(5000, 3))
            rays = np.concatenate([rng.uniform(lo, hi, (5000, 3)), d / np.linalg.norm(d, axis=1)[:, None]], 1)
            out[surface, "rays"] = (e.trace_rays(rays.astype(np.float32))[0], 0)
    return out


def test_no_violations_and_the_same_hits(rtg_lib):
    from rti_gb300 import build, _lib
    ref = _run_all(_lib)
    path = build.build(checked=True)
    keep = _lib._lib
    _lib._lib = None
    try:
        _lib.load(path)
        got = _run_all(_lib)
    finally:
        _lib._lib = keep
    for k, (v, err) in got.items():
        assert err == 0, k
        if "adjoint" in k[1]:
            np.testing.assert_allclose(v, ref[k][0], rtol=1e-9)
        else:
            assert np.array_equal(v, ref[k][0]), k
