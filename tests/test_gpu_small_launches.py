"""Launches of fewer rays than the GPU has lanes for, which are spread over 16
warps per SM in shares of 1 to 32 paths: ray counts on either side of where the
share grows and of where it ends, with every refill packet and schedule, traced
alone, in the window mode, in a batch of ragged jobs and by the adjoint.

Paths depend on the seed and the ray id alone, so counts and tallies are the
oracle's.  Adjoint sums differ by the order of at most 160 000 additions in
double of terms of order one: 1e-9 of the result and of the ray count covers it."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


@pytest.fixture(scope="module")
def trench():
    return scenes.trench_discs(domain=1.2, width=0.4, depth=1.0)


@pytest.fixture(scope="module")
def warps():
    import torch
    return 16 * torch.cuda.get_device_properties(0).multi_processor_count


def _count(warps, k, plus):
    return max(1, warps * k + plus)


PLAIN = 2  # RTG_SCHED_PLAIN
SIZES = [(0, 1), (0, 33), (1, 0), (1, 1), (5, -1), (31, 1), (32, 0), (32, 1), (64, 3)]


def _upload(e, t, **more):
    e.upload_discs(t.points, t.normals, t.radii)
    e.configure(box=(t.box_lo, t.box_hi), sticking=0.15, x_bound=1, y_bound=1, reset=True, **more)


@pytest.mark.parametrize("k,plus", SIZES)
def test_counts_equal_the_oracle(eng, trench, oracle_lib, warps, k, plus):
    n = _count(warps, k, plus)
    _upload(eng, trench)
    s = oracle_lib.Scene(trench.xyzr, trench.normals)
    s.neighbors()
    c = s.trace(oracle_lib.make_config(trench.box_lo, trench.box_hi, sticking=0.15, x_bound=1, y_bound=1, seed=3), 0, n)
    for tpb, packet, schedule in ((128, 1, 0), (64, 8, 0), (256, 32, 0), (128, 1, PLAIN)):
        eng.set_launch_config(threads_per_block=tpb, packet=packet, scheduling=schedule)
        try:
            eng.trace(n, 3)
        finally:
            eng.set_launch_config()
        t = eng.tally()
        assert np.array_equal(eng.hit_counts(), c.counts)
        assert (t.hitc, t.nonhitc, t.total, t.segments, t.nb_deposits, t.errors) == (
            c.hitc, c.nonhitc, c.total, c.segments, c.nb_deposits, 0)


@pytest.mark.parametrize("k,plus", SIZES[::2])
def test_window_counts_equal_the_oracle(eng, trench, oracle_lib, warps, k, plus):
    n = _count(warps, k, plus)
    _upload(eng, trench)
    s = oracle_lib.Scene(trench.xyzr, trench.normals)
    c = s.trace(oracle_lib.make_config(trench.box_lo, trench.box_hi, sticking=0.15, seed=3, window=1,
                                       window_factor=5.0), 0, n)
    eng.set_deposit_mode(1, 5.0)
    try:
        eng.trace(n, 3)
    finally:
        eng.set_deposit_mode(0, 5.0)
    assert np.array_equal(eng.hit_counts(), c.counts) and eng.tally().segments == c.segments


@pytest.mark.parametrize("field", [False, True], ids=["global", "field"])
@pytest.mark.parametrize("k,plus", SIZES[1::3])
def test_adjoint_equals_the_oracle(eng, trench, oracle_lib, warps, k, plus, field):
    n = _count(warps, k, plus)
    rng = np.random.default_rng(n)
    g = rng.uniform(0.5, 1.5, trench.n)
    st = rng.uniform(0.05, 0.4, trench.n).astype(np.float32) if field else None
    _upload(eng, trench)
    if field:
        eng.set_sticking_field(st)
    ds, dn, fg = eng.adjoint(g, n, seed=3)
    s = oracle_lib.Scene(trench.xyzr, trench.normals)
    s.neighbors()
    cfg = oracle_lib.make_config(trench.box_lo, trench.box_hi, sticking=0.15, seed=3)
    ods, odn, ofg, _ = oracle_lib.adjoint(s, cfg, g, 0, n, sticking_field=st, unbiased=True)
    tol = dict(rtol=1e-9, atol=1e-9 * n)
    np.testing.assert_allclose(dn, odn, **tol)
    if field:
        np.testing.assert_allclose(fg, ofg, **tol)
    else:
        np.testing.assert_allclose(ds, ods, **tol)


@pytest.mark.parametrize("k,plus", SIZES[::3])
def test_batch_counts_equal_the_oracle(rtg_lib, trench, oracle_lib, warps, k, plus):
    """Jobs of unequal ray counts, one of them of a single ray, share the launch."""
    from rti_gb300 import Engine
    from rti_gb300.batch import Batch
    n = _count(warps, k, plus)
    rays = [1, n, n // 3 + 1]
    s = oracle_lib.Scene(trench.xyzr, trench.normals)
    s.neighbors()
    e, b = Engine(0), Batch(0)
    try:
        _upload(e, trench)
        jobs = [b.add(e, r, seed=3, config=e.config()) for r in rays]
        b.run(use_graph=False)
        b.synchronize()
        for j, r in zip(jobs, rays):
            cfg = oracle_lib.make_config(trench.box_lo, trench.box_hi, sticking=0.15, seed=3, job=j)
            assert np.array_equal(b.results(j)[1], s.trace(cfg, 0, r).counts)
    finally:
        b.close()
        e.close()
