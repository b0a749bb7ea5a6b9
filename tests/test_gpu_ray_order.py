"""Launches that take their rays by the cell they start in (from 2^21 rays in a
surface as deep as wide, from 2^20 on one that outgrows the L2 cache) against the
same rays in pieces below both limits, which are taken in ascending order, and
one of them against the oracle: on either side of a limit, off the multiples of a
block, from a first ray other than 0, and past the rays ordered at once.

Which rays are traced does not depend on the order, so counts and tallies are
equal; sums differ by the order of additions (1e-9, as everywhere)."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu
PIECE = (1 << 20) - 3
FIELDS = ("hitc", "nonhitc", "total", "segments", "truncated", "nb_deposits", "errors")


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _state(e):
    t = e.tally()
    return e.hit_counts(), [getattr(t, k) for k in FIELDS], [np.array(a) for a in e.accumulators()]


def _pieces(e, begin, end, seed):
    for b in range(begin, end, PIECE):
        e.trace(min(end, b + PIECE) - b, seed, ray_begin=b, accumulate=b != begin)
    return _state(e)


def _same(a, b):
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and a[1][-1] == 0 and a[0].sum() > 0
    for x, y in zip(a[2], b[2]):
        np.testing.assert_allclose(x, y, rtol=1e-9, atol=0)


def _deep(e, **more):
    t = scenes.trench_discs(domain=0.9, width=0.3, depth=1.0)
    e.upload_discs(t.points, t.normals, t.radii)
    e.configure(box=(t.box_lo, t.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True, **more)
    assert t.box_hi[2] - t.box_lo[2] >= max(t.box_hi[0] - t.box_lo[0], t.box_hi[1] - t.box_lo[1])
    return t


@pytest.mark.parametrize("mode", ["neighbours", "window", "directional", "plain", "fixed"])
@pytest.mark.parametrize("begin,n", [(0, (1 << 21) - 1), (0, 1 << 21), (12345, (1 << 21) + 77)])
def test_deep_surface_equals_pieces(eng, begin, n, mode):
    _deep(eng, source_exponent=40.0 if mode == "directional" else 1.0)
    eng.set_deposit_mode(1 if mode == "window" else 0, 5.0)
    eng.set_accumulation(1 if mode == "fixed" else 0)
    if mode == "plain":
        eng.set_launch_config(scheduling=2)
    try:
        eng.trace(n, 5, ray_begin=begin)
        got = _state(eng)
        _same(got, _pieces(eng, begin, begin + n, 5))
    finally:
        eng.set_deposit_mode(0, 5.0)
        eng.set_accumulation(0)
        eng.set_launch_config()


def test_deep_surface_equals_the_oracle(eng, oracle_lib):
    t = _deep(eng)
    n = (1 << 21) + 5
    eng.trace(n, 9)
    s = oracle_lib.Scene(t.xyzr, t.normals)
    s.neighbors()
    c = s.trace(oracle_lib.make_config(t.box_lo, t.box_hi, sticking=0.3, seed=9), 0, n)
    assert np.array_equal(eng.hit_counts(), c.counts) and eng.tally().segments == c.segments


def test_more_rays_than_are_ordered_at_once(eng):
    _deep(eng)
    eng.configure(sticking=0.9)
    n = (1 << 25) + 1001
    eng.trace(n, 1)
    _same(_state(eng), _pieces(eng, 0, n, 1))


def test_surface_beyond_the_cache_equals_pieces(eng):
    n = 1600
    r = scenes.rough_discs(n=n, spacing=0.01, rms=0.02, corr=0.1, seed=3)
    eng.upload_discs(r.points, r.normals, r.radii)
    eng.configure(box=(r.box_lo, r.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
    rays = (1 << 20) + 12345
    eng.trace(rays, 2)
    _same(_state(eng), _pieces(eng, 0, rays, 2))


@pytest.mark.parametrize("field", [False, True], ids=["global", "field"])
def test_adjoint_equals_pieces(eng, field):
    import torch
    t = _deep(eng)
    if field:
        eng.set_sticking_field(np.random.default_rng(0).uniform(0.1, 0.5, t.n).astype(np.float32))
    g = torch.rand(t.n, dtype=torch.float64, device="cuda")
    n, out = (1 << 21) + 9, []
    for cuts in ([0, n], list(range(0, n, PIECE)) + [n]):
        f, s = torch.zeros(t.n, dtype=torch.float64, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for b, e in zip(cuts, cuts[1:]):
            eng.adjoint_device(g.data_ptr(), b, e, 7, f.data_ptr(), s.data_ptr())
        torch.cuda.synchronize()
        out.append((f.cpu().numpy(), s.cpu().numpy()))
    scale = np.abs(out[1][0]).max()
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-9, atol=1e-9 * scale)
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-9, atol=1e-9 * n)


def test_batches_of_one_scene_on_two_streams(rtg_lib):
    """Sequential launches of two batches that share a context, on two streams at
    once: they keep no ray order in it, so neither disturbs the other."""
    import torch
    from rti_gb300 import Engine
    from rti_gb300.batch import Batch
    e, bs = Engine(0), [Batch(0), Batch(0)]
    try:
        _deep(e)
        rays = [(1 << 21) + 7, (1 << 21) + 4099]
        jobs = [b.add(e, r, seed=3 + i, config=e.config()) for i, (b, r) in enumerate(zip(bs, rays))]
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        for b, s in zip(bs, streams):
            b.run_sequential(stream=s.cuda_stream)
        torch.cuda.synchronize()
        for i, (b, j, r) in enumerate(zip(bs, jobs, rays)):
            e.trace(r, 3 + i)
            assert np.array_equal(b.results(j)[1], e.hit_counts())
    finally:
        for b in bs:
            b.close()
        e.close()


def test_without_room_the_rays_are_taken_in_ascending_order(rtg_lib):
    from rti_gb300 import Engine
    with Engine(0) as e:
        _deep(e)
        n = (1 << 21) + 5
        e.inject_alloc_failure(0)
        e.trace(n, 4)
        a = _state(e)
        e.inject_alloc_failure(-1)
        e.trace(n, 4)
        _same(a, _state(e))
