"""The deposit on overlapping neighbour discs, whose list a path walks 32
entries at a time and four centres a load: lists from empty to over a hundred
entries, remainders of four and of 32, radii apart by a factor of 300, and
coordinates large against the discs.

A neighbour that rti's test accepts is never left out, so hit counts and
tallies are the oracle's, whole numbers without a tolerance; the sums differ by
the order of their additions alone (200 000 rays of at most a few hundred
deposits on a disc: below 1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _sheet(rng, n, spread, shift, tilt):
    """A wavy sheet of n discs whose radii reach over `spread` discs, in the
    unit square about `shift`."""
    k = int(np.ceil(np.sqrt(n)))
    i, j = np.divmod(np.arange(n), k)
    x, y = (i + rng.uniform(0.2, 0.8, n)) / k, (j + rng.uniform(0.2, 0.8, n)) / k
    z = 0.1 * np.sin(7 * x) * np.cos(5 * y)
    r = np.full(n, 0.55 * spread / k) if tilt < 1 else 0.002 * 300.0 ** rng.uniform(0, 1, n) / 2
    nrm = np.stack([-0.7 * np.cos(7 * x) * np.cos(5 * y), 0.5 * np.sin(7 * x) * np.sin(5 * y), np.ones(n)], 1)
    nrm += rng.normal(scale=0.1, size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    return (np.stack([x, y, z], 1) + shift).astype(np.float32), nrm.astype(np.float32), r.astype(np.float32)


@pytest.mark.parametrize("shift", [0.0, 1500.0], ids=["near", "far"])
@pytest.mark.parametrize("n,spread,tilt", [(400, 0.3, 0), (900, 1.3, 0), (900, 3.2, 0), (1600, 6.0, 0), (900, 1.0, 1)],
                         ids=["none", "few", "remainders", "hundreds", "mixed-radii"])
def test_neighbour_deposits_equal_the_oracle(eng, oracle_lib, n, spread, tilt, shift):
    rng = np.random.default_rng(n + int(10 * spread))
    p, nrm, r = _sheet(rng, n, spread, shift, tilt)
    lo, hi = (shift, shift, shift - 0.5), (1.0 + shift, 1.0 + shift, 0.5 + shift)
    eng.upload_discs(p, nrm, r)
    eng.configure(box=(lo, hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
    eng.trace(200000, 7)
    s = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm)
    ptr = s.neighbors()[0]
    c = s.trace(oracle_lib.make_config(lo, hi, sticking=0.3, seed=7), 0, 200000)
    t, lengths = eng.tally(), np.diff(ptr)
    assert {0.3: lengths.min() == 0, 1.3: lengths.max() >= 8, 3.2: lengths.max() > 32, 6.0: lengths.max() > 96,
            1.0: lengths.max() > 32}[spread]
    assert np.array_equal(eng.hit_counts(), c.counts)
    assert (t.hitc, t.nonhitc, t.total, t.segments, t.nb_deposits, t.errors) == (
        c.hitc, c.nonhitc, c.total, c.segments, c.nb_deposits, 0)
    assert c.nb_deposits > 0 or spread < 1
    for a, b in zip(eng.accumulators(), (c.s1, c.s2, c.s3, c.s4)):
        np.testing.assert_allclose(a, b, rtol=1e-9, atol=0)
