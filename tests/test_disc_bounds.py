"""Discs whose accepted normals are not of length one (0.999 to 1.001): their boxes
hold the whole disc.

A disc tilted by a little against an axis plane reaches r sin(tilt) out of it,
which r sqrt(1 - n_i^2) understates, to zero even, where the normal is longer than
one.  Rays along the plane meet the rim there; the closest hits are those of the
primitive test over all discs (the same float operations, on the CPU)."""
import numpy as np
import pytest

LENGTHS = [0.9991, 1.0, 1.0005, 1.0009]


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _all_discs(p, nrm, r, rays, tnear):
    """Closest hit over every disc, operation by operation as the primitive test."""
    f = np.float32
    best, who = np.full(len(rays), np.inf, f), np.full(len(rays), -1, np.int32)
    o, d = [rays[:, a] for a in range(3)], [rays[:, 3 + a] for a in range(3)]
    with np.errstate(all="ignore"):
        for i in range(len(p)):
            c, n = p[i], nrm[i]
            dn = d[0] * n[0] + d[1] * n[1] + d[2] * n[2]
            t = ((c[0] - o[0]) * n[0] + (c[1] - o[1]) * n[1] + (c[2] - o[2]) * n[2]) / dn
            q = [(o[a] - c[a]) + d[a] * t for a in range(3)]
            ok = (dn != 0) & (t > f(tnear)) & (q[0] * q[0] + q[1] * q[1] + q[2] * q[2] <= r[i] * r[i]) & (t < best)
            best[ok], who[ok] = t[ok], i
    return who, np.where(who >= 0, best, f(0))


def _tilted(length, axis):
    """Discs tilted by 0.005 to 0.08 against the plane of `axis`, and rays through
    points near their rims that leave the plane by a tenth of the tilt."""
    rng = np.random.default_rng(int(1e4 * length) + axis)
    n, m = 40, 400
    p = (np.arange(n)[:, None] * np.array([[5.0, 3.0, 4.0]]) / n + rng.uniform(-0.2, 0.2, (n, 3))).astype(np.float32)
    r = rng.uniform(0.3, 1.0, n).astype(np.float32)
    tilt = rng.uniform(0.005, 0.08, n)
    turn = rng.uniform(0, 2 * np.pi, n)
    a, b = (axis + 1) % 3, (axis + 2) % 3
    nrm, low = np.zeros((n, 3)), np.zeros((n, 3))  # low: along the disc, down its slope
    nrm[:, axis], nrm[:, a], nrm[:, b] = np.cos(tilt), np.sin(tilt) * np.cos(turn), np.sin(tilt) * np.sin(turn)
    low[:, axis], low[:, a], low[:, b] = -np.sin(tilt), np.cos(tilt) * np.cos(turn), np.cos(tilt) * np.sin(turn)
    k = rng.integers(0, n, m)
    at = p[k] + low[k] * (r[k] * rng.choice([-1, 1], m) * rng.uniform(0.8, 0.99, m))[:, None]
    d = np.cross(low[k], nrm[k]) + rng.uniform(-0.1, 0.1, m)[:, None] * tilt[k][:, None] * nrm[k]
    d /= np.linalg.norm(d, axis=1)[:, None]
    return p, (nrm * length).astype(np.float32), r, np.concatenate([at - 2.0 * d, d], 1).astype(np.float32)


def _check(p, nrm, r, rays, prim, t):
    pc, tc = _all_discs(p, nrm, r, rays, 1e-4)
    hit = pc >= 0
    assert hit.mean() > 0.5
    assert np.array_equal(prim, pc), f"{(prim != pc).sum()} of {len(rays)} rays miss or hit another disc"
    assert np.array_equal(t[hit].view(np.uint32), tc[hit].view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 8], ids=["four-box", "eight-wide"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", LENGTHS)
def test_rims_are_hit(eng, length, axis, width):
    p, nrm, r, rays = _tilted(length, axis)
    eng.set_node_width(width)
    try:
        eng.upload_discs(p, nrm, r)
        prim, t = eng.trace_rays(rays, 1e-4)
    finally:
        eng.set_node_width(0)
    _check(p, nrm, r, rays, prim, t)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", LENGTHS)
def test_rims_are_hit_in_the_oracle(oracle_lib, length, axis):
    p, nrm, r, rays = _tilted(length, axis)
    prim, t = oracle_lib.Scene(np.concatenate([p, r[:, None]], 1), nrm).closest_hit(rays)
    _check(p, nrm, r, rays, prim, t)
