"""Ray ids up to the end of their 64-bit range.

A launch of more rays than are ordered at once takes them in pieces of equal
length, rounded up, so the end of the last piece computed as begin + length can
pass 2^64; the launch ends where it was asked to all the same.  Counts and
tallies equal those of the same rays in two calls of one piece each (2^25 and
2^29 rays and a few more)."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu
FIELDS = ("hitc", "nonhitc", "total", "segments", "truncated", "nb_deposits", "errors")
TOP = 1 << 64


@pytest.fixture(scope="module")
def eng(rtg_lib):
    from rti_gb300 import Engine
    t = scenes.trench_discs(domain=0.9, width=0.3, depth=1.0)
    e = Engine(0)
    e.upload_discs(t.points, t.normals, t.radii)
    e.configure(box=(t.box_lo, t.box_hi), sticking=0.9, x_bound=1, y_bound=1, reset=True)
    yield e
    e.close()


@pytest.mark.parametrize("begin,end", [(TOP - (1 << 25) - 2, TOP - 1), (TOP - (1 << 25) - 3, TOP - 1),
                                       (TOP - (1 << 25) - 3, TOP - 2), (TOP - (1 << 29) - 2, TOP - 1),
                                       (TOP - 4099, TOP - 1)])
def test_trace(eng, begin, end):
    got = []
    for cuts in ([begin, end], [begin, begin + (end - begin) // 2, end]):
        for b, e in zip(cuts, cuts[1:]):
            eng.trace(e - b, 3, ray_begin=b, accumulate=b != begin)
        t = eng.tally()
        got.append((eng.hit_counts(), [getattr(t, k) for k in FIELDS], t.num_rays))
    assert got[0][1] == got[1][1] and got[0][2] == got[1][2] == end - begin and np.array_equal(got[0][0], got[1][0])


def test_adjoint(eng):
    import torch
    begin, end, out = TOP - (1 << 25) - 2, TOP - 1, []
    g = torch.rand(eng.num_primitives, dtype=torch.float64, device="cuda")
    for cuts in ([begin, end], [begin, begin + (end - begin) // 2, end]):
        s = torch.zeros(2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for b, e in zip(cuts, cuts[1:]):
            eng.adjoint_device(g.data_ptr(), b, e, 3, 0, s.data_ptr())
        torch.cuda.synchronize()
        out.append(s.cpu().numpy())
    # one path more or less changes the sums of 3.4e7 by about 3e-8; orders of addition by 1e-13
    np.testing.assert_allclose(out[0], out[1], rtol=1e-10, atol=0)
