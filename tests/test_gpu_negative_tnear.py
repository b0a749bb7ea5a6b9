"""Explicit rays with a negative tnear: boxes wholly behind the origin are not
visited, over either tree (a hit a little behind the origin, within its box, is
accepted as ever)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 8], ids=["four-box", "eight-wide"])
@pytest.mark.parametrize("tnear", [0.0, -1e-3, -1.0, -5.0, -np.inf])
def test_behind_the_origin(rtg_lib, tnear, width):
    from rti_gb300 import Engine
    z = np.array([-3.0, -1.0, 1.0, 3.0])
    p = np.zeros((4, 3), np.float32)
    p[:, 2] = z
    nrm = np.tile(np.float32([0, 0, 1]), (4, 1))
    with Engine(0) as e:
        e.set_node_width(width)
        e.upload_discs(p, nrm, np.full(4, 0.5, np.float32))
        o = np.array([0.0, 2.0, 4.0, -2.0, -4.0], np.float32)
        rays = np.zeros((len(o), 6), np.float32)
        rays[:, 2], rays[:, 5] = o, 1.0
        prim, t = e.trace_rays(rays, tnear)
        ahead = [[k for k in range(4) if z[k] > x] for x in o]
        assert prim.tolist() == [a[0] if a else -1 for a in ahead]
        assert t.tolist() == [z[a[0]] - x if a else 0.0 for a, x in zip(ahead, o)]
        # 1e-5 above a disc: its padded box holds the origin
        rays = np.array([[0, 0, 1.00001, 0, 0, 1]], np.float32)
        prim, t = e.trace_rays(rays, tnear)
        assert prim[0] == (2 if tnear < -1e-4 else 3)
