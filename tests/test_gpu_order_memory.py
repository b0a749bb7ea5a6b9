"""The room of ordered launches (traces and replays that take their rays by the
cell they start in): taken and given back in the order of the stream, so that a
call returns after enqueueing; bounded; given back before an allocation fails;
and which launches are ordered at all."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu
FIELDS = ("hitc", "nonhitc", "total", "segments", "truncated", "nb_deposits", "errors")
ROOM = 4 << 25  # bytes of the ids of the rays that are ordered at once


def _deep(e):
    t = scenes.trench_discs(domain=0.9, width=0.3, depth=1.0)
    e.upload_discs(t.points, t.normals, t.radii)
    e.configure(box=(t.box_lo, t.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
    return t


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _took_room(e, call):
    """Whether the call takes room for an order: it meets a failing allocation, and
    goes on without (the call itself succeeds either way)."""
    from rti_gb300 import RtgError
    e.set_sticking_field(None)
    e.inject_alloc_failure(0)
    call()
    try:
        e.set_sticking_field(np.full(e.num_primitives, 0.3, np.float32))  # takes memory of its own
    except RtgError:
        return False
    finally:
        e.inject_alloc_failure(-1)
        e.set_sticking_field(None)
    return True


def test_which_launches_are_ordered(rtg_lib):
    import torch
    from rti_gb300 import Engine
    with Engine(0) as e:
        t = _deep(e)
        g, s = torch.ones(t.n, dtype=torch.float64, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for n, want in (((1 << 21) - 1, False), (1 << 21, True), ((1 << 25) + 1, True)):
            assert _took_room(e, lambda: e.trace(n, 1)) == want, n
            assert _took_room(e, lambda: e.trace(n, 1)) == want, n  # the second time too
        for n, want in (((1 << 21) - 1, False), (1 << 21, True)):
            assert _took_room(e, lambda: e.adjoint_device(g.data_ptr(), 0, n, 1, 0, s.data_ptr())) == want, n
        r = scenes.rough_discs(n=300, spacing=0.01, rms=0.02, corr=0.1, seed=3)  # flat, in the cache
        e.upload_discs(r.points, r.normals, r.radii)
        e.configure(box=(r.box_lo, r.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
        assert not _took_room(e, lambda: e.trace(1 << 22, 1))
        r = scenes.rough_discs(n=1600, spacing=0.01, rms=0.02, corr=0.1, seed=3)  # flat, beyond the cache
        e.upload_discs(r.points, r.normals, r.radii)
        e.configure(box=(r.box_lo, r.box_hi), sticking=0.3, x_bound=1, y_bound=1, reset=True)
        for n, want in (((1 << 20) - 1, False), (1 << 20, True)):
            assert _took_room(e, lambda: e.trace(n, 1)) == want, n
        torch.cuda.synchronize()


def test_fixed_sums_do_not_depend_on_the_order(rtg_lib):
    from rti_gb300 import Engine
    with Engine(0) as e:
        _deep(e)
        e.set_accumulation(1)
        n = (1 << 21) + 77
        out = []
        for ordered in (True, False):
            if ordered:
                e.trace(n, 4)
            else:
                assert _took_room(e, lambda: e.trace(n, 4))
            tally = e.tally()
            out.append((e.values(), e.hit_counts(), [getattr(tally, k) for k in FIELDS]))
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]) and out[0][2] == out[1][2]


def test_a_larger_launch_does_not_wait_for_the_one_before(rtg_lib):
    import torch
    from rti_gb300 import Engine
    with Engine(0) as e:
        t = _deep(e)
        e.configure(sticking=0.02)
        g = torch.ones(t.n, dtype=torch.float64, device="cuda")
        sums = torch.zeros(2, dtype=torch.float64, device="cuda")
        st, done = torch.cuda.Stream(), torch.cuda.Event()
        for call in (lambda n: e.trace(n, 1, stream=st.cuda_stream),
                     lambda n: e.adjoint_device(g.data_ptr(), 0, n, 1, 0, sums.data_ptr(), stream=st.cuda_stream)):
            call(1 << 21)  # the kernels are loaded
            torch.cuda.synchronize()
            call(1 << 23)  # tens of milliseconds
            done.record(st)
            call((1 << 23) + (1 << 20))
            assert not done.query()
            torch.cuda.synchronize()


def test_capture_on_another_stream_goes_on(rtg_lib):
    """A capture in the global mode forbids calls that could wait for the device,
    of which a trace on another stream makes none."""
    import torch
    from rti_gb300 import Engine
    with Engine(0) as e, Engine(0) as f:
        _deep(f)
        f.trace(1 << 21, 1)  # the kernels are loaded
        _deep(e)
        e.synchronize()
        x = torch.zeros(1000, device="cuda")
        side, own = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            graph.capture_begin(capture_error_mode="global")
            x.add_(1.0)
            e.trace(1 << 23, 1, stream=own.cuda_stream)  # its first ordered launch
            x.add_(1.0)
            graph.capture_end()
        torch.cuda.synchronize()
        counts = e.hit_counts()
        e.trace(1 << 23, 1)
        assert np.array_equal(counts, e.hit_counts())
        graph.replay()
        torch.cuda.synchronize()
        assert bool((x == 2.0).all())


def test_room_is_bounded_and_given_back(rtg_lib):
    import torch
    from rti_gb300 import Engine, RtgError
    with Engine(0) as e:
        t = _deep(e)
        e.configure(sticking=1.0)
        g, s = torch.ones(t.n, dtype=torch.float64, device="cuda"), torch.zeros(2, dtype=torch.float64, device="cuda")
        e.trace(1000, 1)
        e.adjoint_device(g.data_ptr(), 0, 1000, 1, 0, s.data_ptr())
        before = _free()
        for n in (1 << 22, 1 << 24, 1 << 25):
            e.trace(n, 1)
            e.adjoint_device(g.data_ptr(), 0, n, 1, 0, s.data_ptr())
        e.synchronize()
        kept = before - _free()
        assert kept <= ROOM + (40 << 20), kept  # the pool's own pages come on top
        # an allocation that fails gives it back first
        e.inject_alloc_failure(0)
        with pytest.raises(RtgError):
            e.set_sticking_field(np.full(t.n, 0.5, np.float32))
        assert before - _free() <= 8 << 20
        e.trace(1 << 22, 1)
        assert e.hit_counts().sum() > 0
    assert _free() >= before


def test_room_of_a_large_launch_goes_back(rtg_lib):
    """2^27 rays are sorted in four pieces and traced by one launch, whose ids take
    512 MB; of these the context keeps no more than of any other launch."""
    from rti_gb300 import Engine
    n = (1 << 27) + 12345
    with Engine(0) as e:
        _deep(e)
        e.configure(sticking=1.0)
        e.trace(1000, 1)
        before = _free()
        e.trace(n, 1)
        got = e.hit_counts(), e.tally().segments
        assert before - _free() <= ROOM + (40 << 20)
        assert _took_room(e, lambda: e.trace(n, 1))
        assert np.array_equal(got[0], e.hit_counts()) and got[1] == e.tally().segments
