"""The order in which a batch's launch takes its jobs (long paths first) and the
areas that jobs of one surface and box share: stickings up, down and mixed, a
sticking field, an empty job, boxes that differ, with and without a graph.

Results belong to the job as it was added: counts equal the oracle's with the
job's stream, areas those of a single context, without a tolerance."""
import numpy as np
import pytest

from rti_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True], ids=["launch", "graph"])
@pytest.mark.parametrize("sticking", [(0.9, 0.4, 0.1, 0.05), (0.05, 0.1, 0.4, 0.9), (0.4, 0.05, 0.9, 0.4)])
@pytest.mark.parametrize("field", [False, True], ids=["global", "field"])
def test_results_belong_to_the_job(rtg_lib, oracle_lib, sticking, graph, field):
    from rti_gb300 import Engine
    from rti_gb300.batch import Batch
    surf = [scenes.trench_discs(domain=1.2, width=0.4, depth=d) for d in (0.5, 1.5)]
    engines, b, jobs = [], Batch(0), []
    try:
        for t in surf:
            e = Engine(0)
            e.upload_discs(t.points, t.normals, t.radii)
            e.configure(box=(t.box_lo, t.box_hi), x_bound=1, y_bound=1, reset=True)
            engines.append(e)
        sf = None
        if field:
            sf = np.random.default_rng(0).uniform(0.1, 0.6, surf[1].n).astype(np.float32)
            engines[1].set_sticking_field(sf)
        for k, st in enumerate(sticking):
            for i, e in enumerate(engines):
                c = e.config()
                c.sticking = st
                rays = 0 if (k, i) == (2, 0) else 4000 + 1000 * k + i
                jobs.append((b.add(e, rays, seed=11, config=c), i, st, rays))
        b.run(use_graph=graph)
        b.synchronize()
        b.run(use_graph=graph)  # a second run zeroes and traces again
        b.synchronize()
        for j, i, st, rays in jobs:
            t = surf[i]
            _, cnt, areas = b.results(j)
            s = oracle_lib.Scene(t.xyzr, t.normals)
            s.neighbors()
            cfg = oracle_lib.make_config(t.box_lo, t.box_hi, sticking=st, seed=11, job=j)
            assert np.array_equal(cnt, s.trace(cfg, 0, rays, sticking_field=sf if i == 1 else None).counts), j
            assert np.array_equal(areas, engines[i].exposed_areas()), j
    finally:
        b.close()
        for e in engines:
            e.close()
