"""The calls that a user of the flux engine makes, at the sizes they are made.

Every case is one pass through the package's public entry points, as a process
simulator or a calibration loop calls them.  A case names its kind of call:

  device_run  the drop-in call: host arrays in, normalised estimates and hit
              counts out, a context of its own (rti::device::run);
  step        a kept engine takes the surface of a new time step, traces it and
              reads the estimates and hit counts;
  trace       the surface stays, another trace reads the flux and the counts
              (deposit "window": the multi-hit window; accum "fixed": the
              bit-reproducible sums);
  move        the surface moved (same primitives): refit, trace, read;
  rays        closest hits of explicit rays;
  grad        differentiable flux: trace and adjoint replay of a weighted flux,
              with respect to one sticking and the source exponent, or (field)
              to one sticking value per disc;
  batch       ragged trenches and holes, three species each, one batched run.

Surfaces: "trench" (discs on a grid: top, walls, bottom of an extruded trench),
"hole_discs", "hole" (triangle mesh of a cylindrical hole) and "rough" (discs on
a Gaussian height field, one per grid point), each of about `n` primitives.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rti_gb300 import Engine, device_run, scenes
from rti_gb300 import _lib as L
from rti_gb300.autograd import flux
from rti_gb300.batch import Batch

SPECIES = scenes.BATCH_SPECIES  # (sticking, source exponent) of the batched workload
WINDOW = 5.0                    # rti's window length in radii


def _case(name, kind, surface, n, rays, *, aspect=5.0, sticking=0.1, exponent=1.0, reflection="diffuse",
          specular=0.0, bounds="periodic", deposit="neighbors", accum="fp64", tree="karras", field=False, noise=0.0,
          surfaces=1):
    c = {"kind": kind, "surface": surface, "n": n, "rays": rays, "aspect": aspect, "sticking": sticking,
         "exponent": exponent, "reflection": reflection, "specular": specular, "bounds": bounds, "deposit": deposit,
         "accum": accum, "tree": tree, "field": field, "noise": noise, "surfaces": surfaces}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a first try of the drop-in header: rti's default 1024 rays, reflective box, a coarse trench
        _case("run_small", "device_run", "trench", 1500, 1024, aspect=3.0, sticking=0.2, bounds="reflective"),
        # one time step of a feature-scale simulation: 98,301-disc trench, 1e6 rays
        _case("step_trench", "step", "trench", 98_301, 1_000_000),
        # the same step on a triangle mesh (the 200,192-triangle hole) with mixed re-emission
        _case("step_hole", "step", "hole", 200_192, 1_000_000, aspect=10.0, sticking=0.01, reflection="mixed",
              specular=0.1),
        # the benchmark's headline trace: 1e7 rays into the deep hole over the clustered tree
        _case("trace_hole", "trace", "hole", 200_192, 10_000_000, aspect=10.0, sticking=0.01, reflection="mixed",
              specular=0.1, tree="ploc"),
        # directional ions on a disc-sampled hole: cos^50 source, specular walls, reproducible sums
        _case("trace_ions", "trace", "hole_discs", 61_000, 3_000_017, aspect=4.0, sticking=0.5, exponent=50.0,
              reflection="specular", bounds="reflective", accum="fixed", noise=0.01),
        # rti's multi-hit window deposit on a trench
        _case("trace_window", "trace", "trench", 25_000, 300_007, deposit="window", noise=0.01),
        # a wafer-scale rough surface with a sticking value per disc (2048 x 2048 discs, beyond the L2 cache)
        _case("trace_rough", "trace", "rough", 2048 * 2048, 20_000_000, sticking=0.12, field=True, tree="ploc"),
        # a surface advanced by a small step: refit, then few rays
        _case("move_rough", "move", "rough", 301 * 301, 200_003, sticking=0.3),
        # visibility queries from outside the tracer: explicit rays against a mesh
        _case("rays_hole", "rays", "hole", 31_000, 262_144, aspect=4.0),
        # calibration of one sticking value and the source exponent
        _case("grad_hole", "grad", "hole", 200_192, 1_000_000, aspect=10.0, sticking=0.01, reflection="mixed",
              specular=0.1, tree="ploc"),
        # calibration of a sticking field
        _case("grad_field", "grad", "rough", 512 * 512, 1_000_000, sticking=0.12, field=True),
        # several features and species of one step in one launch
        _case("batch_ragged", "batch", "ragged", 100_000, 200_000, aspect=8.0, surfaces=6),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["device_run", "step", "step", "trace", "trace", "trace", "move", "rays", "grad", "batch"])
    if kind == "batch":
        return _case(None, kind, "ragged", logint(10_000, 150_000), logint(20_000, 300_000),
                     aspect=round(rng.uniform(2.0, 14.0), 2), surfaces=rng.randint(2, 7))
    surface = rng.choice(["trench", "hole_discs", "rough"] if kind == "device_run" else
                         ["trench", "hole_discs", "hole", "rough"])
    n = logint(1000, 400_000)
    rays = logint(1000, 100_000) if kind == "device_run" else logint(3000, 3_000_000)
    reflection = rng.choice(["diffuse", "diffuse", "specular", "mixed"])
    field = surface == "rough" and rng.random() < 0.5 and kind in ("trace", "grad")
    window = kind == "trace" and surface != "hole" and rng.random() < 0.2
    if window:
        n, rays = min(n, 100_000), min(rays, 500_000)
    c = _case(None, kind, surface, n, rays, aspect=round(rng.uniform(1.0, 12.0), 2),
              sticking=round(math.exp(rng.uniform(math.log(0.01), 0.0)), 4),
              exponent=rng.choice([1.0, 1.0, 5.0, 50.0]), reflection=reflection,
              specular=round(rng.uniform(0.05, 0.9), 3) if reflection == "mixed" else 0.0,
              bounds=rng.choice(["periodic", "reflective"]), deposit="window" if window else "neighbors",
              accum="fixed" if kind in ("step", "trace") and rng.random() < 0.3 else "fp64",
              tree=rng.choice(["karras", "ploc"]) if kind in ("step", "trace", "grad") else "karras", field=field,
              noise=rng.choice([0.0, 0.01, 0.05]))
    if kind == "rays":
        c["rays"] = min(rays, 1_000_000)
    return c


# ---- surfaces -------------------------------------------------------------


def _hole_mesh(n, aspect, seed):
    """The triangle hole of radius 0.5 in a 2 x 2 cell with about n triangles and
    1 % vertex jitter: rings of the top from the rim to the square border, the
    wall, the bottom with a centre fan (right-handed, normals into the open)."""
    rng = np.random.default_rng(seed)
    depth = float(aspect)
    # 512 x (24 top + 160 wall + 12 bottom rings) at aspect 10 is the benchmark's mesh
    scale = math.sqrt(n / 200_192 / ((24 + 12 + 16 * depth) / 196.0))
    n_th = max(16, 8 * int(round(512 * scale / 8)))
    n_top, n_wall, n_bot = (max(2, int(round(k * scale))) for k in (24, 16 * depth, 12))
    th = np.arange(n_th) * (2 * math.pi / n_th)

    def ring_angles(rows):
        return th[None, :] + 0.01 * (2 * math.pi / n_th) * rng.uniform(-1, 1, (rows, n_th))

    f = (np.arange(1, n_top) / n_top)[:, None] + 0.01 / n_top * rng.uniform(-1, 1, (n_top - 1, n_th))
    a = np.concatenate([th[None], ring_angles(n_top - 1), th[None]])
    f = np.concatenate([np.zeros((1, n_th)), f, np.ones((1, n_th))])
    m = np.maximum(np.abs(np.cos(a)), np.abs(np.sin(a)))
    top = np.stack([np.cos(a) * (0.5 + f * (1.0 / m - 0.5)), np.sin(a) * (0.5 + f * (1.0 / m - 0.5)),
                    np.zeros_like(a)], -1)
    dz = depth / n_wall
    z = -dz * np.arange(1, n_wall + 1)[:, None] + np.zeros((1, n_th))
    a = np.concatenate([ring_angles(n_wall - 1), th[None]])
    z[:-1] += 0.01 * dz * rng.uniform(-1, 1, (n_wall - 1, n_th))
    wall = np.stack([0.5 * np.cos(a), 0.5 * np.sin(a), z], -1)
    dr = 0.5 / n_bot
    a = ring_angles(n_bot - 1)
    r = 0.5 - dr * np.arange(1, n_bot)[:, None] + 0.01 * dr * rng.uniform(-1, 1, (n_bot - 1, n_th))
    bot = np.stack([r * np.cos(a), r * np.sin(a), np.full_like(r, -depth)], -1)
    v = np.concatenate([top.reshape(-1, 3), wall.reshape(-1, 3), bot.reshape(-1, 3), [[0.0, 0.0, -depth]]])

    def quads(inner, outer):  # rows of vertex ids -> two triangles per quad
        i1, o1 = np.roll(inner, -1, -1), np.roll(outer, -1, -1)
        return [np.stack([inner, outer, o1], -1).reshape(-1, 3), np.stack([inner, o1, i1], -1).reshape(-1, 3)]

    ids = np.arange(len(v))
    top_i = ids[:(n_top + 1) * n_th].reshape(n_top + 1, n_th)
    wall_i = np.concatenate([top_i[:1], ids[top_i.size:top_i.size + n_wall * n_th].reshape(n_wall, n_th)])
    bot_i = np.concatenate([wall_i[-1:], ids[top_i.size + n_wall * n_th:-1].reshape(n_bot - 1, n_th)])
    t = quads(top_i[:-1], top_i[1:])
    t += [q[:, ::-1] for q in quads(wall_i[:-1], wall_i[1:])]
    t += quads(bot_i[1:], bot_i[:-1])
    t.append(np.stack([bot_i[-1], np.roll(bot_i[-1], -1), np.full(n_th, len(v) - 1)], -1))
    return {"vertices": v.astype(np.float32), "indices": np.concatenate(t).astype(np.uint32),
            "box": ((-1.0, -1.0, -depth), (1.0, 1.0, 0.1))}


def _rough(n, seed):
    """About n discs (a square grid, spacing 0.01) on a periodic Gaussian height
    field of rms 0.05 and correlation length 0.2."""
    m, s = max(8, int(round(math.sqrt(n)))), 0.01
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.fft.fftfreq(m, d=s, device="cuda", dtype=torch.float64) * (2 * math.pi)
    spec = torch.exp(-(k[:, None] ** 2 + k[None, :] ** 2) * (0.2 ** 2 / 8.0))
    h = torch.fft.ifft2(torch.fft.fft2(torch.randn(m, m, generator=g, device="cuda", dtype=torch.float64))
                        * spec.sqrt()).real
    h = h * (0.05 / h.std())
    gx = (torch.roll(h, -1, 0) - torch.roll(h, 1, 0)) / (2 * s)
    gy = (torch.roll(h, -1, 1) - torch.roll(h, 1, 1)) / (2 * s)
    nrm = torch.nn.functional.normalize(torch.stack([-gx, -gy, torch.ones_like(h)], -1), dim=-1)
    x = torch.arange(m, device="cuda", dtype=torch.float64) * s
    p = torch.stack([x[:, None].expand(m, m), x[None, :].expand(m, m), h], -1)
    p, nrm = p.reshape(-1, 3).float().cpu().numpy(), nrm.reshape(-1, 3).float().cpu().numpy()
    z = p[:, 2]
    return _discs(p, nrm, s, ((-s / 2, -s / 2, float(z.min())), (m * s - s / 2, m * s - s / 2, float(z.max()) + 0.1)))


def _discs(p, nrm, spacing, box):
    return {"points": p, "normals": nrm, "radii": np.full(len(p), spacing * math.sqrt(0.5), dtype=np.float32),
            "box": box}


def _feature(case, seed):
    """A disc-sampled trench (3 x 3 cell, width 1) or hole (2 x 2 cell, diameter 1)
    of depth `aspect`; noise moves the discs along their normals by that share
    of the spacing, as a level set's surface points do."""
    ar = case["aspect"]
    if case["surface"] == "trench":
        m = max(6, int(round(3.0 / math.sqrt(3.0 * (3.0 + 2.0 * ar) / case["n"]))))
        s = 3.0 / m
        surf = scenes.trench_discs(width=1.0, depth=ar, domain=3.0, spacing=s)
    else:
        m = max(8, int(round(2.0 / math.sqrt((4.0 + math.pi * ar) / case["n"]))))
        s = 2.0 / m
        surf = scenes.hole_discs(radius=0.5, depth=ar, cell=2.0, spacing=s)
    off = np.random.default_rng(seed).uniform(-1, 1, (surf.n, 1)) * case["noise"] * s
    return _discs((surf.points + off * surf.normals).astype(np.float32), surf.normals, s, (surf.box_lo, surf.box_hi))


def _surface(case, seed):
    if case["surface"] == "hole":
        return _hole_mesh(case["n"], case["aspect"], seed)
    if case["surface"] == "rough":
        return _rough(case["n"], seed)
    return _feature(case, seed)


def _upload(e, s):
    if "vertices" in s:
        e.upload_triangles(s["vertices"], s["indices"])
    else:
        e.upload_discs(s["points"], s["normals"], s["radii"])


def _settings(case, box):
    b = L.RTG_BOUND_PERIODIC if case["bounds"] == "periodic" else L.RTG_BOUND_REFLECTIVE
    return {"x_bound": b, "y_bound": b, "sticking": case["sticking"], "source_exponent": case["exponent"],
            "reflection": {"diffuse": L.RTG_REFLECT_DIFFUSE, "specular": L.RTG_REFLECT_SPECULAR,
                           "mixed": L.RTG_REFLECT_MIXED}[case["reflection"]],
            "specular_fraction": case["specular"], "box": box}


def _engine(case):
    e = Engine(0)
    if case["tree"] == "ploc":
        e.set_tree_builder(L.RTG_TREE_PLOC)
    if case["accum"] == "fixed":
        e.set_accumulation(L.RTG_ACCUM_FIXED)
    if case["deposit"] == "window":
        e.set_deposit_mode(L.RTG_DEPOSIT_WINDOW, WINDOW)
    return e


def _field(case, seed, n):
    """Sticking values per disc, log-normal odds around the case's sticking."""
    x = np.random.default_rng(seed + 1).normal(math.log(case["sticking"] / (1.001 - case["sticking"])), 0.5, n)
    return (1.0 / (1.0 + np.exp(-x))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind, "seed": int(seed), "rays": case["rays"]}
    if kind == "batch":
        rng = np.random.default_rng(case["surfaces"])  # the features' sizes are the case's, the rest the seed's
        st["batch"], st["engines"] = Batch(0), []
        for i in range(case["surfaces"]):
            one = dict(case, surface="trench" if i % 2 == 0 else "hole_discs",
                       n=case["n"] * rng.uniform(0.3, 1.7), aspect=max(1.0, case["aspect"] * rng.uniform(0.4, 1.6)))
            s = _feature(one, seed + i)
            e = _engine(case)
            _upload(e, s)
            e.configure(**_settings(case, s["box"]))
            st["engines"].append(e)
            for sticking, exponent in SPECIES:
                c = e.config()
                c.sticking, c.source_exponent = sticking, exponent
                st["batch"].add(e, case["rays"], seed=int(seed), config=c)
        return st
    s = _surface(case, seed)
    if kind == "device_run":
        cfg = L.RtgConfig()
        L.load().rtg_config_default(cfg)
        for k, v in _settings(case, s["box"]).items():
            if k != "box":
                setattr(cfg, k, v)
        cfg.box_mode = L.RTG_BOX_EXPLICIT
        cfg.box_lo[:], cfg.box_hi[:] = s["box"]
        st["surface"], st["config"] = s, cfg
        return st
    e = _engine(case)
    st["engine"] = e
    if kind == "step":
        st["surface"], st["settings"] = s, _settings(case, s["box"])
        return st
    if kind == "move":  # the engine holds the surface before the step, `surface` is the one after it
        st["surface"] = dict(s, points=s["points"] + 0.002 * s["normals"]) if "points" in s else \
            dict(s, vertices=s["vertices"] * np.float32(1.001))
    _upload(e, s)
    e.configure(**_settings(case, s["box"]))
    n = e.num_primitives
    if kind == "rays":
        # from points between the top and the bottom, in all directions
        rng = np.random.default_rng(seed + 1)
        lo, hi = np.asarray(s["box"][0]), np.asarray(s["box"][1])
        d = rng.normal(size=(case["rays"], 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        o = lo + (hi - lo) * rng.uniform(0, 1, (case["rays"], 3))
        st["query"] = np.concatenate([o, d], 1).astype(np.float32)
    elif kind == "grad":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        st["weights"] = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        st["sticking"] = torch.from_numpy(_field(case, seed, n)).cuda() if case["field"] else \
            torch.tensor(case["sticking"], dtype=torch.float64)
    elif case["field"]:
        e.set_sticking_field(_field(case, seed, n))
    return st


# ---- one pass -------------------------------------------------------------


def run(st):
    kind = st["kind"]
    if kind == "device_run":
        s = st["surface"]
        return device_run(s["points"], s["normals"], s["radii"], n_rays=st["rays"], seed=st["seed"],
                          config=st["config"])
    if kind == "batch":
        b = st["batch"]
        b.run()
        b.synchronize()
        return [b.results(j) for j in range(len(b))]
    e = st["engine"]
    if kind == "step":
        _upload(e, st["surface"])
        e.configure(**st["settings"])
        e.trace(st["rays"], seed=st["seed"])
        return e.mc_estimates(), e.hit_counts()
    if kind == "trace":
        e.trace(st["rays"], seed=st["seed"])
        return e.values(), e.hit_counts().view(np.int64)  # as torch takes them
    if kind == "move":
        s = st["surface"]
        if "vertices" in s:
            e.update_vertices(s["vertices"])
        else:
            e.update_discs(s["points"], s["normals"], s["radii"])
        e.trace(st["rays"], seed=st["seed"])
        return e.mc_estimates(), e.hit_counts()
    if kind == "rays":
        return e.trace_rays(st["query"])
    s = st["sticking"].detach().requires_grad_(True)
    x = torch.tensor(st["case"]["exponent"], dtype=torch.float64, requires_grad=True)
    s1 = flux(e, s, x, st["rays"], seed=st["seed"])
    (st["weights"] * s1).sum().backward()
    return s1.detach(), s.grad, x.grad


# ---- what a pass cannot do without ------------------------------------------


def _segments(case, sticking):
    """Closest-hit queries per source ray: the query that misses or sticks last
    and the bounces before it, about 0.7 of the aspect ratio in a feature whose
    walls hardly stick (rays that meet the top leave after one)."""
    depth = 0.5 if case["surface"] == "rough" else 0.7 * case["aspect"]
    return 2.0 + (1.0 - sticking) * depth


def work(case):
    n, rays, kind = case["n"], case["rays"], case["kind"]
    levels = max(1.0, math.log2(max(2, n)))
    geometry = 18 if case["surface"] == "hole" else 28  # (vertices and indices) or (centre, normal, radius)
    # per query: two slab tests of a binary tree's path to one leaf and the primitive's test
    query = 2 * 17 * levels + 45
    if kind == "rays":
        return {"bytes": geometry * n + rays * (24 + 8), "flops": rays * query}
    if kind == "batch":
        surfaces = case["surfaces"]
        segs = sum(_segments(case, s) for s, _ in SPECIES)
        return {"bytes": surfaces * n * (geometry + 3 * 20.0), "flops": surfaces * rays * segs * (query + 150)}
    out = {"device_run": 12, "step": 12, "move": 12, "trace": 16, "grad": 16}[kind]
    segs = _segments(case, case["sticking"]) * (2 if kind == "grad" else 1)
    return {"bytes": n * (geometry + out + (4 if case["field"] else 0)), "flops": rays * segs * (query + 150)}


# ---- 64-bit values --------------------------------------------------------


def exact(case, seed):
    """Distances of explicit rays to the closest primitive, in 64 bits, by
    testing every primitive.  The other kinds return Monte Carlo sums over paths
    of float32 decisions, which have no 64-bit counterpart."""
    if case["kind"] != "rays" or case["rays"] * case["n"] > 3e10:
        return None
    s = _surface(case, seed)
    rng = np.random.default_rng(seed + 1)
    lo, hi = np.asarray(s["box"][0]), np.asarray(s["box"][1])
    d = rng.normal(size=(case["rays"], 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = lo + (hi - lo) * rng.uniform(0, 1, (case["rays"], 3))
    q = torch.from_numpy(np.concatenate([o, d], 1).astype(np.float32)).cuda().double()
    best = torch.full((len(q),), math.inf, dtype=torch.float64, device="cuda")
    if "vertices" in s:
        v = torch.from_numpy(s["vertices"]).cuda().double()
        i = torch.from_numpy(s["indices"].astype(np.int64)).cuda()
        a = v[i[:, 0]]
        e1, e2 = v[i[:, 1]] - a, v[i[:, 2]] - a
        nn = torch.linalg.cross(e1, e2)
    else:
        a = torch.from_numpy(s["points"]).cuda().double()
        nn = torch.from_numpy(s["normals"]).cuda().double()
        r2 = torch.from_numpy(s["radii"]).cuda().double() ** 2
    an = (a * nn).sum(1)
    step = max(1, int(6e7) // len(q))
    oo, dd = q[:, :3], q[:, 3:]
    for b in range(0, len(a), step):
        p = slice(b, b + step)
        dn = dd @ nn[p].T
        t = (an[p] - oo @ nn[p].T) / dn
        if "vertices" in s:
            # barycentric weights from the moment o x d: (o - a).(d x e2) and d.((o - a) x e1) over -d.n
            m = torch.linalg.cross(oo, dd)
            w1 = torch.linalg.cross(e2[p], a[p])
            w2 = torch.linalg.cross(a[p], e1[p])
            u = (dd @ w1.T - m @ e2[p].T) / dn
            w = (m @ e1[p].T + dd @ w2.T) / dn
            ok = (u >= 0) & (w >= 0) & (u + w <= 1)
        else:
            # |o + t d - c|^2
            oc = (oo ** 2).sum(1)[:, None] - 2 * (oo @ a[p].T) + (a[p] ** 2).sum(1)
            dc = (oo * dd).sum(1)[:, None] - dd @ a[p].T
            ok = oc + 2 * t * dc + t * t * (dd ** 2).sum(1)[:, None] <= r2[p]
        ok &= t > 1e-4
        best = torch.minimum(best, torch.where(ok, t, math.inf).amin(1))
    return None, torch.where(torch.isinf(best), 0.0, best)
