"""Measured workloads of the TWoS estimator, each through its public entry point.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call (a mesh session, sites, the request), ``run`` is one call and
its outputs, ``work`` what the call cannot do without, and ``exact`` the same
outputs from plain 64-bit numpy / torch where that is affordable.

Sites and sample keys come from the seed; the meshes are fixed per case (a
program opens a geometry once and sends it many requests), so sessions are
kept in a bounded cache as a serving process keeps them.

The cases:

* field-small     the smallest call a driver makes: a handful of probe sites
                  with the default 16 walks each, plain FP64 form
                  (latency: one launch of a few hundred walks);
* field-mixed     the compiled benchmark's field request (384 evaluation
                  points, default affine source, mixed form, host buffers);
* field-headline  the headline workload's mesh, walks and shell
                  (327,680 triangles, 4,096 walks, eps 1e-4) on a tenth of
                  its sites, device-resident as a training or serving loop
                  holds them;
* field-fp64      the plain FP64 form at an ordinary size;
* adjoint         the paired request of the adjoint studies: housing-like
                  geometry, Gaussian heat sources, sensor, Green point,
                  inserted cavities, 713 scout points;
* gradient        the plain-method configuration (unit sphere, Dirichlet
                  data, 64 sites, 1,024 paired walks, FP64);
* diffwos         derivatives with respect to six cavities (the study's
                  gradient request: 256 points, 1,024 walks);
* certify         certified fresh-sample validation of one candidate at the
                  protocol's 65,536 samples;
* rqmc            Array-RQMC on a 7 x 7 grid of sites;
* closest         bulk closest-point queries (feasibility masks, site
                  costs), an odd number of points;
* design          the on-device design loop (scout, shortlist, validate,
                  insert), two iterations;
* batch           uneven meshes, site and walk counts in one call.

``draw`` varies the same requests over sizes, precisions, sources and meshes.
"""
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "walking-into-holes_b200"))

import twos_b200 as tb  # noqa: E402
from twos_b200 import geometry, sources  # noqa: E402

MAX_STEPS = 4096
ROW_FLOATS = ("u", "p", "score", "score_se", "same_index")
ROW_COUNTS = ("steps", "caps")
CAVITY_RADIUS = 0.065
# Centres of the inserted cavities, used in this order (inside every sphere
# mesh and clear of each other; shifted into the box for the housing mesh).
CAVITIES = np.array([[0.21, 0.05, 0.02], [-0.18, 0.12, 0.08], [0.02, -0.24, -0.05],
                     [-0.05, 0.02, 0.26], [0.12, 0.22, -0.19], [-0.25, -0.15, -0.12]])
BOX_CAVITIES = np.array([[0.9, 0.5, 0.5], [1.7, 1.2, 0.35], [2.6, 0.7, 0.6],
                         [3.3, 1.4, 0.45], [0.4, 1.5, 0.7], [2.1, 1.7, 0.3]])
SPHERE_LEVEL_TRIS = {k: 20 * 4 ** k for k in range(0, 8)}


def listed():
    return [
        {"name": "field-small", "kind": "field", "mesh": "noise", "level": 3, "sites": 16, "walks": 16,
         "precision": "fp64", "source": "affine", "cavities": 0, "epsilon": 5e-4, "device": False},
        {"name": "field-mixed", "kind": "field", "mesh": "noise", "level": 5, "sites": 384, "walks": 256,
         "precision": "mixed", "source": "affine", "cavities": 0, "epsilon": 5e-4, "device": False},
        {"name": "field-headline", "kind": "field", "mesh": "noise", "level": 7, "sites": 12259, "walks": 4096,
         "precision": "mixed", "source": "constant", "cavities": 0, "epsilon": 1e-4, "device": True},
        {"name": "field-fp64", "kind": "field", "mesh": "noise", "level": 6, "sites": 2000, "walks": 512,
         "precision": "fp64", "source": "affine", "cavities": 0, "epsilon": 1e-4, "device": False},
        {"name": "adjoint", "kind": "adjoint", "mesh": "box", "level": 0, "sites": 713, "walks": 768,
         "precision": "mixed", "source": "green", "cavities": 4, "epsilon": 5e-4},
        {"name": "gradient", "kind": "gradient", "mesh": "sphere", "level": 4, "sites": 64, "walks": 1024,
         "precision": "fp64", "epsilon": 1e-4},
        {"name": "diffwos", "kind": "diffwos", "mesh": "noise", "level": 5, "sites": 256, "walks": 1024,
         "precision": "mixed", "cavities": 6, "epsilon": 1e-4, "offset": 0.008},
        {"name": "certify", "kind": "certify", "mesh": "noise", "level": 5, "sites": 1, "walks": 65536,
         "cavities": 0, "green": True},
        {"name": "rqmc", "kind": "rqmc", "mesh": "noise", "level": 4, "sites": 49, "walks": 256, "batches": 8,
         "precision": "fp64", "method": "array", "epsilon": 1e-4},
        {"name": "closest", "kind": "closest", "mesh": "noise", "level": 6, "points": 122591, "precision": "fp64"},
        {"name": "design", "kind": "design", "mesh": "sphere", "level": 4, "sites": 20000, "walks": 256,
         "validate_walks": 4096, "shortlist": 64, "iterations": 2, "precision": "mixed"},
        {"name": "batch", "kind": "batch", "mesh": "noise", "jobs": 8, "sites": 600, "walks": 700, "level": 6,
         "precision": "mixed", "epsilon": 1e-4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field", "field", "field", "adjoint", "adjoint", "gradient", "diffwos", "certify", "rqmc",
                       "closest", "design", "batch"])
    precision = rng.choice(["mixed", "fp64"])
    epsilon = rng.choice([1e-3, 5e-4, 1e-4])
    if kind == "field":
        most = 30_000_000 if precision == "mixed" else 2_000_000
        walks = _log_int(rng, 16, 4096)
        return {"kind": kind, "mesh": rng.choice(["noise", "sphere", "box"]), "level": rng.randint(3, 6),
                "sites": min(_log_int(rng, 7, 12000), max(7, most // walks)), "walks": walks,
                "precision": precision, "source": rng.choice(["constant", "affine"]),
                "cavities": rng.choice([0, 0, 1, 3, 6]), "epsilon": epsilon, "device": rng.random() < 0.5}
    if kind == "adjoint":
        most = 2_000_000 if precision == "mixed" else 400_000
        walks = _log_int(rng, 12, 1024)
        return {"kind": kind, "mesh": rng.choice(["box", "noise"]), "level": rng.randint(3, 6),
                "sites": min(_log_int(rng, 15, 4000), max(15, most // walks)), "walks": walks,
                "precision": precision, "source": rng.choice(["green", "green", "exact", "hot"]),
                "cavities": rng.randint(0, 6), "epsilon": epsilon}
    if kind == "gradient":
        return {"kind": kind, "mesh": "sphere", "level": rng.randint(3, 5), "sites": _log_int(rng, 8, 600),
                "walks": _log_int(rng, 64, 1500), "precision": precision, "epsilon": epsilon}
    if kind == "diffwos":
        return {"kind": kind, "mesh": "noise", "level": rng.randint(3, 6), "sites": _log_int(rng, 5, 400),
                "walks": _log_int(rng, 64, 1024), "precision": precision, "cavities": rng.randint(1, 6),
                "epsilon": rng.choice([5e-4, 1e-4]), "offset": rng.choice([0.004, 0.008, 0.02])}
    if kind == "certify":
        return {"kind": kind, "mesh": "noise", "level": rng.randint(3, 6), "sites": rng.randint(1, 6),
                "walks": _log_int(rng, 1024, 16384), "cavities": rng.randint(0, 4), "green": rng.random() < 0.5}
    if kind == "rqmc":
        return {"kind": kind, "mesh": "noise", "level": rng.randint(3, 5), "sites": _log_int(rng, 5, 120),
                "walks": rng.choice([32, 64, 128, 256, 512, 1024]), "batches": rng.randint(2, 8),
                "precision": precision, "method": rng.choice(["array", "mc", "neighbors", "sobol"]),
                "epsilon": epsilon}
    if kind == "closest":
        return {"kind": kind, "mesh": rng.choice(["noise", "sphere", "box"]), "level": rng.randint(3, 6),
                "points": _log_int(rng, 33, 200_000), "precision": precision}
    if kind == "design":
        most = 4_000_000 if precision == "mixed" else 600_000
        walks = _log_int(rng, 24, 1024)
        return {"kind": kind, "mesh": "sphere", "level": rng.randint(3, 4),
                "sites": min(_log_int(rng, 500, 30000), most // walks), "walks": walks,
                "validate_walks": _log_int(rng, 256, 4096) if precision == "mixed" else _log_int(rng, 256, 1024),
                "shortlist": rng.choice([8, 24, 64]), "iterations": rng.randint(1, 3), "precision": precision}
    return {"kind": "batch", "mesh": "noise", "jobs": rng.randint(2, 10), "sites": _log_int(rng, 50, 800),
            "walks": _log_int(rng, 32, 700) if precision == "mixed" else _log_int(rng, 32, 200),
            "level": rng.randint(4, 6), "precision": precision, "epsilon": epsilon}


# ---------------------------------------------------------------- geometry
@functools.lru_cache(maxsize=16)
def _geometry(mesh, level, shape):
    if mesh == "noise":
        return geometry.noise_sphere(level, shape)
    if mesh == "sphere":
        return geometry.icosphere(level)
    V, F, _ = geometry.box_minus_cylinders(h=0.04)
    return V, F


@functools.lru_cache(maxsize=16)
def _session(mesh, level, shape=1):
    V, F = _geometry(mesh, level, shape)
    return tb.Mesh(V, F)


def _sites(mesh, n, seed, shape=1, margin=0.98):
    """n points uniform in the solid, a little off its surface."""
    if mesh == "box":
        c = geometry.cylinder_centres()
        return np.ascontiguousarray(geometry.box_interior_points(n, c, 0.15, seed))
    p = geometry.uniform_ball(n, margin, seed)
    if mesh == "noise":
        p *= (1.0 + 0.15 * geometry.sh_field(p, shape))[:, None]
    return np.ascontiguousarray(p)


def _cavities(case):
    n = case.get("cavities", 0)
    return (BOX_CAVITIES if case["mesh"] == "box" else CAVITIES)[:n].copy() if n else None


def _outside(p, cav, gap):
    keep = np.ones(len(p), bool)
    for c in cav if cav is not None else ():
        keep &= np.linalg.norm(p - c, axis=1) > CAVITY_RADIUS + gap
    return p[keep]


def _heat(mesh):
    if mesh == "box":
        return sources.study_heat([(0.6, 0.5, 0.4, 0.35, 3.0), (1.2, 1.5, 0.6, 0.4, 2.0), (2.4, 1.0, 0.3, 0.3, 2.5)])
    return sources.study_heat([(-0.3, 0.1, 0.0, 0.25, 3.0), (0.2, 0.3, -0.1, 0.3, 2.0), (0.1, -0.3, 0.2, 0.2, 2.5)])


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    cav = _cavities(case)
    state = {"kind": kind, "case": case}
    if kind == "batch":
        meshes, sites, cfgs = [], [], []
        for j in range(case["jobs"]):
            level = 3 + j % (case["level"] - 2)  # 3 .. level, uneven meshes side by side
            shape = 2 + j % 3
            n = max(1, int(case["sites"] * 2.0 ** ((5 * j % 7) / 3.0 - 1.0)))  # half to twice the sites
            meshes.append(_session("noise", level, shape))
            sites.append(_sites("noise", n, seed + j, shape, margin=0.9))  # clear of the coarse chords
            cfgs.append(tb.Config(walks=max(2, int(case["walks"] * 2.0 ** (j % 3 - 1))), precision=case["precision"],
                                  seed=seed + j, epsilon=case["epsilon"], max_steps=MAX_STEPS,
                                  source=sources.constant(1.0)))
        state.update(meshes=meshes, sites=sites, cfgs=cfgs)
        return state
    mesh = _session(case["mesh"], case["level"])
    state["mesh"] = mesh
    if kind == "field":
        state["sites"] = _sites(case["mesh"], case["sites"], seed)
        state["cavities"] = cav
        state["config"] = tb.Config(walks=case["walks"], precision=case["precision"], seed=seed,
                                    epsilon=case["epsilon"], max_steps=MAX_STEPS, cavity_radius=CAVITY_RADIUS,
                                    source=sources.affine() if case["source"] == "affine" else sources.constant(1.0))
        if case["device"]:
            state["d_sites"] = torch.from_numpy(state["sites"]).cuda()
            state["d_rows"] = torch.empty((case["sites"], 7), dtype=torch.float64, device="cuda")
    elif kind == "adjoint":
        hot = case["source"] == "hot"
        exact_source = case["source"] == "exact"
        sensor = (3.2, 1.0, 0.5) if case["mesh"] == "box" else (0.35, 0.18, -0.03)
        state["sites"] = _sites(case["mesh"], case["sites"], seed)
        state["cavities"] = cav
        state["config"] = tb.Config(walks=case["walks"], mode="hot" if hot else "paired",
                                    precision=case["precision"], seed=seed, epsilon=case["epsilon"],
                                    max_steps=MAX_STEPS, cavity_radius=CAVITY_RADIUS,
                                    green="exact" if exact_source else True,
                                    source=_heat(case["mesh"]) if exact_source else sources.housing(),
                                    adjoint=[] if hot else sources.normalized_sensor(sensor, 0.13))
    elif kind == "gradient":
        state["sites"] = geometry.uniform_ball(case["sites"], 0.9, seed)
        state["config"] = tb.Config(walks=case["walks"], mode="paired", precision=case["precision"], seed=seed,
                                    epsilon=case["epsilon"], max_steps=MAX_STEPS, green=True, source=[],
                                    adjoint=sources.ball_mean_density((0.0, 0.0, 0.0), 0.5),
                                    boundary=sources.quadratic((1.0, -1.0, 0.0)) + sources.linear(0.5, 2))
    elif kind == "diffwos":
        p = _outside(_sites("noise", 2 * case["sites"] + 64, seed, margin=0.7), cav, 0.02)
        state["sites"] = np.ascontiguousarray(p[: case["sites"]])
        state["cavities"] = cav
        state["config"] = tb.Config(walks=case["walks"], precision=case["precision"], seed=seed,
                                    epsilon=case["epsilon"], max_steps=MAX_STEPS, cavity_radius=CAVITY_RADIUS,
                                    source=sources.affine())
    elif kind == "certify":
        p = _outside(_sites("noise", 4 * case["sites"] + 32, seed, margin=0.7), cav, 0.02)
        state["sites"] = np.ascontiguousarray(p[: case["sites"]])
        state["cavities"] = cav
        state["config"] = tb.Config(walks=case["walks"], precision="fp64", seed=seed, epsilon=1e-6, max_steps=128,
                                    cavity_radius=CAVITY_RADIUS, green=bool(case["green"]), source=sources.affine())
    elif kind == "rqmc":
        state["sites"] = _sites("noise", case["sites"], seed, margin=0.8)
        state["config"] = tb.Config(walks=case["walks"], precision=case["precision"], seed=seed,
                                    epsilon=case["epsilon"], max_steps=MAX_STEPS, source=[])
        state["u_boundary"] = sources.quadratic((1.0, -1.0, 0.0)) + sources.linear(0.5, 2)
        state["p_boundary"] = sources.linear(1.0, 0, 1.5)
    elif kind == "closest":
        # Points of the solid and of the space around it.
        V, _ = _geometry(case["mesh"], case["level"], 1)
        lo, hi = V.min(0), V.max(0)
        rng = np.random.default_rng(seed)
        state["points"] = lo + (hi - lo) * (rng.random((case["points"], 3)) * 1.2 - 0.1)
    elif kind == "design":
        common = dict(precision=case["precision"], seed=seed, epsilon=1e-4, max_steps=MAX_STEPS,
                      source=sources.constant(1.0))
        state["candidates"] = geometry.uniform_ball(case["sites"], 0.85, seed)
        state["scout"] = tb.Config(walks=case["walks"], stream=0, **common)
        state["validate"] = tb.Config(walks=case["validate_walks"], stream=1, **common)
    return state


def _fields(rows, floats, counts):
    out = {k: np.ascontiguousarray(rows[k]) for k in floats}
    out.update({k: rows[k].astype(np.int64) for k in counts})
    return out


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "field" and case["device"]:
        state["mesh"].estimate_device(state["d_sites"], case["sites"], state["d_rows"], state["config"],
                                      cavities=state["cavities"])
        return {"values": state["d_rows"][:, :5], "counts": state["d_rows"][:, 5:].view(torch.int64)}
    if kind in ("field", "adjoint"):
        rows, _ = state["mesh"].estimate(state["sites"], state["config"], cavities=state["cavities"])
        return _fields(rows, ROW_FLOATS, ROW_COUNTS)
    if kind == "gradient":
        rows, _ = state["mesh"].estimate_gradient(state["sites"], state["config"])
        return _fields(rows, ("u", "p", "grad_u", "grad_p", "cross", "cross_se", "u_se", "p_se"), ROW_COUNTS)
    if kind == "diffwos":
        rows, stats, _ = state["mesh"].diffwos(state["sites"], state["config"], state["cavities"],
                                               diff_offset=case["offset"], strict=False)
        return {"rows": _fields(rows, ("dc", "dc_se", "dR", "dR_se"), ()),
                "stats": _fields(stats, (), stats.dtype.names)}
    if kind == "certify":
        samples, stages, _ = state["mesh"].validate(state["sites"], state["config"], cavities=state["cavities"],
                                                    radius_cap=0.1, value_cap=0.2, strict=False)
        return {"samples": _fields(samples, ("value",), ("steps", "capped", "clipped", "contained")),
                "stages": _fields(stages, ("mean", "mean_steps", "center_clearance_lower", "center_distance"),
                                  ("n", "clipped", "path_caps"))}
    if kind == "rqmc":
        bu, bp, td, _ = state["mesh"].rqmc(state["sites"], state["config"], state["u_boundary"], state["p_boundary"],
                                           method=case["method"], batches=case["batches"])
        return {"batch_u": bu, "batch_p": bp, "td": td}
    if kind == "closest":
        dist, point = state["mesh"].closest_point(state["points"], precision=case["precision"])
        return {"distance": dist, "point": point}
    if kind == "design":
        history, cavities, _ = state["mesh"].design_loop(
            state["candidates"], state["scout"], state["validate"], iterations=case["iterations"],
            shortlist=case["shortlist"], cavity_radius=0.03, z=1.96, accept_threshold=0.02, outer_clearance=0.02,
            pair_gap=0.01)
        return {"history": _fields(history, ("scout_score", "score", "score_se", "lower"),
                                   ("chosen", "accepted", "slot", "n_cavities")),
                "cavities": np.concatenate([cavities, np.zeros((case["iterations"] - len(cavities), 3))])}
    outs, _ = tb.estimate_batch(state["meshes"], state["sites"], state["cfgs"])
    return {k: np.concatenate([o[k].astype(np.int64) if k in ROW_COUNTS else o[k] for o in outs])
            for k in ROW_FLOATS + ROW_COUNTS}


# ---------------------------------------------------------------- work
# A walk-on-spheres step cannot do without its random direction, its radius
# from one triangle's distance, the move and the payoff: about 150 flops.  A
# walk takes about 4 + 2.2 ln(1 / eps) steps in these solids.
STEP_FLOPS = 150.0


def _tris(case):
    return {"box": 43412}.get(case["mesh"]) or SPHERE_LEVEL_TRIS[case["level"]]


def _steps(epsilon):
    return 4.0 + 2.2 * math.log(1.0 / epsilon)


def work(case):
    kind = case["kind"]
    if kind == "closest":
        n = case["points"]
        return {"bytes": 24.0 * n + 32.0 * n + 18.0 * _tris(case), "flops": 60.0 * n}
    if kind == "certify":
        walks = case["sites"] * case["walks"]
        return {"bytes": 16.0 * walks + 18.0 * _tris(case), "flops": walks * 50.0 * STEP_FLOPS}
    if kind == "design":
        walks = case["iterations"] * (case["sites"] * case["walks"] + case["shortlist"] * case["validate_walks"])
        return {"bytes": 24.0 * case["sites"] + 18.0 * _tris(case), "flops": walks * _steps(1e-4) * STEP_FLOPS}
    if kind == "batch":
        walks = 1.5 * case["jobs"] * case["sites"] * case["walks"]
        return {"bytes": 80.0 * case["jobs"] * case["sites"], "flops": walks * _steps(case["epsilon"]) * STEP_FLOPS}
    walks = case["sites"] * case["walks"] * case.get("batches", 1)
    row = {"field": 56, "adjoint": 56, "gradient": 112, "diffwos": 64 * case.get("cavities", 0) + 56, "rqmc": 24}[kind]
    return {"bytes": case["sites"] * (24.0 + row) + 18.0 * _tris(case),
            "flops": walks * _steps(case["epsilon"]) * STEP_FLOPS}


# ---------------------------------------------------------------- exact
def _closest_brute(points, V, F):
    """(distance, closest point) of each point to the triangle soup, FP64, by
    testing every triangle: the interior projection where it falls inside,
    else the nearest of the three clamped edges."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    P = torch.from_numpy(np.ascontiguousarray(points)).to(dev)
    T = torch.from_numpy(V[F.astype(np.int64)]).to(dev)
    a, b, c = T[:, 0], T[:, 1], T[:, 2]
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1)
    inv = torch.where(nn > 0, 1.0 / nn, torch.zeros_like(nn))
    edges = [(a, b - a), (b, c - b), (c, a - c)]
    inner = [torch.linalg.cross(n, e) for _, e in edges]
    inv_e = [1.0 / (e * e).sum(1).clamp_min(1e-300) for _, e in edges]
    dist2 = torch.empty(len(P), dtype=torch.float64, device=dev)
    which = torch.empty(len(P), dtype=torch.int64, device=dev)
    step = max(1, int(4e7 // len(T)))
    for i in range(0, len(P), step):
        p = P[i:i + step]
        inside = torch.ones((len(p), len(T)), dtype=torch.bool, device=dev)
        best = torch.full((len(p), len(T)), math.inf, dtype=torch.float64, device=dev)
        for (o, e), m, ie in zip(edges, inner, inv_e):
            inside &= (p @ m.T - (o * m).sum(1)) >= 0
            t = ((p @ e.T - (o * e).sum(1)) * ie).clamp_(0.0, 1.0)
            d2 = torch.zeros_like(t)
            for k in range(3):
                d2 += (p[:, k:k + 1] - o[:, k] - t * e[:, k]) ** 2
            best = torch.minimum(best, d2)
        h = p @ n.T - (a * n).sum(1)
        best = torch.where(inside, h * h * inv, best)
        dist2[i:i + step], which[i:i + step] = best.min(1)
    # The winning triangle again, without the expanded dot products' rounding.
    a, b, c = T[which, 0], T[which, 1], T[which, 2]
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1, keepdim=True)
    q = P - n * (((P - a) * n).sum(1, keepdim=True) / nn.clamp_min(1e-300))
    inside = (nn > 0).squeeze(1)
    near, near2 = a.clone(), ((P - a) ** 2).sum(1)
    for o, e in ((a, b - a), (b, c - b), (c, a - c)):
        inside &= ((q - o) * torch.linalg.cross(n, e)).sum(1) >= 0
        t = (((P - o) * e).sum(1) / (e * e).sum(1).clamp_min(1e-300)).clamp(0.0, 1.0)
        x = o + t[:, None] * e
        d2 = ((P - x) ** 2).sum(1)
        closer = d2 < near2
        near[closer], near2[closer] = x[closer], d2[closer]
    q = torch.where(inside[:, None], q, near)
    return ((P - q) ** 2).sum(1).sqrt().cpu().numpy(), q.cpu().numpy()


def _philox(k0, k1, c0, c1, c2, c3):
    """Philox4x32-10 (Salmon et al. 2011) on uint64 arrays holding 32-bit words."""
    m = np.uint64(0xFFFFFFFF)
    s = np.uint64(32)
    c = [np.asarray(v, np.uint64) for v in np.broadcast_arrays(c0, c1, c2, c3)]
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> s) ^ c[1] ^ np.uint64(k0), p1 & m, (p0 >> s) ^ c[3] ^ np.uint64(k1), p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _key(seed, stream):
    """SplitMix64 of seed + golden * (stream + 1): the request's sample key."""
    M, g = (1 << 64) - 1, 0x9E3779B97F4A7C15
    x = (seed + g * (stream + 1) + g) & M
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M
    x ^= x >> 31
    return x & 0xFFFFFFFF, x >> 32


def _exact_field(case, seed):
    """The plain FP64 field request walked in numpy: compliance walks with
    the request's counter stream, distances by testing every triangle."""
    V, F = _geometry(case["mesh"], case["level"], 1)
    cav = _cavities(case)
    sites, walks = _sites(case["mesh"], case["sites"], seed), case["walks"]
    k0, k1 = _key(seed, 0)
    n = len(sites) * walks
    site, walk = np.divmod(np.arange(n), walks)
    pos = sites[site].copy()
    u, steps = np.zeros(n), np.zeros(n, np.int64)
    live = np.arange(n)
    while len(live):
        if np.all(steps[live] == 0):
            d = _closest_brute(sites, V, F)[0][site[live]]
        else:
            d = _closest_brute(pos[live], V, F)[0]
        for c in cav if cav is not None else ():
            d = np.minimum(d, np.sqrt(((pos[live] - c) ** 2).sum(1)) - CAVITY_RADIUS)
        go = d > case["epsilon"]
        live, r = live[go], d[go]
        if not len(live):
            break
        f = 1.0 + 0.65 * (pos[live, 1] + 0.5) if case["source"] == "affine" else 1.0
        u[live] += r * r / 6.0 * f
        x, y, z, w = _philox(k0, k1, steps[live].astype(np.uint64), walk[live].astype(np.uint64),
                             site[live].astype(np.uint64), np.uint64(0))
        a = (((x << np.uint64(32)) | y) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
        b = (((z << np.uint64(32)) | w) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
        cz = 1.0 - 2.0 * a
        rad = np.sqrt(np.maximum(0.0, 1.0 - cz * cz))
        pos[live] += r[:, None] * np.stack([rad * np.cos(2 * np.pi * b), rad * np.sin(2 * np.pi * b), cz], 1)
        steps[live] += 1
        if steps[live].max() >= MAX_STEPS:
            return None
    U = u.reshape(len(sites), walks)
    N = float(walks)
    s1, s2 = U.sum(1), (U * U).sum(1)
    leave = ((s1[:, None] - U) ** 2 - (s2[:, None] - U * U)) / ((N - 1) * (N - 2))
    se = np.sqrt((N - 1) / N * ((leave - leave.mean(1, keepdims=True)) ** 2).sum(1))
    rows = {"u": s1 / N, "p": s1 / N, "score": (s1 * s1 - s2) / (N * (N - 1)), "score_se": se, "same_index": s2 / N}
    if case["device"]:
        return {"values": np.stack([rows[k] for k in ROW_FLOATS], 1), "counts": None}
    return {**rows, "steps": None, "caps": None}


def exact(case, seed):
    if case["kind"] == "closest":
        if case["points"] * _tris(case) > 1.2e10:
            return None
        V, F = _geometry(case["mesh"], case["level"], 1)
        dist, point = _closest_brute(prepare(case, seed)["points"], V, F)
        return {"distance": dist, "point": point}
    if case["kind"] == "field" and case["precision"] == "fp64":
        if case["sites"] * case["walks"] * float(_tris(case)) > 4e8:
            return None
        return _exact_field(case, seed)
    return None
