"""Where a closest-point query's bounds are tight: candidate lists that do and
do not fit, and the limits of the searches."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tb(lib_built):
    import twos_b200
    return twos_b200


def _fan(n):
    """A closed double cone: n triangles meet at each apex."""
    t = 2 * np.pi * np.arange(n) / n
    V = np.concatenate([np.c_[np.cos(t), np.sin(t), np.zeros(n)], [[0, 0, 0.5], [0, 0, -0.5]]])
    i = np.arange(n)
    j = (i + 1) % n
    return V, np.concatenate([np.c_[i, j, np.full(n, n)], np.c_[j, i, np.full(n, n + 1)]]).astype(np.uint32)


@pytest.mark.parametrize("shape", ["fan4", "sphere3", "noise5", "sliver", "fan64"])
def test_cells_near_the_surface_have_candidate_lists(tb, monkeypatch, shape):
    """The grid's cells near the surface have candidate lists -- a list holds
    its entry node, one triangle at least and its end, 32 entries at most --
    except where the candidates are too many (around the apex of 64
    triangles), and a session without a grid has none."""
    if shape.startswith("fan"):
        V, F = _fan(int(shape[3:]))
    elif shape == "sliver":
        V, F = tb.geometry.icosphere(4)
        V = V * np.array([1.0, 0.05, 1.0])
    else:
        V, F = tb.geometry.icosphere(3) if shape == "sphere3" else tb.geometry.noise_sphere(5, 2)
    with tb.Mesh(V, F) as m:
        n = m.candidate_lists()
    assert 0 < n["listed_cells"] <= n["near_cells"]
    assert 3 * n["listed_cells"] <= n["entries"] <= 32 * n["listed_cells"]
    if shape == "fan64":
        assert n["listed_cells"] < n["near_cells"]
    monkeypatch.setenv("TWOS_GRID_VERTICES", "0")
    with tb.Mesh(V, F) as m:
        assert set(m.candidate_lists().values()) == {0}


def test_every_open_builds_the_same_lists(tb):
    """The lists' places in memory are taken in any order; their number and
    the walks that read them are the same at every open, and those of queries
    that start at the root."""
    V, F = tb.geometry.noise_sphere(5, 2)
    P = tb.geometry.uniform_ball(60, 0.7, seed=3)
    cfg = tb.Config(walks=200, precision="mixed", seed=5, epsilon=1e-4, max_steps=4096, source=tb.sources.affine())
    seen = []
    for entry in (1, 1, 0):
        with tb.Mesh(V, F) as m:
            m.set_tuning(**dict(m.get_tuning(), entry=entry))
            seen.append((m.candidate_lists(), m.estimate(P, cfg)[0]))
    for n, rows in seen[1:]:
        assert n == seen[0][0]
        np.testing.assert_array_equal(rows, seen[0][1])


@pytest.mark.parametrize("level,jitter", [(1, 0.0), (3, 0.0), (4, 1e-9), (5, 0.0)])
def test_many_nearly_equidistant_triangles_at_once(tb, level, jitter):
    """Points at and beside the centre of a sphere, among others: the number of
    triangles within rounding of the minimum goes from one to far beyond what
    a warp replays, from point to point of one warp.  Every point gets what a
    lane's traversal gives it, alone and among others."""
    V, F = tb.geometry.icosphere(level)
    rng = np.random.default_rng(level)
    P = rng.uniform(-0.3, 0.3, (12000, 3))
    P[::3] = jitter * rng.normal(size=(4000, 3))
    with tb.Mesh(V, F) as m:
        d, q = m.closest_point(np.tile(P, (2, 1)), precision="mixed")  # a lane per point
        dw, qw = m.closest_point(P, precision="mixed")  # a warp per point
        one = [m.closest_point(P[i:i + 1], precision="mixed") for i in (0, 1, 3)]
    assert np.array_equal(d[: len(P)], d[len(P):]) and np.array_equal(d[: len(P)], dw)
    assert np.array_equal(q[: len(P)], qw)
    for i, (di, qi) in zip((0, 1, 3), one):
        assert di[0] == dw[i] and np.array_equal(qi[0], qw[i])


def _cube(n):
    """A rotated cube of half extent about 1, each face n x n squares of two triangles."""
    g = np.linspace(-1.0, 1.0, n + 1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).ravel()
    quads = np.stack([a, a + n + 1, a + n + 2, a + 1], 1)
    V, F = [], []
    for axis in range(3):
        for side in (-1.0, 1.0):
            P = np.zeros((n + 1, n + 1, 3))
            P[..., axis] = side
            P[..., (axis + 1) % 3], P[..., (axis + 2) % 3] = g[:, None], g[None, :]
            q = quads if side > 0 else quads[:, ::-1]
            F.append(np.concatenate([q[:, [0, 1, 2]], q[:, [0, 2, 3]]]) + sum(len(v) for v in V))
            V.append(P.reshape(-1, 3))
    R = np.linalg.qr(np.array([[0.8, 0.3, 0.5], [-0.4, 0.9, 0.1], [-0.4, -0.2, 0.9]]))[0]
    return np.concatenate(V) @ R.T * 0.6, np.concatenate(F).astype(np.uint32)


@pytest.mark.parametrize("shape", ["cube8", "cube60", "sphere4", "graded"])
@pytest.mark.parametrize("query_radius", [0.0, 300.0])
def test_mixed_queries_far_from_the_mesh(tb, shape, query_radius):
    """FP32 bounds lose more to rounding the farther the point is: what a warp
    returns for a point (a small call, a site's first query) stays what a
    lane's traversal returns, from the surface to 10^4 half extents away."""
    if shape.startswith("cube"):
        V, F = _cube(int(shape[4:]))
    else:
        V, F = tb.geometry.icosphere(4)
        if shape == "graded":  # triangles down to 1e-6 of the extent, in a plane
            V = V * 10.0 ** np.clip(6.0 * (V[:, 2:] - 1.0) / 2.0, -6.0, 0.0)
    rng = np.random.default_rng(6)
    out = rng.normal(size=(6000, 3))
    out /= np.linalg.norm(out, axis=1)[:, None]
    on = V[F[rng.integers(0, len(F), 6000)].astype(np.int64)].mean(1)  # far along the faces' own normals, too
    n = np.cross(V[F[:, 1]] - V[F[:, 0]], V[F[:, 2]] - V[F[:, 0]])
    n = n[rng.integers(0, len(n), 6000)]
    n /= np.linalg.norm(n, axis=1)[:, None]
    far = 10.0 ** rng.uniform(-1.0, 4.0, (6000, 1))
    P = np.concatenate([out * far, on + n * far, out * 2.0 ** rng.integers(0, 14, (6000, 1))])
    with tb.Mesh(V, F) as m:
        d, q = m.closest_point(P, precision="mixed", query_radius=query_radius)  # a lane per point
        parts = [m.closest_point(p, precision="mixed", query_radius=query_radius) for p in np.split(P, 6)]
        delta = np.float32(m.info()["mixed_delta"])
        cfg = tb.Config(walks=2, precision="mixed", seed=3, epsilon=1e-30, max_steps=1, query_radius=None,
                        source=tb.sources.constant(6.0))
        got = m.walk_samples(P, cfg)["u"][:, 0].astype(np.float32) if query_radius == 0.0 else None
    dw, qw = (np.concatenate(x) for x in zip(*parts))  # a warp per point
    if query_radius == 0.0:
        assert np.all(np.isfinite(d)) and np.all(np.isfinite(q))
    np.testing.assert_array_equal(dw, d)
    np.testing.assert_array_equal(qw, q)
    if got is not None:
        r = d.astype(np.float32) - delta
        want = np.where(r > np.float32(1e-30), (r * r / np.float32(6)) * np.float32(6), np.float32(0))
        np.testing.assert_array_equal(got, want)


@pytest.fixture(scope="module")
def deep():
    """A closed cone whose rings shrink by a constant factor towards the apex:
    a BVH of the deepest level the builder allows, 24, all of whose levels hold
    a stack entry when an unbounded search reaches the leaf nearest to many
    points (0.2 of those below the apex, 0.1 of those in the cone)."""
    S, R = 32, 800
    r = 1e-8 ** (np.arange(R + 1) / R)
    t = 2 * np.pi * np.arange(S) / S
    V = np.concatenate([np.c_[x * np.cos(t), x * np.sin(t), np.full(S, x)] for x in r] + [[[0, 0, 1], [0, 0, r[-1]]]])
    a = (np.arange(R)[:, None] * S + np.arange(S)).ravel()
    b = (np.arange(R)[:, None] * S + (np.arange(S) + 1) % S).ravel()
    i, j = np.arange(S), (np.arange(S) + 1) % S
    F = [np.c_[a, b, b + S], np.c_[a, b + S, a + S], np.c_[np.full(S, (R + 1) * S), j, i],
         np.c_[np.full(S, (R + 1) * S + 1), R * S + i, R * S + j]]
    rng = np.random.default_rng(1)
    z = 10.0 ** rng.uniform(-8.0, 0.0, (10000, 1))
    inner = np.c_[rng.uniform(-0.6, 0.6, (10000, 2)) * z, z]
    z = 10.0 ** rng.uniform(-3.0, 1.0, (10000, 1))
    outer = np.c_[rng.uniform(-0.5, 0.5, (10000, 2)) * z, -z]
    return V, np.concatenate(F).astype(np.uint32), inner, outer


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("grid", [True, False])
def test_searches_of_the_deepest_hierarchy(tb, deep, monkeypatch, precision, grid):
    """A leaf at depth 24 with an entry held at every level is within the stack:
    closest points (a lane per point against a warp per point) and RQMC, with
    and without the grid's bounds."""
    V, F, inner, outer = deep
    if not grid:
        monkeypatch.setenv("TWOS_GRID_VERTICES", "0")
    cfg = tb.Config(walks=64, precision=precision, seed=2, epsilon=1e-5 if precision == "mixed" else 1e-12,
                    max_steps=4096, source=tb.sources.constant(1.0))
    with tb.Mesh(V, F) as m:
        assert m.info()["bvh_depth"] == 24
        P = np.concatenate([inner, outer])
        d = m.closest_point(P, precision=precision, with_points=False)
        assert np.array_equal(d, np.concatenate([m.closest_point(p, precision=precision, with_points=False)
                                                 for p in np.split(P, 2)]))
        bu, _, _, _ = m.rqmc(inner[:200], cfg, tb.sources.constant(0.0), tb.sources.constant(0.0), method="mc", batches=2)
        assert np.all(np.isfinite(bu))


@pytest.mark.parametrize("grid", [True, False])
def test_certified_searches_of_the_deepest_hierarchy(tb, deep, monkeypatch, grid):
    """Certified walks in the same cone, with and without the grid's bounds."""
    V, F, inner, _ = deep
    if not grid:
        monkeypatch.setenv("TWOS_GRID_VERTICES", "0")
    cfg = tb.Config(walks=64, precision="fp64", seed=2, epsilon=1e-9, max_steps=8, source=tb.sources.constant(1.0))
    with tb.Mesh(V, F) as m:
        sites = inner[m.inside(inner)][:64]
        s, st, _ = m.validate(sites, cfg, radius_cap=1e3, value_cap=1e9, strict=False)
    assert len(sites) == 64 and np.all(s["contained"] == 1)
    assert np.all(s["steps"][st["center_clearance_lower"][:, 0] > 1e-9] > 0)


def test_a_certified_first_distance_that_overruns_is_zero(tb, monkeypatch):
    """A search that gives up certifies nothing: a site whose first distance
    overruns the iteration bound (the centre of a sphere, equidistant to all of
    it; the bound lowered to a hundredth of the visits) has clearance 0, its
    walks take no step, and the call reports the overrun."""
    V, F = tb.geometry.icosphere(5)
    monkeypatch.setenv("TWOS_MAX_ITERATIONS", "200")
    req = tb.Config(walks=64, precision="fp64", seed=2, epsilon=1e-6, max_steps=32,
                    source=tb.sources.constant(1.0)).to_request()
    site = np.zeros((1, 3))
    abi = tb._abi
    samples = np.zeros((1, 64), dtype=abi.CERT_SAMPLE_DTYPE)
    stages = np.zeros((1, abi.VALIDATE_MAX_STAGES), dtype=abi.VALIDATE_STAGE_DTYPE)
    params, n, summ = abi.ValidateParams(0.1, 10.0), ctypes.c_uint32(), abi.Summary()
    with tb.Mesh(V, F) as m:
        rc = abi.load().twos_validate(m._h, ctypes.byref(req), ctypes.byref(params), site.ctypes.data, 1, None, 0,
                                      samples.ctypes.data, stages.ctypes.data, ctypes.byref(n), ctypes.byref(summ))
    assert rc != abi.OK and summ.error_flags & abi.DEVERR_ITER
    assert n.value >= 1 and stages["center_clearance_lower"][0, 0] == 0.0
    assert np.all(samples["steps"] == 0) and np.all(samples["value"] == 0.0)


@pytest.mark.parametrize("radius_cap", [0.02, 0.3])
def test_certified_walks_among_more_boxes_than_a_query_holds(tb, oracle_mod, radius_cap):
    """Around an apex where 64 triangles meet, a query's candidates are tested
    several times before it ends: the oracle's steps and flags exactly, its
    values to the parity tests' 1e-10."""
    V, F = _fan(64)
    sites = np.array([[0.0, 0.0, 0.45], [0.01, 0.0, -0.4], [0.02, -0.03, 0.2]])
    common = dict(walks=200, seed=9, epsilon=1e-6, max_steps=96, cavity_radius=0.05)
    cfg = tb.Config(precision="fp64", green=True, source=tb.sources.constant(1.0), **common)
    with tb.Mesh(V, F) as m:
        s, st, _ = m.validate(sites, cfg, radius_cap=radius_cap, value_cap=0.2, strict=False)
    o = oracle_mod.OracleMesh(V, F).validate(sites, radius_cap, 0.2, rng=oracle_mod.RNG_COUNTER, green=True,
                                             source=[oracle_mod.term(oracle_mod.TERM_CONST, 1.0)], **common)
    for k in ("steps", "capped", "clipped", "contained"):
        assert np.array_equal(s[k].astype(o[k].dtype), o[k]), k
    np.testing.assert_allclose(s["value"], o["value"], rtol=1e-10, atol=0)
    assert np.array_equal(st["center_clearance_lower"][:, 0], o["clearance"])


@pytest.mark.parametrize("k", [30, 34, 37])
@pytest.mark.parametrize("level", [1, 4])
def test_a_scaled_mesh_gives_scaled_results(tb, monkeypatch, level, k):
    """A power of two times every length is a power of two times every FP64
    distance and estimate, bit for bit, and leaves the steps alone, also where
    FP32 has no room for the products of the closest-point arithmetic.  The
    mixed form's distances there are those of a session without a grid."""
    V, F = tb.geometry.icosphere(level)
    rng = np.random.default_rng(level)
    P = rng.uniform(-0.9, 0.9, (20000, 3))
    sites = 0.5 * rng.uniform(-1, 1, (24, 3))
    cav = np.array([[0.3, 0.1, 0.0], [-0.4, 0.2, 0.1]])
    got = []
    for a in (1.0, 2.0 ** k):
        cfg = tb.Config(walks=100, precision="fp64", seed=7, epsilon=1e-4 * a, max_steps=4096, cavity_radius=0.1 * a,
                        query_radius=None, source=tb.sources.constant(1.0))
        with tb.Mesh(V * a, F) as m:
            d = [m.closest_point(p * a, precision="fp64", with_points=False) / a for p in (P, P[:500])]
            rows, _ = m.estimate(sites * a, cfg, cavities=cav * a)
            f = [m.closest_point(p * a, precision="mixed", with_points=False) for p in (P, P[:500])]
        got.append((*d, rows["u"] / a**2, rows["steps"]))
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)
    monkeypatch.setenv("TWOS_GRID_VERTICES", "0")
    with tb.Mesh(V * a, F) as m:
        for x, p in zip(f, (P, P[:500])):
            np.testing.assert_array_equal(x, m.closest_point(p * a, precision="mixed", with_points=False))


@pytest.mark.parametrize("k", [-38, -34, -32, -28])
@pytest.mark.parametrize("level", [1, 3])
@pytest.mark.parametrize("cavities", [False, True])
def test_a_small_mesh_gives_scaled_results(tb, level, k, cavities):
    """The same where the products of the closest-point arithmetic are below
    FP32's normal numbers and the grid's values far off: no search depends
    on its upper bound, and no cavity is taken for nearer than the surface."""
    V, F = tb.geometry.icosphere(level)
    rng = np.random.default_rng(level)
    P = rng.uniform(-0.9, 0.9, (20000, 3))
    sites = 0.5 * rng.uniform(-1, 1, (200, 3))
    cav = np.array([[0.3, 0.1, 0.0], [-0.4, 0.2, 0.1], [0.7, 0.1, 0.1], [-0.1, -0.75, 0.0]]) if cavities else np.zeros((0, 3))
    got = []
    for a in (1.0, 2.0 ** k):
        cfg = tb.Config(walks=100, precision="fp64", seed=7, epsilon=1e-4 * a, max_steps=4096, query_radius=None,
                        cavity_radius=0.1 * a, source=tb.sources.constant(1.0))
        with tb.Mesh(V * a, F) as m:
            d = [m.closest_point(p * a, precision="fp64", with_points=False) / a for p in (P, P[:500])]
            rows, _ = m.estimate(sites * a, cfg, cavities=cav * a)
        got.append((*d, rows["u"] / a**2, rows["steps"]))
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_walks_between_needles(tb, monkeypatch, precision):
    """A cylinder of 3,000 segments: triangles a thousand times longer than
    high, whose FP32 distances at the grid's vertices can be below those at
    the points of a walk.  Every query is answered; the FP64 samples, and all
    closest points, are those without the grid.  (Without it a mixed walk can
    run out of the solid on such triangles.)"""
    n = 3000
    t = 2 * np.pi * np.arange(n) / n
    V = np.concatenate([np.c_[np.cos(t), np.sin(t), np.full(n, -1.0)], np.c_[np.cos(t), np.sin(t), np.full(n, 1.0)],
                        [[0, 0, -1], [0, 0, 1]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    F = np.concatenate([np.c_[i, j, j + n], np.c_[i, j + n, i + n], np.c_[j, i, np.full(n, 2 * n)],
                        np.c_[i + n, j + n, np.full(n, 2 * n + 1)]]).astype(np.uint32)
    R = np.linalg.qr(np.random.default_rng(3).normal(size=(3, 3)))[0]
    rng = np.random.default_rng(6)
    S, P = rng.uniform(-0.5, 0.5, (200, 3)) @ R.T, rng.uniform(-1.3, 1.3, (20000, 3)) @ R.T
    cfg = tb.Config(epsilon=1e-4, max_steps=2000, query_radius=None, walks=64, precision=precision, seed=7,
                    source=tb.sources.constant(1.0))
    got = []
    for grid in (True, False):
        if not grid:
            monkeypatch.setenv("TWOS_GRID_VERTICES", "0")
        with tb.Mesh(V @ R.T, F) as m:
            got.append((m.closest_point(P, precision=precision, with_points=False),
                        m.closest_point(P[:4000], precision=precision, with_points=False),
                        m.walk_samples(S, cfg) if grid or precision == "fp64" else None))
    for x, y in zip(got[0][:2], got[1][:2]):
        np.testing.assert_array_equal(x, y)
    if precision == "fp64":
        for key in got[0][2]:
            np.testing.assert_array_equal(got[0][2][key], got[1][2][key])


@pytest.mark.parametrize("shape", ["cube1", "cube8", "sphere3", "noise4"])
def test_of_equidistant_triangles_the_same_one_is_met(tb, shape):
    """Points of a lattice (on planes of symmetry and edges' normals) and at
    random: the FP64 closest point is the one of a search of the FP64 nodes,
    which a mesh beyond FP32's range takes -- to the bit in a call with few
    points, but for the rounding of points on a common edge in a bulk call."""
    if shape.startswith("cube"):
        n = int(shape[4:])
        V, F = _cube(n)  # its triangles, on the axes again
        g = np.linspace(-1.0, 1.0, n + 1)
        u, v = np.meshgrid(g, g, indexing="ij")
        V = np.concatenate([np.roll(np.stack([np.full_like(u, side), u, v], -1).reshape(-1, 3), axis, axis=1)
                            for axis in range(3) for side in (-1.0, 1.0)])
    else:
        V, F = tb.geometry.icosphere(3) if shape == "sphere3" else tb.geometry.noise_sphere(4, 1)
    t = np.linspace(-1.5, 1.5, 25)
    P = np.stack(np.meshgrid(t, t, t), -1).reshape(-1, 3)
    P = np.concatenate([P, np.random.default_rng(1).uniform(-1.5, 1.5, (4000, 3))])
    a = 2.0 ** 41
    with tb.Mesh(V, F) as m, tb.Mesh(V * a, F) as far:
        d, q = far.closest_point(P * a, precision="fp64")
        small = [m.closest_point(p, precision="fp64") for p in np.array_split(P, 2)]
        bulk = m.closest_point(P, precision="fp64")
    assert len(P) > 16384
    np.testing.assert_array_equal(np.concatenate([x[0] for x in small]), d / a)
    np.testing.assert_array_equal(np.concatenate([x[1] for x in small]), q / a)
    np.testing.assert_array_equal(bulk[0], d / a)
    np.testing.assert_allclose(bulk[1], q / a, rtol=0, atol=2.0 ** -47)


@pytest.mark.parametrize("n", [12000, 20000])
@pytest.mark.parametrize("distance", [1e4, 1e6])
def test_a_far_point_takes_no_longer_than_without_fp32(tb, n, distance):
    """FP32 prunes less the farther a point is: a call with far points takes at
    most twice what it takes for a mesh beyond FP32's range, which is searched
    by the FP64 nodes, and gives its distances."""
    V, F = tb.geometry.noise_sphere(5, 1)
    P = np.random.default_rng(2).normal(size=(n, 3))
    P *= distance / np.linalg.norm(P, axis=1)[:, None]
    got = []
    for a in (1.0, 2.0 ** 41):
        with tb.Mesh(V * a, F) as m:
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                d = m.closest_point(P * a, precision="fp64", with_points=False) / a
                t.append(time.perf_counter() - t0)
        got.append((min(t), d))
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][0] < 2 * got[1][0]


@pytest.mark.parametrize("offset", [1e5, 1e8, 1e9])
def test_a_mesh_far_from_the_origin_is_searched_like_one_at_it(tb, offset):
    """Coordinates a hundred thousand to a billion half extents from the
    origin: candidate lists, and the FP64 distances and estimates of the FP64
    nodes (which the same mesh beyond FP32's range takes)."""
    V, F = tb.geometry.noise_sphere(4, 1)
    V = V + offset * np.array([1.0, -0.7, 0.4])
    rng = np.random.default_rng(5)
    o = V.mean(0)
    P, sites, cav = o + rng.uniform(-1.2, 1.2, (20000, 3)), o + rng.uniform(-0.4, 0.4, (40, 3)), o + np.array([[0.3, 0.1, 0.0], [-0.4, 0.2, 0.1]])
    got = []
    for a in (1.0, 2.0 ** 41):
        cfg = tb.Config(walks=100, precision="fp64", seed=7, epsilon=1e-4 * a, max_steps=4096, cavity_radius=0.1 * a,
                        query_radius=None, source=tb.sources.constant(1.0))
        with tb.Mesh(V * a, F) as m:
            assert (m.candidate_lists()["listed_cells"] > 0) == (a == 1.0)
            d = [m.closest_point(p * a, precision="fp64", with_points=False) / a for p in (P, P[:500])]
            rows = [m.estimate(sites * a, cfg, cavities=c)[0] for c in (None, cav * a)]
        got.append((*d, *(r["u"] / a**2 for r in rows), *(r["steps"] for r in rows)))
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)
