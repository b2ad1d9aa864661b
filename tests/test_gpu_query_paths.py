"""The closest-point query's paths against each other: FP64 queries that prune
in FP32 against those that take the FP64 nodes, and walks spread over few or
all lanes of a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tb(lib_built):
    import twos_b200
    return twos_b200


def _fan(n):
    """A closed double cone: n triangles meet at each apex (more than an FP64
    query holds as candidates)."""
    t = 2 * np.pi * np.arange(n) / n
    V = np.concatenate([np.c_[np.cos(t), np.sin(t), np.zeros(n)], [[0, 0, 0.5], [0, 0, -0.5]]])
    i = np.arange(n)
    j = (i + 1) % n
    return V, np.concatenate([np.c_[i, j, np.full(n, n)], np.c_[j, i, np.full(n, n + 1)]]).astype(np.uint32)


def _points(V, F, seed):
    rng = np.random.default_rng(seed)
    lo, hi = V.min(0), V.max(0)
    on = V[rng.integers(0, len(V), 40)]
    mid = V[F[rng.integers(0, len(F), 40)].astype(np.int64)].sum(1) / 3.0  # triangle centroids
    return np.concatenate([lo + (hi - lo) * rng.random((300, 3)), on * (1 + 1e-9), on, on * 3.0, mid,
                           V.mean(0, keepdims=True), rng.normal(size=(20, 3)) * 1e3])


@pytest.mark.parametrize("shape", ["sphere", "noise", "fan5", "fan64", "sliver"])
@pytest.mark.parametrize("exponent", [-60, 60])
def test_fp32_pruning_gives_the_fp64_minimum(tb, shape, exponent):
    """Scaling by a power of two is exact in FP64, so a mesh too small or too
    large for FP32 pruning (which takes the FP64 nodes) has exactly the scaled
    distances of the original, which prunes in FP32."""
    if shape == "sphere":
        V, F = tb.geometry.icosphere(3)
    elif shape == "noise":
        V, F = tb.geometry.noise_sphere(4, 2)
    elif shape == "sliver":  # needle triangles, aspect 1e-7
        V, F = tb.geometry.icosphere(2)
        V = V * np.array([1.0, 1e-7, 1.0])
    else:
        V, F = _fan(int(shape[3:]))
    P = _points(V, F, 3)
    s = 2.0 ** exponent
    with tb.Mesh(V, F) as a, tb.Mesh(V * s, F) as b:
        da, qa = a.closest_point(P, precision="fp64")
        db, qb = b.closest_point(P * s, precision="fp64")
    assert np.array_equal(da * s, db)
    # The nearest point is unique up to rounding except on the medial axis.
    assert np.max(np.abs(np.linalg.norm(P - qa, axis=1) - da)) <= 4e-16 * 2e3
    assert np.max(np.abs(np.linalg.norm(P * s - qb, axis=1) - db)) <= 4e-16 * 2e3 * s


@pytest.mark.parametrize("offset", [0.0, 1e4, 1e8])
def test_far_points_and_offset_meshes(tb, offset):
    """Points beyond FP32 squares and meshes far from the origin keep their
    FP64 distances (against every triangle's vertices and faces in numpy: the
    sphere's nearest point is a vertex or inside a face, within its sagitta)."""
    V, F = tb.geometry.icosphere(3)
    d = np.array([[1.0, 2.0, -2.0], [0.3, -0.1, 0.95]]) / np.array([[3.0], [1.0]])
    P = np.concatenate([d[:1] * r for r in (2.0, 1e6, 2.0 ** 40, 2.0 ** 55, 1e25)] + [d[1:] * 0.4])
    with tb.Mesh(V + offset, F) as m:
        dist, _ = m.closest_point(P + offset, precision="fp64")
    T = V[F.astype(np.int64)]
    upper = np.min(np.linalg.norm(P[:, None] - V[None], axis=2), axis=1)  # nearest vertex
    n = np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    n /= np.linalg.norm(n, axis=1)[:, None]
    lower = np.maximum(np.linalg.norm(P, axis=1) - 1.0, 0.0)  # outside the unit ball
    scale = 1e-15 * (np.linalg.norm(P, axis=1) + 4 * offset + 1)
    assert np.all(dist <= upper + scale) and np.all(dist >= lower - scale)
    inner = np.min(np.einsum("fk,fk->f", n, T[:, 0]) - P[-1] @ n.T)
    assert abs(dist[-1] - inner) <= 1e-15 * (4 * offset + 4)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_walks_do_not_depend_on_the_lanes_that_run_them(tb, precision):
    """One site per launch (2 to 700 walks: one lane per warp) and all sites in
    one launch (up to all 32 lanes) walk the same samples."""
    V, F = tb.geometry.noise_sphere(3, 1)
    sites = tb.geometry.uniform_ball(200, 0.6, seed=4)
    with tb.Mesh(V, F) as m:
        for walks in (2, 33, 700):
            cfg = tb.Config(walks=walks, precision=precision, seed=6, epsilon=1e-3)
            every = m.walk_samples(sites, cfg)
            for s in (0, 17, 199):
                one = m.walk_samples(sites[s], tb.Config(walks=walks, precision=precision, seed=6, epsilon=1e-3,
                                                         site_offset=s))
                assert np.array_equal(one["u"][0], every["u"][s])
                assert np.array_equal(one["steps"][0], every["steps"][s])


@pytest.mark.parametrize("radius_cap", [0.02, 0.1, 1e3])
@pytest.mark.parametrize("epsilon,n_cav,walks,offset", [(1e-6, 0, 300, 0.0), (1e-6, 2, 33, 0.0), (0.12, 1, 64, 0.0),
                                                        (1e-6, 1, 64, 4e6)])
def test_certified_walks_equal_the_oracle(tb, oracle_mod, radius_cap, epsilon, n_cav, walks, offset):
    """Certified walks over radius caps that skip no query, some and nearly all
    of them, shells up to beyond radius_cap / 0.95, cavities, a site near the
    surface, and a mesh too far from the origin for FP32 pruning: the oracle's
    steps and flags exactly, its values to the parity tests' 1e-10."""
    V, F = tb.geometry.noise_sphere(3, 1)
    V = V + offset
    sites = np.array([[0.05, -0.1, 0.2], [0.3, 0.2, -0.1], [0.0, 0.0, 0.7]]) + offset
    cav = np.array([[-0.2, 0.1, 0.0], [0.1, -0.3, 0.1]])[:n_cav] + offset
    common = dict(walks=walks, seed=8, epsilon=epsilon, max_steps=96, cavity_radius=0.065)
    cfg = tb.Config(precision="fp64", green=True, source=tb.sources.constant(1.0), **common)
    with tb.Mesh(V, F) as m:
        s, st, _ = m.validate(sites, cfg, cavities=cav if n_cav else None, radius_cap=radius_cap, value_cap=0.2,
                              strict=False)
    o = oracle_mod.OracleMesh(V, F).validate(
        sites, radius_cap, 0.2, cavities=cav if n_cav else None, rng=oracle_mod.RNG_COUNTER, green=True,
        source=[oracle_mod.term(oracle_mod.TERM_CONST, 1.0)], **common)
    for k in ("steps", "capped", "clipped", "contained"):
        assert np.array_equal(s[k].astype(o[k].dtype), o[k]), k
    np.testing.assert_allclose(s["value"], o["value"], rtol=1e-10, atol=0)
    assert np.array_equal(st["center_clearance_lower"][:, 0], o["clearance"])


@pytest.mark.parametrize("level,query_radius", [(1, 4.0), (5, 4.0), (5, None), (3, 0.97)])
def test_first_queries_among_equidistant_triangles(tb, oracle_mod, level, query_radius):
    """The centre of a sphere is (nearly) equidistant to every triangle, so the
    warp's common stack fills up: the walks from it and from points beside it
    are the oracle's.  With a query radius below the distance, every walk
    fails the same way."""
    V, F = tb.geometry.icosphere(level)
    sites = np.array([[0.0, 0.0, 0.0], [1e-9, 0.0, 0.0], [0.01, -0.02, 0.015], [0.5, 0.1, -0.2]])
    cfg = tb.Config(walks=20, precision="fp64", seed=12, epsilon=1e-4, source=tb.sources.constant(1.0),
                    query_radius=query_radius)
    with tb.Mesh(V, F) as m:
        if query_radius is not None and query_radius < 1.0:
            with pytest.raises(tb.TwosError, match="closest-point query failed"):
                m.walk_samples(sites[:1], cfg)
            return
        g = m.walk_samples(sites, cfg)
        d64 = m.closest_point(sites, precision="fp64", with_points=False)
        d32 = m.closest_point(sites, precision="mixed", with_points=False)
        delta = m.info()["mixed_delta"]
    o = oracle_mod.OracleMesh(V, F).walk_samples(sites, rng=oracle_mod.RNG_COUNTER, walks=20, seed=12, epsilon=1e-4,
                                                 max_steps=512, source=[oracle_mod.term(oracle_mod.TERM_CONST, 1.0)],
                                                 weight_order=1)
    assert np.array_equal(g["steps"], o["steps"])
    np.testing.assert_allclose(g["u"], o["u"], rtol=1e-10, atol=0)
    assert np.max(np.abs(d64 - d32)) <= delta


@pytest.mark.parametrize("shape", ["tetra", "sphere1", "sphere5", "noise6", "fan5", "fan64", "sliver"])
def test_first_queries_return_the_traversals_value(tb, shape):
    """A site's first distance, found by a whole warp, is the one a lane's
    traversal returns, to the last bit (the cap of one step makes a walk's
    value its first radius; a bulk closest-point call takes a lane per point,
    a small one a warp)."""
    rng = np.random.default_rng(5)
    if shape == "tetra":
        V = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]) - 0.25
        F = np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], dtype=np.uint32)
    elif shape.startswith("sphere"):
        V, F = tb.geometry.icosphere(int(shape[6:]))
    elif shape.startswith("noise"):
        V, F = tb.geometry.noise_sphere(int(shape[5:]), 1)
    elif shape == "sliver":
        V, F = tb.geometry.icosphere(3)
        V = V * np.array([1.0, 1e-3, 1.0])
    else:
        V, F = _fan(int(shape[3:]))
    mid = V[F.astype(np.int64)].mean(1)
    P = np.concatenate([mid[rng.integers(0, len(mid), 2000)] * rng.uniform(0.0, 0.9, (2000, 1)),
                        V[rng.integers(0, len(V), 300)] * rng.uniform(0.0, 0.95, (300, 1)), np.zeros((1, 3))])
    with tb.Mesh(V, F) as m:
        d = m.closest_point(np.tile(P, (9, 1)), precision="mixed", with_points=False)  # a lane per point
        assert np.array_equal(d, np.tile(d[: len(P)], 9))
        d = d[: len(P)]
        assert np.array_equal(d, m.closest_point(P, precision="mixed", with_points=False))  # a warp per point
        d64 = m.closest_point(np.tile(P, (9, 1)), precision="fp64", with_points=False)
        assert np.array_equal(d64, np.tile(m.closest_point(P, precision="fp64", with_points=False), 9))
        delta = np.float32(m.info()["mixed_delta"])
        cfg = tb.Config(walks=2, precision="mixed", seed=3, epsilon=1e-30, max_steps=1, query_radius=None,
                        source=tb.sources.constant(6.0))
        got = m.walk_samples(P, cfg)
    r = d.astype(np.float32) - delta
    # u = r^2/6 * 6 of the first ball, evaluated in FP32 as the walk does.
    want = np.where(r > np.float32(1e-30), (r * r / np.float32(6)) * np.float32(6), np.float32(0))
    assert np.array_equal(got["u"][:, 0].astype(np.float32), want)


@pytest.mark.parametrize("shape", ["tetra", "sphere4", "noise5", "fan5", "fan64", "sliver", "box"])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_candidate_lists_change_no_walk(tb, shape, precision):
    """Queries from the grid cells' candidate lists (the default) against
    queries that traverse from the root (entry=0): the same walks, bit for
    bit -- with cavities, in cells whose candidates are too many for a list
    (around the apex of 64 triangles) and among needle triangles."""
    if shape == "tetra":
        V = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]) - 0.25
        F = np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], dtype=np.uint32)
    elif shape.startswith("sphere"):
        V, F = tb.geometry.icosphere(int(shape[6:]))
    elif shape.startswith("noise"):
        V, F = tb.geometry.noise_sphere(int(shape[5:]), 2)
    elif shape == "sliver":
        V, F = tb.geometry.icosphere(4)
        V = V * np.array([1.0, 0.05, 1.0])
    elif shape == "box":
        V, F, _ = tb.geometry.box_minus_cylinders(h=0.2)
        V = V - V.mean(0)
    else:
        V, F = _fan(int(shape[3:]))
    rng = np.random.default_rng(9)
    mid = V[F.astype(np.int64)].mean(1)
    P = mid[rng.integers(0, len(mid), 150)] * rng.uniform(0.05, 0.98, (150, 1))
    cav = np.array([[0.05, 0.0, 0.02], [-0.1, 0.01, 0.0]])
    with tb.Mesh(V, F) as m:
        keep = m.inside(P)
        P = P[keep][:60]
        for c in (None, cav):
            cfg = tb.Config(walks=500, precision=precision, seed=14, epsilon=1e-4, cavity_radius=0.01, max_steps=4096,
                            source=tb.sources.affine())
            rows = []
            for entry in (1, 0):
                m.set_tuning(**dict(m.get_tuning(), entry=entry))
                rows.append(m.estimate(P, cfg, cavities=c)[0])
            np.testing.assert_array_equal(rows[0], rows[1])
