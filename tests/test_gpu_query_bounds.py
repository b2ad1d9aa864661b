"""Where a closest-point query's bounds are tight: candidate lists that do and
do not fit, and the limits of the searches."""
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
