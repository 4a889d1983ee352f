"""Edges, KEO graph and geometry of meshes at the edges of the device build.

The build scans in tiles of 1024 vertices, gives each vertex a warp and
leaves vertices with more than 84 cells to the host.  Edges and graph are
whole numbers and equal the oracle's.  The geometry comes from inner products
of edges, with a relative error of a few machine epsilons times the condition
of the Gram matrix of squared inner products: 1e-12 of the largest value on
well-shaped cells (as in the parity tests), 1e-9 on the fans, whose angle
theta of 0.05 gives a condition of theta^-4 = 2e5 (5e-11, twenty times under
the bound).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _permuted(x, cells, seed):
    r = np.random.default_rng(seed)
    p = r.permutation(len(x)).astype(np.int32)
    inv = np.empty_like(p)
    inv[p] = np.arange(len(p), dtype=np.int32)
    c = inv[cells][r.permutation(len(cells))]
    return x[p], np.stack([r.permutation(row) for row in c]).astype(np.int32)


def _fan(n):
    """n triangles around one vertex"""
    a = 2 * np.pi * np.arange(n) / n
    x = np.vstack([np.zeros((1, 3)), np.stack([np.cos(a), np.sin(a), 0 * a], 1)])
    k = np.arange(n)
    return x, np.stack([0 * k, 1 + k, 1 + (k + 1) % n], 1).astype(np.int32)


def _spindle(n):
    """n tetrahedra around one edge"""
    x, tri = _fan(n)
    x[0, 2] = -0.5
    x = np.vstack([x, [[0.0, 0.0, 0.5]]])
    return x, np.column_stack([tri, np.full(n, n + 1, np.int32)]).astype(np.int32)


def _mesh(name):
    kind, size = name.split("_")
    n = int(size)
    if kind == "square":
        return _permuted(*O.gen_square(n, 3)[:2], 1) + (1e-12,)
    if kind == "cube":
        return _permuted(*O.gen_cube(n, 4)[:2], 2) + (1e-12,)
    x, c = _fan(n) if kind == "fan" else _spindle(n)
    return _permuted(x, c, 5) + (1e-9,)


# one pair of triangles and six tetrahedra; a full scan tile (32^2) and two
# (33^2); two tiles and a ragged third; 84 and 85 cells at a vertex, and hubs
@pytest.mark.parametrize(
    "name", ["square_2", "cube_1", "square_32", "square_33", "cube_12", "fan_84", "fan_85", "fan_130", "spindle_84",
             "spindle_85", "spindle_120"])
def test_topology_and_geometry_match_oracle(name):
    import nosh_gb300 as ng

    x, c, tol = _mesh(name)
    o = O.finish_mesh(x, c)
    m = ng.mesh(x, c)
    assert np.array_equal(m.my_edges(), o.edges)
    rp, ci = m.build_complex_graph()
    rows = [[v] for v in range(o.N)]
    for a, b in o.edges:
        rows[a].append(b)
        rows[b].append(a)
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum([len(r) for r in rows])]))
    assert np.array_equal(ci, np.concatenate([sorted(r) for r in rows]))
    ln, cov = m.get_edge_data()
    assert np.abs(ln - o.length).max() <= 1e-15 * 4 * np.abs(o.length).max()
    assert np.abs(cov - o.covolume).max() <= tol * np.abs(o.covolume).max()
    cv = m.control_volumes()
    assert np.abs(cv - o.cv).max() <= tol * np.abs(o.cv).max()
    # the scatter maps: every nonzero's edge and sign enter the operator
    A = O.mvp_constant_curl(x)
    psi = np.random.default_rng(9).standard_normal(2 * o.N)
    f = ng.nls(m, A, -1.0, 1.0, 1.0, mu=0.7).compute_f(psi, {"g": 1.0, "mu": 0.7})
    ref = O.Problem(o, A).compute_f(psi, 1.0, 0.7)
    assert np.abs(f - ref).max() <= 10 * tol * np.abs(ref).max()


def _fans(sizes):
    xs, cs, n = [], [], 0
    for k, s in enumerate(sizes):
        x, c = _fan(s)
        xs.append(x + [3.0 * k, 0.0, 0.0])
        cs.append(c + n)
        n += len(x)
    return np.vstack(xs), np.vstack(cs).astype(np.int32)


def test_many_hubs():
    """more hubs than one host thread takes, among vertices that are none"""
    import nosh_gb300 as ng

    x, c = _permuted(*_fans(range(60, 140)), 7)
    o = O.finish_mesh(x, c)
    m = ng.mesh(x, c)
    assert np.array_equal(m.my_edges(), o.edges)
    ln, cov = m.get_edge_data()
    assert np.abs(cov - o.covolume).max() <= 1e-9 * np.abs(o.covolume).max()
    assert np.abs(m.control_volumes() - o.cv).max() <= 1e-9 * np.abs(o.cv).max()


def test_time_of_many_hubs():
    """10000 hubs are found together, in about 6 ms; one after the other, each
    with copies of its own, they take 340, the bound is 100"""
    import time

    import nosh_gb300 as ng

    x, c = _fans([85] * 10000)
    best = 1.0
    for _ in range(4):
        t = time.perf_counter()
        ng.mesh(x, c)
        best = min(best, time.perf_counter() - t)
    assert best < 0.1, best


def test_vertices_outside_every_cell():
    """a vertex of no cell has an empty row, wherever it stands"""
    import nosh_gb300 as ng

    x, c, _ = _mesh("square_5")
    x = np.vstack([[[9.0, 9.0, 0.0]], x[:11], [[8.0, 9.0, 0.0]], x[11:], [[7.0, 9.0, 0.0]]])
    c = c + 1 + (c >= 11)
    o = O.finish_mesh(x, c.astype(np.int32))
    m = ng.mesh(x, c.astype(np.int32))
    assert np.array_equal(m.my_edges(), o.edges)
    rp, _ = m.build_complex_graph()
    d = np.bincount(o.edges.ravel(), minlength=o.N) + 1
    assert np.array_equal(np.diff(rp), d) and d[0] == d[12] == d[-1] == 1
    assert np.all(m.control_volumes()[[0, 12, -1]] == 0.0)


@pytest.mark.parametrize("nvc", [3, 4])
def test_degenerate_cells_are_refused(nvc):
    """a flat cell among good ones, and coordinates that are no numbers"""
    import nosh_gb300 as ng

    x, c = (O.gen_square(4, 1) if nvc == 3 else O.gen_cube(2, 1))[:2]
    for bad in ("flat", "nan", "inf"):
        y = x.copy()
        if bad == "flat":
            y[c[3, 2]] = 0.5 * (y[c[3, 0]] + y[c[3, 1]])
        else:
            y[c[3, 2], 0] = float(bad)
        with pytest.raises(ng.NoshError, match="degenerate cell"):
            ng.mesh(y, c)
