"""The resident V-cycle (levels in a thread-block cluster's shared memory)
against the same cycle with its fine level on the grid, and its symmetry.

Small meshes run the whole cycle resident; with kernel timing on the handle
keeps the fine level on the grid, so the two applies differ in rounding only.
Sizes sit at the edges: a hierarchy of two levels, fewer rows than CTAs, one
row more than a multiple of them, the largest mesh taken whole and the one
after, triangles and tetrahedra, every smoothing degree parity.

Tolerances, before any run: a cycle is about 30 dependent roundings deep and
its intermediate vectors are within a factor of 100 of its result, so FP64
1e-12 and FP32 1e-4 of the largest entry; the symmetry defect relative to
||a|| ||M b|| the same.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

MESHES = {
    "square9": lambda: O.gen_square(9, 3),
    "square17": lambda: O.gen_square(17, 1),
    "square33": lambda: O.gen_square(33, 2),
    "square45": lambda: O.gen_square(45, 4),
    "square46": lambda: O.gen_square(46, 4),
    "square65": lambda: O.gen_square(65, 1),
    "cube4": lambda: O.gen_cube(4, 5),
    "cube11": lambda: O.gen_cube(11, 6),
    "cube17": lambda: O.gen_cube(17, 7),
}


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-4)])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_resident_cycle(name, prec, tol, degree):
    import nosh_gb300 as ng

    x, c, psi = MESHES[name]()
    m = O.finish_mesh(x, c)
    A = O.mvp_constant_curl(m.x)
    model = ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.3, precision=prec)
    model.set_spmv_schedule(ng.SPMV_STAGED)
    model.set_amg_options(smooth_degree=degree, coarse_size=40)
    M = model.create_W_prec()
    M.rebuild({"g": 1.0, "mu": 0.3}, psi)
    rng = np.random.default_rng(11)
    a, b = rng.standard_normal((2, 2 * m.N))
    Ma, Mb = M.apply(a), M.apply(b)
    assert np.isfinite(Ma).all() and a @ Ma > 0 and b @ Mb > 0
    assert abs(a @ Mb - b @ Ma) <= tol * np.linalg.norm(a) * np.linalg.norm(Mb)
    model.profile(True)
    grid = M.apply(a)
    model.profile(False)
    assert np.abs(grid - Ma).max() <= tol * np.abs(grid).max()
    assert np.array_equal(M.apply(a), Ma)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("name", ["square9", "cube11", "square65"])
def test_waits_that_run_out(name, prec):
    """With a bound of 0 polls every wait of the resident cycle gives up at
    once: the call returns NOSH_ERR_CUDA and names the cycle, alone and in a
    solve, and with the bound restored the handle gives the same bits as
    before.  (The warp schedule has no waits of its own.)"""
    import nosh_gb300 as ng

    x, c, psi = MESHES[name]()
    m = O.finish_mesh(x, c)
    A = O.mvp_constant_curl(m.x)
    model = ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.3, precision=prec)
    model.set_spmv_schedule(ng.SPMV_WARP)
    model.set_amg_options(coarse_size=40)
    M = model.create_W_prec()
    M.rebuild({"g": 1.0, "mu": 0.3}, psi)
    a = np.random.default_rng(11).standard_normal(2 * m.N)
    Ma = M.apply(a)
    model.set_stage_wait_limit(0)
    for call in (lambda: M.apply(a), lambda: model.newton(psi.copy(), {"g": 1.0, "mu": 0.3})):
        with pytest.raises(ng.NoshError) as e:
            call()
        assert e.value.code == ng.ERR_CUDA and "resident coarse cycle" in str(e.value)
    model.set_stage_wait_limit(-1)
    M.rebuild({"g": 1.0, "mu": 0.3}, psi)
    assert np.array_equal(M.apply(a), Ma)
    sol = psi.copy()
    st = model.newton(sol, {"g": 1.0, "mu": 0.3}, tol=1e-10)
    assert st["status"] == 0 and np.linalg.norm(O.Problem(m, A).compute_f(sol, 1.0, 0.3)) <= 2e-10


# the first level that runs resident for the mesh alone
FIRST = {"square33": 0, "square45": 0, "square65": 1, "cube11": 0, "cube17": 1}


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-4)])
@pytest.mark.parametrize("name", sorted(FIRST))
def test_resident_against_every_level_on_the_grid(name, prec, tol):
    """A union of equal meshes is block diagonal with equal blocks, so every
    block of its V-cycle is the V-cycle of the mesh alone: the same levels,
    aggregates and Chebyshev bounds.  With so many copies that the coarsest
    level has more than 1024 nodes the union has no level in the resident kernel;
    the mesh alone has all but its fine level there, or that as well.
    Tolerances as above."""
    import nosh_gb300 as ng

    x, c, psi = MESHES[name]()
    m = O.finish_mesh(x, c)
    r = np.random.default_rng(3).standard_normal(2 * m.N)
    p = {"g": 1.0, "mu": 0.3}
    out = []
    for many in (False, True):
        k = 1025 // out[0][1][-1] + 1 if many else 1
        X = np.tile(m.x, (k, 1))
        cells = (m.cells[None] + m.N * np.arange(k)[:, None, None]).reshape(-1, m.cells.shape[1]).astype(np.int32)
        model = ng.nls(ng.mesh(X, cells), O.mvp_constant_curl(X), -1.0, 1.0, 1.0, mu=0.3, precision=prec)
        model.set_spmv_schedule(ng.SPMV_STAGED)
        model.set_amg_options(coarse_size=40)
        if many:
            model.set_systems(m.N * np.arange(k + 1), np.full(k, 0.3))
        M = model.create_W_prec()
        M.rebuild(p, np.tile(psi, k))
        sizes, tail = model.amg_levels()
        out.append((M.apply(np.tile(r, k)).reshape(k, -1), np.array(sizes), tail))
    (alone, sizes, tail), (union, usizes, _) = out
    assert tail == FIRST[name] and np.array_equal(usizes, len(union) * sizes) and usizes[-1] > 1024, (sizes, tail)
    assert np.abs(union - alone).max() <= tol * np.abs(alone).max()
