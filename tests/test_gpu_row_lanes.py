"""Rows shared by several lanes give the products of rows of one lane.

Meshes whose cells are random well-shaped tetrahedra over n vertices (nearly
every pair of vertices shares a cell, which is no geometry but a graph with
rows of up to n - 1): with at least 6 nonzeros a lane, 30 vertices take one
lane a row, 45 two, 62 four and 100 eight; 129 and 131 end in ragged row
blocks, and the row blocks of 300 vertices exceed the staging buffer.

The bound is the sum of rounding errors row by row, against |J| |x|: (n + 20)
machine epsilons of the precision; in FP64 the edge coefficients of oracle and
device differ by their solves (condition of the cells here up to 1e4: 1e-11
relative), which the bound takes for every entry; in FP32 the entries are
rounded once more (one epsilon).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mesh(n):
    r = np.random.default_rng(n)
    x = r.random((n, 3))
    cells = []
    while len(cells) < n * n // 4:
        c = np.stack([r.choice(n, 4, replace=False) for _ in range(64)])
        e = x[c[:, 1:]] - x[c[:, :1]]
        vol = np.abs(np.linalg.det(e))
        size = np.linalg.norm(x[c][:, :, None] - x[c][:, None], axis=3).max(axis=(1, 2))
        cells += list(c[vol > 0.12 * size**3])
    return O.finish_mesh(x, np.array(cells, np.int32))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [30, 45, 62, 100, 129, 131, 300])
def test_jacobian_product_matches_oracle(n, prec):
    import nosh_gb300 as ng

    m = _mesh(n)
    A = O.mvp_constant_curl(m.x)
    r = np.random.default_rng(1)
    psi, x = r.standard_normal(2 * n), r.standard_normal(2 * n)
    model = ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.7,
                   precision=ng.PREC_FP64 if prec == "fp64" else ng.PREC_MIXED)
    model.set_spmv_schedule(ng.SPMV_STAGED)
    P = O.Problem(m, A)
    J = model.create_W_op()
    J.rebuild({"g": 1.0, "mu": 0.7}, psi)
    got = J.apply(x)
    ref = P.jac_apply(psi, 1.0, 0.7, x)
    size = np.abs(P.jac_csr_real(psi, 1.0, 0.7)) @ np.abs(x)
    bound = (n + 20) * 2.0**-53 + 1e-11 if prec == "fp64" else (n + 21) * 2.0**-24 + 1e-11
    assert np.all(np.abs(got - ref) <= bound * size)
    again = J.apply(x)
    assert np.array_equal(got, again)
