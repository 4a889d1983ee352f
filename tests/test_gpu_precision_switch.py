"""An operator rebuilt in one precision and applied in the other.

The FP32 blocks of the Jacobian are written with the FP64 ones on a mixed
handle and rounded from them on the first FP32 apply otherwise: the same
values either way, so the applies agree to the bit.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gen", [lambda: O.gen_square(9, 3), lambda: O.gen_cube(6, 2)], ids=["square9", "cube6"])
@pytest.mark.parametrize("nvec", [1, 3])
def test_jacobian_rebuilt_in_fp64_applied_mixed(gen, nvec):
    import nosh_gb300 as ng

    x, c, psi = gen()
    m = O.finish_mesh(x, c)
    A = O.mvp_constant_curl(m.x)
    P = O.Problem(m, A)
    X = np.random.default_rng(3).standard_normal((nvec, 2 * m.N))
    p = {"g": 1.0, "mu": 0.3}
    out = {}
    for first in (ng.PREC_FP64, ng.PREC_MIXED):
        model = ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.3, precision=first)
        model.set_spmv_schedule(ng.SPMV_STAGED)
        J = model.create_W_op()
        J.rebuild(p, psi)
        model.set_precision(ng.PREC_MIXED)
        mixed = J.apply(X)
        model.set_precision(ng.PREC_FP64)
        out[first] = (mixed, J.apply(X))
    for a, b in zip(out[ng.PREC_FP64], out[ng.PREC_MIXED]):
        assert np.array_equal(a, b)
    for v, w in zip(X, out[ng.PREC_FP64][1]):
        ref = P.jac_apply(psi, 1.0, 0.3, v)
        assert np.abs(w - ref).max() <= 1e-12 * np.abs(ref).max()
