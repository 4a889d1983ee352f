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


def _handle(gen, precision):
    import nosh_gb300 as ng

    x, c, psi = gen()
    m = O.finish_mesh(x, c)
    model = ng.nls(ng.mesh(m.x, m.cells), O.mvp_constant_curl(m.x), -1.0, 1.0, 1.0, mu=0.3, precision=precision)
    model.set_spmv_schedule(ng.SPMV_STAGED)
    model.set_amg_options(coarse_size=10)
    return model, psi, np.random.default_rng(5).standard_normal(2 * m.N)


CYCLES = {"square9": lambda: O.gen_square(9, 3), "cube6": lambda: O.gen_cube(6, 2), "square65": lambda: O.gen_square(65, 1)}


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("gen", sorted(CYCLES))
def test_preconditioner_applied_in_the_other_precision(gen, first):
    """After a rebuild in one precision the V-cycle and the smoother of the
    other are those of a rebuild in it, to the bit: on a hierarchy that the
    other precision has not had yet, and on one that it had at another state."""
    p = {"g": 1.0, "mu": 0.3}
    other = 1 - first
    model, psi, v = _handle(CYCLES[gen], other)
    M = model.create_W_prec()
    M.rebuild(p, psi)
    want = M.apply(v), M.smoother_apply(v)
    model, psi, v = _handle(CYCLES[gen], first)
    M = model.create_W_prec()
    M.rebuild(p, psi)
    model.set_precision(other)
    assert np.array_equal(M.apply(v), want[0]) and np.array_equal(M.smoother_apply(v), want[1])
    # the other precision's hierarchy is now at psi; rebuilt in the first at
    # another state, it follows (its fine level at least: the smoother)
    model.set_precision(first)
    M.rebuild(p, 2.0 * psi)
    model.set_precision(other)
    moved = M.smoother_apply(v)
    model, psi, v = _handle(CYCLES[gen], other)
    M = model.create_W_prec()
    M.rebuild(p, 2.0 * psi)
    assert np.array_equal(moved, M.smoother_apply(v)) and not np.array_equal(moved, want[1])


@pytest.mark.parametrize("gen", sorted(CYCLES))
def test_preconditioner_of_a_mixed_handle_after_an_fp64_solve(gen):
    """An FP64 Newton step leaves the operators at its starting state: the
    mixed handle's V-cycle agrees with that of an FP64 handle rebuilt there (a
    cycle is some 30 roundings deep: 1e-4 of the largest entry in FP32) and is
    positive definite."""
    import nosh_gb300 as ng

    p = {"g": 1.0, "mu": 0.3}
    model, psi, v = _handle(CYCLES[gen], ng.PREC_MIXED)
    model.newton(psi.copy(), p, precision=ng.PREC_FP64, max_newton=1)
    mixed = model.create_W_prec().apply(v)
    model, psi, v = _handle(CYCLES[gen], ng.PREC_FP64)
    M = model.create_W_prec()
    M.rebuild(p, psi)
    fp64 = M.apply(v)
    assert np.isfinite(mixed).all() and v @ mixed > 0
    assert np.abs(mixed - fp64).max() <= 1e-4 * np.abs(fp64).max()


@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("gen", sorted(CYCLES))
def test_a_solve_in_the_other_precision_leaves_the_cycle_alone(gen, first):
    """The V-cycle rebuilt at the same state is the same, to the bit, after a
    solve of the other precision at another state and parameter."""
    p = {"g": 1.0, "mu": 0.3}
    model, psi, v = _handle(CYCLES[gen], first)
    M = model.create_W_prec()
    M.rebuild(p, psi)
    want = M.apply(v)
    model.newton(1.1 * psi, {"g": 1.0, "mu": 0.5}, precision=1 - first)
    M.rebuild(p, psi)
    assert np.array_equal(M.apply(v), want)
