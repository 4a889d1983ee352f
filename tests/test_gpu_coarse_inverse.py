"""The coarsest level's dense inverse at the edges of its 16-pivot steps.

A hierarchy of one level is the inverse itself, so that the preconditioner
solves K_reg x = b.  The inverse is of 2 N real rows: 8, 16 and 18, 32 and 34
take one to three steps with whole and ragged last ones in FP64, 128 is the largest
that the mixed path inverts in FP32, 130 the smallest it inverts in FP64 there;
a batch has blocks of several sizes in one launch.  Forward error bound of a
solve by an explicit inverse: 4 m cond(K) machine epsilons, and the rounding
of the FP32 copy and product (m epsilons of FP32) on the mixed path.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(model, problems, mu, prec, m_max):
    K = [P.kreg_csr_real(psi, 1.0, mu_).toarray() for P, psi, mu_ in problems]
    b = np.random.default_rng(3).standard_normal(sum(len(k) for k in K))
    M = model.create_W_prec()
    M.rebuild({"g": 1.0, "mu": mu}, np.concatenate([psi for _, psi, _ in problems]))
    x = M.apply(b)
    assert len(model.amg_levels()[0]) == 1
    at = 0
    for k in K:
        m = len(k)
        ref = np.linalg.solve(k, b[at:at + m])
        cond = np.linalg.cond(k)
        fp32 = prec == "mixed"
        eps = 2.0**-53 if not fp32 or m_max > 128 else 2.0**-24
        bound = 4 * m * cond * eps + ((m + 2) * 2.0**-24 * np.abs(np.linalg.inv(k)).sum(1).max()
                                      * np.abs(b[at:at + m]).max() / np.abs(ref).max() if fp32 else 0.0)
        assert np.abs(x[at:at + m] - ref).max() <= bound * np.abs(ref).max()
        at += m


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [4, 8, 9, 16, 17, 64, 65, 100])
def test_one_level_preconditioner_is_the_inverse(n, prec):
    import nosh_gb300 as ng

    # a strip of squares cut into triangles, n vertices
    k = (n + 1) // 2
    x = np.array([[i // 2, i % 2, 0.0] for i in range(2 * k)])[:n] + 0.1 * np.random.default_rng(n).random((n, 3))
    c = np.array([[i, i + 1, i + 2] for i in range(n - 2)], np.int32)
    m = O.finish_mesh(x, c)
    A = O.mvp_constant_curl(m.x)
    psi = np.random.default_rng(2).standard_normal(2 * n)
    model = ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.3,
                   precision=ng.PREC_FP64 if prec == "fp64" else ng.PREC_MIXED)
    model.set_amg_options(max_levels=1)
    _check(model, [(O.Problem(m, A), psi, 0.3)], 0.3, prec, 2 * n)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_blocks_of_several_sizes(prec):
    import nosh_gb300 as ng
    from nosh_gb300 import batch

    sides, mus = [2, 3, 4, 6], [0.2, 0.4, 0.6, 0.8]
    x, c, off, _, A, mu = batch.squares(sides, mus, seed0=70)
    model = ng.nls(ng.mesh(x, c), A, -1.0, 1.0, 1.0, mu=0.0,
                   precision=ng.PREC_FP64 if prec == "fp64" else ng.PREC_MIXED)
    model.set_systems(off, mu)
    model.set_amg_options(max_levels=1)
    problems = []
    for k, s in enumerate(sides):
        mk = O.finish_mesh(*O.gen_square(s, 70 + k)[:2])
        psi = np.random.default_rng(k).standard_normal(2 * mk.N)
        problems.append((O.Problem(mk, O.mvp_constant_curl(mk.x)), psi, mus[k]))
    _check(model, problems, 0.0, prec, 72)
