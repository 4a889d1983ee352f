"""DkeoDP from the assembled KEO, and blocks of vectors on the mixed path.

DkeoDP's values are the KEO's times -+ i dp where the KEO stands at the same
parameter, and come from the sines elsewhere: both round the sine, its product
with alpha and that with dp once each, so they agree to five machine epsilons.  A block of
vectors on the device is rounded to FP32 four at a time: each product is the
one of that vector alone, bit for bit, from the host as from the device.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _model(name, prec):
    import nosh_gb300 as ng

    x, c, _ = O.gen_square(9, 5) if name == "square" else O.gen_cube(4, 5)
    m = O.finish_mesh(x, c)
    A = O.mvp_constant_curl(m.x)
    return m, A, ng.nls(ng.mesh(m.x, m.cells), A, -1.0, 1.0, 1.0, mu=0.1, precision=prec)


@pytest.mark.parametrize("name", ["square", "cube"])
def test_dkeo_values_by_both_routes(name):
    import nosh_gb300 as ng

    values = []
    for keo_mu in (0.6, 0.2):
        m, A, model = _model(name, ng.PREC_FP64)
        model.keo.set_parameters({"g": 1.0, "mu": keo_mu})
        model.dkeo_dp.set_parameters({"g": 1.0, "mu": 0.6})
        values.append(model.dkeo_dp.values())
    assert np.abs(values[0] - values[1]).max() <= 5 * 2.0**-52 * np.abs(values[1]).max()
    # and they stay what they are when the KEO moves on
    model.keo.set_parameters({"g": 1.0, "mu": 0.6})
    assert np.array_equal(model.dkeo_dp.values(), values[1])


@pytest.mark.parametrize("nvec", [1, 3, 4, 5, 9])
def test_block_products_are_the_single_ones(nvec):
    torch = pytest.importorskip("torch")
    import nosh_gb300 as ng

    m, A, model = _model("cube", ng.PREC_MIXED)
    psi = np.random.default_rng(1).standard_normal(2 * m.N)
    X = np.random.default_rng(2).standard_normal((nvec, 2 * m.N))
    J = model.create_W_op()
    J.rebuild({"g": 1.0, "mu": 0.6}, psi)
    one = np.stack([J.apply(v) for v in X])
    assert np.array_equal(J.apply(X), one)
    Xd = torch.from_numpy(X).cuda()
    Yd = torch.empty_like(Xd)
    torch.cuda.synchronize()
    J.apply(Xd, Yd)
    assert np.array_equal(Yd.cpu().numpy(), one)
