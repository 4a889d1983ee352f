"""The network's gradient at sizes around the tiles of its backward kernels
(64-row node tiles, 16-row edge passes, one CTA or many), against the torch
reference of tests/test_gpu_learned.py.

Tolerances as there: 3e-3 on the coefficient, 1e-3 on the loss, and for the
gradient (BF16 operands, FP16 messages) a cosine above 0.999 and 3e-2 of its
norm.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_learned import FX, torch_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gen", [lambda: O.gen_square(3, 1), lambda: O.gen_square(8, 1), lambda: O.gen_cube(3, 2),
                                 lambda: O.gen_square(23, 3), lambda: O.gen_cube(9, 4)],
                         ids=["square3", "square8", "cube3", "square23", "cube9"])
def test_gradient_at_tile_edges(gen):
    import nosh_gb300 as ng

    x, c, _ = gen()
    m = O.finish_mesh(x, c)
    model = ng.nls(ng.mesh(m.x, m.cells), O.mvp_constant_curl(m.x), -1.0, 1.0, 1.0, mu=0.5)
    net = ng.mpnn(model)
    p = net.params()
    rng = np.random.default_rng(5)
    X = rng.standard_normal((m.N, FX)).astype(np.float32)
    X[:, 9] = 1.0
    gram = np.array([2.0, 0.5, 1.0])
    rp, ci = model.mesh.build_complex_graph()
    rows = np.repeat(np.arange(m.N), np.diff(rp))
    off = ci != rows
    rp_off = np.concatenate([[0], np.cumsum(np.bincount(rows[off], minlength=m.N))])
    w_ref, loss_ref, g_ref = torch_reference(p, net.edge_features(), rp_off, ci[off], X, gram)
    w = net.forward(X)
    assert abs(w - w_ref) <= 3e-3 * abs(w_ref), (w, w_ref)
    loss, g = net.loss_grad(X, gram)
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref), (loss, loss_ref)
    cos = g @ g_ref / (np.linalg.norm(g) * np.linalg.norm(g_ref))
    assert cos > 0.999 and np.linalg.norm(g - g_ref) < 3e-2 * np.linalg.norm(g_ref), cos
    loss2, g2 = net.loss_grad(X, gram)
    assert loss2 == loss and np.array_equal(g, g2)
