"""Surrogate kernels at the edges of their 32-row tiles: vertex and swap counts around a
tile, degrees around the eight neighbours a pass loads, few and many input features; the
gradient against the numpy restatement, the training step against Adam on that gradient."""
import numpy as np
import pytest

import graphgolf as G
import surrogate_ref as R


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,F,P", [(32, 3, 1, 1), (33, 4, 16, 31), (64, 7, 17, 33), (250, 9, 5, 64), (100, 11, 250, 65),
                                     (4800, 8, 5, 200)])
def test_gradient_and_step_at_tile_edges(n, d, F, P):
    adj = G.random_regular(n if n * d % 2 == 0 else n + 1, d, 3)
    n = len(adj)
    rng = np.random.default_rng(n + P)
    feats = rng.standard_normal((n, F)).astype(np.float32)
    sw = G.gen_swaps(adj, 0, P, 5)
    t = rng.standard_normal(P).astype(np.float32)
    mask = (rng.random(P) < 0.8).astype(np.int32)
    mask[0] = 1
    net = G.Surrogate(n, d, F, seed=2)
    net.set_graph(adj, feats)
    p0 = net.get_params()
    pred = net.predict(sw)
    g, loss = net.grad(sw, t, mask)
    ref = R.Net(adj, feats, bf16=True)
    want_pred, _ = ref.forward(p0.astype(np.float64), sw)
    want_loss, want_g, _ = ref.loss_grad(p0.astype(np.float64), sw, t, mask)
    # both sides round the same operands to bf16; the kernels sum in fp32 in another order,
    # so a later operand may round the other way (2^-8 of it): the bounds of the other tests
    assert np.abs(pred - want_pred).max() <= 1e-2 * np.abs(want_pred).max() + 1e-4
    assert abs(loss - want_loss) <= 1e-2 * abs(want_loss)
    assert np.linalg.norm(g - want_g) <= 2e-2 * np.linalg.norm(want_g)
    step = net.train(sw, t, lr=1e-3, mask=mask)
    assert abs(step - loss) <= 1e-5 * max(1.0, loss)
    p1 = net.get_params()
    big = np.abs(g) > 1e-4 * np.abs(g).max()     # where the first step's sign is not rounding
    assert np.allclose((p1 - p0)[big], (-1e-3 * g / (np.abs(g) + 1e-8))[big], atol=2e-6)
    net.close()
