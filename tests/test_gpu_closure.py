"""The fused closure kernels at the edges of their tiles: the training pass
(32-row tiles, 128 x 64 tiles of the weight gradients, hidden sizes 128 and
256) and the inference (tiles of a few ADOs, hidden sizes that fill a 128-row
block of outputs or leave it ragged) against the numpy restatement.
Tolerances are those of the closure's other tests: every GEMM operand is
rounded to BF16 (2^-8) on both sides, so an activation that rounds to the
neighbouring value moves a gradient by a few 1e-3 of the largest one."""
import numpy as np
import pytest

import libheom_gb300 as lh
import oracle
from libheom_gb300 import configs
from libheom_gb300 import terminator as T
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,batch,kind", [(2, 256, 1, 1), (2, 256, 31, 1), (2, 128, 32, 1), (3, 128, 33, 1),
                                            (5, 256, 97, 1), (7, 256, 129, 1), (7, 128, 64, 0), (7, 256, 1000, 0)])
def test_training_pass_edges(n, h, batch, kind):
    torch = pytest.importorskip("torch")
    n2 = n * n
    din, dout = 4 * n2 + 2 * n, 2 * n2
    rng = np.random.default_rng(100 * n + batch)
    mlp = T.MLP(din, h, dout, seed=n)
    x = rng.standard_normal((batch, din)).astype(np.float32)
    if kind == 1:
        mlp.set_loss(1, n2)
        t = rng.standard_normal((batch, 5 * n2)).astype(np.float32)
        t[:, 4 * n2:] = rng.integers(-1, 2, (batch, n2))
    else:
        t = rng.standard_normal((batch, dout)).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    before = mlp.get_params()
    g, loss = mlp.gradients(xd.data_ptr(), td.data_ptr(), batch)
    gref, lref = mlp_oracle.gradients(before, x.astype(np.float64), t.astype(np.float64), din, h, dout, kind)
    assert abs(loss - lref) <= 1e-3 * abs(lref)
    assert np.abs(g - gref).max() <= 3e-3 * np.abs(gref).max()
    # a step moves every weight by lr g / (|g| + eps) (the first Adam step)
    assert mlp.train_step(xd.data_ptr(), td.data_ptr(), batch, 1e-3) == loss
    step = before - mlp.get_params()
    assert np.abs(step - 1e-3 * g / (np.abs(g) + 1e-8)).max() <= 1e-6


@pytest.mark.parametrize("n,depth,h", [(2, 0, 64), (3, 2, 64), (3, 1, 192), (5, 2, 128), (6, 2, 256)])
def test_inference_tiles(n, depth, h):
    p = configs.spin_boson(depth=depth) if n == 2 else configs.aggregate_24site(n_sites=n, depth=depth)
    din, dout = T.dims(p)
    mlp = T.MLP(din, h, dout, seed=7)
    q = lh.from_params(p)
    rng = np.random.default_rng(n)
    shape = (p.n_hrchy(), n, n)
    rho = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * 0.3
    plain = q.calc_diff(rho)
    T.attach(q, mlp)
    got = q.calc_diff(rho)
    n_tab, _, _ = oracle.Oracle("port").hrchy(p.n_modes, p.max_depth)
    first = int(np.argmax(n_tab.sum(1) == p.max_depth))
    X, _ = mlp_oracle.term_features(p, n_tab, rho, first)
    Y, _ = mlp_oracle.forward(mlp.get_params(), X, din, h, dout)
    bath_of = T._mode_constants(p)[0]
    expect, K = plain.copy(), p.n_modes
    for j, l in enumerate(range(first, p.n_hrchy())):
        for k in range(K):
            v = np.diag(p.V[bath_of[k]])
            sg = np.sign((v[:, None] - v[None, :]).real).ravel()
            C = mlp_oracle.gain_head(Y[j * K + k], sg) * np.abs(sg)
            expect[l] -= 1j * (v[:, None] - v[None, :]) * (C * rho[l].ravel()).reshape(n, n)
    scale = np.abs(plain).max() + np.abs(expect - plain).max()
    assert np.abs(got - expect).max() <= 5e-4 * scale
