"""The MLP's step kernel at shapes around its tiles (columns per pass, rows per pass, terms per
stage, cluster slices): forward and gradients against the FP64 restatement, and whole training
runs against the same steps taken one gh_mlp_grad + gh_mlp_adam_step at a time, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((4, 3), 1), ((4, 1, 3), 33), ((3, 17, 130, 20), 31), ((4, 128, 128, 128, 3), 129), ((2, 129, 40, 17), 260)]


def data(n, nin, nout, seed):
    g = np.random.default_rng(seed)
    return g.uniform(-1, 1, (n, nin)).astype(np.float32), g.normal(size=(n, nout)).astype(np.float32)


@pytest.mark.parametrize("widths,n", SHAPES)
def test_forward_and_gradient(widths, n):
    from gauge_higgs_b200.mlp import MLPEnsemble
    from oracle import mlp_oracle as mo
    net = MLPEnsemble(widths, members=2, seed=5)
    x, y = data(n, widths[0], widths[-1], 1)
    p = net.params()
    g, loss = net.grad(x, y)
    _, _, per = net.predict(x, members=True)
    for m in range(2):
        out, _, _ = mo.forward(p[m], net.widths, x)
        assert np.abs(per[m] - out).max() < 2e-3 * max(1.0, np.abs(out).max())
        lo, go = mo.loss_and_grad(p[m], net.widths, x, y)
        assert abs(loss[m] - lo) < 1e-3 * lo
        assert np.linalg.norm(g[m] - go) < 2e-2 * np.linalg.norm(go)
    net.close()


@pytest.mark.parametrize("widths,n,batch", [(s, max(n, 2), b) for s, n in SHAPES for b in (1000, 24)])
def test_training_is_its_steps(widths, n, batch):
    from gauge_higgs_b200._lib import LIB
    from gauge_higgs_b200.mlp import MLPEnsemble
    x, y = data(n, widths[0], widths[-1], 2)
    a, b = (MLPEnsemble(widths, members=3, seed=7) for _ in range(2))
    epochs, losses = 3, None
    la = a.train(x, y, epochs=epochs, batch=batch, lr=1e-3, seed=7)
    for ep in range(epochs):
        idx, losses = list(range(n)), []
        for i in range(n - 1, 0, -1):
            j = min(int(LIB.gh_rng_uniform(7, LIB.gh_rng_key(0x5348, ep, i, 0, 0)) * (i + 1)), i)
            idx[i], idx[j] = idx[j], idx[i]
        for s in range(0, n, batch):
            losses.append(b.grad(x[idx[s:s + batch]], y[idx[s:s + batch]])[1])
            b.adam_step(1e-3)
    assert np.array_equal(a.params(), b.params())
    assert np.allclose(la, np.mean(losses, axis=0), rtol=1e-6)
    a.close()
    b.close()
