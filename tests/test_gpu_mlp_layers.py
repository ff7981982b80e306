"""The two forms of an MLP call, one cluster per network or one launch per layer: calls far on
either side of the line between them give the same numbers bit for bit.  An ensemble's first
members are those of a smaller ensemble of the same seed, and 48 small networks at a batch in the
thousands run layer by layer where two run in clusters; predictions of many samples run layer by
layer, of a few in clusters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data(n, nin, nout):
    g = np.random.default_rng(4)
    return g.uniform(-1, 1, (n, nin)).astype(np.float32), g.normal(size=(n, nout)).astype(np.float32)


@pytest.mark.parametrize("widths", [(4, 16, 3), (5, 17, 33, 2), (1, 31, 1)])
def test_members_of_large_and_small_ensembles(widths):
    from gauge_higgs_b200.mlp import MLPEnsemble
    x, y = data(4099, widths[0], widths[-1])
    out = []
    for members in (48, 2):
        net = MLPEnsemble(widths, members=members, seed=5)
        g, loss = net.grad(x, y)
        net.adam_step(1e-3)
        last = net.train(x, y, epochs=2, batch=2050, lr=1e-3)
        out.append([a[:2] for a in (g, loss, last, net.params())])
        net.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("widths,n", [((4, 64, 64, 3), 4097), ((3, 1000, 2), 4097), ((1024, 70, 5), 2049)])
def test_predictions_of_many_and_few_samples(widths, n):
    from gauge_higgs_b200.mlp import MLPEnsemble
    x, _ = data(n, widths[0], widths[-1])
    net = MLPEnsemble(widths, members=3, seed=6)
    mean, var, per = net.predict(x, members=True)
    for first in (0, 32, n - 33):
        few = net.predict(x[first:first + 33], members=True)
        for a, b in zip(few, (mean[first:first + 33], var[first:first + 33], per[:, first:first + 33])):
            assert np.array_equal(a, b)
    net.close()


def test_wide_network_at_a_large_batch():
    """Against the FP64 restatement, with the bounds of the other shapes."""
    from gauge_higgs_b200.mlp import MLPEnsemble
    from oracle import mlp_oracle as mo
    widths = (4, 300, 290, 3)
    x, y = data(3001, 4, 3)
    net = MLPEnsemble(widths, members=1, seed=5)
    p = net.params()
    g, loss = net.grad(x, y)
    lo, go = mo.loss_and_grad(p[0], net.widths, x, y)
    assert abs(loss[0] - lo) < 1e-3 * lo
    assert np.linalg.norm(g[0] - go) < 2e-2 * np.linalg.norm(go)
    net.close()


@pytest.mark.parametrize("widths", [(4, 250, 3), (4, 33, 16, 3)])
def test_members_with_small_batches(widths):
    """96 members layer by layer, two with everything in their clusters' shared memory."""
    from gauge_higgs_b200.mlp import MLPEnsemble
    x, y = data(62, widths[0], widths[-1])
    out = []
    for members in (96, 2):
        net = MLPEnsemble(widths, members=members, seed=5)
        g, loss = net.grad(x, y)
        net.adam_step(1e-3)
        last = net.train(x, y, epochs=3, batch=33, lr=1e-3)
        out.append([a[:2] for a in (g, loss, last, net.params())])
        net.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
