"""Ensembles of different widths trained from several threads at once (each call releases the
interpreter): every call succeeds and gives what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_widths():
    from gauge_higgs_b200.mlp import MLPEnsemble
    g = np.random.default_rng(1)
    x, y = g.uniform(-1, 1, (8, 4)).astype(np.float32), g.normal(size=(8, 3)).astype(np.float32)
    errors, stop = [], threading.Event()

    def train(net, n):
        try:
            for _ in range(n):
                net.train(x, y, epochs=1, batch=8, lr=1e-3)
                if stop.is_set():
                    break
        except Exception as e:      # reported by the test's own thread
            errors.append(e)

    steps, wide = 5000, [MLPEnsemble((4, 128, 128, 128, 3), members=1, seed=3) for _ in range(2)]
    narrow = [MLPEnsemble((4, 16, 3), members=1, seed=k) for k in range(6)]
    train(wide[0], steps)
    others = [threading.Thread(target=train, args=(n, 10 ** 9)) for n in narrow]
    for t in others:
        t.start()
    train(wide[1], steps)
    stop.set()
    for t in others:
        t.join()
    assert not errors
    assert np.array_equal(wide[0].params(), wide[1].params())
    for n in wide + narrow:
        n.close()
