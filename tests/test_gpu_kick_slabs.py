"""Kicks cut into slabs (links and momenta beyond L2): every link and site is still done once --
the same P and pi bit for bit as with one-site tiles, whose order is another, and forces of one
kind alone equal the kick's parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rep,N,L,tile", [("fund", 3, [20, 20, 20, 21], None), ("fund", 3, [32, 16, 16, 32], [8, 4, 2, 2]),
                                          ("adj", 3, [20, 20, 20, 20], None), ("fund", 2, [28, 28, 28, 27], None),
                                          ("4", 2, [32, 32, 32, 16], [16, 8, 1, 1])])
def test_every_item_once(rep, N, L, tile):
    import gauge_higgs_b200 as gh
    h = gh.GaugeHiggsHMC(L, gh.make_rep(N, rep), seed=3, precision="fp64", beta=5.0, kappa=0.1, lam=0.5)
    h.hot(0.8)
    h.phi_gaussian(12345, 0.3)
    h.refresh_momenta()
    P0, pi0 = h.P, h.pi
    if tile:
        h.set_tile(tile)
    h.kick(0.05)
    P1, pi1 = h.P, h.pi
    assert not (P1 == P0).any(axis=(1, 2)).all()
    h.P, h.pi = P0, pi0
    h.set_tile([1] * 4)
    h.kick(0.05)
    assert np.array_equal(h.P, P1) and np.array_equal(h.pi, pi1)
    del P0
    F = h.scalar_force()
    assert np.abs(pi0 + 0.05 * F - pi1).max() < 1e-13 * np.abs(pi1).max()
    h.close()


def test_ensemble_beyond_l2():
    import gauge_higgs_b200 as gh
    ext = [[16] * 4, [12, 10, 9, 8], [16, 16, 16, 8], [16] * 4, [17, 16, 16, 16]]
    out = []
    for tile in (None, [1] * 4):
        e = gh.Ensemble(ext, gh.FundamentalRep(3), seeds=range(1, 6), precision="fp64", beta=5.7, kappa=0.1, nmd=2)
        e.hot(0.8)
        e.phi_gaussian(12345, 0.3)
        if tile:
            e.set_tile(tile)
        out.append(e.run(1))
        e.close()
    assert np.array_equal(out[0], out[1])
