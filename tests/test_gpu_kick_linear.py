"""Kick items over consecutive sites (extents that power-of-two tiles do not divide): the same
forces, momenta and pi bit for bit as one-site tiles, at volumes below, at and past the 128
sites of a block, extents of 1 and odd ones, and a ladder of unequal lattices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("L", [[3, 1, 1, 1], [5, 3, 2, 1], [7, 3, 3, 2], [3, 43], [129, 3], [5, 5, 5], [9, 9, 9, 3],
                               [12, 10, 6, 7]])
def test_linear_items_equal_one_site_tiles(L, precision):
    import gauge_higgs_b200 as gh
    for rep in (gh.FundamentalRep(2), gh.AdjointRep(3), gh.GeneralRep(3, [2])):
        h = gh.GaugeHiggsHMC(L, rep, seed=3, precision=precision, beta=5.0, kappa=0.1, lam=0.5)
        h.hot(0.8)
        h.phi_gaussian(12345, 0.3)
        h.refresh_momenta()
        P0, pi0 = h.P, h.pi
        h.kick(0.05)
        P1, pi1 = h.P, h.pi
        assert not np.array_equal(P1, P0)
        h.P, h.pi = P0, pi0
        h.set_tile([1] * len(L))
        h.kick(0.05)
        assert np.array_equal(h.P, P1) and np.array_equal(h.pi, pi1)
        h.close()


def test_linear_items_of_a_batch():
    import gauge_higgs_b200 as gh
    ext = [[4] * 4, [5, 3, 7, 2], [6] * 4, [8, 4, 4, 4]]
    one = []
    for tile in (None, [1] * 4):
        e = gh.Ensemble(ext, gh.FundamentalRep(2), seeds=[1, 2, 3, 4], precision="fp64", beta=2.3, kappa=0.2, nmd=3)
        e.hot(0.8)
        e.phi_gaussian(12345, 0.3)
        if tile:
            e.set_tile(tile)
        rec = e.run(2)
        one.append((rec, [e.get("U", i) for i in range(4)]))
        assert e.autotune(reps=1) > 0
        e.close()
    assert np.array_equal(one[0][0], one[1][0])
    for a, b in zip(one[0][1], one[1][1]):
        assert np.array_equal(a, b)
