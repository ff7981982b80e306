"""The links of a kick cut into slabs (links and momenta beyond L2), against the two forces
computed alone: those launches walk the links-only table, whose order has no slabs' site items."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rep,N,L", [("fund", 3, [20, 20, 20, 21]), ("adj", 3, [20, 20, 20, 20]), ("fund", 2, [28, 28, 28, 27])])
def test_momenta_are_the_sum_of_the_forces(rep, N, L):
    import gauge_higgs_b200 as gh
    h = gh.GaugeHiggsHMC(L, gh.make_rep(N, rep), seed=3, precision="fp64", beta=5.0, kappa=0.1, lam=0.5)
    h.hot(0.8)
    h.phi_gaussian(12345, 0.3)
    h.refresh_momenta()
    P0 = h.P
    h.kick(0.05)
    P1 = h.P
    F = h.gauge_force() + h.matter_link_force()
    h.close()
    # P - eps F, both in a few roundings of numbers of the size of P and of F's terms (beta)
    assert np.abs(P0 - 0.05 * F - P1).max() < 1e-13 * max(np.abs(P1).max(), np.abs(F).max())
    # no link left as it was: a component may keep its value by chance, a whole link not
    assert (P1 != P0).any(axis=2).all()
