"""Contexts that live side by side: what one needs of a kernel does not change under another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spin(n, precision="fp64"):
    import gauge_higgs_b200 as gh
    h = gh.GaugeHiggsHMC([4, 4, 3], gh.GeneralRep(2, [n]), seed=5, precision=precision, beta=2.0, kappa=0.1, lam=0.5, nmd=4, tau=0.2)
    h.hot(0.5)
    h.phi_gaussian(12345, 0.3)
    return h


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_smaller_context_leaves_the_larger_alone(precision):
    a = spin(12, precision)
    want = a.matter_link_force(), a.scalar_force(), a.run(2)
    a.close()
    a, b = spin(12, precision), spin(6, precision)
    got = a.matter_link_force(), a.scalar_force(), a.run(2)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
    a.close()
    b.close()
