"""The heatbath's draws split over four blocks per item: the same bits as whole items, which a
batch too large for the split uses, in volumes around 32 and 128 sites."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rep,N", [("fund", 2), ("adj", 3)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("L", [[1, 1], [31, 1], [8, 4], [127, 1], [43, 3], [5, 7, 4]])
def test_split_draws(rep, N, precision, L):
    import gauge_higgs_b200 as gh
    out = []
    for more in (0, 200):                     # 200 lattices of 8 x 8 x .. sites: 1000 items or more
        ext = [L] + [[16] * len(L)] * more
        e = gh.Ensemble(ext, gh.make_rep(N, rep), seeds=range(7, 8 + more), precision=precision, beta=2.0, kappa=0.1, nmd=2)
        e.hot(0.8)
        e.phi_gaussian(12345, 0.3)
        e.refresh_momenta()
        out.append([e.get(k, 0) for k in ("P", "pi", "phi")])
        rec = e.run(1)                        # and the reject copy taken with the draws
        out[-1] += [e.get("U", 0), rec["dH"][:, 0]]
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
