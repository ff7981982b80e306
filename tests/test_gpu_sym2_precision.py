"""Matter force of the symmetric-tensor irreps on FP32 fields: its sums run in double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_and_columns_cancel():
    """Unit links and phi(x) = i^(x_0 + x_1) v with v real and of weight zero: the tensor of v is
    diagonal and exact at every step, so the force is the difference of equal sums over rows and
    columns.  In double that leaves a few 2^-53 of their size, 4 kappa w |v|^2 (w <= 2)."""
    import gauge_higgs_b200 as gh
    rep = gh.GeneralRep(3, [4, 2])
    L, kappa = [4, 8], 0.117
    cartan = [t for t in rep.T if np.abs(t - np.diag(np.diag(t))).max() < 1e-12]
    zero = [m for m in range(rep.d) if all(abs(t[m, m]) < 1e-12 for t in cartan)]
    assert len(cartan) == 2 and len(zero) == 3
    v = np.zeros(rep.d)
    v[zero] = np.float32(np.random.default_rng(2).normal(size=len(zero)))
    h = gh.GaugeHiggsHMC(L, rep, seed=2, precision="fp32", beta=5.0, kappa=kappa, lam=0.5)
    assert h.rep_path() == "product"
    h.cold()
    x = np.arange(np.prod(L))
    h.phi = (1j ** ((x % L[0] + x // L[0]) % 4))[:, None] * v
    F = h.matter_link_force()
    h.close()
    assert np.abs(F).max() < 1e-14 * 8 * kappa * (v @ v)


@pytest.mark.parametrize("N,rows", [(3, [4, 2]), (2, [4])])
def test_force_of_the_same_fields(N, rows):
    """FP32 against FP64 on the same FP32 fields: the roundings of the links' products and of psi
    remain, about ten of 2^-24 each against the largest of some hundred forces."""
    import gauge_higgs_b200 as gh
    rep = gh.GeneralRep(N, rows)
    h = [gh.GaugeHiggsHMC([5, 4, 3], rep, seed=2, precision=p, beta=5.0, kappa=0.12, lam=0.5) for p in ("fp32", "fp64")]
    h[0].hot(0.7)
    h[0].phi_gaussian(12345, 0.4)
    h[1].U, h[1].phi = h[0].U, h[0].phi
    a, b = (k.matter_link_force() for k in h)
    for k in h:
        k.close()
    assert np.abs(a - b).max() < 2e-6 * np.abs(b).max()
