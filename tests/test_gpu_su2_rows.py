"""SU(2) links read by their first row in the kick, and the exponential's series in the drift on
both sides of its r = 1/2 limit: against the oracle (FP64) and the FP64 result (FP32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("L", [[2, 3], [5, 4, 3], [3, 2, 5, 4]])
@pytest.mark.parametrize("rep", ["fund", "adj", "none"])
def test_forces(orc, rep, L):
    import gauge_higgs_b200 as gh
    from oracle.oracle import REP_ADJ, REP_FUND
    D = len(L)
    U = orc.hot_start(D, 2, L, 5, 0.9)
    r = None if rep == "none" else gh.make_rep(2, rep)
    out = {}
    for prec in ("fp64", "fp32"):
        h = (gh.GaugeHMC(L, 2, seed=5, precision=prec, beta=2.3) if r is None else
             gh.GaugeHiggsHMC(L, r, seed=5, precision=prec, beta=2.3, kappa=0.2, lam=0.5))
        h.U = U
        F = h.gauge_force()
        if r is not None:
            h.phi_gaussian(12345, 0.5)
            F = F + h.matter_link_force()
            out[prec] = (F, h.scalar_force())
            phi = h.phi
        else:
            out[prec] = (F,)
        h.close()
        if prec == "fp64":
            Fo = orc.gauge_force(D, 2, L, U, 2.3)
            if r is not None:
                o = orc.rep(REP_FUND if rep == "fund" else REP_ADJ, 2)
                Fo = Fo + orc.matter_force(D, 2, L, o, U, phi, 0.2)
                assert rel(out[prec][1].reshape(-1), orc.scalar_force(D, 2, L, o, U, phi, 0.2, 0.5).reshape(-1)) < 1e-12
            assert rel(F.reshape(-1), Fo.reshape(-1)) < 1e-12
    for a, b in zip(out["fp32"], out["fp64"]):
        assert rel(a, b) < 2e-6


@pytest.mark.parametrize("scale", [0.0, 1e-9, 0.1, 0.99, 1.01, 3.0, 40.0])
def test_drift_exponential(scale):
    # P = 2 r n, so the exponential's angle at eps = 1/2 is r / 2; scale is r
    import gauge_higgs_b200 as gh
    L = [4, 5]
    g = np.random.default_rng(4)
    n = g.normal(size=(20, 2, 3))
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    for prec, tol in (("fp64", 2e-15), ("fp32", 2e-7)):
        h = gh.GaugeHMC(L, 2, seed=1, precision=prec)
        h.hot(0.9)
        U0 = h.U
        P = 2 * scale * n
        if prec == "fp32":
            P = P.astype(np.float32).astype(np.float64)
        h.P = P
        h.drift(0.5)
        v = 0.5 * P
        r = 0.5 * np.linalg.norm(v, axis=-1)[..., None, None]
        H = 0.5 * np.stack([np.stack([v[..., 2], v[..., 0] - 1j * v[..., 1]], -1), np.stack([v[..., 0] + 1j * v[..., 1], -v[..., 2]], -1)], -2)
        E = np.cos(r) * np.eye(2) + 1j * np.sinc(r / np.pi) * H
        # beyond the series (r > 1/2: sincos, as before it) the angle's own rounding, 3 units in
        # the last place of r from its sum of squares and root, enters as 3 r 2^-53
        far = 3 * float(r.max()) * 2.0 ** -53 if scale > 1 else 0.0
        assert np.abs(h.U - E @ U0).max() < tol + far
        h.close()
