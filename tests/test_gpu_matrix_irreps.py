"""The register path of the one-fold adjoint product (k_gen_pair with U Phi U^dag): a basis with
complex entries against the library's real one, and the FP32 force's error against FP64 on the
same links at volumes around a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("N,rows", [(3, [2, 1]), (2, [2]), (3, [2]), (3, [1, 1])])
def test_complex_basis(N, rows):
    import gauge_higgs_b200 as gh
    rep = gh.GeneralRep(N, rows)
    g = np.random.default_rng(5)
    V, _ = np.linalg.qr(g.normal(size=(rep.d, rep.d)) + 1j * g.normal(size=(rep.d, rep.d)))
    mixed = gh.GeneralRep(N, rows, T=np.einsum("ki,aij,lj->akl", V.conj(), rep.T, V), W=V @ rep.W)
    out = []
    for r, B in ((rep, np.eye(rep.d)), (mixed, V.conj())):
        h = gh.GaugeHiggsHMC([5, 3, 3], r, seed=2, beta=5.0, kappa=0.12, lam=0.5)
        if r is rep:
            h.hot(0.7)
            h.phi_gaussian(12345, 0.4)
            U, phi = h.U, h.phi
        else:
            h.U, h.phi = U, phi @ B.T
        out.append((h.rep_path(), h.matter_link_force(), h.scalar_force() @ B.conj(), h.measure()["S_H"]))
        h.close()
    assert out[0][0] == out[1][0] and out[0][0] in ("product", "pair")
    for a, b in zip(out[0][1:], out[1][1:]):
        assert rel(np.asarray(b), np.asarray(a)) < 1e-12


@pytest.mark.parametrize("L", [[1, 1], [127, 1], [43, 3], [4, 4, 8]])
def test_fp32_force_against_fp64(L):
    # rounding of the FP32 fields and of a handful of 3 x 3 products: a few 2^-24 of the largest entry
    import gauge_higgs_b200 as gh
    out = []
    for prec in ("fp32", "fp64"):
        h = gh.GaugeHiggsHMC(L, gh.GeneralRep(3, [2, 1], real=True), seed=6, precision=prec, beta=5.0, kappa=0.12, lam=0.5)
        if out:
            h.U, h.phi = U, phi
        else:
            h.hot(0.7)
            h.phi_gaussian(12345, 0.4)
            U, phi = h.U, h.phi
        out.append((h.matter_link_force(), h.scalar_force()))
        h.close()
    assert rel(out[0][0], out[1][0]) < 2e-6 and rel(out[0][1], out[1][1]) < 2e-6
