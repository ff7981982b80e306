"""Irreps of the two-fold adjoint product as symmetric tensors (k_gen_sym2): against the tensor
path at volumes around the 32 links of a block, and against the same irrep in a basis that
mixes weights, which has no sparse tensor form and runs on the product kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def forces(h):
    h.hot(0.7)
    h.phi_gaussian(12345, 0.4)
    return h.matter_link_force(), h.scalar_force(), h.measure()["S_H"]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-5)])
@pytest.mark.parametrize("N,rows,L", [(3, [4, 2], [1, 1]), (3, [4, 2], [31, 1]), (3, [4, 2], [8, 4]), (3, [4, 2], [3, 11, 1]),
                                      (2, [4], [13, 5])])
def test_equals_tensor_path(N, rows, L, precision, tol):
    import gauge_higgs_b200 as gh
    h = gh.GaugeHiggsHMC(L, gh.GeneralRep(N, rows), seed=2, precision=precision, beta=5.0, kappa=0.12, lam=0.5)
    assert h.rep_path() == "product"
    a = forces(h)
    try:
        h.set_rep_path("tensor")
    except gh.GaugeHiggsError:
        h.set_rep_path("closed_form")
    b = forces(h)
    assert rel(a[0], b[0]) < tol and rel(a[1], b[1]) < tol and abs(a[2] - b[2]) <= tol * abs(b[2])
    h.close()


def test_mixed_basis_keeps_the_product_kernel():
    import gauge_higgs_b200 as gh
    rep = gh.GeneralRep(3, [4, 2])
    g = np.random.default_rng(3)
    V, _ = np.linalg.qr(g.normal(size=(27, 27)) + 1j * g.normal(size=(27, 27)))
    mixed = gh.GeneralRep(3, [4, 2], T=np.einsum("ki,aij,lj->akl", V.conj(), rep.T, V), W=V @ rep.W)
    L, out = [3, 5, 3], []
    for r, B in ((rep, np.eye(27)), (mixed, V.conj())):
        h = gh.GaugeHiggsHMC(L, r, seed=2, beta=5.0, kappa=0.12, lam=0.5)
        assert h.rep_path() == "product"
        if r is rep:
            h.hot(0.7)
            h.phi_gaussian(12345, 0.4)
            U, phi = h.U, h.phi
        else:
            h.U, h.phi = U, phi @ B.T
        out.append((h.matter_link_force(), h.scalar_force() @ B.conj(), h.measure()["S_H"]))
        h.close()
    for a, b in zip(*out):
        assert rel(np.asarray(b), np.asarray(a)) < 1e-12
