"""SU(2) {n} through k_gen_spin: forces and hopping action against D(U) = exp(i w.T) with w read
off the link, at volumes around the 32 links of a block, and the multi-invariant potential's
w against its superoperator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def d_matrix(T, U):
    """exp(i w.T_R) for U = cos r + i sin r n.sigma, w = 2 r n ([V, 2, 2] -> [V, d, d])."""
    s = np.stack([U[:, 0, 1].imag + U[:, 1, 0].imag, U[:, 0, 1].real - U[:, 1, 0].real, U[:, 0, 0].imag - U[:, 1, 1].imag], 1) / 2
    sn = np.linalg.norm(s, axis=1)
    r = np.arctan2(sn, 0.5 * (U[:, 0, 0] + U[:, 1, 1]).real)
    w = 2 * s * np.where(sn > 1e-300, r / np.maximum(sn, 1e-300), 1.0)[:, None]
    e, v = np.linalg.eigh(np.einsum("va,aij->vij", w, T))
    return np.einsum("vik,vk,vjk->vij", v, np.exp(1j * e), v.conj())


@pytest.mark.parametrize("n,L", [(5, [1, 1]), (6, [31, 1]), (8, [8, 4]), (12, [3, 11]), (12, [5, 4, 3]), (13, [3, 2, 2, 3]), (17, [4, 3])])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 3e-6)])
def test_forces(n, L, precision, tol):
    import gauge_higgs_b200 as gh
    rep, D, V = gh.GeneralRep(2, [n]), len(L), int(np.prod(L))
    kappa, lam, f = 0.11, 0.5, None
    h = gh.GaugeHiggsHMC(L, rep, seed=3, precision=precision, beta=2.0, kappa=kappa, lam=lam)
    assert h.rep_path() == "closed_form"
    h.hot(0.8)
    h.phi_gaussian(12345, 0.3)
    U, phi = h.U, h.phi
    F, S, m = h.matter_link_force(), h.scalar_force(), h.measure()
    A = None
    if n <= 8:
        ch = gh.CasimirChannels(rep)
        f = np.linspace(0.05, 0.15, ch.n_channels())
        h.potential = gh.MultiInvariantPotential(ch, f, 0.07)
        A = ch.superop(f)
        S2 = h.scalar_force()
    h.close()
    st = np.cumprod([1] + L[:-1])
    s = np.arange(V)
    Fo, hop, sh = np.zeros((V, D, 3)), 0.0, np.zeros_like(phi)
    for mu in range(D):
        x = s // st[mu] % L[mu]
        fw = np.where(x + 1 < L[mu], s + st[mu], s - x * st[mu])
        Dm = d_matrix(rep.T, U[:, mu])
        psi = np.einsum("vij,vj->vi", Dm, phi[fw])
        back = np.zeros_like(psi)
        back[fw] = np.einsum("vji,vj->vi", Dm.conj(), phi)
        Fo[:, mu] = 2 * kappa * np.imag(np.einsum("vi,aij,vj->va", phi.conj(), rep.T, psi))
        sh += 2 * kappa * (psi + back)
        hop += np.real(np.sum(phi.conj() * psi))
    n2 = (np.abs(phi) ** 2).sum(1)
    So = sh - 2 * (1 + 2 * lam * (n2 - 1))[:, None] * phi
    assert np.abs(F - Fo).max() < tol * np.abs(Fo).max()
    assert np.abs(S - So).max() < tol * np.abs(So).max()
    assert abs(m["L_link"] - hop / (V * D)) < tol * max(1.0, n2.mean())
    if A is not None:
        M = np.einsum("vi,vj->vij", phi, phi.conj()).reshape(V, -1)
        w = np.einsum("vij,vj->vi", (M @ A.T).reshape(V, rep.d, rep.d), phi)
        So = sh + 2 * 0.07 * phi - 2 * w
        assert np.abs(S2 - So).max() < max(tol, 1e-11) * np.abs(So).max()
