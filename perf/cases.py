"""The work that a program built on this framework has it do, as cases that can be timed and
compared: whole HMC measurement loops over the gauge groups, representations, integrators,
precisions and lattice sizes that the drivers, the tests and the benchmark run, a batched
tempering ladder, a driver with host-resident fields, and the training of the coupling-scan
surrogate.

A lattice case is the drivers' measurement loop: a trajectory, its record, the Polyakov loop;
after the last trajectory the configuration is taken as device tensors (whole planes by
gh_halo_pack, in the precision the fields are held in).  `exact` is the same computation in
plain torch, complex128."""
import ctypes
import math

import numpy as np
import torch

import gauge_higgs_b200 as gh
from gauge_higgs_b200._lib import LIB, check
from gauge_higgs_b200.mlp import MLPEnsemble

OMELYAN = 0.1931833275037836
# 13 channel couplings and mu^2 of the SU(2) spin-6 (2I) potential
F2I = [0.1182, 0.0819, 0.0353, 0.0274, 0.1550, 0.0828, 0.0157, 0.0702, 0.1083, 0.1143, 0.0189, 0.1124, 0.0595]
MU2 = 0.065


def _case(name, N, rep, L, prec, beta, kappa, nmd, ntraj=1, integ="omelyan", tau=1.0, lam=0.5, kind="loop"):
    return {"name": name, "kind": kind, "N": N, "rep": rep, "L": L, "prec": prec, "beta": beta, "kappa": kappa,
            "lam": lam, "nmd": nmd, "tau": tau, "integ": integ, "ntraj": ntraj}


def listed():
    return [
        # the reference's small validation run: SU(2) + fundamental, 6^4, leapfrog; each launch is a
        # few microseconds of work, so launches and latency are what a user waits for
        _case("su2_fund_6x4_f64", 2, "fund", "6x6x6x6", "fp64", 2.3, 0.20, 20, 4, "leapfrog"),
        # a kappa ladder over unequal extents, one batch with swaps on the device: how the
        # transition is located
        _case("su2_ladder_f32", 2, "fund", "6,8,10,12", "fp32", 2.3, 0.22, 20, 4, kind="ladder"),
        # SU(3) + fundamental at 16^4 in the two precisions: the configuration that rates are quoted on
        _case("su3_fund_16x4_f32", 3, "fund", "16x16x16x16", "fp32", 5.7, 0.10, 16, 3),
        _case("su3_fund_16x4_f64", 3, "fund", "16x16x16x16", "fp64", 5.7, 0.10, 16, 2),
        # the largest lattice the benchmark runs: fields far beyond L2
        _case("su3_fund_32x4_f32", 3, "fund", "32x32x32x32", "fp32", 5.7, 0.10, 16),
        # a host program that keeps U and phi in its own memory, uploaded and downloaded around
        # every trajectory; ragged extents
        _case("su3_fund_host_f64", 3, "fund", "14x14x14x18", "fp64", 5.7, 0.10, 16, kind="host"),
        # adjoint Higgs, odd extents
        _case("su3_adj_9x9x9x12_f64", 3, "adj", "9x9x9x12", "fp64", 5.7, 0.10, 20),
        # the general-irrep configuration's three representations at its size
        _case("su3_sextet_12x4_f64", 3, "2", "12x12x12x12", "fp64", 5.7, 0.10, 20),
        _case("su3_octet_12x4_f32", 3, "2,1:real", "12x12x12x12", "fp32", 5.7, 0.10, 20),
        _case("su3_27plet_12x4_f64", 3, "4,2:real", "12x12x12x12", "fp64", 5.7, 0.10, 20),
        # SU(2) spin 6 with the 13-channel potential, the SU(2) -> 2I breaking study's point at 8^4
        _case("su2_spin6_8x4_f64", 2, "12m", "8x8x8x8", "fp64", 2.0, 0.10, 40),
        # the coupling-scan surrogate: five networks fitted to a campaign's points, then evaluated
        # on a kappa grid
        {"name": "surrogate_fit", "kind": "fit", "n": 208, "members": 5, "hidden": 128, "epochs": 20, "batch": 32,
         "grid": 401},
    ]


def draw(rng):
    """One more case of the same ranges: group, representation, precision and integrator as
    the drivers take them, extents of 3 to 24 (odd ones among them) in two to four dimensions."""
    if rng.random() < 0.12:
        return {"kind": "fit", "n": rng.randint(60, 200), "members": rng.randint(2, 5), "hidden": rng.choice([48, 64, 100, 128]),
                "epochs": rng.randint(4, 16), "batch": rng.choice([24, 32, 48, 64]), "grid": rng.randint(50, 500)}
    prec = rng.choice(["fp64", "fp32"])
    integ = rng.choice(["omelyan", "omelyan", "leapfrog"])
    nmd = rng.randint(10, 24)
    if rng.random() < 0.12:
        sizes = sorted(rng.sample(range(4, 13), rng.randint(2, 4)))
        c = _case("", 2, "fund", ",".join(map(str, sizes)), prec, round(rng.uniform(2.1, 2.5), 3), 0.22, nmd, 2, integ,
                  kind="ladder")
    else:
        N = rng.choice([2, 3, 3])
        reps = ["fund", "fund", "adj", "none", "12m"] if N == 2 else ["fund", "fund", "fund", "adj", "none", "2",
                                                                      "2,1:real", "4,2:real"]
        rep = rng.choice(reps)
        # sites: spread over their logarithm; the irreps of large dimension stop earlier
        top = {"4,2:real": 12 ** 4, "12m": 8 ** 4, "2": 16 ** 4, "2,1:real": 16 ** 4, "adj": 16 ** 4}.get(rep, 24 ** 4)
        v = math.exp(rng.uniform(math.log(4 ** 4), math.log(top)))
        D = rng.choice([4, 4, 4, 4, 4, 4, 3, 2])
        if D < 4:
            v = min(v, 24.0 ** D)
        L, left = [], v
        for mu in range(D):
            x = left ** (1.0 / (D - mu)) * (rng.uniform(0.75, 1.35) if mu + 1 < D else 1.0)
            L.append(max(3, min(24, int(round(x)))))
            left = max(1.0, left / L[-1])
        if rep == "12m":        # the stiff potential: small steps
            nmd, beta, kappa = 40, 2.0, 0.1
        else:
            beta, kappa = (round(rng.uniform(2.0, 2.5), 3), round(rng.uniform(0.1, 0.3), 3)) if N == 2 else (
                round(rng.uniform(5.5, 6.0), 3), round(rng.uniform(0.05, 0.15), 3))
        kind = "host" if rng.random() < 0.15 else "loop"
        big = float(np.prod(L)) > 10 ** 5 or rep in ("4,2:real", "2,1:real", "12m")
        c = _case("", N, rep, "x".join(map(str, L)), "fp64" if kind == "host" else prec, beta, kappa, nmd,
                  1 if big or kind == "host" else rng.randint(1, 3), integ, kind=kind)
    c.pop("name")
    return c


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _lattices(case):
    """(extents, kappa) of every lattice of the case: one, or four kappas for each size."""
    if case["kind"] != "ladder":
        return [([int(x) for x in case["L"].split("x")], case["kappa"])]
    return [([int(s)] * 4, case["kappa"] + 0.03 * i) for s in case["L"].split(",") for i in range(4)]


def _rep(case):
    r = case["rep"]
    return None if r == "none" else gh.make_rep(case["N"], "12" if r == "12m" else r)


def _seeds(case, seed):
    return [int(seed) + 1 + 1000 * i for i in range(len(_lattices(case)))]


def _real(case):
    return case["rep"] == "adj" or case["rep"].endswith(":real")


def _fit_data(case, seed):
    """Points (beta, kappa, lambda, 1/L) in units of the scan's box and smooth observables of
    them with measurement noise, standardised: what a campaign hands to the fit."""
    g = torch.Generator().manual_seed(int(seed))
    x = torch.rand(case["n"], 4, generator=g, dtype=torch.float64) * 2 - 1
    t = x[:, 1] + 0.3 * x[:, 0] + 0.2 * x[:, 2]
    y = torch.stack([torch.tanh(3 * t), 2 * torch.exp(-8 * t * t) + 0.3 * x[:, 3], 0.5 * x[:, 0] + 0.2 * torch.tanh(2 * t)], 1)
    y = y + 0.02 * torch.randn(y.shape, generator=g, dtype=torch.float64)
    y = (y - y.mean(0)) / y.std(0)
    grid = torch.zeros(case["grid"], 4, dtype=torch.float64)
    grid[:, 1] = torch.linspace(-1, 1, case["grid"], dtype=torch.float64)
    grid[:, 3] = float(torch.rand(1, generator=g))
    return x.float().numpy(), y.float().numpy(), grid.float().numpy()


def _widths(case):
    return (4, case["hidden"], case["hidden"], case["hidden"], 3)


def prepare(case, seed):
    if case["kind"] == "fit":
        x, y, grid = _fit_data(case, seed)
        return {"case": case, "net": MLPEnsemble(_widths(case), case["members"], int(seed) + 1), "x": x, "y": y, "grid": grid}
    lats, rep = _lattices(case), _rep(case)
    common = dict(precision=case["prec"], beta=case["beta"], tau=case["tau"], nmd=case["nmd"], integ=case["integ"])
    if case["kind"] == "ladder":
        h = gh.Ensemble([L for L, _ in lats], rep, seeds=_seeds(case, seed), kappa=[k for _, k in lats], lam=case["lam"], **common)
        h.enable_tempering(True)
    elif rep is None:
        h = gh.GaugeHMC(lats[0][0], case["N"], seed=_seeds(case, seed)[0], **common)
    else:
        h = gh.GaugeHiggsHMC(lats[0][0], rep, seed=_seeds(case, seed)[0], kappa=case["kappa"], lam=case["lam"], **common)
    if case["rep"] == "12m":
        h.potential = gh.MultiInvariantPotential(gh.CasimirChannels(rep), F2I, MU2)
    h.hot(0.8)
    if rep is not None:
        h.phi_gaussian(12345, 0.3)
    state = {"case": case, "h": h}
    if case["kind"] == "host":          # the program's own fields, in pinned memory
        state["keep"] = []
        for k in ("U", "phi") if rep is not None else ("U",):
            v = h.get(k)
            p = torch.empty(v.shape, dtype=torch.complex128).pin_memory()
            p.copy_(torch.from_numpy(v))
            state["keep"].append(p)
            state[k] = p.numpy()
    else:
        state["snap"] = [_planes(case, h, i, L) for i, (L, _) in enumerate(lats)]
    return state


def _planes(case, h, lat, L):
    """Device tensors for every plane x_nu = const of one lattice's U and phi, nu the shortest
    direction: [plane][component * site, padded to 16 bytes] complex."""
    nu = min(range(len(L)), key=lambda m: L[m])
    n = int(np.prod(L)) // L[nu]
    dt = torch.complex128 if case["prec"] == "fp64" else torch.complex64
    out = {"lat": lat, "nu": nu, "n": L[nu]}
    for f, ncomp in ((0, len(L) * case["N"] ** 2),) + (((1, h.d),) if h.d else ()):
        out[f] = torch.zeros((L[nu], (n * ncomp + 1) // 2 * 2), dtype=dt, device="cuda")
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _configuration(s):
    """U and phi of every lattice into the program's device tensors."""
    ctx, got = s["h"].ctx.h, []
    for p in s["snap"]:
        for f in (0, 1):
            if f in p:
                row = p[f].stride(0) * p[f].element_size()
                for x in range(p["n"]):
                    check(LIB.gh_halo_pack(ctx, p["lat"], f, p["nu"], x, ctypes.c_void_p(p[f].data_ptr() + x * row)), ctx)
        got.append({"U": p[0], "phi": p[1]} if 1 in p else {"U": p[0]})
    return got


def _table(rows, case):
    """The records as a table, dH first.  With FP32 fields dH is the difference of two sums of
    10^5 to 10^7 whose last digits are the fields' rounding: three digits of it mean something,
    so it is kept apart, in half precision."""
    if case["prec"] == "fp64":
        return {"records": np.array(rows, np.float64)}
    t = np.array(rows, np.float64)
    return {"records": t[:, 1:].astype(np.float32), "dH": t[:, 0].astype(np.float16)}


def _row(r):
    return [float(r[k]) for k in ("dH", "accepted", "traj", "plaquette", "L_phi", "L_link", "kappa", "beta")]


def run(s):
    case = s["case"]
    if case["kind"] == "fit":
        net = s["net"]
        loss = net.train(s["x"], s["y"], epochs=case["epochs"], batch=case["batch"], lr=1e-3, seed=7)
        mean, var, per = net.predict(s["grid"], members=True)
        return {"loss": loss, "params": net.params(), "mean": mean, "var": var, "per_member": per}
    h = s["h"]
    if case["kind"] == "host":
        r = h.trajectory_host(s["U"], s.get("phi"))
        row = [r.dH, r.accepted, r.traj, r.plaquette, r.L_phi, r.L_link, r.kappa, r.beta]
        return {**_table([row], case), "U": s["U"], **({"phi": s["phi"]} if "phi" in s else {})}
    if case["kind"] == "ladder":
        rec = h.run(case["ntraj"])
        return {**_table([_row(r) for t in rec for r in t], case), "lattices": _configuration(s)}
    rows = []
    for _ in range(case["ntraj"]):
        r = h.run(1)[0, 0]
        rows.append(_row(r) + [h.polyakov_loop()])
    return {**_table(rows, case), "lattices": _configuration(s)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the configuration (and for the fit the data and parameters) in and out once per
    pass.  Flops: the reference's force and update arithmetic with complex N x N products, the
    irreps' hops as applications of their smallest tensor form."""
    if case["kind"] == "fit":
        w = _widths(case)
        P = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
        steps = case["epochs"] * -(-case["n"] // case["batch"])
        fwd = 2.0 * sum(a * b for a, b in zip(w[:-1], w[1:])) * case["members"]
        return {"bytes": 4.0 * (case["members"] * (2 * P + 3 * case["grid"]) + 7 * case["n"] + 10 * case["grid"]),
                "flops": fwd * (3.0 * case["n"] * case["epochs"] + case["grid"]) + 12.0 * P * case["members"] * steps}
    N, total = case["N"], {"bytes": 0.0, "flops": 0.0}
    d, hop = {"none": (0, 0.0), "fund": (N, 8.0 * N * N), "adj": (N * N - 1, 16.0 * N ** 3), "2": (6, 16.0 * 27),
              "2,1:real": (8, 16.0 * 27), "4,2:real": (27, 16.0 * 216), "12m": (13, 8.0 * 169)}[case["rep"]]
    mm = 8.0 * N ** 3
    for L, _ in _lattices(case):
        D, V = len(L), float(np.prod(L))
        real = 8.0 if case["prec"] == "fp64" else 4.0
        kick = D * ((4 * (D - 1) + 1) * mm + 2 * hop + 8.0 * d * N + 4 * N * N) + 12.0 * d * D
        drift = D * (5 * mm) + 4.0 * d
        steps = case["ntraj"] * case["nmd"] * (1 if case["integ"] == "leapfrog" else 2)
        total["flops"] += V * ((steps + case["ntraj"]) * kick + steps * drift)
        total["bytes"] += V * 4.0 * real * (D * N * N + d)
    return total


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _mix(x):
    """splitmix64 of 64-bit integers (int64 tensors, wrapping arithmetic)."""
    x = x + _i64(0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _i64(0xBF58476D1CE4E5B9)
    x = (x ^ _shr(x, 27)) * _i64(0x94D049BB133111EB)
    return x ^ _shr(x, 31)


def _t(v):
    return v if isinstance(v, torch.Tensor) else torch.tensor(_i64(int(v)), dtype=torch.int64, device=_dev())


def _key(*parts):
    g = _i64(0x9E3779B97F4A7C15)
    h = _mix(_t(parts[0]))
    for p in list(parts[1:]) + [0] * (5 - len(parts)):
        h = _mix(h ^ (_t(p) + g))
    return h


def _uniform(seed, k):
    return (_shr(_mix(_t(seed) ^ _mix(k)), 11).double() + 0.5) * (1.0 / 9007199254740992.0)


def _gauss(seed, k):
    u1, u2 = _uniform(seed, _mix(k * 2 + 1)), _uniform(seed, _mix(k * 2 + 2))
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)


def _mm(a, b):
    """Products of small matrices: one fused broadcast multiply and sum per column of a."""
    r = a[..., :, 0:1] * b[..., 0:1, :]
    for k in range(1, a.shape[-1]):
        r = r + a[..., :, k:k + 1] * b[..., k:k + 1, :]
    return r


def _dag(a):
    return a.conj().transpose(-1, -2)


def _generators(N):
    T = []
    pairs = [(j, k) for j in range(N) for k in range(j + 1, N)]
    for s in (0, 1):
        for j, k in pairs:
            m = np.zeros((N, N), complex)
            m[j, k], m[k, j] = (0.5, 0.5) if s == 0 else (-0.5j, 0.5j)
            T.append(m)
    for l in range(1, N):
        c = math.sqrt(2.0 / (l * (l + 1)))
        T.append(np.diag([0.5 * c] * l + [-0.5 * c * l] + [0.0] * (N - l - 1)).astype(complex))
    return torch.tensor(np.array(T), device=_dev())


def _expi(H):
    """exp(iH) of Hermitian H: scaling and squaring around a Taylor series."""
    n = float(H.abs().pow(2).sum((-1, -2)).max().sqrt())
    s = max(0, math.ceil(math.log2(max(n, 1e-30) / 0.25)))
    A = 1j * H / 2 ** s
    E = torch.eye(H.shape[-1], dtype=H.dtype, device=H.device).expand(H.shape).clone()
    term = E
    for k in range(1, 15):
        term = _mm(term, A) / k
        E = E + term
    for _ in range(s):
        E = _mm(E, E)
    return E


def _permutations(blocks, n):
    """All permutations of range(n) that keep each block, with their signs."""
    from itertools import permutations
    out = [(list(range(n)), 1)]
    for b in blocks:
        nxt = []
        for p, sg in out:
            for q in permutations(range(len(b))):
                inv = sum(q[i] > q[j] for i in range(len(q)) for j in range(i + 1, len(q)))
                g = list(p)
                for i, j in enumerate(q):
                    g[b[i]] = b[j]
                nxt.append((g, sg * (-1) ** inv))
        out = nxt
    return out


def _basis(N, rows):
    """Orthonormal basis of the irrep inside n tensor slots, [d][N^n]: the Young symmetriser
    (rows symmetrised, then columns antisymmetrised) of every basis tensor in index order,
    orthonormalised in that order."""
    n = sum(rows)
    if len(rows) == 1:
        idx = np.indices((N,) * n).reshape(n, -1).T
        hist = np.array([[int((t == v).sum()) for v in range(N)] for t in idx])
        kinds = sorted({tuple(h) for h in hist}, reverse=True)
        W = np.array([(hist == np.array(k)).all(1).astype(float) for k in kinds])
        return torch.tensor(W / np.sqrt(W.sum(1, keepdims=True)), device=_dev()).to(torch.complex128)
    rb, cb, pos = [], [[] for _ in range(rows[0])], 0
    for r in rows:
        rb.append(list(range(pos, pos + r)))
        for j in range(r):
            cb[j].append(pos + j)
        pos += r
    eye = np.eye(N ** n).reshape((N ** n,) + (N,) * n)
    sym = np.zeros_like(eye)
    for p, _ in _permutations(rb, n):
        sym += np.transpose(eye, [0] + [1 + x for x in np.argsort(p)])
    c = np.zeros_like(eye)
    for p, sg in _permutations(cb, n):
        c += sg * np.transpose(sym, [0] + [1 + x for x in np.argsort(p)])
    W = []
    for v in c.reshape(N ** n, -1):
        for _ in range(2):
            for w in W:
                v = v - (w @ v) * w
        norm = np.linalg.norm(v)
        if norm > 1e-9:
            W.append(v / norm)
    return torch.tensor(np.array(W), device=_dev()).to(torch.complex128)


class _Plain:
    """One lattice of a case, everything in 64 bits."""

    def __init__(self, case, L, kappa, seed):
        self.c, self.L, self.D, self.N, self.seed = case, L, len(L), case["N"], seed
        self.V = int(np.prod(L))
        self.beta, self.kappa, self.lam = case["beta"], kappa, case["lam"]
        dev = _dev()
        self.T = _generators(self.N)
        self.ng = len(self.T)
        s = np.arange(self.V)
        x, st = [], []
        for mu in range(self.D):
            st.append(int(np.prod(L[:mu])))
            x.append(s // st[-1] % L[mu])
        self.x = x
        self.fw = [torch.tensor(np.where(x[m] + 1 < L[m], s + st[m], s - x[m] * st[m]), device=dev) for m in range(self.D)]
        self.bw = [torch.tensor(np.where(x[m] > 0, s - st[m], s + (L[m] - 1) * st[m]), device=dev) for m in range(self.D)]
        self.site = torch.tensor(s, device=dev)
        self.rep = case["rep"]
        self.real = _real(case)
        r = self.rep
        if r == "none":
            self.d = 0
        elif r == "fund":
            self.d, self.TR = self.N, self.T
        elif r == "adj":
            self.d = self.ng
            self.TR = torch.stack([2 * torch.einsum("bij,cji->bc", self.T, a @ self.T - self.T @ a) for a in self.T])
        else:
            rows = [12] if r == "12m" else [int(v) for v in r.split(":")[0].split(",")]
            self.n = sum(rows)
            self.W = _basis(self.N, rows)
            self.d = self.W.shape[0]
            self.TR = torch.stack([self.W.conj() @ self._derivation(a).T for a in self.T])
        if r == "12m":
            self.A = self._channels(F2I)
        P = []
        for mu in range(self.D):
            P.append(torch.stack([0.8 * _gauss(seed, _key(1, self.site, mu, a)) for a in range(self.ng)], 1))
        self.U = [_expi(torch.einsum("va,aij->vij", p.to(torch.complex128), self.T)) for p in P]
        self.phi = self._vector(12345, 0.3) if self.d else None
        self.traj = 0

    def _vector(self, stream, sigma):
        re, im = [], []
        for k in range(self.d):
            re.append(sigma * _gauss(self.seed, _key(stream, self.site, 2 * k)))
            im.append(torch.zeros_like(re[0]) if self.real else sigma * _gauss(self.seed, _key(stream, self.site, 2 * k + 1)))
        return torch.complex(torch.stack(re, 1), torch.stack(im, 1))

    def _derivation(self, a):
        """a acting on every slot of each basis tensor, [d][N^n]."""
        d, out = self.d, 0
        for sl in range(self.n):
            w = self.W.reshape(d, self.N ** sl, self.N, -1)
            out = out + torch.einsum("ij,dajb->daib", a, w).reshape(d, -1)
        return out

    def _channels(self, f):
        """sum_c 2 f_c P_c on d x d matrices, P_c the eigenprojectors of sum_a [T^a, [T^a, .]]
        in ascending order of eigenvalue."""
        d, one = self.d, torch.eye(self.d, dtype=torch.complex128, device=_dev())
        C = 0
        for a in self.TR:
            ad = torch.kron(a, one) - torch.kron(one, a.T.contiguous())
            C = C + ad @ ad
        w, v = np.linalg.eigh(C.cpu().numpy())
        A, c, last = np.zeros((d * d, d * d), complex), -1, None
        cuts = []
        for i, e in enumerate(w):
            if last is None or e - last > 1e-4:
                cuts.append(i)
            last = e
        for c, i in enumerate(cuts):
            j = cuts[c + 1] if c + 1 < len(cuts) else len(w)
            A += 2 * f[c] * v[:, i:j] @ v[:, i:j].conj().T
        return torch.tensor(A, device=_dev())

    # ---- D(U) v and D(U)^dag v, [V][d] ----
    def hop(self, U, v, dag=False):
        M = _dag(U) if dag else U
        if self.rep == "fund":
            return _mm(M, v[..., None])[..., 0]
        if self.rep == "adj":
            Phi = torch.einsum("va,aij->vij", v, self.T)
            return 2 * torch.einsum("aij,vji->va", self.T, _mm(_mm(M, Phi), _dag(M)))
        if self.rep == "12m":       # exp(i w.T_R) with w from U = cos r + i sin r n.sigma
            a = torch.stack([2 * torch.einsum("ij,vji->v", t, M).imag for t in self.T], 1)
            sn = 0.5 * a.pow(2).sum(1, keepdim=True).sqrt()
            cs = 0.5 * (M[:, 0, 0] + M[:, 1, 1]).real[:, None]
            r = torch.atan2(sn, cs)
            w = a * torch.where(sn > 1e-150, r / sn.clamp_min(1e-150), torch.ones_like(sn))
            return torch.matmul(torch.matrix_exp(1j * torch.einsum("va,aij->vij", w.to(torch.complex128), self.TR)), v[..., None])[..., 0]
        out = []
        for z, m in zip(v.split(32768), M.split(32768)):
            t = z @ self.W
            for sl in range(self.n):
                t = torch.matmul(m[:, None], t.reshape(len(z), self.N ** sl, self.N, -1)).reshape(len(z), -1)
            out.append(t @ self.W.conj().T)
        return torch.cat(out)

    # ---- actions and forces ----
    def staples(self, mu):
        S = 0
        for nu in range(self.D):
            if nu == mu:
                continue
            f, g, b = self.fw[mu], self.fw[nu], self.bw[nu]
            S = S + _mm(_mm(self.U[nu][f], _dag(self.U[mu][g])), _dag(self.U[nu]))
            S = S + _mm(_mm(_dag(self.U[nu][f][b]), _dag(self.U[mu][b])), self.U[nu][b])
        return S

    def kick(self, eps):
        F = [(self.beta / self.N) * torch.einsum("aij,vji->va", self.T, _mm(self.U[mu], self.staples(mu))).imag
             for mu in range(self.D)]
        if self.d:
            Fp = self.potential()[1]
            for mu in range(self.D):
                psi = self.hop(self.U[mu], self.phi[self.fw[mu]])
                g = -2 * torch.stack([(self.phi.conj() * (psi @ a.T)).sum(1).imag for a in self.TR], 1)
                F[mu] = F[mu] - self.kappa * g
                Fp = Fp + 2 * self.kappa * (psi + self.hop(self.U[mu], self.phi, True)[self.bw[mu]])
            self.pi = self.pi + eps * Fp
        self.P = [p - eps * f for p, f in zip(self.P, F)]

    def potential(self):
        """sum V(phi) and -2 dV/dphi^*."""
        n2 = self.phi.abs().pow(2).sum(1)
        if self.rep == "12m":
            M = torch.einsum("vi,vj->vij", self.phi, self.phi.conj()).reshape(self.V, -1)
            w = torch.matmul((M @ self.A.T).reshape(self.V, self.d, self.d), self.phi[..., None])[..., 0]
            return float((-MU2 * n2 + 0.5 * (self.phi.conj() * w).sum(1).real).sum()), 2 * MU2 * self.phi - 2 * w
        return float((n2 + self.lam * (n2 - 1) ** 2).sum()), -2 * (1 + 2 * self.lam * (n2 - 1))[:, None] * self.phi

    def drift(self, eps):
        self.U = [_mm(_expi(torch.einsum("va,aij->vij", (eps * p).to(torch.complex128), self.T)), u) for p, u in zip(self.P, self.U)]
        if self.d:
            self.phi = self.phi + eps * self.pi

    def measure(self):
        tr = 0.0
        for mu in range(self.D):
            for nu in range(mu + 1, self.D):
                a = _mm(self.U[mu], self.U[nu][self.fw[mu]])
                b = _mm(self.U[nu], self.U[mu][self.fw[nu]])
                tr += float((a * b.conj()).real.sum())
        npl = self.V * self.D * (self.D - 1) // 2
        H = 0.5 * sum(float(p.pow(2).sum()) for p in self.P) + self.beta / self.N * (self.N * npl - tr)
        o = {"plaq": tr / (self.N * npl), "L_phi": 0.0, "L_link": 0.0}
        if self.d:
            h = sum(float((self.phi.conj() * self.hop(self.U[m], self.phi[self.fw[m]])).real.sum()) for m in range(self.D))
            H += 0.5 * float(self.pi.abs().pow(2).sum()) + self.potential()[0] - 2 * self.kappa * h
            o["L_phi"] = float(self.phi.abs().pow(2).sum()) / self.V
            o["L_link"] = h / (self.V * self.D)
        o["H"] = H
        return o

    def trajectory(self):
        pure = not self.d
        st = _key(0xA1 if pure else 0xC3, self.traj)
        self.P = [torch.stack([_gauss(self.seed, _key(st, self.site, mu, a)) for a in range(self.ng)], 1) for mu in range(self.D)]
        if not pure:
            self.pi = self._vector(_key(0xD4, self.traj), 1.0)
        old = (self.U, self.phi)
        a = self.measure()
        n, eps = self.c["nmd"], self.c["tau"] / self.c["nmd"]
        if self.c["integ"] == "leapfrog":
            self.kick(0.5 * eps)
            for i in range(n):
                self.drift(eps)
                self.kick(eps if i + 1 < n else 0.5 * eps)
        else:
            self.kick(OMELYAN * eps)
            for i in range(n):
                self.drift(0.5 * eps)
                self.kick((1 - 2 * OMELYAN) * eps)
                self.drift(0.5 * eps)
                self.kick(2 * OMELYAN * eps if i + 1 < n else OMELYAN * eps)
        b = self.measure()
        dH = b["H"] - a["H"]
        self.traj += 1
        coin = float(_uniform(self.seed, _key(0xB2 if pure else 0xE5, self.traj)))
        acc = dH <= 0 or coin < math.exp(-dH)
        if not acc:
            self.U, self.phi = old
        self.last = b if acc else a
        return [dH, float(acc), float(self.traj), self.last["plaq"], self.last["L_phi"], self.last["L_link"], self.kappa, self.beta]

    def polyakov(self):
        t = self.D - 1
        s = torch.tensor(np.nonzero(self.x[t] == 0)[0], device=_dev())
        P = self.U[t][s]
        for _ in range(1, self.L[t]):
            s = self.fw[t][s]
            P = _mm(P, self.U[t][s])
        return float(P.diagonal(dim1=-2, dim2=-1).sum(-1).real.mean()) / self.N

    def planes(self):
        nu = min(range(self.D), key=lambda m: self.L[m])
        out = {}
        for k, f in (("U", torch.stack(self.U, 1).reshape(self.V, -1)), ("phi", self.phi)):
            if f is not None:
                rows = torch.stack([f[torch.tensor(np.nonzero(self.x[nu] == p)[0], device=_dev())].T.reshape(-1) for p in range(self.L[nu])])
                out[k] = torch.nn.functional.pad(torch.view_as_real(rows), (0, 0, 0, rows.shape[1] % 2))
                out[k] = torch.view_as_complex(out[k].contiguous())
        return out


def _swaps(lats, ladder, counter, swap_seed=0x5A7AB1EC):
    """Exchanges of kappa between neighbours of each size's ladder: even pairs, then odd."""
    for order in ladder:
        for start in (0, 1):
            for k in range(start, len(order) - 1, 2):
                a, b = lats[order[k]], lats[order[k + 1]]
                delta = (a.kappa - b.kappa) * 2 * a.V * a.D * (a.last["L_link"] - b.last["L_link"])
                counter += 1
                if delta <= 0 or float(_uniform(swap_seed, _key(0x57A9, counter))) < math.exp(-delta):
                    a.kappa, b.kappa = b.kappa, a.kappa
                    order[k], order[k + 1] = order[k + 1], order[k]
    return counter


def _exact_fit(case, seed):
    x, y, grid = (torch.tensor(v, dtype=torch.float64, device=_dev()) for v in _fit_data(case, seed))
    w, M, n = _widths(case), case["members"], case["n"]
    shapes, params = list(zip(w[:-1], w[1:])), []
    for l, (i, o) in enumerate(shapes):
        e = torch.arange(o * i, device=_dev())
        lim = np.float32(1) / np.sqrt(np.float32(i))
        u = [((2 * _uniform(int(seed) + 1, _key(0x4D4C50, m, l, e)) - 1).float() * float(lim)).double() for m in range(M)]
        params += [torch.stack(u).reshape(M, o, i), torch.zeros(M, 1, o, dtype=torch.float64, device=_dev())]
    for p in params:
        p.requires_grad_()

    def net(v):
        v = v.expand(M, *v.shape)
        for l in range(len(shapes)):
            v = v @ params[2 * l].transpose(1, 2) + params[2 * l + 1]
            if l + 1 < len(shapes):
                v = v * torch.sigmoid(v)
        return v

    m1, m2, t = [torch.zeros_like(p) for p in params], [torch.zeros_like(p) for p in params], 0
    for ep in range(case["epochs"]):
        idx, u = list(range(n)), _uniform(7, _key(0x5348, ep, torch.arange(n, device=_dev()))).tolist()
        for i in range(n - 1, 0, -1):
            j = min(int(u[i] * (i + 1)), i)
            idx[i], idx[j] = idx[j], idx[i]
        sums, batches = 0, 0
        for s in range(0, n, case["batch"]):
            at = torch.tensor(idx[s:s + case["batch"]], device=_dev())
            loss = (net(x[at]) - y[at]).pow(2).mean((1, 2))
            grads = torch.autograd.grad(loss.sum(), params)
            t, sums, batches = t + 1, sums + loss.detach(), batches + 1
            with torch.no_grad():
                for p, g, a, b in zip(params, grads, m1, m2):
                    a.mul_(0.9).add_(g, alpha=0.1)
                    b.mul_(0.999).add_(g * g, alpha=0.001)
                    p -= 1e-3 * (a / (1 - 0.9 ** t)) / ((b / (1 - 0.999 ** t)).sqrt() + 1e-8)
    with torch.no_grad():
        per = net(grid)
        flat = torch.cat([p.reshape(M, -1) for p in params], 1)
    return {"loss": sums / batches, "params": flat, "mean": per.mean(0), "var": per.var(0, unbiased=False), "per_member": per}


def exact(case, seed):
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    lats = _lattices(case)
    heavy = {"4,2:real": 120.0, "2,1:real": 8.0, "2": 4.0, "12m": 12.0}.get(case["rep"], 1.0)
    if sum(float(np.prod(L)) for L, _ in lats) * case["nmd"] * case["ntraj"] * heavy > 6e7:
        return None                     # over about 20 seconds in plain torch
    lats = [_Plain(case, L, k, s) for (L, k), s in zip(lats, _seeds(case, seed))]
    if case["kind"] == "host":
        rows = [lats[0].trajectory()]
        return {"records": np.array(rows), "U": torch.stack(lats[0].U, 1),
                **({"phi": lats[0].phi} if lats[0].d else {})}
    rows, counter = [], 0
    sizes = sorted({tuple(p.L) for p in lats})
    ladder = [sorted((i for i, p in enumerate(lats) if tuple(p.L) == s), key=lambda i: lats[i].kappa) for s in sizes]
    for _ in range(case["ntraj"]):
        if case["kind"] == "ladder":
            rows += [p.trajectory() for p in lats]
            counter = _swaps(lats, ladder, counter)
        else:
            rows.append(lats[0].trajectory() + [lats[0].polyakov()])
    rows = np.array(rows)
    if case["prec"] != "fp64":          # an FP32 trajectory's dH has no 64-bit counterpart
        return {"records": rows[:, 1:], "dH": None, "lattices": [p.planes() for p in lats]}
    return {"records": rows, "lattices": [p.planes() for p in lats]}
