"""The framework's work as timed cases: what a program that uses it has it do.

An exact-diagonalisation run builds the sector of its states and the Hamiltonian on it, finds
the ground state, runs Lanczos recurrences and shifted solves for the spectra, and evaluates
continued fractions; on large bases it trains a small network and ranks states with it.  Each
kind of case is one of these stages through the entry point that a program calls; ``spectra`` is a
whole drop-in call.  Models are the package's seeded Anderson models: 6 2p and 10 3d
spin-orbitals with 10 bath spin-orbitals per level, from one level (26 spin-orbitals) over five
(66) to thirty (316), at most two bath holes.
"""

import math

import numpy as np
import torch

from impuritymodel_gb300 import finite, models, pruning, spectra
from impuritymodel_gb300.engine import DeviceOp, get_engine, make_restrictions

# ---------------------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------------------


def listed():
    return [
        # the smallest whole call: XAS of the 26-spin-orbital model through the dict API, three
        # polarisations of three thermal states; launches, copies and host work dominate
        dict(name="spectra_xas26", kind="spectra", levels=1, family="xas", states=3, krylov=150, points=2000),
        # the core-hole sector of the 66-spin-orbital model (360 states): expansion and CSR of
        # a sector that fits one SM many times over, latency
        dict(name="sector_xas66", kind="sector", levels=5, family="xas"),
        # the photoemission sector of the 316-spin-orbital model: 462 120 states, 4.7 M entries
        dict(name="sector_ps316", kind="sector", levels=30, family="ps"),
        # three lowest eigenpairs of the 66-spin-orbital model (1770 states), FP64
        dict(name="ground_66", kind="ground", levels=5, pairs=3),
        # the ground state of the 316-spin-orbital model (47 895 states), FP64
        dict(name="ground_316", kind="ground", levels=30, pairs=1),
        # RIXS final states: 3 polarisations x 5 states x 50 incoming energies, upstream's
        # recurrence of 150 steps on the 1770-state sector, FP64 (the drop-in default)
        dict(name="lanczos_rixs66", kind="lanczos", levels=5, runs=750, krylov=150),
        # Green's-function recurrences on a sector too large for one SM's shared memory; three
        # polarisations of one state
        dict(name="lanczos_316", kind="lanczos", levels=30, runs=3, krylov=100),
        # RIXS intermediate states: 15 right-hand sides at 50 incoming energies, core-hole sector
        dict(name="shifted_rixs66", kind="shifted", levels=5, rhs=15, shifts=50),
        # RIXS spectra: 750 runs at 4000 loss energies, 150 coefficients each, FP64
        dict(name="cfrac_rixs66", kind="cfrac", runs=750, krylov=150, points=4000),
        # H x for 16 complex64 vectors on the 462 120-state sector
        dict(name="hv_ps316", kind="hv", levels=30, family="ps", vectors=16, mixed=True),
        # the basis-ranking network: forward, backward and Adam, eight batches of 4096
        dict(name="net_train", kind="train", samples=32768, batch=4096),
        # ranking the states of a large expansion layer
        dict(name="net_rank", kind="rank", samples=462120),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["spectra", "sector", "sector", "ground", "lanczos", "lanczos", "shifted", "cfrac", "hv", "hv",
                       "train", "rank"])
    if kind == "spectra":
        family = rng.choice(["xas", "ps"])
        return dict(kind=kind, levels=rng.randint(1, 5 if family == "xas" else 2), family=family,
                    states=rng.randint(1, 5), krylov=_log(rng, 20, 150), points=_log(rng, 100, 4000))
    if kind == "sector":
        return dict(kind=kind, levels=_log(rng, 1, 30), family=rng.choice(["xas", "ps", "xps"]))
    if kind == "ground":
        levels = _log(rng, 1, 30)
        return dict(kind=kind, levels=levels, pairs=rng.randint(1, 4 if levels <= 10 else 1))
    if kind == "lanczos":
        if rng.random() < 0.5:
            return dict(kind=kind, levels=rng.randint(1, 5), runs=_log(rng, 1, 750), krylov=_log(rng, 20, 150))
        return dict(kind=kind, levels=rng.randint(22, 30), runs=_log(rng, 1, 8), krylov=_log(rng, 20, 80))
    if kind == "shifted":
        return dict(kind=kind, levels=rng.randint(1, 6), rhs=_log(rng, 1, 15), shifts=_log(rng, 1, 100))
    if kind == "cfrac":
        return dict(kind=kind, runs=_log(rng, 1, 750), krylov=_log(rng, 10, 150), points=_log(rng, 100, 4000))
    if kind == "hv":
        return dict(kind=kind, levels=_log(rng, 5, 30), family=rng.choice(["ground", "xps", "ps"]),
                    vectors=_log(rng, 1, 32), mixed=rng.random() < 0.5)
    if kind == "train":
        batch = 128 * _log(rng, 2, 64)
        return dict(kind=kind, samples=max(batch, _log(rng, 1000, 32768)), batch=batch)
    return dict(kind=kind, samples=_log(rng, 100, 462120))


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------


def _model(levels, seed):
    # bath ranges of the package's 66- and 316-spin-orbital models
    e, v = ((-8.0, 2.0), (0.1, 0.8)) if levels > 10 else ((-5.0, 0.0), (0.3, 1.5))
    return models.Model(levels, e, v, seed, 2)


def _generator(eng, seed):
    g = torch.Generator(device=eng.device)
    g.manual_seed(int(seed))
    return g


class _Problem:
    """A seeded model with its compiled operator, restrictions and sorted ground basis."""

    def __init__(self, eng, levels, seed):
        self.mod = _model(levels, seed)
        self.n_orb = self.mod.n_spin_orbitals
        self.basis = finite.get_basis(*self.mod.basis_args())
        self.dop = DeviceOp(self.mod.hOp, eng.device)
        self.restr = make_restrictions(self.mod.restrictions, self.n_orb)
        self.sorted_basis = finite._SortedBasis(eng, list(self.basis), self.n_orb)

    def transition_ops(self, family):
        return {"xas": self.mod.xas_ops, "ps": self.mod.ps_ops, "xps": lambda: self.mod.ps_ops(l=1)}[family]()

    def starts(self, eng, family, seed):
        """States that a transition operator makes of half of the ground basis."""
        b = self.sorted_basis.sorted
        pick = torch.rand(b.shape[0], device=eng.device, generator=_generator(eng, seed)) < 0.5
        pick[0] = True
        b = b[pick].contiguous()
        amps = torch.zeros((b.shape[0], 2), dtype=torch.float64, device=eng.device)
        amps[:, 0] = 1.0
        ops = [DeviceOp(t, eng.device) for t in self.transition_ops(family)]
        outs = eng.apply_vectors_multi([b], [amps], ops, self.restr, 0.0)
        return eng.sort_unique(torch.cat([o[0][0] for o in outs], 0).contiguous())

    def hamiltonian(self, eng, family, seed):
        if family == "ground":
            return eng.build_csr(self.sorted_basis.sorted, self.dop, None)
        return spectra.Sector(eng, self.dop, self.restr, self.starts(eng, family, seed)).csr


def _vectors(eng, n, runs, seed):
    v = torch.randn((n, runs), dtype=torch.complex128, device=eng.device, generator=_generator(eng, seed))
    return v / torch.linalg.vector_norm(v, dim=0)


def _product_states(eng, n, seed):
    """Occupations of the 316-spin-orbital ground sector's kind: 6 2p and 8-10 3d electrons, two bath
    holes at most, as padded words [n, 5]."""
    g = _generator(eng, seed)
    occ = torch.ones((n, 320), dtype=torch.bool, device=eng.device)
    occ[:, 316:] = False
    holes = torch.randint(0, 3, (n,), device=eng.device, generator=g)
    d = torch.rand((n, 10), device=eng.device, generator=g).argsort(1)
    bath = torch.randint(0, 300, (n, 2), device=eng.device, generator=g)
    for k in range(2):  # two 3d holes less one for each bath hole
        occ[torch.arange(n, device=eng.device), 6 + d[:, k]] = holes > k
        occ[torch.arange(n, device=eng.device), 16 + bath[:, k]] &= holes <= k
    shifts = torch.arange(63, -1, -1, device=eng.device)
    return (occ.view(n, 5, 64).to(torch.int64) << shifts).sum(2)


def _omega(points):
    return np.linspace(-2.0, 12.0, points)


def prepare(case, seed):
    eng = get_engine()
    eng.reset_status()
    kind = case["kind"]
    s = dict(kind=kind, eng=eng, case=case)
    if kind == "spectra":
        p = _Problem(eng, case["levels"], seed)
        rng = np.random.default_rng(seed)
        psis = []
        for _ in range(case["states"]):  # weights spread over the orders of magnitude an eigenstate has
            a = rng.normal(size=len(p.basis)) * 10.0 ** (-3.0 * rng.random(len(p.basis)))
            a /= np.linalg.norm(a)
            psis.append({b: complex(x) for b, x in zip(p.basis, a) if x * x >= 1e-7})
        s.update(n=p.n_orb, h=p.mod.hOp, t=p.transition_ops(case["family"]), psis=psis,
                 es=-700.0 + 0.01 * np.arange(case["states"]), w=np.linspace(-25.0, 25.0, case["points"]),
                 restrictions=p.mod.restrictions)
    elif kind == "sector":
        p = _Problem(eng, case["levels"], seed)
        s.update(p=p, starts=p.starts(eng, case["family"], seed))
    elif kind == "ground":
        p = _Problem(eng, case["levels"], seed)
        s.update(csr=p.hamiltonian(eng, "ground", seed))
    elif kind == "lanczos":
        csr = _Problem(eng, case["levels"], seed).hamiltonian(eng, "ground", seed)
        s.update(csr=csr, v0=_vectors(eng, csr.n, case["runs"], seed),
                 k=np.full(case["runs"], min(case["krylov"], csr.n), dtype=np.int32))
    elif kind == "shifted":
        csr = _Problem(eng, case["levels"], seed).hamiltonian(eng, "xas", seed)
        d = csr.val_r[torch.repeat_interleave(torch.arange(csr.n, device=eng.device),
                                              csr.row_ptr[1:] - csr.row_ptr[:-1]) == csr.col]
        w = float(d.min().item()) + np.linspace(-10.0, 20.0, case["shifts"])
        rng = np.random.default_rng(seed)
        # incoming energies above each eigenstate's energy, core-hole lifetime 0.2 eV
        zs = w[None, :] + 0.1 * rng.random((case["rhs"], 1)) + 0.2j
        s.update(csr=csr, y=_vectors(eng, csr.n, case["rhs"], seed).t().contiguous(), zs=zs)
    elif kind == "cfrac":
        rng = np.random.default_rng(seed)
        R, K = case["runs"], case["krylov"]
        to = lambda x: torch.from_numpy(x).to(eng.device)  # noqa: E731
        s.update(alpha=to(-700.0 + 5.0 * rng.normal(size=(R, K))), beta=to(0.2 + 6.0 * rng.random((R, K))),
                 k=rng.integers(max(1, K // 2), K + 1, size=R).astype(np.int32), w=_omega(case["points"]),
                 e=-700.0 + rng.random(R), scale=0.1 + rng.random(R))
        s["k"][: (R + 1) // 2] = K
    elif kind == "hv":
        csr = _Problem(eng, case["levels"], seed).hamiltonian(eng, case["family"], seed)
        x = _vectors(eng, csr.n, case["vectors"], seed)
        s.update(csr=csr.mixed() if case["mixed"] else csr, x=x.to(torch.complex64) if case["mixed"] else x)
    else:
        s.update(states=_product_states(eng, case["samples"], seed), net=pruning.BasisNet(eng, seed=seed))
        if kind == "train":
            g = _generator(eng, seed + 1)
            s["log_w"] = -14.0 * torch.rand(case["samples"], device=eng.device, generator=g)
    return s


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------


def run(s):
    kind, eng, case = s["kind"], s["eng"], s["case"]
    if kind == "spectra":
        finite.clear_sector_cache()  # a new model's first spectra: no sector of an earlier call
        return spectra.getSpectra(s["n"], s["h"], s["t"], s["psis"], s["es"], s["w"], 0.2, s["restrictions"],
                                  krylovSize=case["krylov"])
    if kind == "sector":
        sec = spectra.Sector(eng, s["p"].dop, s["p"].restr, s["starts"])
        return dict(basis=sec.basis, row_ptr=sec.csr.row_ptr, col=sec.csr.col, val=sec.csr.val_r)
    if kind == "ground":
        es, X = finite.eig_lowest(eng, s["csr"], case["pairs"])
        return dict(es=es, vectors=X)
    if kind == "lanczos":
        return eng.lanczos(s["csr"], s["v0"], s["k"])
    if kind == "shifted":
        n = s["csr"].n
        return eng.shifted_solve(s["csr"], s["y"], s["zs"], 1e-10, min(6 * n + 50, 2000))[0]
    if kind == "cfrac":
        return eng.cfrac(s["alpha"], s["beta"], s["k"], s["w"], 0.05, s["e"], s["scale"])
    if kind == "hv":
        return eng.spmv(s["csr"], s["x"], precision=1 if case["mixed"] else 0)
    net = s["net"]
    if kind == "train":
        losses = net.train(s["states"], s["log_w"], epochs=1, batch=case["batch"])
        return dict(losses=torch.stack(losses), parameters=net.P, gradients=net.G, m=net.m, v=net.v)
    return net.predict(s["states"])


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------


def _sector_size(levels, family):
    """States and stored entries of a sector with at most two bath holes."""
    nb = 10 * levels
    if family == "xas":  # one 2p hole, nine or ten 3d electrons
        n = 6 * (10 + nb)
    elif family == "ps":
        n = 120 + 45 * nb + 10 * (nb * (nb - 1) // 2)
    else:
        n = 45 + 10 * nb + nb * (nb - 1) // 2
        n *= 6 if family == "xps" else 1
    return n, n * (6 if family == "xas" else 10)


def work(case):
    kind = case["kind"]
    if kind in ("spectra", "sector", "ground", "lanczos", "shifted", "hv"):
        family = case.get("family", "xas" if kind == "shifted" else "ground")
        n, nnz = _sector_size(case["levels"], family)
        words = (16 + 10 * case["levels"] + 63) // 64
        matrix = 12 * nnz + 8 * n
    if kind == "spectra":
        runs = case["states"] * (3 if family == "xas" else 10)
        k = min(case["krylov"], n)
        return dict(bytes=8 * words * n + 16 * runs * case["points"],
                    flops=runs * k * (4 * nnz + 20 * n) + 15 * runs * k * case["points"])
    if kind == "sector":
        return dict(bytes=8 * words * n * 2 + matrix, flops=0)
    if kind == "ground":  # about 100 steps, each vector orthogonalised against the ones before it
        return dict(bytes=matrix + 16 * n * case["pairs"], flops=100 * (4 * nnz + 20 * n) + 8 * 100 * 100 * n)
    if kind == "lanczos":
        runs, k = case["runs"], min(case["krylov"], n)
        return dict(bytes=matrix + 16 * n * runs + 16 * runs * k, flops=runs * k * (4 * nnz + 20 * n))
    if kind == "shifted":
        rhs, nz = case["rhs"], case["shifts"]
        return dict(bytes=matrix + 16 * n * rhs * (1 + nz), flops=rhs * n * (4 * nnz + 20 * n + 8 * n * nz))
    if kind == "cfrac":
        runs, k, nw = case["runs"], case["krylov"], case["points"]
        return dict(bytes=16 * runs * k + 16 * runs * nw, flops=15 * runs * k * nw)
    if kind == "hv":
        vec = (8 if case["mixed"] else 16) * n * case["vectors"]
        return dict(bytes=(8 if case["mixed"] else 12) * nnz + 8 * n + 2 * vec, flops=4 * nnz * case["vectors"])
    rows = case["samples"]
    gemm = 2 * rows * 256 * (320 + 256)
    if kind == "train":
        rows = rows // case["batch"] * case["batch"]
        return dict(bytes=44 * rows + 16 * 147969 * 2 * (rows // case["batch"]), flops=3 * gemm)
    return dict(bytes=44 * rows, flops=gemm)


# ---------------------------------------------------------------------------------------
# The same in 64 bits, without the package's code
# ---------------------------------------------------------------------------------------


def _csr_apply(csr, x):
    rows = torch.repeat_interleave(torch.arange(csr.n, device=x.device), csr.row_ptr[1:] - csr.row_ptr[:-1])
    y = torch.zeros((csr.n, x.shape[1]), dtype=torch.complex128, device=x.device)
    for c in range(0, x.shape[1], 4):
        part = x[:, c:c + 4].to(torch.complex128)
        y[:, c:c + 4].index_add_(0, rows, csr.val_r.view(-1, 1) * part[csr.col.to(torch.int64)])
    return y


def _dense(csr):
    rows = torch.repeat_interleave(torch.arange(csr.n, device=csr.col.device), csr.row_ptr[1:] - csr.row_ptr[:-1])
    h = torch.zeros((csr.n, csr.n), dtype=torch.float64, device=csr.col.device)
    h[rows, csr.col.to(torch.int64)] = csr.val_r
    return h


def _occupied(states, words):
    """Bit i of word i // 64 counted from its top is orbital i: [n, 64 * words] bool."""
    shifts = torch.arange(63, -1, -1, device=states.device)
    return ((states.unsqueeze(2) >> shifts) & 1).reshape(states.shape[0], 64 * words).to(torch.float64)


def _network(net_p, x):
    h1 = torch.relu(x @ net_p["W1"].t() + net_p["b1"])
    h2 = torch.relu(h1 @ net_p["W2"].t() + net_p["b2"])
    return h2 @ net_p["w3"] + net_p["b3"]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("spectra", "sector", "lanczos"):
        # the sector's numbers are sums in a given order; the recurrences lose orthogonality, after
        # which their coefficients are no function of the inputs that 64 bits determine
        return None
    if kind == "ground":
        if case["levels"] > 8:
            return None
        h = _dense(prepare(case, seed)["csr"])
        return dict(es=torch.linalg.eigvalsh(h)[: case["pairs"]].cpu().numpy(), vectors=None)
    if kind == "shifted":
        s = prepare(case, seed)
        es, u = torch.linalg.eigh(_dense(s["csr"]))
        u = u.to(torch.complex128)
        c = s["y"] @ u
        zs = torch.from_numpy(s["zs"]).to(c.device)
        return torch.stack([(c[r] / (zs[r].unsqueeze(1) - es)) @ u.t() for r in range(case["rhs"])])
    if kind == "cfrac":
        s = prepare(case, seed)
        dev = s["alpha"].device
        to = lambda x: torch.from_numpy(np.asarray(x)).to(dev)  # noqa: E731
        z = to(s["w"]).unsqueeze(0) + to(s["e"]).unsqueeze(1) + 0.05j
        g = torch.zeros_like(z)
        k = to(s["k"]).unsqueeze(1)
        for i in range(case["krylov"] - 1, -1, -1):
            a, b = s["alpha"][:, i:i + 1], s["beta"][:, i:i + 1]
            d = z - a - torch.where(k - 1 > i, b * b, torch.zeros_like(b)) * g
            g = torch.where(k > i, 1.0 / d, g)
        return to(s["scale"]).unsqueeze(1) * g
    if kind == "hv":
        s = prepare(case, seed)
        return _csr_apply(s["csr"], s["x"])
    s = prepare(case, seed)
    net = s["net"]
    p = {k: v.to(torch.float64).clone() for k, v in net.p.items()}
    if kind == "rank":
        return torch.cat([_network(p, _occupied(x, 5)) for x in s["states"].split(65536)])
    return _train_exact(p, s, case)


def _train_exact(p, s, case):
    """The same shuffled batches, mean squared error and Adam steps in 64 bits."""
    batch, n = case["batch"], case["samples"]
    names = list(p)
    gen = torch.Generator(device=s["states"].device)
    gen.manual_seed(0)
    perm = torch.randperm(n, device=s["states"].device, generator=gen)
    for v in p.values():
        v.requires_grad_(True)
    m = [torch.zeros_like(p[k]) for k in names]
    v2 = [torch.zeros_like(p[k]) for k in names]
    losses, grads = [], None
    for t, b0 in enumerate(range(0, n - batch + 1, batch), 1):
        idx = perm[b0:b0 + batch]
        loss = ((_network(p, _occupied(s["states"][idx], 5)) - s["log_w"][idx].to(torch.float64)) ** 2).mean()
        grads = torch.autograd.grad(loss, [p[k] for k in names])
        losses.append(loss.detach())
        lr = 1e-3 * math.sqrt(1.0 - 0.999 ** t) / (1.0 - 0.9 ** t)
        with torch.no_grad():
            for q, k in enumerate(names):
                m[q].mul_(0.9).add_(0.1 * grads[q])
                v2[q].mul_(0.999).add_(0.001 * grads[q] ** 2)
                p[k] -= lr * m[q] / (v2[q].sqrt() + 1e-8)
    flat = lambda xs: torch.cat([x.detach().reshape(-1) for x in xs])  # noqa: E731
    # late in training the residuals are small, and the gradients are mostly the rounding of the
    # BF16 activations: 64 bits say nothing about them
    return dict(losses=torch.stack(losses), parameters=flat([p[k] for k in names]), gradients=None, m=None, v=flat(v2))
