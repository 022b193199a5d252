"""Kernels at the sizes where their tiles, remainders and dispatch rules change."""

import numpy as np
import pytest
import scipy.sparse
import torch

pytestmark = pytest.mark.gpu


def _random_csr(eng, n, seed, complex_vals=False, heavy=()):
    """Hermitian CSR with 2-9 entries a row, rows of ``heavy`` linked to 40 others each."""
    from impuritymodel_gb300.engine import CsrMatrix

    rng = np.random.default_rng(seed)
    h = {}
    for i in range(n):
        h[(i, i)] = complex(rng.normal() * 3.0)
        for j in rng.integers(0, n, size=40 if i in heavy else 2):
            if i != j:
                v = complex(rng.normal(), rng.normal() if complex_vals else 0.0)
                h[(i, int(j))] = v
                h[(int(j), i)] = v.conjugate()
    keys = sorted(h)
    rows = np.array([k[0] for k in keys])
    col = torch.tensor([k[1] for k in keys], dtype=torch.int32, device=eng.device)
    vals = np.array([h[k] for k in keys])
    rp = torch.from_numpy(np.searchsorted(rows, np.arange(n + 1)).astype(np.int64)).to(eng.device)
    if complex_vals:
        csr = CsrMatrix(rp, col, val_c=torch.from_numpy(np.stack([vals.real, vals.imag], 1)).to(eng.device).contiguous())
    else:
        csr = CsrMatrix(rp, col, val_r=torch.from_numpy(np.ascontiguousarray(vals.real)).to(eng.device))
    import scipy.sparse

    return csr, scipy.sparse.csr_matrix((vals, (rows, [k[1] for k in keys])), shape=(n, n))


def _recurrence(H, v, K):
    """Upstream's three-term recurrence in NumPy (finite.py:1974-1992)."""
    alpha, beta = [], []
    p, bp = np.zeros_like(v), 0.0
    for _ in range(K):
        y = H @ v
        a = np.vdot(v, y).real
        w = y - a * v - bp * p
        alpha.append(a)
        bp = np.linalg.norm(w)
        beta.append(bp)
        p, v = v, w / bp
    return np.array(alpha), np.array(beta)


@pytest.mark.parametrize("n,R,K,precision,cplx", [
    (4300, 1, 12, 0, False),    # 256-thread blocks, one run
    (4300, 33, 12, 0, False),   # two run tiles, the second of one run
    (9000, 31, 3, 0, True),     # a run tile that does not divide the block
    (40011, 3, 12, 0, False),   # 512-thread blocks, one pass, a ragged last row
    (40011, 7, 12, 1, True),    # complex64 vectors and values
    (14620, 30, 12, 0, False),  # several passes of 17 rows: the last rows in the middle of a group of 8
    (12000, 16, 1, 0, False),   # a single step: alpha only
    (12000, 16, 2, 1, False),
])
def test_grid_wide_lanczos(eng, n, R, K, precision, cplx):
    csr, H = _random_csr(eng, n, n + R, cplx, heavy=(0, 1, 2, 5, n // 2, n - 1))
    g = np.random.default_rng(R)
    v = g.normal(size=(n, R)) + 1j * g.normal(size=(n, R))
    v /= np.linalg.norm(v, axis=0)
    k = np.full(R, K, dtype=np.int32)
    a, b = eng.lanczos(csr, torch.from_numpy(v).to(eng.device), k, precision=precision)
    a, b = a.cpu().numpy(), b.cpu().numpy()
    # a dozen steps of an unconverged recurrence amplify rounding by less than 1e3
    tol = (1e-12 if precision == 0 else 6e-5) * abs(H).sum(1).max()
    for r in {0, R // 2, R - 1}:
        ar, br = _recurrence(H, v[:, r], K)
        assert np.abs(a[r] - ar).max() < tol
        assert np.abs(b[r, : K - 1] - br[: K - 1]).max(initial=0.0) < tol


def _fraction(alpha, beta, k, omega, delta, e, scale):
    """The continued fraction of upstream's getGreen (spectra.py:678-680), from its end."""
    g = np.zeros((len(k), len(omega)), dtype=np.complex128)
    for r, kl in enumerate(k):
        x = np.zeros(len(omega), dtype=np.complex128)
        for i in range(kl - 1, -1, -1):
            d = omega + e[r] + 1j * delta - alpha[r, i]
            x = 1.0 / (d - (beta[r, i] ** 2 * x if i != kl - 1 else 0.0))
        g[r] = scale[r] * x
    return g


@pytest.mark.parametrize("R,K,nw,delta", [
    (1, 1, 1, 0.1),         # one coefficient, one frequency
    (5, 7, 3, -0.2),        # several runs a block, negative broadening, ragged lengths
    (130, 9, 1, 0.05),      # more runs than a block holds
    (3, 150, 129, 0.05),    # a second tile of one frequency
    (2, 1030, 200, 0.05),   # more coefficients than one stage holds
    (4, 60, 100, 1e-11),    # below the scaled form's smallest broadening
    (4, 400, 64, 40.0),     # a broadening far above the spread of the coefficients
])
def test_continued_fraction(eng, R, K, nw, delta):
    g = np.random.default_rng(K + nw)
    alpha = -700.0 + 5.0 * g.normal(size=(R, K))
    beta = 0.1 + 6.0 * g.random((R, K))
    k = g.integers(1, K + 1, size=R).astype(np.int32)
    k[0] = K
    beta[np.arange(R), k - 1] = np.nan  # no part of the fraction
    omega, e, scale = np.linspace(-8.0, 9.0, nw), -700.0 + g.random(R), 0.5 + g.random(R)
    to = lambda x: torch.from_numpy(x).to(eng.device)  # noqa: E731
    got = eng.cfrac(to(alpha), to(beta), k, omega, delta, e, scale).cpu().numpy()
    want = _fraction(alpha, beta, k, omega, delta, e, scale)
    # NumPy rounds omega + e at 700 eV (1.1e-13); a pole of width delta turns that into 1.1e-13 / delta
    tol = 1e-12 + (4e-13 / abs(delta) if abs(delta) > 1e-9 else 1e-6)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("n,words", [
    (1, 5), (127, 5), (129, 5),        # one tile, a ragged one, a second of one state
    (130, 2), (300, 7),                # fewer and more words than the network reads
    (152 * 128, 5), (152 * 128 + 1, 5),  # one tile a CTA, then two
    (100001, 5),
])
def test_rank_in_one_launch(eng, n, words):
    from impuritymodel_gb300.pruning import BasisNet, pad_words

    net = BasisNet(eng, seed=n)
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    net.p["b1"].copy_(torch.randn(256, device=eng.device, generator=g))
    net.p["b2"].copy_(torch.randn(256, device=eng.device, generator=g))
    states = torch.randint(-(1 << 62), 1 << 62, (n, words), device=eng.device, generator=g) * 2
    states[:, -1] |= 1  # the last column of the last word
    got = net.predict(states)
    # layer by layer: the same roundings and K order, the head's 256 products summed in another order
    # (at most 14 roundings deep there, 22 here)
    pad = (-n) % 128
    X, _ = net.inputs(torch.cat([pad_words(states), states.new_zeros((pad, 5))], 0))
    want, (_, _, H2, _) = net.forward(X)
    bound = 36 * 2.0 ** -24 * (H2.double().abs() @ net.p["w3"].double().abs() + net.p["b3"].double().abs())
    assert got.shape == (n,)
    assert bool(((got.double() - want[:n].double()).abs() <= bound[:n]).all())


def _random_operator(rng, n_orb, n_terms, cplx):
    """Terms of 0 to 4 operators with repeated orbitals, spectators and several terms an output."""
    op = {}
    while len(op) < n_terms:
        kind = rng.integers(0, 8)
        i, j, k, l = (int(x) for x in rng.integers(0, n_orb, size=4))
        key = [((i, "c"), (j, "a")), ((i, "c"), (k, "c"), (k, "a"), (j, "a")), ((k, "a"), (k, "c"), (i, "c"), (j, "a")),
               ((i, "c"), (j, "c"), (l, "a"), (k, "a")), ((i, "c"), (i, "a")), ((i, "c"), (j, "c"), (i, "a"), (j, "a")),
               ((i, "a"),), ((i, "c"), (j, "a"), (j, "c"))][kind]
        v = float(rng.normal()) if rng.random() > 0.1 else -0.0
        op[key] = complex(v, rng.normal()) if cplx else v
    return op


def _two_pass(eng, states, dop, restr, weight_min, basis, filt, conj):
    """edgpu_apply_columns: a count and a fill launch."""
    import ctypes as C

    from impuritymodel_gb300 import _lib as L
    from impuritymodel_gb300.engine import _ptr

    n, w = states.shape
    rp = C.byref(restr) if restr is not None else None
    nb = 0 if basis is None else basis.shape[0]
    counts = torch.empty(n, dtype=torch.int64, device=eng.device)
    cap = 256
    while True:
        eng.reset_status()
        L.check(eng.lib.edgpu_apply_columns(w, _ptr(states), n, C.byref(dop.terms), rp, weight_min, _ptr(basis), nb,
                                            filt, None, _ptr(counts), None, None, None, 0, cap, _ptr(eng.status),
                                            eng.stream), "apply_columns")
        if int(eng.status.item()) == 0:
            break
        cap *= 4
    offs = eng.scan(counts)
    tot = int(offs[-1].item())
    s = torch.empty((tot, w), dtype=torch.int64, device=eng.device)
    i = torch.empty(tot, dtype=torch.int64, device=eng.device)
    v = torch.empty((tot, 2), dtype=torch.float64, device=eng.device)
    if tot:
        L.check(eng.lib.edgpu_apply_columns(w, _ptr(states), n, C.byref(dop.terms), rp, weight_min, _ptr(basis), nb,
                                            filt, _ptr(offs), None, _ptr(s), _ptr(i), _ptr(v), int(conj), cap,
                                            _ptr(eng.status), eng.stream), "apply_columns")
    return offs, s, i, v


@pytest.mark.parametrize("n,n_orb,n_terms,cplx,filled", [
    (1, 10, 1, False, 0.5),        # one state, one term
    (3, 63, 40, True, 0.5),
    (33, 64, 700, False, 0.9),     # a full word
    (700, 26, 900, False, 0.4),    # a dense operator: more outputs than the first arena holds
    (5000, 130, 3000, False, 0.95),  # table lookups, many groups
    (257, 316, 2500, True, 0.97),
    (40, 512, 8192, False, 0.9),   # eight words, the largest plan
])
def test_one_pass_application(eng, n, n_orb, n_terms, cplx, filled):
    from impuritymodel_gb300 import _lib as L
    from impuritymodel_gb300.engine import DeviceOp, make_restrictions

    rng = np.random.default_rng(n + n_terms)
    dop = DeviceOp(_random_operator(rng, n_orb, n_terms, cplx), eng.device)
    w = (n_orb + 63) // 64
    occ = np.zeros((n, 64 * w), dtype=np.uint8)
    occ[:, :n_orb] = rng.random((n, n_orb)) < filled
    words = np.packbits(occ, axis=1).view(">u8").astype(np.uint64).reshape(n, w)
    basis = eng.sort_unique(eng.upload_states(np.unique(words, axis=0)))
    # the basis and what one application adds to it, so that lookups hit
    _, more, _, _ = eng.apply_columns(basis[:200].contiguous(), dop, None, 0.0, want_states=True)
    wide = eng.sort_unique(torch.cat([basis, more], 0))
    restr = make_restrictions({frozenset(range(0, n_orb, 2)): (0, n_orb // 2), frozenset(range(5)): (1, 4)}, n_orb)
    for filt, b, r, wmin, conj in ((L.FILTER_NONE, None, None, 0.0, False), (L.FILTER_IN_BASIS, wide, None, 1e-12, True),
                                   (L.FILTER_NOT_IN_BASIS, basis, restr, 0.5, False)):
        want = _two_pass(eng, basis, dop, r, wmin, b, filt, conj)
        got = eng.apply_columns(basis, dop, r, wmin, basis=b, filt=filt, want_states=True, want_index=True,
                                want_vals=True, conj=conj)
        for g, x in zip(got, want):
            assert torch.equal(g.view(torch.int64), x.view(torch.int64))


@pytest.mark.parametrize("n,K,cplx,locked", [
    (5, 5, False, 0),         # fewer rows than a lane group, the whole space
    (300, 40, True, 0),       # two row chunks, complex H
    (1770, 60, False, 3),     # seven chunks, deflated vectors
    (1300, 1100, False, 0),   # more coefficients than shared memory keeps
    (5000, 50, False, 0),     # more chunks than every block adds up itself
    (30001, 24, False, 0),    # a chunk per SM, a ragged last one, four lanes a row
    (65536, 8, False, 0),     # the largest sector of the cooperative form
])
def test_reorthogonalised_steps(eng, n, K, cplx, locked):
    csr, H = _random_csr(eng, n, n, cplx, heavy=(0, n // 2) if n > 100 else ())
    g = np.random.default_rng(n)
    Q, _ = np.linalg.qr(g.normal(size=(n, locked + 1)) + 1j * g.normal(size=(n, locked + 1)))
    lock = torch.from_numpy(np.ascontiguousarray(Q[:, :locked].T)).to(eng.device) if locked else None
    v0 = torch.from_numpy(np.ascontiguousarray(Q[:, locked])).to(eng.device)
    V, a, b = eng.krylov_reorth(csr, v0, K, chunk=16, locked=lock)
    k = len(a)
    V = V.cpu().numpy()
    assert k == min(K, n - locked)
    # orthonormal to working precision (the dot products of n terms round by up to n eps, about sqrt(n) eps)
    every = np.concatenate([Q[:, :locked].T, V])
    gram = every.conj() @ every.T
    assert np.abs(gram - np.eye(len(every))).max() < 20 * np.sqrt(n) * 2.3e-16 + 1e-14
    # H V = V T + beta v e^T on the complement of the locked vectors, to rounding
    R = H @ V.T
    R -= Q[:, :locked] @ (Q[:, :locked].conj().T @ R)
    T = np.diag(a) + np.diag(b[: k - 1], 1) + np.diag(b[: k - 1], -1)
    R -= V.T @ T
    scale = abs(H).sum(1).max()
    assert np.abs(R[:, : k - 1]).max() < 1e-13 * scale
    if k < n - locked and K < 1000:
        assert abs(np.linalg.norm(R[:, k - 1]) - b[k - 1]) < 1e-12 * scale or b[k - 1] == 0.0


@pytest.mark.parametrize("n,nz,cplx,precision", [
    (1, 1, False, 0),       # one state: the space is exhausted at once
    (33, 5, True, 0),       # a second slice of one row, complex H
    (360, 512, False, 0),   # the most shifts: two rounds of coefficients
    (700, 3, False, 0),     # more rows than threads
    (3000, 2, True, 0),     # entries that do not fit in shared memory
    (360, 50, False, 3),    # double-float recurrence, same coefficients
])
def test_shifted_solves(eng, n, nz, cplx, precision):
    import scipy.sparse.linalg as spl

    csr, H = _random_csr(eng, n, n + nz, cplx, heavy=(0, n // 3) if n > 100 else ())
    g = np.random.default_rng(nz)
    Y = g.normal(size=(3, n)) + 1j * g.normal(size=(3, n))
    Y[1] = 0.0
    zs = g.uniform(-8.0, 8.0, size=(3, nz)) + 0.5j
    X, m = eng.shifted_solve(csr, torch.from_numpy(Y).to(eng.device), zs, 1e-10, min(6 * n + 50, 2000), precision)
    X, m = X.cpu().numpy(), m.cpu().numpy()
    assert m[1] == 0 and not X[1].any()
    for r in (0, 2):
        assert 1 <= m[r] <= min(6 * n + 50, 2000)
        for q in {0, nz // 2, nz - 1}:
            x = spl.spsolve(scipy.sparse.identity(n, format="csc") * zs[r, q] - H.tocsc(), Y[r]) if n > 1 else \
                Y[r] / (zs[r, q] - H[0, 0])
            # residual below 1e-10 |y|, and |(z - H)^{-1}| <= 1 / Im z; as much again for the rounding
            assert np.linalg.norm(X[r, q] - x) <= 4e-10 * np.linalg.norm(Y[r])


@pytest.mark.parametrize("n,R,nz,cplx", [
    (65, 30, 65, True),    # clusters of 4, as many shifts as their CTAs share
    (300, 70, 7, False),   # clusters of 2
    (1300, 60, 2, False),  # clusters of 2, several rows a thread
    (90, 160, 3, False),   # a CTA a right-hand side
])
def test_shifted_solves_on_clusters(eng, n, R, nz, cplx):
    csr, _ = _random_csr(eng, n, n + R, cplx, heavy=(0, n // 3))
    g = np.random.default_rng(R)
    Y = g.normal(size=(R, n)) + 1j * g.normal(size=(R, n))
    Y[R // 2] = 0.0
    zs = g.uniform(-8.0, 8.0, size=(R, nz)) + 0.5j
    X, m = eng.shifted_solve(csr, torch.from_numpy(Y).to(eng.device), zs, 1e-10, min(6 * n + 50, 2000), 0)
    some = [0, 1, R // 2, R - 1]
    X1, m1 = eng.shifted_solve(csr, torch.from_numpy(Y[some]).to(eng.device), zs[some], 1e-10, min(6 * n + 50, 2000), 0)
    X, X1 = X.cpu().numpy()[some], X1.cpu().numpy()
    assert int(m[R // 2]) == 0 and not X[2].any() and not X1[2].any()
    for q in (0, 1, 3):
        # either residual is below 1e-10 |y|, and |(z - H)^{-1}| <= 1 / Im z; as much again for the rounding
        assert np.linalg.norm(X[q] - X1[q], axis=-1).max() <= 8e-10 * np.linalg.norm(Y[some[q]])


@pytest.mark.parametrize("batch,words", [(128, 5), (384, 2), (4096, 5)])
def test_training_step(eng, batch, words):
    """One fused step against the layer-by-layer calls."""
    from impuritymodel_gb300.pruning import BasisNet

    g = torch.Generator(device=eng.device)
    g.manual_seed(batch)
    states = torch.randint(-(1 << 62), 1 << 62, (batch, words), device=eng.device, generator=g) * 2
    log_w = -14.0 * torch.rand(batch, device=eng.device, generator=g)
    one, two = BasisNet(eng, seed=1), BasisNet(eng, seed=1)
    losses = one.train(states, log_w, epochs=1, batch=batch)
    order = torch.Generator(device=eng.device)
    order.manual_seed(0)
    perm = torch.randperm(batch, device=eng.device, generator=order)
    X, Xt = two.inputs(states[perm].contiguous(), transposed=True)
    loss = two.gradients(X, Xt, log_w[perm].contiguous())
    two.adam_step()
    # every gradient but b3's (the last) in the same order of additions
    for a, b in ((one.G, two.G), (one.P, two.P), (one.m, two.m), (one.v, two.v)):
        assert torch.equal(a[:-1], b[:-1])
    for name in ("W1b", "W2b", "W2t"):
        assert torch.equal(getattr(one, name), getattr(two, name))
    # sums of `batch` terms of one size in two orders, both trees over 256 chains
    depth = 2.0 ** -24 * (batch / 128 + 16)
    bound = depth * float((2.0 / batch * (one.predict(states) - log_w).abs()).sum() + 1.0)
    assert abs(float(one.G[-1] - two.G[-1])) <= bound
    assert len(losses) == 1 and abs(float(losses[0] - loss)) <= depth * abs(float(loss))


@pytest.mark.parametrize("R,mapping", [
    (1, None), (3, None), (5, None),       # odd: a run per thread
    (10, None), (34, None),                # row kernel, two runs per thread
    (2, ("sched", 256, 16, 4, 128, 0)), (64, ("sched", 0, 32, 8, 256, 0)),
    (4, ("pages", 256, 16, 4, 512, 0)), (16, ("pages", 4096, 16, 8, 256, 3)), (32, ("pages", 0, 16, 4, 1024, 1)),
])
@pytest.mark.parametrize("cplx", [False, True])
def test_shifted_product(eng, R, mapping, cplx):
    """y = H x from the float32 copy of H - shift I, shift x added in the same launch."""
    n = 1003
    csr, H = _random_csr(eng, n, R, cplx, heavy=(0, 1, 500))
    diag = csr.col == torch.repeat_interleave(torch.arange(n, device=eng.device), csr.row_ptr[1:] - csr.row_ptr[:-1])
    (csr.val_c[:, 0] if cplx else csr.val_r)[diag] -= 700.0
    H = H - 700.0 * scipy.sparse.identity(n)
    csr.mixed()
    assert abs(csr.mixed_shift + 700.0) < 1.0
    g = np.random.default_rng(R)
    x = (g.normal(size=(n, R)) + 1j * g.normal(size=(n, R))).astype(np.complex64)
    y = eng.spmv(csr, torch.from_numpy(x).to(eng.device), precision=1, mapping=mapping).cpu().numpy()
    # float32: values and products round by 2^-24 each, sums of up to ~90 terms in any order
    A = abs(H - csr.mixed_shift * scipy.sparse.identity(n))
    bound = 2.0 ** -24 * (95 * (A @ abs(x)) + 4 * 701.0 * abs(x)) * 2
    assert (abs(y - H @ x.astype(np.complex128)) <= bound).all()


@pytest.mark.parametrize("n,words,flips,ones,packs", [
    (8193, 5, 3, False, True),     # a few zeros in full states, the smallest size beyond one CTA
    (50001, 5, 3, True, True),     # a few ones in empty states
    (20000, 1, 2, False, True),    # one word: two passes and a gather instead of eight passes
    (20000, 8, 6, False, True),    # the widest fields: 60 bits
    (20000, 8, 7, True, False),    # too many positions for one key
    (9001, 2, 40, False, False),   # dense states
])
def test_sort_of_sparse_states(eng, n, words, flips, ones, packs):
    import ctypes as C

    g = np.random.default_rng(n + words)
    bits = np.zeros((n, 64 * words), dtype=np.uint8)
    for _ in range(flips):  # fewer positions where some coincide; a third of the states twice
        bits[np.arange(n), g.integers(3, 64 * words - 2, size=n)] = 1
    bits[: n // 3] = bits[n - n // 3:]
    bits[:, :3] = (1, 0, 1)
    if not ones:
        bits[:, 3:] ^= 1
    keys = np.packbits(bits, axis=1).view(">u8").astype(np.uint64).reshape(n, words)
    t = eng.upload_states(keys)
    payload = torch.arange(n, dtype=torch.int32, device=eng.device) * 3
    stats = torch.empty(2 * words + 2, dtype=torch.int64, device=eng.device)
    eng.lib.edgpu_state_stats(words, t.data_ptr(), n, stats.data_ptr(), eng.stream)
    arr = (C.c_uint64 * (2 * words + 2))(*[int(x) for x in stats.cpu().numpy().view(np.uint64)])
    assert (eng.lib.edgpu_sort_packing(words, arr) > 0) == packs
    eng.sort_states(t, payload)
    order = np.lexsort(keys.T[::-1])  # stable, first word most significant
    assert np.array_equal(t.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(payload.cpu().numpy(), 3 * order)


@pytest.mark.parametrize("n,extra,K", [
    (9, 0, 7),       # less than a warp of rows
    (33, 0, 20),     # fewer rows than threads, one row in the second slice
    (513, 0, 40),    # a second pass of one row
    (1770, 0, 40),
    (4240, 0, 24),   # near the largest sector that fits
    (700, 40, 24),   # rows of 40 more entries: several lengths
    (60, 90, 24),    # a row longer than the sector (repeated columns): no sliced copy
])
def test_runs_on_sliced_rows(eng, n, extra, K):
    """Long calls (sliced rows) give every run the bits that it has in a short call (CSR rows)."""
    from impuritymodel_gb300.engine import CsrMatrix

    rng = np.random.default_rng(n + extra)
    rows, cols = [np.arange(n)], [np.arange(n)]
    for _ in range(2):
        i, j = rng.integers(0, n, size=(2, n))
        rows += [i, j]
        cols += [j, i]
    for i in (0, n // 2):
        j = rng.integers(0, n, size=extra)
        rows += [np.full(extra, i), j]
        cols += [j, np.full(extra, i)]
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    o = np.argsort(rows, kind="stable")
    rows, cols = rows[o], cols[o]
    vals = np.cos(1.0 + 7.0 * np.minimum(rows, cols) + 3.0 * np.maximum(rows, cols)) + 4.0 * (rows == cols)
    rp = torch.from_numpy(np.searchsorted(rows, np.arange(n + 1)).astype(np.int64)).to(eng.device)
    csr = CsrMatrix(rp, torch.from_numpy(cols.astype(np.int32)).to(eng.device),
                    val_r=torch.from_numpy(vals).to(eng.device))
    R = torch.cuda.get_device_properties(eng.device).multi_processor_count + 5
    v = rng.normal(size=(n, R)) + 1j * rng.normal(size=(n, R))
    v = torch.from_numpy(v / np.linalg.norm(v, axis=0)).to(eng.device)
    k = np.full(R, K, dtype=np.int32)
    k[1], k[2] = 0, max(1, K // 2)
    a, b = eng.lanczos(csr, v, k, precision=0)
    some = [0, 1, 2, R // 2, R - 1]
    k1 = np.minimum(k[some], 7)
    a1, b1 = eng.lanczos(csr, v[:, some].contiguous(), k1, precision=0)
    for q, r in enumerate(some):
        assert torch.equal(a[r, :k1[q]], a1[q, :k1[q]])
        assert torch.equal(b[r, :max(k1[q] - 1, 0)], b1[q, :max(k1[q] - 1, 0)])
    H = scipy.sparse.csr_matrix((vals, (rows, cols)), shape=(n, n))
    ar, br = _recurrence(H, v[:, 0].cpu().numpy(), min(K, 12))
    m = min(K, 12)
    # a dozen steps of an unconverged recurrence amplify rounding by less than 1e3
    assert np.abs(a[0, :m].cpu().numpy() - ar[:m]).max() < 1e-12 * max(abs(H).sum(1).max(), 1.0)


@pytest.mark.parametrize("n,R,K,cplx,extra", [
    (4267, 1, 12, False, 0),      # four threads a row, most of the block idle
    (4300, 32, 12, False, 0),     # as many runs as a block sums
    (30000, 2, 12, True, 0),      # two threads a row
    (47895, 8, 12, False, 0),     # several rows a thread
    (47895, 3, 12, False, 3000),  # a block's entries beyond its shared memory, repeated columns
    (20000, 5, 1, False, 0),      # a single step: alpha only
])
def test_grid_wide_lanczos_in_one_launch(eng, n, R, K, cplx, extra):
    """The cooperative form against the two launches a step (which the timed entry point keeps)."""
    from impuritymodel_gb300.engine import CsrMatrix

    rng = np.random.default_rng(n + R)
    rows, cols = [np.arange(0, n, 2)], [np.arange(0, n, 2)]  # odd diagonals are 0, some rows empty
    for _ in range(2):
        i, j = rng.integers(0, n, size=(2, n // 2))
        rows += [i, j]
        cols += [j, i]
    for i in (0, n // 3):
        j = rng.integers(0, n // 8, size=extra) * 8 % n
        rows += [np.full(extra, i), j]
        cols += [j, np.full(extra, i)]
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    o = np.argsort(rows, kind="stable")
    rows, cols = rows[o], cols[o]
    lo, hi = np.minimum(rows, cols), np.maximum(rows, cols)
    vals = np.cos(1.0 + 7.0 * lo + 3.0 * hi) / (1.0 + extra ** 0.5) + 4.0 * (rows == cols)
    rp = torch.from_numpy(np.searchsorted(rows, np.arange(n + 1)).astype(np.int64)).to(eng.device)
    col = torch.from_numpy(cols.astype(np.int32)).to(eng.device)
    if cplx:
        im = np.sign(cols - rows) * np.sin(5.0 * lo + hi)
        csr = CsrMatrix(rp, col, val_c=torch.from_numpy(np.stack([vals, im], 1)).to(eng.device).contiguous())
    else:
        csr = CsrMatrix(rp, col, val_r=torch.from_numpy(vals).to(eng.device))
    v = rng.normal(size=(n, R)) + 1j * rng.normal(size=(n, R))
    v = torch.from_numpy(v / np.linalg.norm(v, axis=0)).to(eng.device)
    k = np.full(R, K, dtype=np.int32)
    a, b = eng.lanczos(csr, v, k, precision=0)
    a1, b1 = eng.lanczos(csr, v, k, precision=0, timing=[])
    norm = np.bincount(rows, weights=np.abs(vals) + (np.abs(im) if cplx else 0.0)).max()
    # a dozen steps of an unconverged recurrence amplify rounding by less than 1e3
    assert (a - a1).abs().max().item() < 1e-12 * norm
    assert K == 1 or (b - b1)[:, :K - 1].abs().max().item() < 1e-12 * norm


@pytest.mark.parametrize("n,words,kinds", [
    (2, 1, 1),       # one key twice
    (33, 2, 20),     # a ragged second warp
    (1025, 5, 700),  # a network of 2048 keys, several blocks of heads
    (2048, 8, 2048),  # the longest keys
    (8192, 2, 5000),  # the largest that one CTA sorts
])
def test_sorted_unique_in_one_launch(eng, n, words, kinds):
    """Against the separate sort and compaction."""
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    pool = torch.randint(-(1 << 62), 1 << 62, (kinds, words), device=eng.device, generator=g) * 2
    pool[0] = -1  # the padding's key
    keys = pool[torch.randint(0, kinds, (n,), device=eng.device, generator=g)]
    assert eng.lib.edgpu_sort_unique_fits(words, n) == 1
    wide = torch.cat([keys, keys], 1)
    k, p = keys.clone(), torch.arange(n, dtype=torch.int32, device=eng.device)
    eng.sort_states(k, p)
    want, _, _ = eng.unique_sorted(k, p)
    before = keys.clone()
    assert torch.equal(eng.sort_unique(keys), want) and torch.equal(keys, before)
    assert torch.equal(eng.sort_unique(wide[:, :words]), want)  # strided rows


@pytest.mark.parametrize("n,n_orb,n_terms,cplx,filled", [
    (19501, 130, 400, False, 0.95),  # four states a batch, the last ones ragged
    (20000, 200, 2500, True, 0.97),  # complex operator
    (20500, 26, 900, False, 0.4),    # more outputs than a batch's scratch holds: one by one
])
def test_candidates_of_several_states(eng, n, n_orb, n_terms, cplx, filled, monkeypatch):
    if n_orb == 26:
        monkeypatch.setattr(eng, "scratch_entries", 64)
    test_one_pass_application(eng, n, n_orb, n_terms, cplx, filled)
