"""Calls in the forms that a dispatch rule or a kept plan could get wrong: cut into chunks, under
inference mode, on tables written in place, with inputs of another length, type or place."""

import pytest
import torch

from .test_gpu_kernel_edges import _random_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,cplx,locked", [
    (40, 30, False, 0),
    (300, 41, True, 0),
    (1770, 50, False, 3),   # deflated vectors ahead of the run's own
    (9000, 22, False, 0),   # several rows a lane group
])
def test_reorthogonalised_steps_of_any_chunk(eng, n, K, cplx, locked):
    """Where the host cuts a run into launches depends on its residuals: no bit may."""
    csr, _ = _random_csr(eng, n, n + K, cplx, heavy=(0,))
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    Q, _ = torch.linalg.qr(torch.randn((n, locked + 1), dtype=torch.complex128, device=eng.device, generator=g))
    lock = Q[:, :locked].t().contiguous() if locked else None
    v0 = Q[:, locked].contiguous()
    V, a, b = eng.krylov_reorth(csr, v0, K, chunk=K, locked=lock)
    for chunk in (1, 7):
        W, c, d = eng.krylov_reorth(csr, v0, K, chunk=chunk, locked=lock)
        assert (a == c).all() and (b == d).all()
        assert torch.equal(torch.view_as_real(V), torch.view_as_real(W))


def _hopping(n_orb, value=0.3):
    """A ring of hops and a density-density term per neighbour."""
    op = {}
    for i in range(n_orb):
        j = (i + 1) % n_orb
        op[((i, "c"), (i, "a"))] = 0.1 * i
        op[((i, "c"), (j, "a"))] = value
        op[((j, "c"), (i, "a"))] = value
        op[((i, "c"), (j, "c"), (j, "a"), (i, "a"))] = 0.7
    return op


def _start(eng, words=(0b1011 << 60,)):
    import numpy as np

    return eng.upload_states(np.array([words], dtype=np.uint64))


def test_application_of_tables_from_inference_mode(eng):
    """Tensors made there count no versions; a plan of them is not kept."""
    from impuritymodel_gb300 import ops as _ops  # noqa: F401  (registers torch.ops.edgpu)
    from impuritymodel_gb300.engine import DeviceOp

    b0 = _start(eng)
    plain = DeviceOp(_hopping(9), eng.device)
    basis, order = eng.expand(b0, plain, None)
    csr = eng.build_csr(basis, plain, None)
    with torch.inference_mode():
        dop = DeviceOp(_hopping(9), eng.device)
        inside = eng.expand(b0, dop, None) + tuple(getattr(eng.build_csr(basis, dop, None), k)
                                                   for k in ("row_ptr", "col", "val_r"))
        none = torch.zeros(0, dtype=torch.int32, device=eng.device)
        mask = torch.zeros((0, 8), dtype=torch.int64, device=eng.device)
        ops = torch.ops.edgpu.build_csr(basis, dop.ops, dop.coeff, dop.flags, none, none, mask, 1e-12)
    outside = eng.build_csr(basis, dop, None)  # the same tensors after the mode has ended
    again = eng.build_csr(basis, plain, None)  # a plan made outside, read again
    with torch.inference_mode():
        again_inside = eng.build_csr(basis, plain, None)
    assert torch.equal(inside[0], basis) and torch.equal(inside[1], order)
    for got in (inside[2:], ops, (outside.row_ptr, outside.col, outside.val_r), (again.row_ptr, again.col, again.val_r),
                (again_inside.row_ptr, again_inside.col, again_inside.val_r)):
        for x, y in zip(got, (csr.row_ptr, csr.col, csr.val_r)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("full,empty", [(16, 17), (64, 64), (70, 70), (64, 128)])  # outputs: 272, 4096, 4900, 8192
def test_application_of_more_outputs_than_the_scratch(eng, full, empty, cplx):
    """Hops from `full` to `empty` orbitals: as many outputs of one state as terms, in their order."""
    import numpy as np

    from impuritymodel_gb300.engine import DeviceOp

    hops = [(i, j) for i in range(full, full + empty) for j in range(full)]
    amp = [0.5 + k + (0.25j * k if cplx else 0.0) for k in range(len(hops))]
    dop = DeviceOp({((i, "c"), (j, "a")): v for (i, j), v in zip(hops, amp)}, eng.device)
    occ = np.zeros((1, 256), dtype=np.uint8)
    occ[0, :full] = 1
    words = lambda o: np.packbits(o, axis=1).view(">u8").astype(np.uint64)  # noqa: E731
    state = eng.upload_states(words(occ))
    before = eng.scratch_entries
    offs, out, _, vals = eng.apply_columns(state, dop, None, 0.0, want_states=True, want_vals=True)
    want = np.repeat(occ, len(hops), axis=0)
    for k, (i, j) in enumerate(hops):
        want[k, i], want[k, j] = 1, 0
    # j orbitals below the annihilated one, then full - 1 below the created one
    sign = np.array([(-1.0) ** (j + full - 1) for _, j in hops])
    assert offs.tolist() == [0, len(hops)]
    assert np.array_equal(out.cpu().numpy().view(np.uint64), words(want))
    v = vals.cpu().numpy()
    assert np.array_equal(v[:, 0] + 1j * v[:, 1], sign * np.array(amp))
    # what that call needed is no other call's
    assert eng.scratch_entries == before
    basis, _ = eng.expand(_start(eng), DeviceOp(_hopping(9), eng.device), None)
    assert basis.shape == (84, 1)  # three particles on nine orbitals


def test_application_follows_its_tables(eng):
    """Tables written in place between two applications: coefficients that become complex, orbitals
    beyond the states' words."""
    from impuritymodel_gb300.engine import DeviceOp

    b0 = _start(eng, (0b1011 << 60, 0))  # two words
    dop = DeviceOp(_hopping(9), eng.device)
    cols = lambda d: eng.apply_columns(b0, d, None, 0.0, want_states=True, want_vals=True)  # noqa: E731
    cols(dop)
    dop.coeff[:, 1] = 0.5 * dop.coeff[:, 0]
    want = DeviceOp({k: v * (1 + 0.5j) for k, v in _hopping(9).items()}, eng.device)
    for x, y in zip(cols(dop), cols(want)):
        assert x is None and y is None or torch.equal(x, y)
    basis, _ = eng.expand(b0, want, None)
    one, two = eng.build_csr(basis, dop, None), eng.build_csr(basis, want, None)
    assert torch.equal(one.val_c, two.val_c) and torch.equal(one.col, two.col)
    dop.coeff[:, 1] = 0.0  # real again
    one, two = eng.build_csr(basis, dop, None), eng.build_csr(basis, DeviceOp(_hopping(9), eng.device), None)
    assert torch.equal(one.val_r, two.val_r) and torch.equal(one.col, two.col)
    # a hop to an orbital that the words do not hold: the kernel for general tables only empties the
    # other one, and the plan has no group for it
    near, far = ((1, "c"), (0, "a")), ((200, "c"), (0, "a"))
    dop.ops[list(_hopping(9)).index(near)] = DeviceOp({far: 0.3}, eng.device).ops[0]
    moved = DeviceOp({(far if t == near else t): v for t, v in _hopping(9).items()}, eng.device)
    for x, y in zip(cols(dop), cols(moved)):
        assert x is None and y is None or torch.equal(x, y)


@pytest.fixture(scope="module")
def refusing(eng, tmp_path_factory):
    """A copy of the library whose cooperative and cluster launches are refused, by the linker's
    stand-ins for the two runtime calls, as where a program holds only a part of the SMs."""
    import glob
    import os
    import subprocess

    from impuritymodel_gb300 import _lib as L
    from impuritymodel_gb300 import nvcc_build

    out = tmp_path_factory.mktemp("refusing")
    src = out / "refuse.cu"
    src.write_text("""
#include <cuda_runtime.h>
static int refused = 0;
extern "C" cudaError_t __wrap_cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  ++refused;
  return cudaErrorCooperativeLaunchTooLarge;
}
extern "C" cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
  ++refused;
  return cudaErrorInvalidClusterSize;
}
extern "C" int launches_refused() { return refused; }
""")
    so = str(out / "librefusing.so")
    objs = glob.glob(os.path.join(nvcc_build.BUILD_DIR, "*.o"))
    subprocess.run([nvcc_build._nvcc(), *nvcc_build.ARCH, "-Xcompiler", "-fPIC", "-shared", "-o", so, str(src), *objs,
                    "-cudart", "static", "-Xlinker", "--wrap=cudaLaunchCooperativeKernel", "-Xlinker",
                    "--wrap=cudaLaunchKernelExC"], check=True, capture_output=True)
    return L.load(so)


@pytest.mark.parametrize("n,R,K,cplx", [(4300, 1, 12, False), (20000, 3, 12, True), (47895, 8, 9, False)])
def test_large_sectors_where_cooperative_launches_are_refused(eng, refusing, monkeypatch, n, R, K, cplx):
    """The two launches a step take the call, to the rounding of another order of sums."""
    csr, H = _random_csr(eng, n, n + R, cplx, heavy=(0, 1, n // 2))
    g = torch.Generator(device=eng.device)
    g.manual_seed(R)
    v = torch.randn((n, R), dtype=torch.complex128, device=eng.device, generator=g)
    v /= torch.linalg.vector_norm(v, dim=0)
    a, b = eng.lanczos(csr, v, [K] * R)
    before = refusing.launches_refused()
    monkeypatch.setattr(eng, "lib", refusing)
    a1, b1 = eng.lanczos(csr, v, [K] * R)
    assert refusing.launches_refused() == before + 1
    # a dozen steps of an unconverged recurrence amplify rounding by less than 1e3
    tol = 1e-12 * abs(H).sum(1).max()
    assert (a - a1).abs().max().item() < tol and (b - b1)[:, :K - 1].abs().max().item() < tol


@pytest.mark.parametrize("n,R,cplx", [(40, 2, False), (360, 15, False), (360, 70, True)])
def test_shifted_solves_where_cluster_launches_are_refused(eng, refusing, monkeypatch, n, R, cplx):
    csr, _ = _random_csr(eng, n, n + R, cplx, heavy=(0,))
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    y = torch.randn((R, n), dtype=torch.complex128, device=eng.device, generator=g)
    y /= torch.linalg.vector_norm(y, dim=1, keepdim=True)
    zs = torch.linspace(-8.0, 8.0, 3 * R, dtype=torch.float64).view(R, 3).numpy() + 0.5j
    X, _ = eng.shifted_solve(csr, y, zs, 1e-10, min(6 * n + 50, 2000))
    before = refusing.launches_refused()
    monkeypatch.setattr(eng, "lib", refusing)
    X1, _ = eng.shifted_solve(csr, y, zs, 1e-10, min(6 * n + 50, 2000))
    assert refusing.launches_refused() > before
    # either residual is below 1e-10, and |(z - H)^{-1}| <= 1 / Im z; as much again for the rounding
    assert torch.linalg.vector_norm(X - X1, dim=2).max().item() <= 8e-10


@pytest.mark.parametrize("n,R,K,precision", [
    (1770, 3, 40, 0),    # one SM
    (4300, 2, 25, 0),    # one cooperative launch
    (47895, 3, 30, 0),
    (5000, 33, 10, 0),   # two launches a step
    (5000, 40, 10, 1),
])
def test_timed_lanczos_is_the_plain_one(eng, n, R, K, precision):
    csr, _ = _random_csr(eng, n, n + R, heavy=(0, n // 2))
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    v = torch.randn((n, R), dtype=torch.complex128, device=eng.device, generator=g)
    v /= torch.linalg.vector_norm(v, dim=0)
    a, b = eng.lanczos(csr, v, [K] * R, precision=precision)
    timing = []
    a1, b1 = eng.lanczos(csr, v, [K] * R, precision=precision, timing=timing)
    assert torch.equal(a, a1) and torch.equal(b, b1)
    assert timing[0]["spmm_ms"] > 0.0 and timing[0]["axpy_ms"] >= 0.0 and timing[0]["normalize_ms"] == 0.0


def test_a_read_status_is_spent(eng):
    """What one call set and answered for is no later call's error."""
    import numpy as np

    from impuritymodel_gb300 import _lib as L
    from impuritymodel_gb300.engine import CsrMatrix, DeviceOp
    from impuritymodel_gb300.pruning import BasisNet

    n = 12
    csr = CsrMatrix(torch.arange(n + 1, device=eng.device), torch.arange(n, dtype=torch.int32, device=eng.device),
                    val_r=torch.arange(n, dtype=torch.float64, device=eng.device))
    v = torch.zeros(n, dtype=torch.complex128, device=eng.device)
    v[3] = 1.0
    net, dop = BasisNet(eng, seed=0), DeviceOp(_hopping(9), eng.device)
    eng.reset_status()

    def rank():
        basis, _ = eng.expand(_start(eng, (0b1011 << 60, 0, 0, 0, 0)), dop, None)
        assert net.predict(basis).shape == (84,)

    V, a, b = eng.krylov_reorth(csr, v, 8, chunk=2)  # an eigenvector: the space is exhausted at once
    assert len(a) == 1 and a[0] == 3.0 and b[0] == 0.0
    rank()
    with pytest.raises(L.EdgpuError):
        eng.lanczos(csr, v.view(n, 1), [4])
    rank()
    zs = np.full((1, 1), 3.5 + 0.1j)
    y = torch.ones((1, n), dtype=torch.complex128, device=eng.device)
    with pytest.warns(UserWarning):
        eng.shifted_solve(csr, y, zs, 1e-13, 2)
    rank()


@pytest.mark.parametrize("what", ["arena", "larger arena", "table"])
def test_application_without_room_for_its_arena(eng, monkeypatch, what):
    """The two passes, which keep nothing but the outputs, take the call."""
    from impuritymodel_gb300 import _lib as L
    from impuritymodel_gb300.engine import DeviceOp

    op = _hopping(26)
    # refused: the first arena, the one for 45 outputs a state that follows, the hash table of the basis
    op.update({((i, "c"), (j, "a")): 0.01 * (i + 1) * (j + 1) for i in range(26) for j in range(26) if (i - j) % 26 > 1})
    dop = DeviceOp(op, eng.device)
    basis, _ = eng.expand(_start(eng, (0b1011 << 60,)), dop, None)
    assert basis.shape == (2600, 1)
    want_c = eng.apply_columns(basis, dop, None, 0.0, want_states=True, want_vals=True)
    want = eng.build_csr(basis, dop, None)
    entry, first = eng.lib.edgpu_apply_groups_entry_bytes(), 16 * 2600 + 4096
    assert want.nnz > first
    empty = torch.empty

    def refuse(*size, **kw):
        big = entry * (first + 1 if what == "larger arena" else first)
        if kw.get("dtype") == torch.uint8 and size[0] >= big if what != "table" else size == (8192,):
            raise torch.cuda.OutOfMemoryError("refused")
        return empty(*size, **kw)

    monkeypatch.setattr(eng, "TABLE_MIN_BASIS", 1)
    monkeypatch.setattr(torch, "empty", refuse)
    got = eng.build_csr(basis, dop, None)
    got_c = eng.apply_columns(basis, dop, None, 0.0, want_states=True, want_vals=True)
    for k in ("row_ptr", "col", "val_r"):
        assert torch.equal(getattr(got, k), getattr(want, k))
    for x, y in zip(got_c, want_c):
        assert x is None and y is None or torch.equal(x, y)
    assert L.EDGPU_OK == int(eng.status.item())


@pytest.mark.parametrize("terms", [1, 33, 1025, 9000])
@pytest.mark.parametrize("cplx,top", [(False, -1), (True, 700), (False, 1023)])
def test_what_the_host_reads_of_tables(eng, terms, cplx, top):
    """Imaginary parts and the largest orbital, the last term alone deciding; unused slots hold none."""
    from types import SimpleNamespace

    from impuritymodel_gb300 import _lib as L

    ops = torch.zeros(terms, dtype=torch.int64, device=eng.device)
    ops[:-1] = 0x0000_03FF_8005_C007  # orbital 1023 in a slot that is not in use
    coeff = torch.zeros((terms, 2), dtype=torch.float64, device=eng.device)
    coeff[:, 0], coeff[:, 1] = 1.0, -0.0
    flags = torch.zeros(terms, dtype=torch.int32, device=eng.device)
    if top >= 0:
        ops[-1] = (0x8000 | top) << 32
    if cplx:
        coeff[-1, 1] = float("nan") if terms == 33 else 1e-300
    op = SimpleNamespace(ops=ops, coeff=coeff, flags=flags, n_terms=terms,
                         terms=L.Terms(ops.data_ptr(), coeff.data_ptr(), flags.data_ptr(), terms))
    eng.read_tables(op)
    assert op.is_real == (not cplx) and op.max_orbital == max(top, 7 if terms > 1 else -1)


@pytest.mark.parametrize("n,R,precision", [
    (1770, 3, 0), (1770, 160, 0),  # one SM, CSR and sliced rows
    (5000, 3, 0),                  # one cooperative launch
    (5000, 40, 0), (5000, 3, 1),   # two launches a step
])
def test_a_bad_run_keeps_to_itself(eng, n, R, precision):
    """A start vector with a NaN or an infinity, or of zeros: its status, and the other runs' bits."""
    from impuritymodel_gb300 import _lib as L

    K = 9
    csr, _ = _random_csr(eng, n, n + R, heavy=(0, n // 2))
    g = torch.Generator(device=eng.device)
    g.manual_seed(n)
    v = torch.randn((n, R), dtype=torch.complex128, device=eng.device, generator=g)
    v /= torch.linalg.vector_norm(v, dim=0)
    a, b = eng.lanczos(csr, v, [K] * R, precision=precision)
    others = [r for r in range(R) if r != 1]
    for value, status in ((float("nan"), L.EDGPU_ERR_NAN), (float("inf"), L.EDGPU_ERR_NAN), (0.0, L.EDGPU_ERR_BREAKDOWN)):
        w = v.clone()
        w[slice(None) if value == 0.0 else n // 2, 1] = value
        with pytest.raises(L.EdgpuError) as err:
            eng.lanczos(csr, w, [K] * R, precision=precision)
        assert err.value.status == status
        a1, b1 = eng.lanczos(csr, w, [K] * R, precision=precision, check=False)
        assert torch.equal(a[others], a1[others]) and torch.equal(b[others, :K - 1], b1[others, :K - 1])
        if value != 0.0:
            assert not bool(torch.isfinite(a1[1]).any())
    eng.reset_status()
