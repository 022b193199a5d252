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
