"""The blocked Gram and Cholesky kernels of the FP32 re-orthonormalisation
at the edges of their row blocks, stages and cluster splits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,dims,shift", [
    (1, (8, 8, 8), 0), (4, (4, 4, 4), 0), (5, (6, 6, 6), 1), (8, (8, 6, 12), 0), (9, (16, 16, 16), 0),
    (12, (4, 6, 2), 0), (13, (24, 24, 24), 1), (16, (16, 16, 8), 0), (17, (32, 32, 32), 0), (20, (32, 32, 32), 1),
    (21, (16, 16, 16), 0), (24, (24, 24, 24), 0), (25, (8, 8, 8), 1), (33, (32, 32, 16), 0), (64, (12, 12, 12), 0)])
def test_qr_at_block_edges(N, dims, shift):
    """Orthonormal orbitals and log R_ii that reproduce the Gram determinant,
    for row counts around the blocks of four, volumes below one stage and
    split over 1 to 8 CTAs, and orbitals that start 8 bytes past a 16-byte
    boundary (shift); the tolerances are those of the kernel's other tests.
    A configuration's result is the same bits alone and in a batch."""
    import nrcps_b200 as nb
    ctx = nb.default_context()
    nconf, V = 5, int(np.prod(dims))
    g = torch.Generator(device=ctx.device).manual_seed(N + V)
    a = torch.randn((nconf, N, V), dtype=torch.complex64, device=ctx.device, generator=g)
    a[:, 1:] += 0.9 * a[:, :1]
    buf = torch.zeros(a.numel() + 1, dtype=a.dtype, device=ctx.device)
    psi = buf[shift:shift + a.numel()].view(a.shape)
    psi.copy_(a)
    assert psi.data_ptr() % 16 == 8 * shift
    log_r = nb.reorthonormalise(psi, ctx=ctx)
    q, p = psi.to(torch.complex128), a.to(torch.complex128)
    eye = torch.eye(N, dtype=torch.complex128, device=ctx.device)
    for c in range(nconf):
        assert (q[c].conj() @ q[c].T - eye).abs().max().item() < 5e-5, c
        want = torch.linalg.slogdet(p[c].conj() @ p[c].T)[1].item()
        assert abs(2 * log_r[c].sum().item() - want) <= 1e-5 * abs(want) + 1e-5, c
    alone = a[3:4].clone() if not shift else None
    if alone is not None:
        one = nb.reorthonormalise(alone, ctx=ctx)
        assert torch.equal(alone[0], psi[3]) and torch.equal(one[0], log_r[3])


def test_singular_gram_matrix_is_marked():
    """A configuration whose orbitals are zero has no Cholesky factor: NaN in
    its log R_ii, the other configurations untouched by it."""
    import nrcps_b200 as nb
    ctx = nb.default_context()
    psi = torch.randn((3, 7, 512), dtype=torch.complex64, device=ctx.device)
    psi[1] = 0
    log_r = nb.reorthonormalise(psi, ctx=ctx)
    assert torch.isnan(log_r[1]).all() and torch.isfinite(log_r[[0, 2]]).all()
