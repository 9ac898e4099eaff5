"""The error of the leading minors against extended precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _minors(S):
    """Leading minors by Gaussian elimination in numpy's long double (64-bit
    mantissa), partial pivoting."""
    n, N, _ = S.shape
    out = np.empty((n, N), np.clongdouble)
    for m in range(1, N + 1):
        A = S[:, :m, :m].astype(np.clongdouble)
        d, r = np.ones(n, np.clongdouble), np.arange(n)
        for j in range(m):
            k = np.argmax(np.abs(A[:, j:, j]), axis=1) + j
            t = A[r, k].copy()
            A[r, k] = A[r, j]
            A[r, j] = t
            d *= np.where(k != j, -1, 1) * A[:, j, j]
            if j + 1 < m:
                el = A[:, j + 1:, j] / A[:, j, j][:, None]
                A[:, j + 1:, j + 1:] -= el[:, :, None] * A[:, j, None, j + 1:]
        out[:, m - 1] = d
    return out


@pytest.mark.parametrize("N", [8, 16, 24, 32])
def test_no_further_off_than_one_rounding_per_update(N):
    """Matrices 1 + 0.3 G / sqrt(N): an entry is updated by products an order
    below it, each rounding it once by eps / sqrt(12) in the mean, and a minor
    gathers those of up to N pivots: an rms relative error below eps / sqrt(12)
    sqrt(N (N + 1) / 2).  The kernel in registers may lie a tenth above the one in
    shared memory; a second rounding per update puts it 1.4 times there."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ptr
    ctx = nb.default_context()
    g = torch.Generator().manual_seed(N)
    G = torch.randn((600, N, N), dtype=torch.complex128, generator=g)
    S = (torch.eye(N) + 0.3 * G / N ** 0.5).contiguous()
    exact = _minors(S.numpy())
    dev = S.to(ctx.device)
    room = torch.empty(2 * dev.numel() + 2, dtype=torch.float64, device=ctx.device)[1:]
    assert room.data_ptr() % 16 == 8  # matrices on 8 bytes take the kernel in shared memory
    room[:2 * dev.numel()] = torch.view_as_real(dev).reshape(-1)
    other = torch.empty((600, N), dtype=torch.complex128, device=ctx.device)
    ctx.check(lib().nrcps_slater_dets(ctx.handle, _ptr(room), None, N, 600, 0, 0, _ptr(other)))

    def rms(d):
        e = np.abs(d.cpu().numpy().astype(np.clongdouble) - exact) / np.abs(exact)
        return float(np.sqrt(np.mean(e.astype(np.float64) ** 2)))

    got, ref = rms(nb.slater_dets(dev, ctx=ctx)), rms(other)
    assert ref <= 2.2e-16 / 12 ** 0.5 * (N * (N + 1) / 2) ** 0.5
    assert got <= 1.1 * ref
