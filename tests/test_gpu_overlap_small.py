"""The CUDA-core overlap in small volumes and with few sources or orbitals: its
two kernels give the same sums, as accurate as those of 256 threads."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("ns,nt,vol", [(10, 1, 4096), (33, 1, 512), (3, 33, 4096), (2, 70, 1728), (19, 5, 1728),
                                       (8, 33, 1728), (9, 10, 5000), (17, 18, 700)])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_same_bits_by_either_kernel(ctx, ns, nt, vol, precision):
    """From one configuration to thousands both kernels and every split come up."""
    import nrcps_b200 as nb
    g = torch.Generator(device=ctx.device).manual_seed(ns * 100 + nt)
    dt = torch.complex128 if precision == "f64" else torch.complex64
    most = min(3000, (1 << 24) // (nt * vol))
    src = torch.randn((ns, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((most, nt, vol), dtype=dt, device=ctx.device, generator=g)
    ctx.set_option("overlap.tc", 0)
    try:
        whole = nb.overlap(src, psi, ctx)
        for n in (1, 3, 20, 75, 300):
            if n < most:
                assert torch.equal(nb.overlap(src, psi[:n], ctx), whole[:n]), n
    finally:
        ctx.set_option("overlap.tc", 1)
    c = most - 1
    p = psi[c].to(torch.complex128)
    size = src.abs() @ p.abs().T
    assert ((whole[c] - src.conj() @ p.T).abs() <= 1e-13 * size).all()


@pytest.mark.parametrize("n,vol", [(7, 512), (10, 512), (19, 512), (19, 1728), (10, 4096), (24, 4096)])
def test_error_in_small_volumes(ctx, n, vol):
    """Against sums of 256 threads a site apart, a warp's tree and eight warps in
    a row.  The variance of a sum's roundings goes with half the length of its
    chains: 12.5 such units against 12.5 in 8^3, 17 against 17 in 12^3, at worst 25.5
    against 26 in 16^3; of 200 numbers and more an rms scatters by some percent, so
    that 1.25 holds where 1.7 (32 sites a lane, N = 19) would not."""
    import nrcps_b200 as nb
    g = torch.Generator(device=ctx.device).manual_seed(n + vol)
    src = torch.randn((n, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((4, n, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    got = nb.overlap(src, psi, ctx).cpu().numpy()
    a, b = src.cpu().numpy().conj(), psi.cpu().numpy()
    want = a.astype(np.clongdouble) @ b.astype(np.clongdouble).transpose(0, 2, 1)

    def threads(x, y):
        """sum of the real products x y over the sites in that order, in doubles"""
        pad = -vol % 256
        p = np.pad(x[None, :, None] * y[:, None], ((0, 0), (0, 0), (0, 0), (0, pad)))
        s = np.zeros(p.shape[:3] + (256,))
        for k in range(0, vol + pad, 256):
            s = s + p[..., k:k + 256]
        s = s.reshape(p.shape[:3] + (8, 32))
        while s.shape[-1] > 1:
            s = s[..., : s.shape[-1] // 2] + s[..., s.shape[-1] // 2:]
        t = np.zeros(p.shape[:3])
        for w in range(8):
            t = t + s[..., w, 0]
        return t

    ref = threads(a.real, b.real) - threads(a.imag, b.imag)
    err = np.sqrt(np.mean(((got.real - want.real).astype(np.float64)) ** 2))
    assert err <= 1.25 * np.sqrt(np.mean(((ref - want.real).astype(np.float64)) ** 2))
