"""Fields that are real at some sites and complex at others through the fused
steps, which ask a chunk of sites at a time whether its weights are real."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("L", [8, 16, 24, 32, 48])
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("mode,trap", [(2, False), (2, True), (0, False)])
@pytest.mark.parametrize("nconf", [1, 160])
def test_mixed_fields(ctx, L, precision, mode, trap, nconf):
    """Against the same step from torch's FP64 transforms of the same orbitals.
    A 3-D transform rounds a value some 3 log2 L times (17 at L = 48) with
    errors that add up as their squares; 2^-53 (2^-24) x 40 of the norm holds
    two of them and the factors.  One configuration and more than SMs."""
    import nrcps_b200 as nb
    if nconf > 1 and L == 48:
        nconf = 40
    V = L ** 3
    g = torch.Generator(device=ctx.device).manual_seed(L + nconf)
    dt = torch.complex64 if precision == "f32" else torch.complex128
    psi = torch.randn((nconf, L, L, L), dtype=dt, device=ctx.device, generator=g)
    k = torch.rand(V, dtype=torch.float64, device=ctx.device, generator=g) + 0.5
    phi = torch.randn((nconf * V, 2), dtype=torch.float64, device=ctx.device, generator=g)
    run = torch.arange(nconf * V, device=ctx.device) // (3 * L * L)  # whole chunks of a pencil, and parts of some
    phi[:, 1] *= (run % 2 == 0) | (torch.rand(nconf * V, device=ctx.device, generator=g) < 0.01)
    if mode == 0:
        phi /= V
    pos = torch.rand(V, dtype=torch.float64, device=ctx.device, generator=g) if trap else None
    a = 0.3
    w = torch.view_as_complex(phi).reshape(nconf, L, L, L)
    if mode == 2:
        w = (1 + a * w) / V
    if trap:
        w = w * pos.reshape(L, L, L)
    kk = k.reshape(L, L, L)
    want = kk * torch.fft.ifftn(w * torch.fft.fftn(kk * psi.to(torch.complex128), dim=(1, 2, 3)), dim=(1, 2, 3),
                                norm="forward")
    nb.propagate(psi, 1, k, phi, a, mode, 0, V, pos, ctx)
    err = torch.linalg.vector_norm(psi - want) / torch.linalg.vector_norm(want)
    assert err < 40 * 2.0 ** (-24 if precision == "f32" else -53)
