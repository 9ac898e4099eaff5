"""Pair matrices of one set of FP32 orbitals (csrc/pair_sym.cu): edges of its
tiles and blocks, and its error against the general kernel's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


def _matrix(ctx, x, y, w, opp):
    import ctypes

    import nrcps_b200 as nb
    from nrcps_b200 import _capi as C
    nconf, n, vol = x.shape
    out = torch.full((nconf, n, n), float("nan"), dtype=torch.complex128, device=ctx.device)
    o32 = opp.to(torch.int32)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (x, y, w, o32, out)]
    ctx.check(nb.lib().nrcps_pair_matrix(ctx.handle, p[0], p[1], n, nconf, vol, p[2], p[3], C.F32, p[4]),
              "pair_matrix")
    return out


def _inputs(ctx, n, vol, nconf, positive):
    g = torch.Generator(device=ctx.device).manual_seed(n + vol + nconf)
    psi = torch.randn((nconf, n, vol), dtype=torch.complex64, device=ctx.device, generator=g)
    if positive:
        psi = (psi.abs() * (1 + 0.1j)).to(torch.complex64)
    i = torch.arange(vol, device=ctx.device)
    opp = (vol - i) % vol
    w = torch.rand(vol, dtype=torch.float64, device=ctx.device, generator=g) + 0.1
    return psi, torch.where(i < opp, w, w[opp]), opp


# volumes from the first that this kernel takes, whole tiles of 128 sites and not,
# more configurations than clusters fit
@pytest.mark.parametrize("n,vol,nconf", [(9, 4096, 2), (10, 4097, 1), (13, 4225, 3), (15, 6000, 40), (16, 8192, 30),
                                         (17, 4096, 24), (20, 5001, 9), (19, 4224, 200)])
def test_edges(ctx, n, vol, nconf):
    """A real sum is a chain of at most 8 products, one join and three tree levels
    in FP32 on weights and weighted orbitals rounded once each: 14 roundings, two
    products per term, so 28 x 2^-24 of the sum of moduli."""
    psi, w, opp = _inputs(ctx, n, vol, nconf, False)
    out = _matrix(ctx, psi, psi, w, opp)
    for c in sorted({0, nconf // 2, nconf - 1}):
        x = psi[c].to(torch.complex128)
        size = (x.abs() * w) @ x[:, opp].abs().T
        assert ((out[c] - (x * w) @ x[:, opp].T).abs() <= 28 * 2.0 ** -24 * size).all()
    assert torch.equal(out, out.transpose(1, 2))


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("n,vol", [(9, 4096), (10, 13824), (13, 13824), (16, 13824), (20, 32768)])
def test_error_is_the_general_kernels(ctx, n, vol, positive):
    """Positive orbitals, as those without nodes are, leave every rounding of a
    sum at its whole size.  The general kernel, which takes two sets of orbitals,
    sums chains of 14 and more products; rms errors of hundreds of entries scatter
    by some percent, 1.2 allows for it."""
    psi, w, opp = _inputs(ctx, n, vol, 8, positive)
    x = psi.to(torch.complex128)
    want = torch.einsum("csv,ctv->cst", x * w, x[:, :, opp])
    size = torch.einsum("csv,ctv->cst", x.abs() * w, x[:, :, opp].abs())
    own, general = (_matrix(ctx, psi, y, w, opp) for y in (psi, psi.clone()))
    rms = [(((s - want).abs() / size) ** 2).mean().sqrt() for s in (own, general)]
    assert rms[0] <= 1.2 * rms[1]
