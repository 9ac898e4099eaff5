"""The overlap with up to ten dense sources (csrc/overlap_few.cu) at the edges
of its blocks, groups of orbitals, tiles and splits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("ns,nt,vol,nconf", [
    (1, 1, 16, 1), (5, 5, 128, 3), (6, 5, 144, 700), (5, 6, 512, 9), (10, 10, 4096, 1), (10, 23, 4096, 5),
    (3, 11, 1728, 2), (10, 10, 13824, 30), (10, 10, 32768, 60)])
def test_overlap_of_few_sources(ctx, ns, nt, vol, nconf):
    """A real sum is a chain of at most 32 products, one join and five tree
    levels in FP32, on sources rounded once: 39 roundings, so 39 x 2^-24 of the
    sum of moduli bounds each part and 56 x 2^-24 the complex value."""
    import nrcps_b200 as nb
    g = torch.Generator(device=ctx.device).manual_seed(ns * 100 + nt + vol)
    src = torch.randn((ns, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((nconf, nt, vol), dtype=torch.complex64, device=ctx.device, generator=g)
    got = nb.overlap(src, psi, ctx)
    p = psi.to(torch.complex128)
    want = torch.einsum("sv,ctv->cst", src.conj(), p)
    size = torch.einsum("sv,ctv->cst", src.abs(), p.abs())
    assert ((got - want).abs() <= 56 * 2.0 ** -24 * size).all()
