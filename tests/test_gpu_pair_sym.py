"""The packed pair kernel of one set of FP32 orbitals at the edges of its
blocks, tiles and windows of tiles."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


# block counts 2 to 4, full and padded; a volume below one tile, not whole
# tiles, one block of many configurations, a partner table that is no mirror;
# the last: 308 tiles of one CTA, more than one window
@pytest.mark.parametrize("n,vol,nconf,mirror", [
    (9, 64, 2, True), (10, 216, 5, False), (13, 1000, 3, True), (15, 512, 700, True), (16, 4096, 1, False),
    (20, 1728, 9, True), (10, 13824, 2, False), (16, 39304, 148, True)])
def test_pair_matrix_of_one_set(ctx, n, vol, nconf, mirror):
    """Every real sum is a chain of at most 12 products, one join and five tree
    levels in FP32 on weights and weighted orbitals rounded once each: at most
    20 roundings, on a component that has two products per term, so 40 x 2^-24
    of the sum of moduli bounds it.  Symmetric by construction."""
    import nrcps_b200 as nb
    from nrcps_b200 import _capi as C
    g = torch.Generator(device=ctx.device).manual_seed(n + vol)
    psi = torch.randn((nconf, n, vol), dtype=torch.complex64, device=ctx.device, generator=g)
    opp = torch.arange(vol, device=ctx.device)
    if mirror:
        opp = (vol - opp) % vol
    else:  # a random involution: half the sites in pairs, the rest their own partners
        p = torch.randperm(vol, device=ctx.device, generator=g)[: vol // 4 * 2]
        opp[p[0::2]], opp[p[1::2]] = p[1::2].clone(), p[0::2].clone()
    w = torch.rand(vol, dtype=torch.float64, device=ctx.device, generator=g) + 0.1
    w = torch.where(torch.arange(vol, device=ctx.device) < opp, w, w[opp])
    out = torch.full((nconf, n, n), float("nan"), dtype=torch.complex128, device=ctx.device)
    o32 = opp.to(torch.int32)
    ctx.check(nb.lib().nrcps_pair_matrix(ctx.handle, *(ctypes.c_void_p(t.data_ptr()) for t in (psi, psi)), n, nconf,
                                         vol, ctypes.c_void_p(w.data_ptr()), ctypes.c_void_p(o32.data_ptr()), C.F32,
                                         ctypes.c_void_p(out.data_ptr())), "pair_matrix")
    for c in sorted({0, nconf // 2, nconf - 1}):
        x = psi[c].to(torch.complex128)
        want = (x * w) @ x[:, opp].T
        size = (x.abs() * w) @ x[:, opp].abs().T
        assert ((out[c] - want).abs() <= 40 * 2.0 ** -24 * size).all()
    assert torch.equal(out, out.transpose(1, 2))
