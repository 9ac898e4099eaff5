"""The tiled CUDA-core overlap and the segment-per-minor determinants at the
edges of their tiles, segments and chunks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("ns,nt,vol,nconf", [
    (1, 1, 8, 3), (4, 4, 512, 1), (5, 3, 216, 7), (7, 7, 4096, 1), (16, 32, 4096, 2), (19, 19, 32768, 1),
    (19, 19, 576, 700), (33, 33, 13824, 1), (33, 20, 1000, 5), (1, 40, 2048, 1), (130, 2, 999, 1), (24, 25, 8191, 2)])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_overlap_tiles(ctx, ns, nt, vol, nconf, precision):
    """S = <src|psi> summed in FP64 against the same sum in torch: every
    product is exact to 2^-53 and a sum of V terms rounds by at most V eps of
    the sum of moduli (by sqrt(V) eps in the mean); 1e-13 of that sum holds
    the largest V here.  Tiles that do not fill, chunks of one cluster and of
    many, one source or orbital against many."""
    import nrcps_b200 as nb
    g = torch.Generator(device=ctx.device).manual_seed(ns * 1000 + vol)
    dt = torch.complex128 if precision == "f64" else torch.complex64
    src = torch.randn((ns, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((nconf, nt, vol), dtype=dt, device=ctx.device, generator=g)
    ctx.set_option("overlap.tc", 0)
    try:
        got = nb.overlap(src, psi, ctx)
    finally:
        ctx.set_option("overlap.tc", 1)
    p = psi.to(torch.complex128)
    want = torch.einsum("sv,ctv->cst", src.conj(), p)
    size = torch.einsum("sv,ctv->cst", src.abs(), p.abs())
    assert ((got - want).abs() <= 1e-13 * size).all()


@pytest.mark.parametrize("N", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 31, 32])
@pytest.mark.parametrize("mode,log", [(0, False), (1, False), (0, True)])
def test_minors_by_segments_against_the_thread_kernel(ctx, N, mode, log):
    """Orders around the segments of 8, 16 and 32 lanes and the groups of four
    columns, batches that leave segments empty, against the thread-per-minor
    kernel; matrices 1 + 0.3 G have condition numbers of a few hundred at
    most, so 1e-11 relative is N eps times that with room."""
    import nrcps_b200 as nb
    g = torch.Generator(device=ctx.device).manual_seed(N)
    S = torch.eye(N, dtype=torch.complex128, device=ctx.device) + 0.3 * torch.randn(
        (37, N, N), dtype=torch.complex128, device=ctx.device, generator=g) / N ** 0.5
    S[5] *= 1e-170  # squares of the moduli underflow
    S[6] *= 1e170   # ... overflow
    P = torch.randn((37, N, N), dtype=torch.complex128, device=ctx.device, generator=g) if mode else None
    out = []
    try:
        for warp in (1, 0):
            ctx.set_option("lu.warp", warp)
            out.append(nb.slater_dets(S, P, mode=mode, log=log, ctx=ctx).cpu().numpy())
    finally:
        ctx.set_option("lu.warp", 1)
    a, b = out
    if log:  # the same determinant: moduli, and phases up to whole turns
        assert np.max(np.abs(a.real - b.real)) < 1e-9
        assert np.max(np.abs(np.exp(1j * a.imag) - np.exp(1j * b.imag))) < 1e-9
        return
    ok = np.isfinite(b) & (np.abs(b) > 1e-290)
    assert ok[np.arange(37) != 5][:5].all()
    assert np.max(np.abs(a[ok] - b[ok]) / np.abs(b[ok])) < 1e-11


def test_minors_ties_zero_pivots_and_zero_rows(ctx):
    """Exact ties, zero pivots (ludcmp's 1e-20) and all-zero rows (NaN) in
    every segment size, bit for bit the thread kernel's."""
    import nrcps_b200 as nb
    mats = []
    for N in (32,):
        ones = torch.ones((N, N), dtype=torch.complex128)
        perm = torch.eye(N, dtype=torch.complex128).flip(0)
        zero = torch.eye(N, dtype=torch.complex128)
        zero[11] = 0
        mats = [torch.eye(N, dtype=torch.complex128), ones, perm, zero]
    S = torch.stack(mats).to(ctx.device)
    out = []
    try:
        for warp in (1, 0):
            ctx.set_option("lu.warp", warp)
            out.append(nb.slater_dets(S, ctx=ctx).cpu().numpy())
    finally:
        ctx.set_option("lu.warp", 1)
    nan = np.isnan(out[1])
    assert np.array_equal(np.isnan(out[0]), nan) and nan.any()
    assert np.allclose(out[0][~nan], out[1][~nan], rtol=1e-13, atol=0.0)
