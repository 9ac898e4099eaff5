"""Arrays of complex doubles that start on 8 bytes: every double pointer that
the calls take, not only those on 16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _on_eight(t):
    """A copy of complex128 t whose storage starts at an odd double, as doubles."""
    flat = torch.view_as_real(t.contiguous()).reshape(-1)
    room = torch.empty(flat.numel() + 2, dtype=torch.float64, device=t.device)
    room = room[1:] if room.data_ptr() % 16 == 0 else room
    room[:flat.numel()] = flat
    assert room.data_ptr() % 16 == 8
    return room


@pytest.mark.parametrize("N", [3, 8, 19, 32])
@pytest.mark.parametrize("mode,which", [(0, "S"), (1, "S"), (1, "P")])
def test_minors(N, mode, which):
    """Matrices 1 + 0.3 G against the same on 16 bytes (another kernel: N eps
    times condition numbers of a few hundred)."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ptr
    ctx = nb.default_context()
    g = torch.Generator(device=ctx.device).manual_seed(N)
    S = torch.eye(N, dtype=torch.complex128, device=ctx.device) + 0.3 * torch.randn(
        (5, N, N), dtype=torch.complex128, device=ctx.device, generator=g) / N ** 0.5
    P = torch.randn((5, N, N), dtype=torch.complex128, device=ctx.device, generator=g) if mode else None
    want = nb.slater_dets(S, P, mode=mode, ctx=ctx)
    s, p = (_on_eight(S) if which == "S" else S), (_on_eight(P) if which == "P" else P)
    got = torch.empty_like(want)
    ctx.check(lib().nrcps_slater_dets(ctx.handle, _ptr(s), _ptr(p), N, 5, mode, 0, _ptr(got)))
    assert ((got - want).abs() <= 1e-11 * want.abs()).all()


@pytest.mark.parametrize("N", [1, 5, 19, 33, 64])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_reorthonormalise_scratch(N, dtype):
    """The caller's scratch on 8 bytes: the same bits as on 16."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ptr
    ctx = nb.default_context()
    g = torch.Generator(device=ctx.device).manual_seed(N)
    psi = torch.randn((3, N, 512), dtype=dtype, device=ctx.device, generator=g)
    want, logR = psi.clone(), torch.zeros((3, N), dtype=torch.float64, device=ctx.device)
    nb.reorthonormalise(want, logR, ctx)
    got, log8 = psi.clone(), torch.zeros_like(logR)
    work = _on_eight(torch.zeros((3, N, N), dtype=torch.complex128, device=ctx.device))
    ctx.check(lib().nrcps_reorthonormalise(ctx.handle, _ptr(got), N, 512, 3, 0 if dtype == torch.complex128 else 1,
                                           _ptr(work), _ptr(log8)))
    assert torch.equal(got, want) and torch.equal(log8, logR)


@pytest.mark.parametrize("nconf", [1, 6, 200])
def test_overlap_into_eight_bytes(nconf):
    """S on 8 bytes from one CTA, a cluster and many CTAs per configuration:
    the same bits as on 16."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ptr
    ctx = nb.default_context()
    ns, nt, vol = 19, 18, 13824
    g = torch.Generator(device=ctx.device).manual_seed(nconf)
    src = torch.randn((ns, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((nconf, nt, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    want = torch.view_as_real(nb.overlap(src, psi, ctx)).reshape(-1)
    out = _on_eight(torch.zeros((nconf, ns, nt), dtype=torch.complex128, device=ctx.device))
    ctx.check(lib().nrcps_overlap(ctx.handle, _ptr(src), ns, _ptr(psi), nt, nconf, vol, 0, _ptr(out)))
    assert torch.equal(out[:want.numel()], want)
