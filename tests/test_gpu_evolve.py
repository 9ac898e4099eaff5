"""Potential / Interaction::Evolve and Interaction::Initialize by one launch
(the fused step with k = 1, or an orbital per CTA) and by pencil passes,
against torch's transforms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# every extent on every axis, cubes with and without a fused step, lattices
# that fit a CTA's shared memory and that do not
DIMS = [(2, 4, 6), (6, 2, 48), (48, 8, 2), (4, 48, 12), (12, 6, 24), (24, 16, 8), (16, 32, 4), (32, 12, 16),
        (8, 24, 32), (8, 8, 8), (12, 12, 12), (16, 16, 16), (24, 24, 24), (32, 32, 32), (32, 32, 48), (48, 48, 48)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_evolve_against_torch(dims, precision):
    """One step and one Initialize with a complex field: FP64 transforms of at
    most 48^3 points round by a few eps log2 V (1e-14 of the norm with room),
    FP32 ones by 1e-6 of it."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    ctx = nb.default_context()
    V, batch = int(np.prod(dims)), 3
    g = torch.Generator(device=ctx.device).manual_seed(V)
    rnd = lambda *s: torch.randn(s, dtype=torch.complex128, device=ctx.device, generator=g)  # noqa: E731
    fft = lambda x: torch.fft.fftn(x, dim=(-3, -2, -1))  # noqa: E731
    back = lambda x: torch.fft.ifftn(x, dim=(-3, -2, -1), norm="forward")  # noqa: E731
    tol = 1e-14 if precision == "f64" else 1e-6
    b = nb.Fourier(batch, dims, precision, ctx)
    psi = rnd(batch, *dims).to(b.b.dtype)
    d3, prec = _ip(_dims(dims)), 0 if precision == "f64" else 1

    def check(got, want, bound):
        assert (torch.linalg.vector_norm(got - want) <= bound * torch.linalg.vector_norm(want)).item()

    fld = rnd(*dims) / V
    b.b.copy_(psi)
    ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(b.b), batch, d3, _ptr(fld), prec))
    check(b.b.to(torch.complex128), back(fld * fft(psi.to(torch.complex128))), tol)
    pot = torch.rand(dims, dtype=torch.float64, device=ctx.device, generator=g) / V
    b.b.copy_(psi)
    ctx.check(lib().nrcps_potential_evolve(ctx.handle, _ptr(b.b), batch, d3, _ptr(pot), prec))
    check(b.b.to(torch.complex128), back(pot * fft(psi.to(torch.complex128))), tol)
    if precision == "f64":
        phi, out = rnd(*dims), torch.empty(dims, dtype=torch.complex128, device=ctx.device)
        ctx.check(lib().nrcps_interaction_initialize(ctx.handle, _ptr(phi), _ptr(pot), d3, _ptr(out)))
        check(out, (1 + fft(pot * back(phi))) / V, 1e-14)


def test_evolve_many_orbitals_and_a_capture():
    """More orbitals than the one-CTA kernel takes (pencil passes), and a step
    captured into a graph on a context that has made no table before."""
    import nrcps_b200 as nb
    ctx = nb.Context(0)
    dims = (8, 4, 6)
    fld = torch.randn((*dims, 2), dtype=torch.float64, device=ctx.device)
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    d3 = _ip(_dims(dims))
    big = torch.randn((1000, *dims), dtype=torch.complex128, device=ctx.device)
    one = big[:5].clone()
    for t, n in ((big, 1000), (one, 5)):
        ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(t), n, d3, _ptr(fld), 0))
    assert torch.allclose(big[:5], one, rtol=1e-12, atol=1e-12)
    s = torch.cuda.Stream()
    cube = _ip(_dims((16, 16, 16)))
    f16 = torch.randn((4096, 2), dtype=torch.float64, device=ctx.device)
    psi = torch.randn((2, 16, 16, 16), dtype=torch.complex128, device=ctx.device)
    start = psi.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.use_current_stream()
        ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(psi), 2, cube, _ptr(f16), 0))
    ctx.use_current_stream()
    psi.copy_(start)
    graph.replay()
    torch.cuda.synchronize()
    ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(start), 2, cube, _ptr(f16), 0))
    assert (torch.linalg.vector_norm(psi - start) <= 1e-14 * torch.linalg.vector_norm(start)).item()
    ctx.close()
