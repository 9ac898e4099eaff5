"""The class API's Evolve and Initialize under options and buffers that the
faster paths do not take."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fft(x):
    return torch.fft.fftn(x, dim=(-3, -2, -1))


def _back(x):
    return torch.fft.ifftn(x, dim=(-3, -2, -1), norm="forward")


def _close(got, want, bound):
    return (torch.linalg.vector_norm(got - want) <= bound * torch.linalg.vector_norm(want)).item()


@pytest.mark.parametrize("L", [24, 32])
@pytest.mark.parametrize("options", [{"fused.kind": 4}, {"fused.kind": 12}, {"fused.kind": 11, "fused.cluster": 8},
                                     {"fused.cluster": 2}, {"propagate.fused": 0}])
def test_initialize_and_evolve_under_forced_variants(L, options):
    """Variants that FP64 orbitals do not have (or that exist for neither
    precision): the calls run on their other path and leave no error text.
    FP64 transforms of 32^3 points round by a few eps log2 V."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    ctx = nb.Context(0)
    dims = (L, L, L)
    d3, V = _ip(_dims(dims)), L ** 3
    g = torch.Generator(device=ctx.device).manual_seed(L)
    phi = torch.randn(dims, dtype=torch.complex128, device=ctx.device, generator=g)
    c = torch.rand(dims, dtype=torch.float64, device=ctx.device, generator=g) / V
    psi = torch.randn((2, *dims), dtype=torch.complex128, device=ctx.device, generator=g)
    for name, value in options.items():
        ctx.set_option(name, value)
    out = torch.empty_like(phi)
    ctx.check(lib().nrcps_interaction_initialize(ctx.handle, _ptr(phi), _ptr(c), d3, _ptr(out)))
    assert _close(out, (1 + _fft(c * _back(phi))) / V, 1e-14)
    here = phi.clone()  # in place
    ctx.check(lib().nrcps_interaction_initialize(ctx.handle, _ptr(here), _ptr(c), d3, _ptr(here)))
    assert _close(here, (1 + _fft(c * _back(phi))) / V, 1e-14)
    b = psi.clone()
    ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(b), 2, d3, _ptr(phi), 0))
    assert _close(b, _back(phi * _fft(psi)), 1e-14)
    b = psi.clone()
    ctx.check(lib().nrcps_potential_evolve(ctx.handle, _ptr(b), 2, d3, _ptr(c), 0))
    assert _close(b, _back(c * _fft(psi)), 1e-14)
    assert lib().nrcps_last_error(ctx.handle) in (b"", None)
    ctx.close()


@pytest.mark.parametrize("dims", [(8, 8, 8), (4, 6, 12), (24, 24, 24)])
def test_initialize_from_a_field_on_eight_bytes(dims):
    """A field that starts at an odd double of its buffer: the same values."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    ctx = nb.default_context()
    d3, V = _ip(_dims(dims)), int(np.prod(dims))
    g = torch.Generator(device=ctx.device).manual_seed(V)
    room = torch.randn(2 * V + 1, dtype=torch.float64, device=ctx.device, generator=g)
    lat = room[1:]
    assert lat.data_ptr() % 16 == 8
    c = torch.rand(dims, dtype=torch.float64, device=ctx.device, generator=g) / V
    out = torch.empty(dims, dtype=torch.complex128, device=ctx.device)
    ctx.check(lib().nrcps_interaction_initialize(ctx.handle, _ptr(lat), _ptr(c), d3, _ptr(out)))
    phi = torch.view_as_complex(lat.clone().view(*dims, 2))
    assert _close(out, (1 + _fft(c * _back(phi))) / V, 1e-14)
