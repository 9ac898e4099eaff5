"""Contexts of two host threads running the same kernels at different sizes."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_two_threads_with_kernels_of_different_sizes():
    """Evolve, overlap and re-orthonormalisation in two threads, a large and a
    small shape each: the shared memory that one asks for is not taken from
    the other.  A launch that fails raises; results are those of one thread."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    shapes = [((2, 4, 6), 5, 16), ((24, 12, 16), 30, 64)]  # lattice, sources, QR orbitals (64 KB of matrix)
    errors, out = [], {}

    def inputs(k, device):
        dims, n, m = shapes[k]
        g = torch.Generator(device=device).manual_seed(k)
        V = dims[0] * dims[1] * dims[2]
        rnd = lambda *s: torch.randn(s, dtype=torch.complex128, device=device, generator=g)  # noqa: E731
        return dims, rnd(3, *dims), rnd(*dims) / V, rnd(n, V), rnd(2, n, V), rnd(2, m, 512)

    def work(k, rounds):
        ctx = nb.Context(0)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            ctx.use_current_stream()
            dims, psi, fld, src, orb, q = inputs(k, ctx.device)
            d3, idle = _ip(_dims(dims)), torch.zeros_like(psi)
            for _ in range(20 * rounds):  # (the calls alone: their launches fail or do not)
                ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(idle), 3, d3, _ptr(fld), 0))
            for _ in range(rounds):
                e, r = psi.clone(), q.clone()
                ctx.check(lib().nrcps_interaction_evolve(ctx.handle, _ptr(e), 3, d3, _ptr(fld), 0))
                S = nb.overlap(src, orb, ctx)
                logR = nb.reorthonormalise(r, None, ctx)
            stream.synchronize()
        ctx.close()
        return e, S, r, logR

    def run(k):
        try:
            out[k] = work(k, 200)
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    want = [work(k, 1) for k in range(2)]
    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert all(torch.equal(a, b) for a, b in zip(out[k], want[k]))


def test_first_calls_beside_another_threads_capture():
    """A first Evolve (a table of ones) and a first overlap of one configuration
    (a buffer of sums) in one thread while another captures a graph: neither
    call fails, nor does the capture."""
    import nrcps_b200 as nb
    from nrcps_b200.api import lib, _ip, _dims, _ptr
    ctx = nb.Context(0)
    L = 16
    d3 = _ip(_dims((L, L, L)))
    g = torch.Generator(device=ctx.device).manual_seed(5)
    psi = torch.randn((2, L, L, L), dtype=torch.complex128, device=ctx.device, generator=g)
    pot = torch.rand((L, L, L), dtype=torch.float64, device=ctx.device, generator=g) / L ** 3
    src = torch.randn((19, 13824), dtype=torch.complex128, device=ctx.device, generator=g)
    orb = torch.randn((1, 19, 13824), dtype=torch.complex128, device=ctx.device, generator=g)
    S = torch.empty((1, 19, 19), dtype=torch.complex128, device=ctx.device)
    x = torch.zeros(64, device=ctx.device)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ctx.use_current_stream()
    other = nb.Context(0)
    want = psi.clone()
    other.check(lib().nrcps_potential_evolve(other.handle, _ptr(want), 2, d3, _ptr(pot), 0))
    want_S = nb.overlap(src, orb, other)
    torch.cuda.synchronize()
    errors = []

    def work():
        try:
            ctx.check(lib().nrcps_potential_evolve(ctx.handle, _ptr(psi), 2, d3, _ptr(pot), 0))
            ctx.check(lib().nrcps_overlap(ctx.handle, _ptr(src), 19, _ptr(orb), 19, 1, 13824, 0, _ptr(S)))
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # (other threads' unsafe calls would end it)
        x.add_(1.0)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x.mul_(2.0)
    assert not errors, errors
    graph.replay()
    torch.cuda.synchronize()
    assert x.eq(2.0).all() and torch.equal(psi, want) and torch.equal(S, want_S)
    ctx.close()
    other.close()
