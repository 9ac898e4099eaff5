"""Chunk sums of the CUDA-core overlap on several streams and in graphs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(n, device, vol=32768, N=19, seed=0):
    g = torch.Generator(device=device).manual_seed(seed)
    src = torch.randn((N, vol), dtype=torch.complex128, device=device, generator=g)
    psi = torch.randn((n, 1, N, vol), dtype=torch.complex128, device=device, generator=g)
    return src, psi


def test_two_streams_of_one_context():
    """Overlaps queued on two streams in turn, nothing between them: each the
    bits it has alone."""
    import nrcps_b200 as nb
    ctx = nb.Context(0)
    src, psi = _inputs(8, ctx.device)
    want = [nb.overlap(src, p, ctx) for p in psi]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for k in range(40):
        with torch.cuda.stream(streams[k % 2]):
            ctx.use_current_stream()
            got.append(nb.overlap(src, psi[k % 8], ctx))
    torch.cuda.synchronize()
    ctx.use_current_stream()
    assert all(torch.equal(g, want[k % 8]) for k, g in enumerate(got))
    ctx.close()


def test_graph_beside_direct_calls():
    """A captured overlap replayed while direct calls run on another stream;
    sums of 32768 products round by 1e-13 of the sum of moduli at most."""
    import nrcps_b200 as nb
    ctx = nb.Context(0)
    src, psi = _inputs(4, ctx.device, seed=1)
    want = [nb.overlap(src, p, ctx) for p in psi]
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        ctx.use_current_stream()
        out = nb.overlap(src, psi[0], ctx)
    ctx.use_current_stream()
    got = []
    for k in range(20):
        with torch.cuda.stream(s):
            graph.replay()
        got.append(nb.overlap(src, psi[1 + k % 3], ctx))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[1 + k % 3]) for k, g in enumerate(got))
    size = torch.einsum("sv,ctv->cst", src.abs(), psi[0].abs())
    assert ((out - want[0]).abs() <= 1e-13 * size).all()
    ctx.close()


def test_two_ensembles_on_two_streams():
    """Dense-source FP64 ensembles of one context, their graphs running at the
    same time: the determinants each gives alone."""
    import numpy as np
    import nrcps_b200 as nb
    ctx = nb.Context(0)
    rs = np.random.default_rng(2)
    src = rs.standard_normal((19, 24 ** 3)) + 1j * rs.standard_normal((19, 24 ** 3))
    job = nb.EnsembleJob(L=24, T=8, n_conf=1, precision="f64")
    streams = [torch.cuda.Stream() for _ in range(2)]
    es, alone = [], []
    for k in range(2):
        with torch.cuda.stream(streams[k]):
            ctx.use_current_stream()
            es.append(nb.Ensemble(job, sources=src, ctx=ctx))
            alone.append(es[k].run(k).clone())
        torch.cuda.synchronize()
    for _ in range(5):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                ctx.use_current_stream()
                es[k].run(k)
        torch.cuda.synchronize()
        assert all(torch.equal(a, e.dets) for a, e in zip(alone, es))
    ctx.use_current_stream()
    for e in es:
        e.close()
    ctx.close()
