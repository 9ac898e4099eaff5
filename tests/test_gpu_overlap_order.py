"""The CUDA-core overlap's order of summation: given by the shape, not by the
batch, the buffer at hand or a capture; what FP32 orbitals may differ by."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nt,vol", [(19, 19, 13824), (7, 7, 4096), (3, 2, 5000), (33, 20, 1000), (16, 40, 4096),
                                       (5, 9, 700), (7, 7, 13824), (2, 2, 13824), (4, 5, 2048), (10, 10, 1728)])
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_same_bits_in_every_batch(ns, nt, vol, precision):
    """One configuration alone (many CTAs), in batches that give it a cluster
    or one CTA, and in a graph: the same bits."""
    import nrcps_b200 as nb
    ctx = nb.Context(0)
    g = torch.Generator(device=ctx.device).manual_seed(ns * 100 + nt)
    dt = torch.complex128 if precision == "f64" else torch.complex64
    src = torch.randn((ns, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    batch = [1, 2, 40, 100, 700] if vol * nt < 1 << 17 else [1, 2, 30, 90]
    psi = torch.randn((max(batch), nt, vol), dtype=dt, device=ctx.device, generator=g)
    ctx.set_option("overlap.tc", 0)
    want = nb.overlap(src, psi[:1], ctx)
    for n in batch:
        got = nb.overlap(src, psi[:n], ctx)
        assert torch.equal(got[:1], want), n
        assert torch.equal(got[n - 1:], nb.overlap(src, psi[n - 1:n], ctx)), n
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        ctx.use_current_stream()
        out = nb.overlap(src, psi[:1], ctx)
    ctx.use_current_stream()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    ctx.close()


@pytest.mark.parametrize("precision,nt,vol", [("f64", 1600000, 4), ("f32", 700000, 16)])
def test_very_many_orbitals(precision, nt, vol):
    """More tiles and groups of orbitals than a grid has in y: accepted as by a
    block per orbital.  Sums of at most 16 products, in FP32 or better."""
    import nrcps_b200 as nb
    ctx = nb.default_context()
    g = torch.Generator(device=ctx.device).manual_seed(nt)
    dt = torch.complex128 if precision == "f64" else torch.complex64
    src = torch.randn((1, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((1, nt, vol), dtype=dt, device=ctx.device, generator=g)
    got = nb.overlap(src, psi, ctx)
    p = psi.to(torch.complex128)
    want = torch.einsum("sv,ctv->cst", src.conj(), p)
    size = torch.einsum("sv,ctv->cst", src.abs(), p.abs())
    assert ((got - want).abs() <= (1e-14 if precision == "f64" else 3e-6) * size).all()


@pytest.mark.parametrize("n,vol,batch", [(10, 13824, 130), (7, 4096, 700), (10, 4096, 5), (4, 32768, 40)])
def test_fp32_alone_and_in_a_batch(n, vol, batch):
    """FP32 orbitals and up to ten sources: kernel and split follow the batch.
    The tensor-core kernel is held to 1e-6 of the largest |S|, the packed one
    to 56 x 2^-24 of the sum of moduli (39 roundings a real part): a
    configuration alone and in a batch are within the two of each other."""
    import nrcps_b200 as nb
    ctx = nb.default_context()
    g = torch.Generator(device=ctx.device).manual_seed(n * 1000 + batch)
    src = torch.randn((n, vol), dtype=torch.complex128, device=ctx.device, generator=g)
    psi = torch.randn((batch, n, vol), dtype=torch.complex64, device=ctx.device, generator=g)
    got = nb.overlap(src, psi, ctx)
    for c in (0, batch - 1):
        alone = nb.overlap(src, psi[c:c + 1], ctx)[0]
        size = src.abs() @ psi[c].to(torch.complex128).abs().T
        bound = 1e-6 * alone.abs().max() + 56 * 2.0 ** -24 * size
        assert ((got[c] - alone).abs() <= bound).all()
