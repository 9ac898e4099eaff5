"""The fused step that holds a 16^3 orbital in one CTA
(csrc/fused_one.cu) against the cluster kernel it stands in for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("precision,nconf,batch", [("f64", 223, 1), ("f64", 64, 7), ("f64", 199, 5), ("f32", 445, 1),
                                                   ("f32", 127, 7), ("f32", 199, 10)])
@pytest.mark.parametrize("field,off0", [("z2", 0), ("z2", 37), ("z2_pos", 3), ("z2_pos_no_table", 0), ("real", 1),
                                        ("complex", 0), ("fld", 2), ("table", 3), ("z2_exact", 5)])
def test_one_cta_step_is_bit_identical_to_the_cluster_kernel(ctx, precision, nconf, batch, field, off0):
    """Just enough orbitals for the kernel (half of three or six per SM), a few
    more than it has slots and several rounds, every class of field, windows at
    odd offsets: the same bits as kind 0 on pairs of CTAs."""
    import nrcps_b200 as nb
    L, V = 16, 16 ** 3
    if field == "table" and precision == "f64":
        pytest.skip("FP32 weight tables are for FP32 orbitals")
    g = torch.Generator(device=ctx.device).manual_seed(nconf + off0)
    psi = torch.randn((nconf * batch, L, L, L), device=ctx.device, generator=g,
                      dtype=torch.complex128 if precision == "f64" else torch.complex64)
    kinv = torch.from_numpy(1.0 / nb.kinetic_table((L, L, L))).to(ctx.device)
    pos, mode, a, zpos = None, 1, 0.3, 1
    n_sites = nconf * (V - 1) + V + 64  # configurations V - 1 apart: every alignment
    if field.startswith("z2"):
        f = torch.randint(-2 ** 31, 2 ** 31, (n_sites // 32 + 2,), dtype=torch.int32, device=ctx.device, generator=g)
        a = 0.5 if field == "z2_exact" else 0.3
        if "pos" in field:
            pos = torch.rand(V, dtype=torch.float64, device=ctx.device, generator=g)
            zpos = 0 if field == "z2_pos_no_table" else 1
    elif field == "table":
        mode, f = 3, torch.randn(n_sites, device=ctx.device, generator=g) / V
    else:
        mode = 0 if field == "fld" else 2
        f = torch.randn((n_sites, 2), dtype=torch.float64, device=ctx.device, generator=g)
        if field == "real":
            f[:, 1] = 0
    out = []
    try:
        ctx.set_option("fused.zpos", zpos)
        for kind, cluster in ((-1, 0), (0, 2)):
            ctx.set_option("fused.kind", kind)
            ctx.set_option("fused.cluster", cluster)
            q = psi.clone()
            nb.propagate(q, batch, kinv, f, a, mode, off0, V - 1, pos, ctx)
            out.append(q)
        ctx.synchronize()
    finally:
        ctx.set_option("fused.zpos", 1)
        ctx.set_option("fused.kind", -1)
        ctx.set_option("fused.cluster", 0)
    assert ctx.fused_choice(precision, L) == (14, 1)
    assert torch.equal(*out)
