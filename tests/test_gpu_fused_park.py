"""The fused step that holds a 32^3 FP32 orbital in one SM
(csrc/fused_park.cu) against the cluster kernel it stands in for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    return nb.default_context()


@pytest.mark.parametrize("nconf,batch", [(100, 1), (37, 4), (33, 9), (199, 3)])
@pytest.mark.parametrize("field,off0", [("z2", 0), ("z2", 37), ("z2_general_a", 5), ("z2_pos", 0), ("z2_pos", 3),
                                        ("z2_pos_no_table", 0), ("real", 1), ("complex", 0), ("table", 0),
                                        ("table", 3), ("fld", 2)])
def test_one_sm_step_is_bit_identical_to_the_cluster_kernel(ctx, nconf, batch, field, off0):
    """Batches of less than one, exactly one, and more than one orbital per SM
    (148), every class of field, windows at odd offsets: the same bits as kind
    11 on clusters of eight, the same operations in the same order."""
    import nrcps_b200 as nb
    L, V = 32, 32 ** 3
    g = torch.Generator(device=ctx.device).manual_seed(nconf + off0)
    psi = torch.randn((nconf * batch, L, L, L), dtype=torch.complex64, device=ctx.device, generator=g)
    kinv = torch.from_numpy(1.0 / nb.kinetic_table((L, L, L))).to(ctx.device)
    pos, mode, a, zpos = None, 1, 0.5, 1
    n_sites = nconf * (V - 1) + V + 64  # configurations V - 1 apart: every alignment
    if field.startswith("z2"):
        f = torch.randint(-2 ** 31, 2 ** 31, (n_sites // 32 + 2,), dtype=torch.int32, device=ctx.device, generator=g)
        a = 0.5 if field == "z2" else 0.3
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
        if field == "fld":
            f /= V
    out = []
    try:
        ctx.set_option("fused.zpos", zpos)
        for kind, cluster in ((-1, 0), (11, 8)):
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
    assert ctx.fused_choice("f32", L) == (13, 1)
    assert torch.equal(*out)
