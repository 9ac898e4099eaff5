"""Which fused kernel a batch runs: the tests that compare the kernels holding a
whole orbital with the cluster kernels rely on their batches running the former."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import nrcps_b200 as nb
    c = nb.Context(0)
    yield c
    c.close()


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("precision,per_sm", [("f64", 3), ("f32", 6)])
def test_one_cta_kernel_from_an_eighth_of_a_wave(ctx, precision, per_sm):
    slots = _sms() * per_sm
    assert ctx.fused_choice(precision, 16, slots // 8)[0] not in (13, 14)
    for n in (slots // 8 + 1, slots // 2, slots, slots + 1, 1 << 20, None):
        assert ctx.fused_choice(precision, 16, n) == (14, 1)


def test_parked_kernel_where_the_last_wave_is_two_thirds_full(ctx):
    s = _sms()
    for n in (1, 2 * s // 3, s + 1, 4 * s // 3):
        assert ctx.fused_choice("f32", 32, n)[0] == 11
    for n in (2 * s // 3 + 1, s, 4 * s // 3 + 1, 2 * s, 19456, None):
        assert ctx.fused_choice("f32", 32, n) == (13, 1)
    assert ctx.fused_choice("f64", 32, 19456)[0] not in (13, 14)


@pytest.mark.parametrize("precision,n", [("f64", 223), ("f64", 448), ("f64", 995), ("f32", 445), ("f32", 889),
                                         ("f32", 1990)])
def test_batches_of_the_one_cta_comparison(ctx, precision, n):
    assert ctx.fused_choice(precision, 16, n) == (14, 1)


@pytest.mark.parametrize("n", [100, 148, 297, 597])
def test_batches_of_the_parked_comparison(ctx, n):
    if _sms() != 148:
        pytest.skip("batches chosen for 148 SMs")
    assert ctx.fused_choice("f32", 32, n) == (13, 1)


def test_a_forced_variant_is_what_runs(ctx):
    ctx.set_option("fused.kind", 0)
    try:
        assert ctx.fused_choice("f32", 16, 10000)[0] == 0
        assert ctx.fused_choice("f32", 32, 10000)[0] in (0, -1)
    finally:
        ctx.set_option("fused.kind", -1)
