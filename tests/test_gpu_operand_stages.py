"""The 16-bit-conversion GEMM's operand stages of one unit (256-wide tiles) and two (128, 192): odd and even numbers of units of
codes and of the 16-bit tail, one row block and an odd number of them on CTA pairs, more stages than the rings hold, two half-filled
chunks per unit, several tiles per CTA.  Every width gives the same bits (the K order of an element does not depend on it)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,tail", [(64, 0), (128, 0), (192, 0), (128, 64), (192, 72), (320, 64), (448, 136), (576, 192), (1280, 200), (2240, 320)])
@pytest.mark.parametrize("mode,M", [("sym", 1), ("asym", 129), ("int8", 385), ("sym", 700)])
def test_every_tile_width_gives_the_same_bits(mode, M, D, tail, monkeypatch):
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    m = {"sym": ops.INT4_SYM, "asym": ops.INT4_ASYM, "int8": ops.INT8_ASYM}[mode]
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, M, 1160, ops.ActFormat(m, D, tail_len=tail), D + M)
    lay = act.layout
    folded = ops.fold_weight_scales_f16(pk, ops.pad_tail_weight(w_tail, lay.tail_pitch, 1160, "cuda"), lay.tail_total)
    out = []
    for bn in ("128", "192", "256"):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        out.append(ops.gemm_w4a4_int_f16(act, pk, folded, bias.cuda()))
    ops.check_status()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


# stage counts of a tile that are odd and even, on CTAs with one to four tiles: the converter groups' turns run on across tiles
@pytest.mark.parametrize("D", [64, 192, 320])
@pytest.mark.parametrize("bn", ["128", "192", "256"])
def test_turns_of_the_converter_groups_run_on(bn, D, monkeypatch):
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, 9000, 1160, ops.ActFormat(ops.INT4_ASYM, D, tail_len=0), 5)
    folded = ops.fold_weight_scales_f16(pk, None, 0)
    monkeypatch.setenv("DIROTQ_GF_BN", bn)
    y = ops.gemm_w4a4_int_f16(act, pk, folded, bias.cuda())
    monkeypatch.setenv("DIROTQ_GF_BN", "128")
    part = torch.cat([ops.gemm_w4a4_int_f16(a, pk, folded, bias.cuda()) for a in
                      (ops.quantize_act(x[i:i + 3000].cuda(), act.fmt) for i in (0, 3000, 6000))])
    ops.check_status()
    assert torch.equal(y, part)


@pytest.mark.parametrize("bn", ["128", "192"])
@pytest.mark.parametrize("quant,a_sym,H", [("int4", True, 5), ("int4", False, 70), ("int8", False, 7), ("int8", False, 6), ("int4", True, 3)])
def test_half_chunks_in_stages_of_two_units(bn, quant, a_sym, H, monkeypatch):
    from dirotq_b200 import backend
    from dirotq_b200.wrapper import ActQuantWrapper
    import test_gpu_models
    monkeypatch.setenv("DIROTQ_GF_BN", bn)
    monkeypatch.setattr(ActQuantWrapper, "forward", backend._fused_forward_b200)
    test_gpu_models.test_short_per_head_groups_share_operand_stages(quant, a_sym, H, 300, monkeypatch)
