"""The two ways a row's scales reach the 16-bit-conversion GEMM -- the scales themselves, or records of the folding kernel (long
calls of siblings, 256-wide tiles) -- give the same bits, from any scales and from any address; and the rotation kernel's packed
quantiser agrees with the oracle where a group lies far from zero or is clipped; 16-bit channels copied in the quantiser's
launch or behind it."""
import dataclasses
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


# rows and widths around the tiles (128 rows, a stage of four 64-slot chunks, a tail of 64), one to five chunks, ragged ends; rows
# around an octet of scales, 100 and 192 chunks (96 of them are in flight when the epilogue warps read a tile's scales)
@pytest.mark.parametrize("M,D,tail", [(1, 128, 8), (129, 320, 0), (257, 384, 72), (300, 1152, 64), (520, 4608, 320), (39, 6464, 64),
                                      (137, 12288, 0)])
@pytest.mark.parametrize("mode", ["sym", "asym", "int8"])
def test_both_scale_routes_give_the_same_bits(mode, M, D, tail, monkeypatch):
    from dirotq_b200 import ops
    from gpu_helpers import gemm_on_records, kernel_names
    from test_gpu_gemm import _setup_int
    m = {"sym": ops.INT4_SYM, "asym": ops.INT4_ASYM, "int8": ops.INT8_ASYM}[mode]
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, M, 264, ops.ActFormat(m, D, tail_len=tail), 71)
    lay = act.layout
    # rows 2^-24 .. 2^24 apart, and groups of one row 2^-12 apart: scales whose records are subnormal or zero
    s = act.scales[: lay.n_scales * act.ldm * 2].view(torch.bfloat16).view(lay.n_scales, act.ldm)
    rows = torch.arange(act.ldm, device="cuda")
    s *= torch.exp2(((rows * 7) % 49 - 24).float()).to(torch.bfloat16)
    s[::2] *= torch.exp2(-((rows * 5) % 13).float()).to(torch.bfloat16)
    if M > 1:
        s[:, M // 2] = 0
    wt = ops.pad_tail_weight(w_tail, lay.tail_pitch, 264, "cuda")
    folded = ops.fold_weight_scales_f16(pk, wt, lay.tail_total)
    bias = bias.cuda()
    run = lambda a: ops.gemm_w4a4_int_f16(a, pk, folded, bias)
    on_records = lambda: gemm_on_records(act, pk, folded, bias)
    want = on_records()
    assert torch.isfinite(want.float()).all()
    for bn in ("128", "192", "256"):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        assert torch.equal(run(act), want), bn
    ops.check_status()
    # what each route launches beside the GEMM: the folding kernel (with the panel's pre-pass, where there is no resident panel), or
    # none
    pre = lambda fn: [re.search("fold_expand|fold_scales|expand_weight_panel|$", n)[0] for n in kernel_names(fn)
                      if "2dq" in n and "gemm_int_f16" not in n]
    assert pre(on_records) == ["fold_expand"] and pre(lambda: run(act)) == ["expand_weight_panel"]
    folded.panel = ops.expand_weight_panel_f16(pk, folded)
    assert torch.equal(on_records(), want)
    assert pre(on_records) == ["fold_scales"] and pre(lambda: run(act)) == []

    def shifted(t):                                   # the same values at an address that is no multiple of 16
        if t is None:
            return None
        buf = torch.empty(t.numel() + 16, dtype=torch.uint8, device="cuda")[2:2 + t.numel()]
        return buf.copy_(t)
    moved = dataclasses.replace(act, scales=shifted(act.scales), zeros=shifted(act.zeros))
    assert moved.scales.data_ptr() % 16
    for bn in ("128", "256"):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        assert torch.equal(run(moved), want)
    ops.check_status()


# Nine tiles and more per CTA: the table of row powers, four tiles deep and written one tile ahead, goes round more than twice.
# One operand stage per tile (converter groups take alternate tiles), two (a chunk and the tail), five.
@pytest.mark.parametrize("D,tail", [(64, 0), (128, 64), (320, 0)])
@pytest.mark.parametrize("mode", ["sym", "asym", "int8"])
def test_row_powers_of_many_tiles_per_cta(mode, D, tail, monkeypatch):
    from dirotq_b200 import ops
    from gpu_helpers import gemm_on_records
    from test_gpu_gemm import _setup_int
    M, N = 34300, 1032                               # 134 x 5 tiles of 256 columns on 74 pairs of SMs
    m = {"sym": ops.INT4_SYM, "asym": ops.INT4_ASYM, "int8": ops.INT8_ASYM}[mode]
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, M, N, ops.ActFormat(m, D, tail_len=tail), 75)
    lay = act.layout
    s = act.scales[: lay.n_scales * act.ldm * 2].view(torch.bfloat16).view(lay.n_scales, act.ldm)
    rows = torch.arange(act.ldm, device="cuda")
    s *= torch.exp2(((rows // 3 * 7) % 49 - 24).float()).to(torch.bfloat16)     # a wrong tile's or row's power shows
    folded = ops.fold_weight_scales_f16(pk, ops.pad_tail_weight(w_tail, lay.tail_pitch, N, "cuda"), lay.tail_total)
    bias = bias.cuda()
    want = gemm_on_records(act, pk, folded, bias)
    for bn in ("128", "192", "256"):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        assert torch.equal(ops.gemm_w4a4_int_f16(act, pk, folded, bias), want), bn
    ops.check_status()


@pytest.mark.parametrize("quant,H", [("int4", 5), ("int4", 70), ("int8", 7)])
@pytest.mark.parametrize("a_sym", [True, False])
@pytest.mark.parametrize("M", [1, 300])
def test_both_scale_routes_with_half_chunks(quant, a_sym, H, M, monkeypatch):
    """Two half-filled chunks per operand stage, odd and even head counts: one to eighteen raw stages."""
    from dirotq_b200 import backend, dit, ops
    from dirotq_b200.synth import synth_activations
    from gpu_helpers import forward_on_records
    ld = dit.LayerDef("attn1.to_out.0", H * 32, 264, kind="perhead", tail=4, heads=H, head_dim=32)
    w = dit.make_wrapped_linear(ld, quant, 77, "cuda", a_sym=a_sym)
    backend.preconvert_rotations_to_device(torch.nn.ModuleDict({"l": w}), "cuda")
    st, x = w._b200_state, synth_activations(M, H * 32, torch.Generator().manual_seed(H)).cuda()
    x *= torch.exp2((torch.arange(M, device="cuda") % 49 - 24).float()).to(torch.bfloat16)[:, None]
    want = forward_on_records(st, x)
    assert torch.isfinite(want.float()).all()
    for bn in ("128", "192", "256"):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        assert torch.equal(backend.linear_forward(st, x), want), bn
    ops.check_status()


def test_unforced_call_of_five_rounds_of_192_wide_pairs(monkeypatch):
    """15360 x 1152 x 1152: 192-wide tiles on CTA pairs, five rounds, by the dispatch's own choice."""
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, 15360, 1152, ops.ActFormat(ops.INT4_ASYM, 1152, tail_len=64), 76)
    lay = act.layout
    folded = ops.fold_weight_scales_f16(pk, ops.pad_tail_weight(w_tail, lay.tail_pitch, 1152, "cuda"), lay.tail_total)
    y = ops.gemm_w4a4_int_f16(act, pk, folded, bias.cuda())
    monkeypatch.setenv("DIROTQ_GF_BN", "256")
    assert torch.equal(y, ops.gemm_w4a4_int_f16(act, pk, folded, bias.cuda()))
    ops.check_status()


@pytest.mark.parametrize("M,D,tail", [(5, 128, 0), (131, 320, 40), (300, 1152, 64)])
@pytest.mark.parametrize("mode,clip", [("sym", 1.0), ("sym", 0.3), ("asym", 1.0), ("asym", 0.3)])
def test_rotation_epilogue_quantises_groups_far_from_zero_as_the_oracle(mode, clip, M, D, tail):
    from gpu_helpers import assert_act_matches_oracle
    from dirotq_b200 import ops
    g = torch.Generator().manual_seed(72)
    x = torch.randn(M, D, generator=g)
    x[::3] += torch.tensor([3.0, -40.0, 700.0])[torch.arange(D) // 64 % 3]      # offsets from within to far outside the spread
    x[1, :64] = 0
    x[2, 64:128] = -1e-7
    x = x.to(torch.bfloat16)
    fmt = ops.ActFormat(ops.INT4_SYM if mode == "sym" else ops.INT4_ASYM, D, tail_len=tail, clip_ratio=clip)
    buf = ops.rotate_quantize(x.cuda(), torch.eye(D).to(torch.bfloat16).cuda(), fmt)     # x_rot is x itself
    ops.check_status()
    assert_act_matches_oracle(buf, x)


# the quantise-only kernels copy the 16-bit channels in their own launch (groups of 64, NVFP4; whole 16-byte pieces) or a launch behind
@pytest.mark.parametrize("M", [1, 33, 515])
@pytest.mark.parametrize("mode,group,D,tail", [("INT4_SYM", 64, 136, 8), ("INT4_ASYM", 64, 4608, 512), ("INT4_SYM", 64, 136, 12),
                                               ("INT4_SYM", 32, 136, 8), ("INT8_ASYM", 64, 192, 64), ("NVFP4_HW", 16, 136, 8),
                                               ("NVFP4_HW", 16, 1152, 20)])
def test_quantise_only_kernels_copy_the_16_bit_channels(mode, group, D, tail, M):
    from gpu_helpers import assert_act_matches_oracle
    from dirotq_b200 import ops
    x = torch.randn(M, D, generator=torch.Generator().manual_seed(73)).to(torch.bfloat16)
    fmt = ops.ActFormat(getattr(ops, mode), D, tail_len=tail, group_size=group)
    assert_act_matches_oracle(ops.quantize_act(x.cuda(), fmt), x)
