"""The two ways a row's scales reach the 16-bit-conversion GEMM -- records of the folding kernel (CTA pairs), or the scales
themselves (single CTAs) -- give the same bits, from any scales and from any address; and the rotation kernel's packed
quantiser agrees with the oracle where a group lies far from zero or is clipped; 16-bit channels copied in the quantiser's
launch or behind it."""
import dataclasses

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
    run = lambda a: ops.gemm_w4a4_int_f16(a, pk, folded, bias.cuda())
    out = {}
    for bn, pair in (("256", "1"), ("128", "0"), ("192", "0"), ("256", "0")):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        monkeypatch.setenv("DIROTQ_GF_PAIR", pair)
        out[bn, pair] = run(act)
    ops.check_status()
    assert torch.isfinite(out["256", "1"].float()).all()
    for k, y in out.items():
        assert torch.equal(y, out["256", "1"]), k

    def shifted(t):                                   # the same values at an address that is no multiple of 16
        if t is None:
            return None
        buf = torch.empty(t.numel() + 16, dtype=torch.uint8, device="cuda")[2:2 + t.numel()]
        return buf.copy_(t)
    moved = dataclasses.replace(act, scales=shifted(act.scales), zeros=shifted(act.zeros))
    assert moved.scales.data_ptr() % 16
    for bn, pair in (("128", "0"), ("256", "1")):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        monkeypatch.setenv("DIROTQ_GF_PAIR", pair)
        assert torch.equal(run(moved), out["256", "1"])
    ops.check_status()


# Nine tiles and more per CTA: the table of row powers, four tiles deep and written one tile ahead, goes round more than twice.
# One operand stage per tile (converter groups take alternate tiles), two (a chunk and the tail), five.
@pytest.mark.parametrize("D,tail", [(64, 0), (128, 64), (320, 0)])
@pytest.mark.parametrize("mode", ["sym", "asym", "int8"])
def test_row_powers_of_many_tiles_per_cta(mode, D, tail, monkeypatch):
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    M, N = 34300, 1032                               # 268 x 5 tiles of 256 columns on 148 SMs
    m = {"sym": ops.INT4_SYM, "asym": ops.INT4_ASYM, "int8": ops.INT8_ASYM}[mode]
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, M, N, ops.ActFormat(m, D, tail_len=tail), 75)
    lay = act.layout
    s = act.scales[: lay.n_scales * act.ldm * 2].view(torch.bfloat16).view(lay.n_scales, act.ldm)
    rows = torch.arange(act.ldm, device="cuda")
    s *= torch.exp2(((rows // 3 * 7) % 49 - 24).float()).to(torch.bfloat16)     # a wrong tile's or row's power shows
    folded = ops.fold_weight_scales_f16(pk, ops.pad_tail_weight(w_tail, lay.tail_pitch, N, "cuda"), lay.tail_total)
    bias = bias.cuda()
    out = {}
    for bn, pair in (("256", "1"), ("128", "0"), ("192", "0"), ("256", "0")):
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
        monkeypatch.setenv("DIROTQ_GF_PAIR", pair)
        out[bn, pair] = ops.gemm_w4a4_int_f16(act, pk, folded, bias)
    ops.check_status()
    for k, y in out.items():
        assert torch.equal(y, out["256", "1"]), k


def test_unforced_call_of_five_single_cta_rounds(monkeypatch):
    """15360 x 1152 x 1152: 192-wide tiles on single CTAs, five rounds, by the dispatch's own choice."""
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, 15360, 1152, ops.ActFormat(ops.INT4_ASYM, 1152, tail_len=64), 76)
    lay = act.layout
    folded = ops.fold_weight_scales_f16(pk, ops.pad_tail_weight(w_tail, lay.tail_pitch, 1152, "cuda"), lay.tail_total)
    y = ops.gemm_w4a4_int_f16(act, pk, folded, bias.cuda())
    monkeypatch.setenv("DIROTQ_GF_BN", "256")
    monkeypatch.setenv("DIROTQ_GF_PAIR", "1")
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
