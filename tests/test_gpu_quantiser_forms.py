"""The packed quantisers where they can go wrong: every E2M1 decision of the hardware conversion, 8-bit groups near and far from
zero, values that are no numbers, per-head groups of one, two and more blocks with tails that take each store path."""
import pytest
import torch

from oracle import dirotq_oracle as O

pytestmark = pytest.mark.gpu


def _ops():
    from dirotq_b200 import ops
    return ops


def _bf16(bits):
    return bits.to(torch.int16).view(torch.bfloat16)


# Every bf16 maximum over twenty octaves (so every micro-scale, clamped ones among them) with every value from it down to a 128th
# of it, both signs; tensor scales inside and outside the range of the hardware conversion
@pytest.mark.parametrize("T", [1.0, 0.5, 2.0 ** -62, 2.0 ** 61])
def test_nvfp4_codes_of_every_value(T):
    ops = _ops()
    from gpu_helpers import assert_act_matches_oracle
    amax = torch.arange(20 * 128) + ((127 - 8) << 7)
    down = torch.arange(900)
    v = (amax[:, None] - down).clamp_min(0)
    v = torch.cat([v, v | 0x8000], 1).reshape(amax.numel(), -1, 15)                # fifteen values beside each group's maximum
    x = torch.cat([amax[:, None, None].expand(-1, v.shape[1], 1), v], 2).reshape(-1, 1024)
    x = _bf16(x) * T
    fmt = ops.ActFormat(ops.NVFP4_HW, 1024, group_size=16, tensor_scale=T)
    assert_act_matches_oracle(ops.quantize_act(x.cuda(), fmt), x)


def test_values_that_are_no_numbers_get_the_same_codes_as_before():
    ops = _ops()
    from gpu_helpers import decode_act
    x = torch.randn(8, 64, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    bad = x.clone()
    bad[1, 5], bad[2, 17], bad[3, 40] = float("nan"), float("inf"), -float("inf")
    buf = ops.ActFormat(ops.NVFP4_HW, 64, group_size=16)
    good, got = decode_act(ops.quantize_act(x.cuda(), buf)), decode_act(ops.quantize_act(bad.cuda(), buf))
    assert torch.equal(good["codes"][[0, 4, 5, 6, 7]], got["codes"][[0, 4, 5, 6, 7]])
    assert got["codes"][1, 0, 5] == 0 and got["codes"][2, 1, 1] == 7 and got["codes"][3, 2, 8] == 0
    assert got["scale"][2, 1] == 448 and got["scale"][3, 2] == 448
    x[1, 5] = x[1, 6]                                       # the maximum and the other codes do not see a NaN
    assert torch.equal(torch.cat([decode_act(ops.quantize_act(x.cuda(), buf))["codes"][1, 0, :5], got["codes"][1, 0, 6:]]),
                       torch.cat([got["codes"][1, 0, :5], got["codes"][1, 0, 6:]]))
    f8 = ops.ActFormat(ops.INT8_ASYM, 64)
    a, b = decode_act(ops.quantize_act(x.cuda(), f8)), decode_act(ops.quantize_act(bad.cuda(), f8))
    keep = torch.arange(64) != 5
    assert b["codes"][1, 0, 5] == 0 and torch.equal(a["codes"][1, 0, keep], b["codes"][1, 0, keep])


@pytest.mark.parametrize("H,d,tail", [(0, 64, 0), (0, 64, 40), (16, 72, 9), (10, 32, 4), (3, 128, 16)])
@pytest.mark.parametrize("rotated", [False, True])
@pytest.mark.parametrize("clip", [1.0, 0.3])
def test_8_bit_groups_near_and_far_from_zero(H, d, tail, rotated, clip):
    ops = _ops()
    from gpu_helpers import assert_act_matches_oracle
    M, D = 131, (H * d if H else 5 * d)
    x = torch.randn(M, D, generator=torch.Generator().manual_seed(75))
    x[::3] += torch.tensor([1.2, -1.5, 700.0, 9.0])[torch.arange(D) // d % 4]       # zero points of some hundred, up to thousands
    x[1::7] = x[1::7].abs() + 0.5
    x = x.to(torch.bfloat16)
    fmt = ops.ActFormat(ops.INT8_ASYM, D, tail_len=tail, num_heads=H, head_dim=d if H else 0, clip_ratio=clip)
    if rotated:
        buf = ops.rotate_quantize(x.cuda(), torch.eye(D).to(torch.bfloat16).cuda(), fmt)         # x_rot is x itself
    else:
        buf = ops.quantize_act(x.cuda(), fmt)
    ops.check_status()
    assert_act_matches_oracle(buf, x)


# one block (28, 29 and 32 of 32), two (63 of 64, whole), three, four; tails by 16-byte, 8-byte, staged and single stores
@pytest.mark.parametrize("H,d,tail", [(10, 32, 4), (9, 32, 3), (6, 48, 16), (16, 72, 9), (7, 64, 1), (5, 72, 8), (3, 96, 17), (3, 128, 15),
                                      (3, 128, 16), (2, 128, 30)])
@pytest.mark.parametrize("mode", ["INT4_SYM", "INT4_ASYM", "INT8_ASYM"])
def test_per_head_blocks_and_tails(H, d, tail, mode):
    ops = _ops()
    from gpu_helpers import assert_act_matches_oracle
    M, D = 301, H * d
    x = O.synth_activations(M, D, torch.Generator().manual_seed(76))
    fmt = ops.ActFormat(getattr(ops, mode), D, tail_len=tail, num_heads=H, head_dim=d)
    buf = ops.rotate_quantize(x.cuda(), torch.eye(D).to(torch.bfloat16).cuda(), fmt)
    ops.check_status()
    assert_act_matches_oracle(buf, x)
