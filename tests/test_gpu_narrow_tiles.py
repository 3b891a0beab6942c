"""The last column of the rotation kernel's and the bf16 GEMM's tiles, as wide as the layer needs: widths around the tiles and
their quarters, one row block and many, grids that share factors with the number of columns."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 64, 72, 192, 256, 264, 320, 384, 392, 448, 520, 1152, 1160])
@pytest.mark.parametrize("M,K", [(1, 64), (129, 192), (4736, 128), (19000, 64)])
def test_bf16_gemm_with_a_narrow_last_column(N, M, K):
    from dirotq_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + M)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    y = ops.gemm_bf16(x, w, b)
    ops.check_status()
    ref = x.float() @ w.float().t() + b.float()
    # one rounding to bf16 (half an ulp of 8 bits: 2^-8 of the value at most), and two fp32 sums of K terms in different orders: K roundings
    # of 2^-24 each, of at most the sum of the magnitudes
    terms = x.float().abs() @ w.float().abs().t() + b.float().abs()
    err = (y.float() - ref).abs()
    assert bool((err <= ref.abs() * 2.0 ** -8 + terms * (K * 2.0 ** -23)).all()), float(err.max())


@pytest.mark.parametrize("form", ["single", "pair"])
@pytest.mark.parametrize("D,tail", [(64, 0), (320, 64), (1152, 64), (2240, 320), (392, 8)])
@pytest.mark.parametrize("mode", ["INT4_SYM", "INT8_ASYM", "NVFP4_HW"])
def test_rotation_with_a_narrow_last_column(D, tail, mode, form, monkeypatch):
    from dirotq_b200 import ops
    from gpu_helpers import assert_act_matches_oracle
    from oracle import dirotq_oracle as O
    monkeypatch.setenv("DIROTQ_ROTATE_TILE", form)
    g = torch.Generator().manual_seed(D)
    x = O.synth_activations(1500, D, g).cuda()
    U = O.random_orthogonal(D, g).to(torch.bfloat16).cuda()
    fmt = ops.ActFormat(getattr(ops, mode), D, tail_len=tail, group_size=16 if mode == "NVFP4_HW" else 64)
    buf, x_rot = ops.rotate_quantize(x, U.T.contiguous(), fmt, want_x_rot=True)
    ops.check_status()
    assert rel_l2(x_rot.float().cpu(), (x.float() @ U.float()).cpu()) < 4e-3
    assert_act_matches_oracle(buf, x_rot.cpu())
    assert torch.equal(buf.codes, ops.rotate_quantize(x, U.T.contiguous(), fmt).codes)       # and so without the rotated tensor
