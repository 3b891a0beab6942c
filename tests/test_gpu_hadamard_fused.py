"""Hadamard layers whose transform and quantiser are one launch: the workspace (codes, scales, zero points, 16-bit channels) and
the output are, byte for byte, those of the two launches it stands for."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _patched(monkeypatch):
    from dirotq_b200 import backend, wrapper
    monkeypatch.setattr(wrapper.ActQuantWrapper, "forward", backend._fused_forward_b200)


def _layer(quant, sym, low, tail, N, flips):
    from dirotq_b200 import dit
    w = dit.make_wrapped_linear(dit.LayerDef("proj", low + tail, N, kind="norot", tail=tail), quant, low + tail, "cuda", a_sym=sym)
    w.use_hadamard, w.hadamard_low_dim, w.hadamard_sign_flips = True, low, flips
    return w


def _inputs(M, D, g):
    x = torch.randn(M, D, generator=g) * torch.exp2(torch.randint(-6, 7, (M, 1), generator=g).float())
    x = x.to(torch.bfloat16)
    x[0] = 0.0
    if M > 5:
        x[1] = -0.0
        x[2, ::2], x[2, 1::2] = 1.0, 1.0                      # one channel takes everything, the others are exact zeros
        x[3, 5] = float("inf")
        x[4, 7] = float("nan")
        x[5] = 3.0e38                                          # overflows in the butterflies
    return x.cuda()


def _both(st, x, low, flips):
    """(workspace, output) of the fused launch and of the separate ones."""
    from dirotq_b200 import _lib, ops
    M, lib, lin = x.shape[0], _lib.lib(), C.byref(st.c_struct())
    size = lib.dirotq_linear_workspace_bytes(lin, M)
    status, stream = ops.status_word(x.device).data_ptr(), torch.cuda.current_stream().cuda_stream
    out = []
    for fused in (True, False):
        ws = torch.full((size + 512,), 0x5A, dtype=torch.uint8, device="cuda")
        y = torch.zeros(M, st.out_features, dtype=torch.bfloat16, device="cuda")
        fp = None if flips is None else flips.data_ptr()
        if fused:
            rc = lib.dirotq_linear_forward_hadamard(lin, x.data_ptr(), low, fp, M, y.data_ptr(), ws.data_ptr(), size, status, stream)
        else:
            h = ops.hadamard_low(x, low, flips)
            rc = lib.dirotq_linear_forward(lin, h.data_ptr(), M, y.data_ptr(), ws.data_ptr(), size, status, stream)
        assert rc == 0
        torch.cuda.synchronize()
        out.append((ws, y))
    ops.check_status()
    return out


@pytest.mark.parametrize("quant,sym", [("int4", True), ("int4", False), ("int8", False), ("nvfp4", True)])
@pytest.mark.parametrize("low,tail", [(1024, 128), (1024, 0), (2048, 192), (2048, 8), (4096, 512), (4096, 1032)])
def test_one_launch_gives_the_bytes_of_two(quant, sym, low, tail):
    """Row counts around a warp's share (two rows of 1024, one of the others), a last warp partly empty, and more rows than the
    chip has warps; with and without sign flips; zeros, infinities, NaN and sums that overflow."""
    g = torch.Generator().manual_seed(low + tail)
    flips = (torch.randint(0, 2, (low,), generator=g).float() * 2 - 1)
    w = _layer(quant, sym, low, tail, 72, flips)
    from dirotq_b200 import backend
    w(torch.zeros(1, 4, low + tail, dtype=torch.bfloat16, device="cuda"))
    st = w._b200_state
    for M in (1, 2, 3, 149, 4801):
        assert backend._fuses_hadamard(st, M) == (low < 4096 or M > 148)
        if not backend._fuses_hadamard(st, M):
            continue
        x = _inputs(M, low + tail, g)
        for f in (flips.to(torch.bfloat16).cuda(), None):
            (ws, y), (ws_ref, y_ref) = _both(st, x, low, f)
            assert torch.equal(ws, ws_ref), (M, f is None)
            assert torch.equal(y.view(torch.int16), y_ref.view(torch.int16)), (M, f is None)


def test_layers_it_does_not_cover_keep_the_separate_launches():
    """Transforms of other lengths, or that do not end where the quantised channels do, or few rows of 4096: refused by the library before any launch,
    and run as before by the layer."""
    from dirotq_b200 import _lib, backend
    g = torch.Generator().manual_seed(1)
    for low, D, tail in [(512, 576, 64), (8192, 8192, 0), (1024, 1152, 64), (1024, 1088, 128), (4096, 4608, 512)]:
        w = _layer("int4", True, D - tail, tail, 64, None)
        w.hadamard_low_dim = low
        x = torch.randn(5, D, generator=g).to(torch.bfloat16).cuda()
        y = w(x)
        st = w._b200_state
        assert not backend._fuses_hadamard(st, 5)
        assert _lib.lib().dirotq_linear_forward_hadamard(C.byref(st.c_struct()), x.data_ptr(), low, None, 5, y.data_ptr(), None, 0,
                                                         None, None) == -2
        from dirotq_b200 import ops
        h = ops.hadamard_low(x, low)
        w.use_hadamard = False
        st.hadamard_low_dim = 0
        assert torch.equal(backend.linear_forward(st, h), y)
