"""Bounded waits: with a limit of a few thousand cycles some role of every kernel that waits on the device gives up (the
first accumulator of these reductions takes several microseconds, a poll that sleeps may take as long).  The kernel reports
it, awaits what it has in flight -- copies, tensor-core work, in both CTAs of a pair -- gives its tensor memory back and
returns, and what runs next is untouched by it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _int_gemm(mode, M, N, D, tail, exact=False, records=False):
    from dirotq_b200 import ops
    from test_gpu_gemm import _setup_int
    m = {"sym": ops.INT4_SYM, "asym": ops.INT4_ASYM, "int8": ops.INT8_ASYM}[mode]
    x, act, dec, qw, sw, pk, w_tail, bias = _setup_int(ops, M, N, ops.ActFormat(m, D, tail_len=tail), 61)
    lay, b = act.layout, bias.cuda()
    wt = ops.pad_tail_weight(w_tail, lay.tail_pitch, N, "cuda")
    if exact:
        return lambda: ops.gemm_w4a4_int(act, pk, wt, b)
    folded = ops.fold_weight_scales_f16(pk, wt, lay.tail_total)
    if records:
        from gpu_helpers import gemm_on_records
        return lambda: gemm_on_records(act, pk, folded, b)
    return lambda: ops.gemm_w4a4_int_f16(act, pk, folded, b)


def _nvfp4_gemm(M, N, D, tail):
    from dirotq_b200 import ops
    g = torch.Generator().manual_seed(62)
    act = ops.quantize_act(torch.randn(M, D, generator=g).to(torch.bfloat16).cuda(),
                           ops.ActFormat(ops.NVFP4_HW, D, tail_len=tail, group_size=16))
    lay = act.layout
    pk = ops.pack_weight_nvfp4_rowscale((torch.randn(N, lay.q_len, generator=g) * 0.02).cuda())
    wt = ops.pad_tail_weight((torch.randn(N, tail, generator=g) * 0.02).to(torch.bfloat16) if tail else None, lay.tail_pitch, N, "cuda")
    return lambda: ops.gemm_w4a4_nvfp4(act, pk, wt, None)


def _bf16_gemm(M, N, K):
    from dirotq_b200 import ops
    g = torch.Generator().manual_seed(63)
    x, w = (torch.randn(r, K, generator=g).to(torch.bfloat16).cuda() for r in (M, N))
    return lambda: ops.gemm_bf16(x, w, None)


def _rotate_quantize(mode, M, D):
    from dirotq_b200 import ops
    g = torch.Generator().manual_seed(64)
    m = {"sym": ops.INT4_SYM, "nvfp4": ops.NVFP4_HW}[mode]
    x, r = (torch.randn(n, D, generator=g).to(torch.bfloat16).cuda() for n in (M, D))
    fmt = ops.ActFormat(m, D, tail_len=64, group_size=16 if mode == "nvfp4" else 64)
    buf = ops.alloc_act(fmt, M, x.device)
    return lambda: (ops.rotate_quantize(x, r, fmt, out=buf), buf.codes)[1]


_KERNELS = {
    "int exact": ({}, lambda: _int_gemm("asym", 300, 264, 4608, 64, exact=True)),
    "int 128": ({"DIROTQ_GF_BN": "128"}, lambda: _int_gemm("sym", 300, 264, 12288, 320)),
    "int 192": ({"DIROTQ_GF_BN": "192"}, lambda: _int_gemm("int8", 300, 264, 12288, 320)),
    "int 256": ({"DIROTQ_GF_BN": "256"}, lambda: _int_gemm("asym", 300, 264, 12288, 320)),
    "int 256, many tiles": ({"DIROTQ_GF_BN": "256"}, lambda: _int_gemm("int8", 5000, 2056, 3072, 384)),
    "int records": ({}, lambda: _int_gemm("sym", 300, 264, 12288, 320, records=True)),
    "int records, many tiles": ({}, lambda: _int_gemm("int8", 5000, 2056, 3072, 384, records=True)),
    "nvfp4 single": ({"DIROTQ_NVFP4_TILE": "single"}, lambda: _nvfp4_gemm(300, 264, 12288, 320)),
    "nvfp4 pair 128": ({"DIROTQ_NVFP4_TILE": "pair128"}, lambda: _nvfp4_gemm(300, 264, 12288, 320)),
    "nvfp4 pair 256": ({"DIROTQ_NVFP4_TILE": "pair256"}, lambda: _nvfp4_gemm(5000, 2056, 12288, 64)),
    "gemm single": ({"DIROTQ_ROTATE_TILE": "single"}, lambda: _bf16_gemm(300, 264, 12288)),
    "gemm pair": ({"DIROTQ_ROTATE_TILE": "pair"}, lambda: _bf16_gemm(300, 264, 12288)),
    "rotate single": ({"DIROTQ_ROTATE_TILE": "single"}, lambda: _rotate_quantize("sym", 300, 4608)),
    "rotate pair": ({"DIROTQ_ROTATE_TILE": "pair"}, lambda: _rotate_quantize("nvfp4", 5000, 4608)),
}


@pytest.mark.parametrize("kernel", list(_KERNELS))
def test_every_waiting_kernel_gives_up_and_leaves_nothing_behind(kernel, monkeypatch):
    from dirotq_b200 import _lib, ops
    env, make = _KERNELS[kernel]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    call = make()
    good = call().clone()
    ops.check_status()
    for limit in (1024, 4096, 8192, 16384):          # gives up on the first tile, or, where a limit allows it, further on
        try:
            ops.set_wait_limit_cycles(limit)
            y = call()
            torch.cuda.synchronize()                 # returns: nothing hangs
        finally:
            ops.set_wait_limit_cycles(0)
        code = int(ops.status_word("cuda")[0].item())
        assert 0 <= code <= 6 and (code > 0 or limit > 1024)
        if code:
            assert code != 5, "the teardown's own waits ran out"
            with pytest.raises(RuntimeError, match="timeout"):
                ops.check_status()
        else:
            assert torch.equal(y, good)
        for _ in range(3):
            assert torch.equal(call(), good)         # shared and tensor memory are whole again, and the status is clean
        ops.check_status()
    assert _lib.lib().dirotq_status_string(5)
