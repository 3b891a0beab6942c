"""The quantising epilogue's stores crowd the queue that the converters' shared-memory loads wait in: a raw stage handed back before
those loads have returned is overwritten under them.  Codes, scales and zero points, again and again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [None, "128", "256"])
@pytest.mark.parametrize("quant,a_sym", [("int4", True), ("int4", False), ("nvfp4", True)])
def test_handed_codes_are_the_same_every_time(quant, a_sym, bn, monkeypatch):
    from dirotq_b200 import backend, dit, ops
    from dirotq_b200.synth import synth_activations
    from dirotq_b200.wrapper import ActQuantWrapper
    monkeypatch.setattr(ActQuantWrapper, "forward", backend._fused_forward_b200)
    if bn:
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
    M, D, F = 1100, 1536, 6144
    up = dit.make_wrapped_linear(dit.LayerDef("ff.net.0.proj", D, F, tail=192), quant, 91, "cuda", a_sym=a_sym)
    down = dit.make_wrapped_linear(dit.LayerDef("ff.net.2", F, 256, kind="norot", source="ff"), quant, 92, "cuda", a_sym=a_sym)
    ff, root = torch.nn.Module(), torch.nn.Module()
    ff.net = torch.nn.ModuleList([dit.GeluProj(up), torch.nn.Identity(), down])
    root.add_module("ff", ff)
    backend.preconvert_rotations_to_device(root, "cuda")
    backend.fuse_gelu_modules(root)
    x = synth_activations(M, D, torch.Generator().manual_seed(5)).reshape(1, M, D).cuda()
    with torch.no_grad():
        want = ff.net[2](ff.net[0](x)).clone()                    # two steps: no hand-off
        assert backend.fuse_ffn_quantise(root, keep_hidden=False) == 1
        wrong = sum(not torch.equal(ff.net[2](ff.net[0](x)), want) for _ in range(120))
    ops.check_status()
    assert wrong == 0


# A zero point is a load of its own, the last of a chunk where chunks are half padding (70 heads of 28 + 4 channels).  The record
# route, whose converters read scale and zero point as one word, says what is right.
@pytest.mark.parametrize("bn", [None, "128", "192", "256"])
@pytest.mark.parametrize("kind", ["hidden", "perhead"])
@pytest.mark.parametrize("quant", ["int4", "int8"])
def test_zero_points_are_the_same_every_time(quant, kind, bn, monkeypatch):
    from dirotq_b200 import backend, dit, ops
    from dirotq_b200.synth import synth_activations
    from gpu_helpers import forward_on_records
    M, D = 3000, 2240
    ld = dit.LayerDef("attn1.to_out.0", D, D, kind="perhead", tail=4, heads=70, head_dim=32) if kind == "perhead" else \
        dit.LayerDef("attn1.to_q", D, D, tail=320)
    w = dit.make_wrapped_linear(ld, quant, 93, "cuda", a_sym=False)
    root = torch.nn.ModuleDict({"l": w})
    backend.preconvert_rotations_to_device(root, "cuda")
    st, x = w._b200_state, synth_activations(M, D, torch.Generator().manual_seed(6)).cuda()
    want = forward_on_records(st, x)
    if bn:
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
    wrong = sum(not torch.equal(backend.linear_forward(st, x), want) for _ in range(120))
    ops.check_status()
    assert wrong == 0
