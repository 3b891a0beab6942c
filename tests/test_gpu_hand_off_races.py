"""The quantising epilogue's stores crowd the queue that the converters' shared-memory loads wait in: a raw stage handed back before
those loads have returned is overwritten under them.  Codes and scales of a feed-forward pair, again and again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [None, "128", "256"])
@pytest.mark.parametrize("quant", ["int4", "nvfp4"])
def test_handed_codes_are_the_same_every_time(quant, bn, monkeypatch):
    from dirotq_b200 import backend, dit, ops
    from dirotq_b200.synth import synth_activations
    from dirotq_b200.wrapper import ActQuantWrapper
    monkeypatch.setattr(ActQuantWrapper, "forward", backend._fused_forward_b200)
    if bn:
        monkeypatch.setenv("DIROTQ_GF_BN", bn)
    M, D, F = 1100, 1536, 6144
    up = dit.make_wrapped_linear(dit.LayerDef("ff.net.0.proj", D, F, tail=192), quant, 91, "cuda")
    down = dit.make_wrapped_linear(dit.LayerDef("ff.net.2", F, 256, kind="norot", source="ff"), quant, 92, "cuda")
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
