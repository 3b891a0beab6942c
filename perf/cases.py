"""The work a user of this package has it do, as cases of one pass each.

Three kinds of case, all through the public entry points (backend.patch_forward, preconvert_rotations_to_device, the
fuse_* switches, then calls of the patched wrappers or of a model-shaped step):

  layer    one wrapped linear: rotation / FWHT / nothing in front, quantised GEMM, bias
  linears  every wrapped linear of one transformer block in block order, with the producer-side fusions a pipeline
           switches on (GELU in the epilogue, q / k / v as one GEMM): what one block of a denoising step costs here
  step     model-shaped blocks with attention, modulation, norms and residuals around the wrapped linears

Shapes are those of dit.py and denoise.py (hidden sizes 1152, 2240, 3072 with their feed-forwards); rows are
batch x tokens of the image sizes these models are run at.  Weights are random codes and scales of those shapes,
activations Gaussian with a planted low-rank subspace and a few heavy-tailed channels.
"""
import math

import torch

from dirotq_b200 import backend, denoise, dit

# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # a 256-pixel image on the 1152-wide model, one attention projection: the smallest call a pipeline makes
        dict(name="layer-1152-rows256-int4", kind="layer", front="hidden", quant="int4", d_in=1152, d_out=1152, tail=64,
             rows=256),
        # output projection of a text stream (512 tokens) with its per-head rotation, FP4
        dict(name="layer-3072-rows512-perhead-nvfp4", kind="layer", front="perhead", quant="nvfp4", d_in=3072, d_out=3072,
             tail=16, heads=24, rows=512),
        # asymmetric activations, an up-projection at a token count that fits no tile (47 x 85 patches)
        dict(name="layer-1152-4608-rows3995-int4asym", kind="layer", front="hidden", quant="int4a", d_in=1152, d_out=4608,
             tail=64, rows=3995),
        # a down-projection under an online Hadamard transform of its first 4096 channels (--hadamard-layers)
        dict(name="layer-4608-1152-hadamard-int4", kind="layer", front="hadamard", quant="int4", d_in=4608, d_out=1152,
             tail=512, rows=4096),
        # one 1024-pixel image through a 2240-wide block (32x autoencoder: 1024 tokens), W4A4
        dict(name="linears-2240-b1-int4", kind="linears", family="sana", quant="int4", batch=1, tokens=1024),
        # the same block at the batch of the throughput configuration, W4A8
        dict(name="linears-2240-b16-w4a8", kind="linears", family="sana", quant="int8", batch=16, tokens=1024),
        # one 1024-pixel image through the linears of a 1152-wide block: the share of one GPU of eight
        dict(name="linears-1152-b1-int4", kind="linears", family="pixart", quant="int4", batch=1, tokens=4096),
        # the same block at batch 8, the headline configuration, in both formats
        dict(name="linears-1152-b8-int4", kind="linears", family="pixart", quant="int4", batch=8, tokens=4096),
        dict(name="linears-1152-b8-nvfp4", kind="linears", family="pixart", quant="nvfp4", batch=8, tokens=4096),
        # a whole block under classifier-free guidance (two samples) at a wide aspect ratio (48 x 84 patches)
        dict(name="step-1152-b2-int4", kind="step", family="pixart", quant="int4", batch=2, tokens=4032, text=300),
        # one double-stream and two single-stream blocks, one image with 512 text tokens, INT4
        dict(name="step-3072-b1-int4", kind="step", family="flux", quant="int4", batch=1, tokens=4096, text=512),
        # the same blocks at batch 4, FP4
        dict(name="step-3072-b4-nvfp4", kind="step", family="flux", quant="nvfp4", batch=4, tokens=4096, text=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("layer", "layer", "linears", "linears", "step"))
    if kind == "layer":
        front = rng.choice(("hidden", "hidden", "hidden", "perhead", "norot", "hadamard", "w4a16"))
        c = dict(kind=kind, front=front)
        if front == "hidden":
            d_in = rng.choice((1152, 2240, 3072))
            d_out = rng.choice((d_in, d_in, 4 * d_in, 3 * d_in, 8 * rng.randint(40, 600)))
            c.update(quant=rng.choice(("int4", "int4", "int4a", "int8", "nvfp4")), d_in=d_in, d_out=d_out,
                     tail={1152: rng.choice((64, 144)), 2240: 320, 3072: 384}[d_in])
        elif front == "perhead":
            heads, d, tail = rng.choice(((16, 72, 9), (70, 32, 4), (24, 128, 16)))
            c.update(quant=rng.choice(("int4", "int4a") + (("nvfp4",) if d == 128 else ("int8",))), d_in=heads * d,
                     d_out=heads * d, tail=tail, heads=heads)
        elif front == "norot":
            d_in, d_out = rng.choice(((4608, 1152), (12288, 3072)))
            c.update(quant=rng.choice(("int4", "int4a", "nvfp4")), d_in=d_in, d_out=d_out,
                     tail=rng.choice((0, d_in // 8)))
        elif front == "hadamard":
            d_in, d_out, low = rng.choice(((4608, 1152, 4096), (1152, 1152, 1024), (2240, 2240, 2048)))
            c.update(quant=rng.choice(("int4", "int4a", "nvfp4")), d_in=d_in, d_out=d_out, tail=d_in - low)
        else:
            d_in, d_out = rng.choice(((4608, 1152), (1152, 1152), (12288, 3072)))
            c.update(quant=rng.choice(("int4", "nvfp4")), d_in=d_in, d_out=d_out, tail=0)
        c["rows"] = _log_int(rng, 16, 18432 if c["d_in"] >= 3072 else 32768)
        return c
    if kind == "linears":
        family = rng.choice(("pixart", "sana"))
        quant = rng.choice(("int4", "nvfp4") if family == "pixart" else ("int4", "int8", "nvfp4"))
        if family == "pixart":
            return dict(kind=kind, family=family, quant=quant, batch=_log_int(rng, 1, 8), tokens=_log_int(rng, 256, 4096))
        return dict(kind=kind, family=family, quant=quant, batch=_log_int(rng, 1, 16), tokens=_log_int(rng, 256, 1024))
    family = rng.choice(("pixart", "flux"))
    return dict(kind=kind, family=family, quant=rng.choice(("int4", "nvfp4")),
                batch=rng.randint(1, 4) if family == "pixart" else rng.randint(1, 2), tokens=_log_int(rng, 1024, 4096),
                text=300 if family == "pixart" else rng.choice((256, 512)))


# ---------------------------------------------------------------------------------------------------------------------
# inputs and prepared modules
# ---------------------------------------------------------------------------------------------------------------------
def _activations(shape, gen, rank=32, heavy=8):
    """N(0, 1) plus a rank-32 subspace of 20x variance plus 8 Student-t(3) channels (synth.py's distribution, on the GPU)."""
    D = shape[-1]
    M = math.prod(shape[:-1])
    kw = dict(generator=gen, device="cuda")
    v = torch.linalg.qr(torch.randn(D, rank, **kw))[0]
    x = torch.randn(M, D, **kw).addmm_(torch.randn(M, rank, **kw) * math.sqrt(19.0), v.t())
    ch = torch.randperm(D, **kw)[:heavy]
    chi = torch.randn(M, heavy, 3, **kw).square().sum(-1) / 3.0
    x[:, ch] = torch.randn(M, heavy, **kw) / chi.sqrt()
    return x.to(torch.bfloat16).reshape(shape)


def _layer(case, seed):
    quant, front, d_in, tail = case["quant"], case["front"], case["d_in"], case["tail"]
    kind = "norot" if front == "hadamard" else front
    heads = case.get("heads", 0)
    ld = dit.LayerDef("proj", d_in, case["d_out"], kind=kind, tail=tail, heads=heads, head_dim=d_in // heads if heads else 0)
    w = dit.make_wrapped_linear(ld, "int4" if quant == "int4a" else quant, seed, "cuda", a_sym=quant != "int4a")
    if front == "hadamard":
        low = d_in - tail
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        w.use_hadamard, w.hadamard_low_dim = True, low
        w.hadamard_sign_flips = torch.randint(0, 2, (low,), generator=gen, device="cuda").float() * 2 - 1
    return w


def _block(case):
    return dit.pixart_block() if case["family"] == "pixart" else dit.sana_block()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    weights = 1000 * (seed + 1)
    backend.patch_forward()
    if case["kind"] == "step":
        step = denoise.DenoiseStep(case["family"], case["quant"], "cuda", n_blocks=1, seed=weights, prepare=True)
        D, B = step.shape["dim"], case["batch"]
        backend.fuse_gelu_modules(step)
        backend.fuse_ffn_quantise(step, keep_hidden=False)      # inside these blocks only the down-projection reads it
        backend.fuse_sibling_gemms(step)
        temb = torch.randn(B, D if case["family"] == "flux" else 6 * D, generator=gen, device="cuda") * 0.1
        return dict(kind="step", step=step, inputs=(_activations((B, case["tokens"], D), gen),
                                                    _activations((B, case["text"], D), gen), temb.to(torch.bfloat16)))
    if case["kind"] == "layer":
        step, x = _layer(case, weights), _activations((1, case["rows"], case["d_in"]), gen)
    else:
        block = _block(case)
        step = dit.LinearPathStep(block, 1, case["quant"], "cuda", seed=weights)
        x = _activations((case["batch"], case["tokens"], block[0].in_f), gen)
    backend.preconvert_rotations_to_device(step, "cuda")
    for w in step.modules():                                    # the synthetic dense data is not kept beside the packed form
        if isinstance(w, dit.ActQuantWrapper):
            w._b200_explicit = None
            w.rotation = w.rotation_per_head = None
    if case["kind"] == "linears":
        backend.fuse_gelu_modules(step)
        backend.fuse_sibling_gemms(step)
    return dict(kind=case["kind"], step=step, inputs=(x,))


def run(state):
    step, inputs = state["step"], state["inputs"]
    with torch.no_grad():
        if state["kind"] != "linears":
            return step(*inputs)
        # LinearPathStep.forward for one block, every layer's output handed back
        x, outs, ff = inputs[0], [], None
        for i, ld in enumerate(step.block):
            if ld.source == "ff":
                outs.append(step.layers[i](ff))
            elif i in step.heads:
                ff = step.heads[i](x)
                outs.append(ff)
            else:
                outs.append(step.layers[i](x))
        return outs


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _weight_bytes(ld, quant):
    low = ld.in_f - (ld.heads * ld.tail if ld.kind == "perhead" else ld.tail)
    group = 16 if quant == "nvfp4" else 64
    n = ld.out_f * (low * 0.5 + low / group * (1 if quant == "nvfp4" else 2) + (ld.in_f - low) * 2 + 2)
    if ld.kind == "hidden":
        n += 2 * ld.in_f * ld.in_f
    elif ld.kind == "perhead":
        n += 2 * ld.in_f * ld.head_dim
    return n


def _flops(lds, M):
    """Linears plus rotations; q, k and v of one attention are rotated once."""
    total, rotated = 0.0, set()
    for ld in lds:
        total += dit.linear_ops(ld, M)
        parent, _, leaf = ld.name.rpartition(".")
        qkv = leaf in ("to_q", "to_k", "to_v", "add_q_proj", "add_k_proj", "add_v_proj") and ld.kind == "hidden"
        key = (parent, leaf.startswith("add")) if qkv else None
        if key is None or key not in rotated:
            total += dit.rotation_ops(ld, M)
        rotated.add(key)
    return total


def work(case):
    if case["kind"] == "layer":
        M, d_in, d_out, tail = case["rows"], case["d_in"], case["d_out"], case["tail"]
        heads = case.get("heads", 0)
        ld = dit.LayerDef("proj", d_in, d_out, kind="norot" if case["front"] in ("hadamard", "w4a16") else case["front"],
                          tail=tail, heads=heads, head_dim=d_in // heads if heads else 0)
        return {"bytes": 2 * M * (d_in + d_out) + _weight_bytes(ld, case["quant"]), "flops": _flops([ld], M)}
    if case["kind"] == "linears":
        M, block = case["batch"] * case["tokens"], _block(case)
        return {"bytes": 2 * M * (block[0].in_f + sum(ld.out_f for ld in block)) +
                sum(_weight_bytes(ld, case["quant"]) for ld in block), "flops": _flops(block, M)}
    B, T, S, quant = case["batch"], case["tokens"], case["text"], case["quant"]
    if case["family"] == "pixart":
        D = 1152
        block = dit.pixart_block()
        flops = _flops(block, B * T) + 4.0 * B * T * (T + S) * D + 4.0 * B * S * D * D
        return {"bytes": 2 * B * (2 * T + S + 6) * D + sum(_weight_bytes(ld, quant) for ld in block) + 4 * D * D, "flops": flops}
    D = 3072
    double, single = dit.flux_double_block(k_down=0), dit.flux_single_block(k_down=0)
    flops = _flops(double, B * T) + _flops(double, B * S) + 2 * _flops(single, B * (T + S)) + \
        3 * 4.0 * B * (T + S) * (T + S) * D + 2.0 * B * D * 18 * D
    weights = 2 * sum(_weight_bytes(ld, quant) for ld in double) + 2 * sum(_weight_bytes(ld, quant) for ld in single)
    return {"bytes": 2 * B * (2 * T + S + 1) * D + weights + 2 * 18 * D * D, "flops": flops}


def tolerance(case):
    """bf16 outputs of one quantised linear agree to a few 1e-3 between correct implementations (one bf16 rounding of the
    rotated tensor moves a few values across a 4-bit boundary); through a chain of blocks such flips add up."""
    return {"rel": 2e-2} if case["kind"] == "step" else {"rel": 1e-2}
