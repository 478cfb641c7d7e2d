"""The work that users of this library have it do, as cases that can be timed and compared.

Four layer families (CP4 conv2d, three-factor CP conv2d, reshaped-CP conv2d, CP dense), each as inference (one forward
operator call) and as training (forward and all gradients); the CP4 convolution also as the one-call training step.

``listed()`` holds the named cases, ``draw(rng)`` more of the same ranges:

    CP4 conv    N 1-64, channels 8-512, images 7-64 (square or not), 3x3 (forward also 5x5), rank 4-128
    CP3 conv    the same, 3x3, rank 4-64
    rCP conv    N 1-32, two or three channel modes of 2-16, up to 256 channels, images 7-32, 3x3, rank 4-64
    CP dense    batch 1-4096, two to four modes of 4-16, up to 4096 features, rank 4-256

Inputs have the value distributions of the benchmark configurations: images uniform in [-1, 1], dense inputs and
upstream gradients normal, CP4 factors normal with deviation 1/sqrt(F*F*C), rCP factors 0.3, dense factors 0.35; the
layer cases start from the layers' own initialisation.
"""
import math

import torch

import paralleltnnlayers_b200 as P
from paralleltnnlayers_b200 import layers

# the most multiply-adds x 2 of a drawn case: those of the largest listed one (the 4096 x 4096 dense layer, trained)
MAX_FLOPS = 1.04e11


def _conv(name, op, N, C, T, H, W, F, R):
    return {"name": name, "family": name.split("_")[0], "op": op, "N": N, "C": C, "T": T, "H": H, "W": W, "F": F, "R": R}


def listed():
    return [
        # one small image through one layer: latency of a single call
        _conv("cp4_forward_one_image", "forward", 1, 16, 16, 32, 32, 3, 8),
        # inference with a wide 5x5 layer on an odd image size (the second layer of the AlexNet list)
        _conv("cp4_forward_48to256_55x55_5x5", "forward", 8, 48, 256, 55, 55, 5, 16),
        # inference with the benchmark's layer
        _conv("cp4_forward_64_56x56", "forward", 32, 64, 64, 56, 56, 3, 16),
        # the benchmark's training step, one call
        _conv("cp4_step_64_56x56", "step", 32, 64, 64, 56, 56, 3, 16),
        # a later stage of the same network: many channels, small images, a larger rank
        _conv("cp4_step_256_14x14", "step", 64, 256, 256, 14, 14, 3, 32),
        # the last stage, as a module under autograd
        _conv("cp4_layer_512_7x7", "layer", 64, 512, 512, 7, 7, 3, 64),
        # an odd image size, different channel counts and a rank that is no power of two (the third AlexNet layer)
        _conv("cp4_layer_256to384_27x27", "layer", 16, 256, 384, 27, 27, 3, 50),
        # the three-factor layer at the rank its compression rule gives for 128 channels
        _conv("cp3_layer_128_28x28", "layer", 32, 128, 128, 28, 28, 3, 56),
        # the reshaped-CP operator at the shape the reference's operator has, a small batch
        {"name": "rcp_forward_16_32x32", "family": "rcp", "op": "forward", "N": 8, "cdims": "4x4", "tdims": "4x4", "H": 32,
         "W": 32, "F": 3, "R": 11},
        # training the reshaped-CP layer of the benchmark configurations
        {"name": "rcp_layer_256_28x28", "family": "rcp", "op": "layer", "N": 32, "cdims": "4x8x8", "tdims": "4x8x8", "H": 28,
         "W": 28, "F": 3, "R": 16},
        # the dense operator at the reference's shape, a serving batch
        {"name": "dense_forward_4096to64", "family": "dense", "op": "forward", "B": 64, "idims": "16x16x16", "odims": "4x4x4",
         "R": 137},
        # training the dense layer of the benchmark configurations
        {"name": "dense_layer_4096", "family": "dense", "op": "layer", "B": 4096, "idims": "8x8x8x8", "odims": "8x8x8x8",
         "R": 32},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Channel counts are mostly multiples of 16 in practice; some are not."""
    c = _log_int(rng, lo, hi)
    return max(16, c // 16 * 16) if rng.random() < 0.7 else c


def _draw_conv(rng, family):
    op = rng.choice(["forward", "layer"] if family == "cp3" else ["forward", "step", "layer"])
    C = _channels(rng, 8, 512)
    H = rng.randint(7, 64)
    return {"family": family, "op": op, "N": _log_int(rng, 1, 64), "C": C, "T": C if rng.random() < 0.5 else _channels(rng, 8, 512),
            "H": H, "W": H if rng.random() < 0.7 else rng.randint(7, 64),
            "F": 5 if (family == "cp4" and op == "forward" and rng.random() < 0.25) else 3,
            "R": _log_int(rng, 4, 64 if family == "cp3" else 128)}


def _modes(rng, order, lo, hi, most):
    while True:
        d = [rng.choice([k for k in (2, 3, 4, 5, 6, 8, 10, 12, 16) if lo <= k <= hi]) for _ in range(order)]
        if math.prod(d) <= most:
            return "x".join(map(str, d))


def _draw_rcp(rng):
    order = rng.choice([2, 2, 3])
    H = rng.randint(7, 32)
    cd = _modes(rng, order, 2, 16, 256)
    return {"family": "rcp", "op": rng.choice(["forward", "layer"]), "N": _log_int(rng, 1, 32), "cdims": cd,
            "tdims": cd if rng.random() < 0.5 else _modes(rng, order, 2, 16, 256), "H": H,
            "W": H if rng.random() < 0.7 else rng.randint(7, 32), "F": 3, "R": _log_int(rng, 4, 64)}


def _draw_dense(rng):
    order = rng.choice([2, 3, 3, 4])
    idims = _modes(rng, order, 4, 16, 4096)
    return {"family": "dense", "op": rng.choice(["forward", "layer"]), "B": _log_int(rng, 1, 4096), "idims": idims,
            "odims": idims if rng.random() < 0.5 else _modes(rng, order, 4, 16, 4096), "R": _log_int(rng, 4, 256)}


def draw(rng):
    while True:
        family = rng.choice(["cp4", "cp4", "cp4", "cp3", "rcp", "dense"])
        case = _draw_rcp(rng) if family == "rcp" else _draw_dense(rng) if family == "dense" else _draw_conv(rng, family)
        w = work(case)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= 6e8:
            return case


def _dims(text):
    return [int(v) for v in text.split("x")]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0):
        return torch.randn(*shape, generator=gen, device="cuda") * std

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device="cuda") * 2 - 1

    family, op, R = case["family"], case["op"], case["R"]
    torch.manual_seed(seed)   # the layers draw their initial factors from the default generator
    if family == "dense":
        idims, odims = _dims(case["idims"]), _dims(case["odims"])
        I, O = math.prod(idims), math.prod(odims)
        x = normal(case["B"], I)
        if op == "forward":
            return {"call": P.dense_cp, "args": (x, *[normal(i, o, R, std=0.35) for i, o in zip(idims, odims)])}
        layer = layers.CPDense(I, O, rank=R, input_shape=idims, output_shape=odims).cuda()
        return {"layer": layer, "x": x.requires_grad_(), "dy": normal(case["B"], O)}
    N, H, W, F = case["N"], case["H"], case["W"], case["F"]
    if family == "rcp":
        cd, td = _dims(case["cdims"]), _dims(case["tdims"])
        C, T = math.prod(cd), math.prod(td)
        x = uniform(N, C, H, W)
        if op == "forward":
            A = [normal(c, t, R, std=0.3) for c, t in zip(cd, td)]
            return {"call": P.conv2d_rcp_fused_nchw, "args": (x, *A, normal(F, F, R, std=0.3))}
        layer = layers.RCPConv2d(C, T, F, rank=R, input_shape=cd, output_shape=td).cuda()
        return {"layer": layer, "x": x.requires_grad_(), "dy": normal(N, T, H, W)}
    C, T, pad = case["C"], case["T"], (F - 1) // 2
    std = 1.0 / math.sqrt(F * F * C)
    x = uniform(N, C, H, W)
    if op == "layer":
        make = layers.CP4Conv2d if family == "cp4" else layers.CPConv2d
        return {"layer": make(C, T, F, rank=R).cuda(), "x": x.requires_grad_(), "dy": normal(N, T, H, W)}
    if family == "cp3":
        K = (normal(T, R, std=std), normal(C, R, std=std), normal(F, F, R, std=std))
        return {"call": P.cp3_conv2d_forward, "args": (x, *K, pad)}
    K = tuple(normal(d, R, std=std) for d in (T, C, F, F))
    if op == "step":
        return {"call": P.cp4_conv2d_step, "args": (x, normal(N, T, H, W), *K, pad)}
    return {"call": P.cp4_conv2d_forward, "args": (x, *K, pad)}


def run(state):
    if "call" in state:
        return state["call"](*state["args"])
    layer, x = state["layer"], state["x"]
    y = layer(x)
    # the gradients of a training step: input (for the layer below) and every factor
    return (y, *torch.autograd.grad(y, (x, *layer.parameters()), state["dy"]))


def work(case):
    """Inputs read once and results written once; the multiply-adds of each direction in the factored form, or with the
    weight multiplied out first where that is less (large ranks)."""
    family, R = case["family"], case["R"]
    if family == "dense":
        idims, odims, B = _dims(case["idims"]), _dims(case["odims"]), case["B"]
        macs, a, b = 0, 1, math.prod(idims)
        for i, o in zip(idims, odims):      # mode by mode: every remaining input entry meets the mode's outputs
            macs += a * b * o
            a, b = a * o, b // i
        I, O = math.prod(idims), math.prod(odims)
        flops = 2 * min(B * R * macs, (B + R) * I * O)
        n_in, n_out = B * I, B * O
        n_par = R * sum(i * o for i, o in zip(idims, odims))
    else:
        px, F = case["N"] * case["H"] * case["W"], case["F"]
        if family == "rcp":
            cd, td = _dims(case["cdims"]), _dims(case["tdims"])
            C, T = math.prod(cd), math.prod(td)
            macs, a, b = C * F * F, 1, C
            for c, t in zip(cd, td):
                macs += a * b * t
                a, b = a * t, b // c
            n_par = R * (sum(c * t for c, t in zip(cd, td)) + F * F)
            flops = 2 * min(px * R * macs, (px + R) * C * T * F * F)
        else:
            C, T = case["C"], case["T"]
            macs = C + T + (2 * F if family == "cp4" else F * F)
            n_par = R * (C + T + (2 * F if family == "cp4" else F * F))
            flops = 2 * px * R * macs
        n_in, n_out = px * C, px * T
    if case["op"] == "forward":
        return {"bytes": 4 * (n_in + n_out + n_par), "flops": flops}
    # training: x and dy read, y and dx written, the factors read and their gradients written
    return {"bytes": 4 * 2 * (n_in + n_out + n_par), "flops": 3 * flops}


def tolerance(case):
    """fp32 in, fp32 out: relative 1e-5 for outputs that sum some thousands of products.  Factor gradients sum up to 1e5
    pixels or samples times the channels, in an order of the implementation's own choice; those of the rCP and dense
    layers also pass through a weight-sized gradient whose fp32 sums over the batch a tensor core truncates rather than
    rounds (a bias of up to half an ulp per addition, 2**-24 times some hundreds of additions)."""
    if case["op"] == "forward":
        return {"rel": 1e-5}
    return {"rel": 5e-5 if case["family"] in ("rcp", "dense") else 2e-5}
