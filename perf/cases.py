"""Workloads of the pair-stack hot path, as a user of the package runs them.

Three public entry points: :func:`turbo_attention`, :func:`turbo_trimul` and
:func:`pair_block.pair_stack_block`; each as inference (no gradients) and as one training pass
(forward, then the gradients of every differentiable input for a given output gradient).

Where the sizes come from: the training crop N = 384 and the blocks at N = 768 and N = 1536 (H = 4, D = 32,
C = 128) are the benchmark's configurations; D in {16, 32, 64}, C in {32, 64, 96, 128}, N = 257, batched inputs
and both storage orders of q / k / v are the shapes the parity tests cover; the other lengths are generic (a target
has the length it has, so most are odd).  ``O`` (outer rows) equals ``N``: the pair tensor is square.
"""
from __future__ import annotations

import math

import torch

from openfold3_triangle_kernel_b200 import turbo_attention, turbo_trimul
from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
from openfold3_triangle_kernel_b200.synthetic import block_params, trimul_weights


def _attention(name, mode, N, B=1, H=4, D=32, layout="seq", bias="bf16"):
    return dict(name=name, op="attention", mode=mode, B=B, N=N, H=H, D=D, layout=layout, bias=bias)


def _trimul(name, mode, N, B=1, C=128, direction="outgoing"):
    return dict(name=name, op="trimul", mode=mode, B=B, N=N, C=C, direction=direction)


def _block(name, mode, N, B=1, C=128, H=4, D=32):
    return dict(name=name, op="block", mode=mode, B=B, N=N, C=C, H=H, D=D)


def listed():
    return [
        # a peptide: the call is latency, not work
        _attention("attention_infer_n20", "infer", 20),
        # a stack of templates: several small pair tensors at once, narrow heads, one bias per batch entry
        _attention("attention_train_b4_n128_d16", "train", 128, B=4, D=16),
        # ragged length with wide heads and an fp32 bias
        _attention("attention_train_n257_d64", "train", 257, D=64, layout="head", bias="fp32"),
        # the training crop
        _attention("attention_train_n384", "train", 384, layout="head"),
        # inference on a large target, q / k / v as views of the projections' [B, O, N, H, D] output
        _attention("attention_infer_n1021", "infer", 1021),
        # a small crop with the narrow channel width, training
        _trimul("trimul_train_n56_c64", "train", 56, C=64),
        # the training crop
        _trimul("trimul_train_n384", "train", 384),
        # inference on a target whose length is not a multiple of anything
        _trimul("trimul_infer_n517", "infer", 517, direction="incoming"),
        # inference on a large target
        _trimul("trimul_infer_n1024", "infer", 1024),
        # a whole block on a small crop: many short operations in a row
        _block("block_train_n72_c64", "train", 72, C=64, D=16),
        # a whole block in training at the larger crop
        _block("block_train_n768", "train", 768),
        # a whole block in inference on the largest target
        _block("block_infer_n1536", "infer", 1536),
    ]


#: largest N drawn per operator and mode
_LARGEST = {("attention", "infer"): 1536, ("attention", "train"): 768, ("trimul", "infer"): 1536,
            ("trimul", "train"): 1024, ("block", "infer"): 1024, ("block", "train"): 768}


def draw(rng):
    op = rng.choice(("attention", "trimul", "block"))
    mode = rng.choice(("infer", "train"))
    lo, hi = math.log(16), math.log(_LARGEST[op, mode])
    N = int(round(math.exp(rng.uniform(lo, hi))))
    B = rng.choice((1, 1, 2, 4)) if N <= 256 else 1
    if op == "attention":
        case = _attention("", mode, N, B=B, H=rng.choice((4, 4, 8)) if N <= 512 else 4, D=rng.choice((16, 32, 32, 64)),
                          layout=rng.choice(("seq", "head")), bias=rng.choice(("bf16", "bf16", "fp32")))
    elif op == "trimul":
        case = _trimul("", mode, N, B=B, C=rng.choice((32, 64, 96, 128, 128, 128)),
                       direction=rng.choice(("outgoing", "incoming")))
    else:
        C, D = rng.choice(((64, 16), (128, 32), (128, 32)))
        case = _block("", mode, N, B=B, C=C, D=D)
    del case["name"]
    return case


def _mask(gen, B, N):
    """Pair mask [B, N, N]: 1, with a random trailing 0..10 % of the residues of each entry (padding) at 0."""
    keep = N - (torch.rand(B, generator=gen, device="cuda") * 0.1 * N).floor()
    seq = (torch.arange(N, device="cuda")[None, :] < keep[:, None]).float()
    return seq[:, :, None] * seq[:, None, :]


def _params(tree, gen, grad):
    """Weights on the GPU; the norm vectors get the small spread that trained ones have."""
    if isinstance(tree, dict):
        return {k: _params(v, gen, grad) for k, v in tree.items()}
    t = tree.cuda()
    if t.ndim == 1:
        t = t + 0.1 * torch.randn(t.shape, generator=gen, device="cuda")
    return t.requires_grad_(grad)


def _flat(tree):
    return [x for v in tree.values() for x in _flat(v)] if isinstance(tree, dict) else [tree]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, N, train = case["B"], case["N"], case["mode"] == "train"

    def normal(*shape, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)

    state = dict(case=case, train=train)
    mask = _mask(gen, B, N)
    if case["op"] == "attention":
        H, D = case["H"], case["D"]
        for n in ("q", "k", "v"):
            if case["layout"] == "head":
                t = normal(B, N, H, N, D)
            else:
                t = normal(B, N, N, H, D).transpose(2, 3)  # a [B, O, N, H, D] projection seen as [B, O, H, N, D]
            state[n] = t.requires_grad_(train)
        dtype = torch.float32 if case["bias"] == "fp32" else torch.bfloat16
        state["bias"] = normal(B, 1, H, N, N, dtype=dtype).requires_grad_(train)
        # the padded keys of every row drop out; in the padded rows too the real keys stay, so no row is empty
        state["mask"] = (1e9 * (mask[:, :1, :] - 1)).expand(B, N, N).reshape(B, N, 1, 1, N).contiguous()
        if train:
            state["d_out"] = normal(B, N, N, H, D)
        state["leaves"] = [state[n] for n in ("q", "k", "v", "bias")]
        return state
    C = case["C"]
    state["z"] = normal(B, N, N, C).requires_grad_(train)
    state["mask"] = mask
    if case["op"] == "trimul":
        state["params"] = _params(trimul_weights(C, seed), gen, train)
    else:
        state["params"] = _params(block_params(C, case["H"], case["D"], seed), gen, train)
    if train:
        state["d_out"] = normal(B, N, N, C) * mask.unsqueeze(-1).bfloat16()  # losses leave the padding out
    state["leaves"] = [state["z"]] + _flat(state["params"])
    return state


def _forward(s):
    case = s["case"]
    if case["op"] == "attention":
        return turbo_attention(s["q"], s["k"], s["v"], pair_bias=s["bias"], res_mask=s["mask"])
    if case["op"] == "trimul":
        return turbo_trimul(s["z"], case["direction"], s["mask"], **s["params"])
    return pair_stack_block(s["z"], s["mask"], s["params"], case["H"])


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return [out.detach(), *torch.autograd.grad(out, state["leaves"], state["d_out"])]


def work(case):
    """Forward: 4 N^2 D per attention plane; 12 C^2 per pair (six C x C projections) and 2 N C (the contraction) for
    the multiplicative update; the block adds its Linears.  Backward: 2.5 times the plane's forward (five products),
    twice the forward elsewhere.  Bytes: inputs and outputs of the call, intermediates not counted."""
    B, N, train = case["B"], case["N"], case["mode"] == "train"
    R = B * N * N
    times = 3 if train else 1
    if case["op"] == "attention":
        H, D = case["H"], case["D"]
        planes, bias = 4 * R * H * N * D, R * H * (4 if case["bias"] == "fp32" else 2)
        return dict(flops=planes * (3.5 if train else 1),
                    bytes=2 * R * H * D * (8 if train else 4) + bias * (2 if train else 1) + 4 * R)
    C = case["C"]
    pair = 2 * R * C * (4 if train else 2) + 4 * R
    tri = times * (12 * R * C * C + 2 * R * N * C)
    tri_weights = 4 * (6 * C * C + 4 * C) * (2 if train else 1)
    if case["op"] == "trimul":
        return dict(flops=tri, bytes=pair + tri_weights)
    H, D = case["H"], case["D"]
    linears = 10 * R * C * H * D + 2 * R * C * H
    weights = 4 * (5 * C * H * D + C * H + 2 * C) * (2 if train else 1)
    return dict(flops=2 * (tri + 4 * R * H * N * D * (3.5 if train else 1) + times * linears),
                bytes=pair + 2 * (tri_weights + weights))


def tolerance(case):
    """bf16 results of bf16 products: 1e-2; gradients through several bf16 intermediates and a block of four updates
    add up to twice that, the gradients of a block (each about 1.4e-2 from an fp64 evaluation) to 2.5e-2."""
    if case["op"] == "block":
        return {"rel": 2.5e-2 if case["mode"] == "train" else 2e-2}
    return {"rel": 2e-2 if case["op"] == "trimul" and case["mode"] == "train" else 1e-2}
