"""Timed workloads of triangle self-attention: the calls a model makes, from the smallest to the
largest, and a generator of further cases of the same ranges.

A case names one problem:

    n, h, d, batch   pair extent, heads, head dim, leading batch
    dtype            "bf16", "fp16" or "fp32"
    mask             "none", "random" (5 % of the keys dropped, never a whole row) or "padding"
                     (the last ``pad`` per cent of the residues are padding, as keys and as rows)
    layout           "dense": q, k, v, bias and dO lie as (batch, heads, n, n, ...);
                     "projection": they are views of what a linear layer wrote, (batch, n, n, heads, ...)
    node             "starting" or "ending"
    backward         forward and all gradients (a training step), or the forward alone (inference)
"""

import math

import torch

from trifast_b200 import triangle_attention
from trifast_b200.torch import triangle_attention_ending_node

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
TOLERANCE = {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}

# Most work of a drawn case, as 14 b h n^3 d: that of the largest listed one (n = 2048), and that
# of the listed head-dim-128 training step where full precision or head dim 128 is asked for.
MOST = 14 * 4 * 2048**3 * 32
MOST_WIDE = 14 * 4 * 512**3 * 128


def _case(name, n, h=4, d=32, dtype="bf16", batch=1, mask="none", pad=0, layout="dense",
          node="starting", backward=True):
    case = dict(n=n, h=h, d=d, dtype=dtype, batch=batch, mask=mask, pad=pad, layout=layout,
                node=node, backward=backward)
    return dict(case, name=name) if name else case


def listed():
    return [
        # Unit-test sized training step in full precision: bound by launches and host work.
        _case("train_n32_fp32", 32, dtype="fp32", mask="random"),
        # A small chain at inference, one of many layers' calls: latency.
        _case("infer_n64", 64, layout="projection", backward=False),
        # A small crop, two samples of odd extent, narrow heads.
        _case("train_b2_n97_d16_fp16", 97, h=8, d=16, dtype="fp16", batch=2, mask="random"),
        # The usual training crop.
        _case("train_n256", 256),
        # Fine-tuning crop, ending node, straight from the projections.
        _case("train_n384_ending", 384, layout="projection", node="ending", mask="padding", pad=5),
        # Larger crop, the batch padded to a common extent.
        _case("train_n512_pad", 512, mask="padding", pad=15),
        # The headline shape.
        _case("train_n1024", 1024),
        # Large complexes in training: the largest case.
        _case("train_n2048_pad", 2048, mask="padding", pad=10),
        # Inference on a chain of any length, straight from the projections.
        _case("infer_n733", 733, layout="projection", mask="padding", pad=3, backward=False),
        # Inference of a model with more and wider heads.
        _case("infer_n1024_h8_d64_fp16", 1024, h=8, d=64, dtype="fp16", mask="random", backward=False),
        # Training without mixed precision.
        _case("train_n256_fp32", 256, dtype="fp32"),
        # The widest head.
        _case("train_n512_d128", 512, d=128),
    ]


def draw(rng):
    dtype = rng.choice(["bf16"] * 6 + ["fp16"] * 2 + ["fp32"] * 2)
    d = rng.choice([16, 32, 32, 32, 32, 32, 64, 64, 128])
    h = rng.choice([1, 2, 4, 4, 4, 8])
    batch = rng.choice([1, 1, 1, 2])
    backward = rng.random() < 0.6
    most = MOST_WIDE if dtype == "fp32" or d == 128 else MOST
    largest = min(2048, int((most / (14 * batch * h * d)) ** (1 / 3)))
    n = round(math.exp(rng.uniform(math.log(16), math.log(largest))))
    if rng.random() < 0.3:      # crops and padded batches are mostly whole multiples
        n = max(16, n // 16 * 16)
    mask = rng.choice(["none", "random", "padding"])
    return _case(None, n, h, d, dtype, batch, mask, rng.randint(1, 30) if mask == "padding" else 0,
                 rng.choice(["dense", "projection"]),
                 rng.choice(["starting", "starting", "ending"]), backward)


def _valid(case):
    return max(1, case["n"] * (100 - case["pad"]) // 100)


def prepare(case, seed):
    """Unit-variance q, k, v, bias and dO, as normalised activations through a linear layer give."""
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    b, h, n, d = case["batch"], case["h"], case["n"], case["d"]
    projection, grad = case["layout"] == "projection", case["backward"]

    def pair(*last):
        shape = (b, n, n, h) + last if projection else (b, h, n, n) + last
        t = torch.randn(shape, generator=g, device=dev, dtype=DTYPES[case["dtype"]])
        if projection:
            t = t.permute((0, 3, 1, 2) + ((4,) if last else ()))
        return t

    state = {"q": pair(d), "k": pair(d), "v": pair(d), "bias": pair()}
    if grad:
        state["leaves"] = [t.requires_grad_(True) for t in state.values()]
        state["do"] = pair(d)
    mask = torch.zeros((b, n, n), dtype=torch.bool, device=dev)
    if case["mask"] == "random":
        mask = torch.rand((b, n, n), generator=g, device=dev) < 0.05
        mask.diagonal(dim1=1, dim2=2).fill_(False)
    elif case["mask"] == "padding":
        mask[:, _valid(case):] = True
        mask[:, :, _valid(case):] = True
    state["mask"] = mask
    state["op"] = triangle_attention_ending_node if case["node"] == "ending" else triangle_attention
    return state


def run(state):
    s = state
    if "do" not in s:
        with torch.no_grad():
            return s["op"](s["q"], s["k"], s["v"], s["bias"], s["mask"])
    o = s["op"](s["q"], s["k"], s["v"], s["bias"], s["mask"])
    return (o.detach(),) + torch.autograd.grad(o, s["leaves"], s["do"])


def work(case):
    """Every input read once, every output written once; the products over the open keys of the
    rows that have one (a padded row has the mean of its values, which needs no product)."""
    b, h, n, d = case["batch"], case["h"], case["n"], case["d"]
    size = DTYPES[case["dtype"]].itemsize
    rows = keys = _valid(case)
    vectors, maps = (8, 2) if case["backward"] else (4, 1)
    return {"bytes": b * (h * n * n * (vectors * d + maps) * size + n * n),
            "flops": (14 if case["backward"] else 4) * b * h * rows * n * keys * d}


def tolerance(case):
    """Weights and score gradients are rounded to the data type between the two products (16 bits),
    or stay in 32 bits throughout."""
    return {"rel": TOLERANCE[case["dtype"]]}
