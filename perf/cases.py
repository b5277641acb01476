"""Workloads of the 2D-CrossScan selective scan, as the programs that use this package run it.

Two operators, both through their differentiable public entry points:

* ``selective_scan_2d``: one scan orientation over K groups of channels (a caller that folds the
  corner directions into the channels itself, the way the operator is called by a VMamba-style block);
* ``cross_scan_2d``: all four corner directions and the trainable fusion weights in one call.

A training case is the forward and the gradients of every input, an evaluation case the forward under
``torch.no_grad()``.  Sizes are batch x K x D channels x N states per channel on an H x W feature map;
they come from ``cs2d.synthetic.CONFIGS`` (backbone stages, detection and segmentation maps) and, for
the small and the ragged ones, from the shapes the tests use.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "official-cross-scan_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cs2d  # noqa: E402

_DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _case(name, op, mode, dtype, batch, k, d, n, h, w):
    c = {"op": op, "mode": mode, "dtype": dtype, "batch": batch, "k": k, "d": d, "n": n, "h": h, "w": w}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: the CPU-checkable correctness size, where launches and host work are everything
        _case("tiny_train_fp32", "scan", "train", "fp32", 1, 4, 8, 4, 8, 8),
        # one image through a first-stage block at serving time
        _case("one_image_eval_bf16", "cross", "eval", "bf16", 1, 4, 192, 16, 56, 56),
        # VMamba-T stage 1, the configuration the headline metric is quoted on
        _case("stage1_train_fp32", "scan", "train", "fp32", 32, 4, 192, 16, 56, 56),
        # ImageNet-224 backbone stages at batch 128: 16 states on the second stage ...
        _case("stage2_n16_train_bf16", "scan", "train", "bf16", 128, 4, 384, 16, 28, 28),
        # ... a single state on the first, third and fourth stage (large map, 28-byte rows, 14-byte rows)
        _case("stage1_n1_train_bf16", "scan", "train", "bf16", 128, 4, 192, 1, 56, 56),
        _case("stage3_n1_train_bf16", "scan", "train", "bf16", 128, 4, 768, 1, 14, 14),
        _case("stage4_n1_train_bf16", "scan", "train", "bf16", 128, 4, 1536, 1, 7, 7),
        # the same backbone evaluated on a batch
        _case("stage1_n1_eval_bf16", "scan", "eval", "bf16", 64, 4, 192, 1, 56, 56),
        # a four-corner block of the second stage with a single state, as a training step calls it
        _case("stage2_n1_cross_train_bf16", "cross", "train", "bf16", 64, 4, 384, 1, 28, 28),
        # detection-scale map: few images, long rows
        _case("detection_train_bf16", "scan", "train", "bf16", 2, 4, 192, 16, 200, 336),
        # segmentation-scale training step with fusion weights: the largest
        _case("segmentation_cross_train_bf16", "cross", "train", "bf16", 16, 4, 384, 16, 128, 128),
        # nothing divides anything: odd rows, an odd number of states and of channels, half precision
        _case("ragged_train_fp16", "scan", "train", "fp16", 3, 4, 51, 7, 45, 61),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["scan", "scan", "cross"])
    mode = rng.choice(["train", "train", "eval"])
    dtype = rng.choice(["fp32", "bf16", "bf16", "fp16"])
    n = rng.choice([1, 1, 16, 16, _log(rng, 1, 16), _log(rng, 1, 16)])
    h = _log(rng, 7, 224)
    w = min(336, max(7, int(round(h * rng.choice([1.0, 1.0, rng.uniform(0.6, 1.7)])))))
    d = _log(rng, 8, 1536)
    batch = _log(rng, 1, 128)
    k = 4 if op == "cross" else rng.choice([1, 4, 4])
    # no more work than the largest listed case: fewer images, then fewer channels.  A pixel of a channel
    # costs its N states and, whatever N is, its own traffic; rows off the usual widths cost more.
    limit = 1.0e9
    per_image = lambda dd: k * dd * (n + 3) * h * w
    batch = max(1, min(batch, int(limit / per_image(d))))
    if batch * per_image(d) > limit:
        d = max(8, int(d * limit / (batch * per_image(d))))
    return _case(None, op, mode, dtype, batch, k, d, n, h, w)


def prepare(case, seed):
    b, k, d, n, h, w = (case[x] for x in ("batch", "k", "d", "n", "h", "w"))
    dtype, dev = _DTYPES[case["dtype"]], "cuda"
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    dim = k * d

    def randn(*shape):
        return torch.randn(shape, generator=gen, device=dev, dtype=torch.float32).to(dtype)

    cross = case["op"] == "cross"
    # activations, raw delta (softplus runs inside the operator) and the input-dependent B and C
    s = {"u": randn(b, d if cross else dim, h, w), "delta": randn(b, dim, h, w),
         "B": randn(b, k, n, h, w), "C": randn(b, k, n, h, w)}
    # parameters: S4D-real A, log-uniform time steps through the inverse softplus, D near 1, fusion weights near 1/K
    s["A"] = -torch.arange(1, n + 1, dtype=torch.float32, device=dev).repeat(dim, 1).contiguous()
    s["A"] = s["A"] * (0.9 + 0.2 * torch.rand(dim, n, generator=gen, device=dev))
    dt = torch.exp(torch.rand(dim, generator=gen, device=dev) * (math.log(0.1) - math.log(1e-3)) + math.log(1e-3))
    s["delta_bias"] = dt + torch.log(-torch.expm1(-dt))
    s["D"] = 1.0 + 0.1 * torch.randn(dim, generator=gen, device=dev)
    if cross:
        s["w"] = (1.0 + 0.1 * torch.randn(k, d, generator=gen, device=dev)) / k
    names = ["u", "delta", "A", "B", "C"] + (["w"] if cross else []) + ["D", "delta_bias"]
    if case["mode"] == "train":
        s["dout"] = randn(*s["u"].shape)
        for x in names:
            s[x].requires_grad_(True)
    s["args"] = [s[x] for x in names]
    s["op"] = cs2d.cross_scan_2d if cross else cs2d.selective_scan_2d
    s["mode"] = case["mode"]
    return s


def run(s):
    if s["mode"] == "eval":
        with torch.no_grad():
            return s["op"](*s["args"], True)
    out = s["op"](*s["args"], True)
    return [out.detach(), *torch.autograd.grad(out, s["args"], s["dout"])]


def work(case):
    b, k, d, n, h, w = (case[x] for x in ("batch", "k", "d", "n", "h", "w"))
    es = 4 if case["dtype"] == "fp32" else 2
    px, dim = b * h * w, k * d
    image = d if case["op"] == "cross" else dim          # channels of u, y (and their gradients)
    par = dim * (n + 2) + (dim if case["op"] == "cross" else 0)
    # forward: u, delta, B, C read, y written; per scanned element the transition (a product, an
    # exponential), the input term, both recurrences and the contribution to y
    nbytes = px * es * (2 * image + dim + 2 * k * n) + 4 * par
    flops = px * dim * (16 * n + 8)
    if case["mode"] == "train":
        # the gradient of y read, a gradient written for every input; forward and gradients are one pass,
        # its inputs are counted once
        nbytes += px * es * (2 * image + dim + 2 * k * n) + 4 * par
        flops += px * dim * (40 * n + 12)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # fp32: the recurrences and the sums over channels, states and the batch are 32-bit in any order;
    # 16-bit inputs: every result is rounded to the type once
    return {"fp32": {"rel": 2e-5, "max": 2e-3}, "fp16": {"rel": 1e-3, "max": 2e-2},
            "bf16": {"rel": 6e-3, "max": 1e-1}}[case["dtype"]]
