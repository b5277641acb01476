"""Host side of the 2D-CrossScan selective scan: the reference's operator API.

``fwd`` and ``bwd`` take the same positional arguments, apply the same checks
and return the same lists as the two pybind functions of the reference
extension ``selective_nd_scan_cuda_oflex``
(``kernels/selective_nd_scan/src/cusoflex/selective_scan_oflex.cpp:179-284``
and ``:286-440``).  They allocate the outputs with torch and call the C-ABI
library on the current CUDA stream (in native code, ``csrc/cs2d_torch.cpp``); all
arithmetic happens in the CUDA kernels, there is no PyTorch or CPU fallback.
``_problem`` describes a problem to the C ABI for the callers that own their
buffers (``cs2d.parallel``, ``cs2d.host``).

Differences a caller can observe:
* the three saved tensors ``x, x_v, x_sd`` returned by ``fwd`` are opaque in
  the reference too; here ``x_v`` carries the row checkpoints and ``x`` /
  ``x_sd`` are empty.  ``bwd`` does not modify them (the reference overwrites
  them, so there a second ``bwd`` on the same tensors is invalid);
* ``A_decay`` must be positive.
"""
from __future__ import annotations

import torch

from . import _lib

_DT = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}
MAX_DSTATE = 16


def _problem(u, delta, A, B, C, D, delta_bias, A_decay, delta_softplus, out_dtype, who, shared_u_dim=None):
    """The C ABI's description of a problem, after the checks that the operators make (``shared_u_dim``: ``u`` holds the channels
    of one group, read by all groups, ``shared_u_dim`` in all)."""
    raw = _lib.native().problem(u, delta, A, B, C, D, delta_bias, A_decay, bool(delta_softplus), out_dtype, who,
                                shared_u_dim is not None)
    p = _lib.Problem.from_buffer_copy(raw)
    if shared_u_dim is not None and p.dim != shared_u_dim:
        raise RuntimeError("u must have dim / n_groups channels")
    return p


def _raise_on(rc, what):
    if rc != 0:
        raise RuntimeError(f"cs2d {what} failed ({rc}): {_lib.last_error()}")


def fwd(u, delta, A, B, C, D_=None, delta_bias_=None, delta_softplus=False, out_float=False, A_decay_=None):
    """Selective nd scan forward.  Returns ``[out, x, x_v, x_sd]``.

    Under ``torch.use_deterministic_algorithms(True)`` the state is the one that the deterministic backward reads;
    the kernels that write it differ from the others in the last bits of ``out``.
    """
    return _lib.native().fwd(u, delta, A, B, C, D_, delta_bias_, bool(delta_softplus), bool(out_float), A_decay_, None)


def fwd_only(u, delta, A, B, C, D_=None, delta_bias_=None, delta_softplus=False, out_float=False, A_decay_=None):
    """Forward that no backward will follow: returns ``out`` alone.

    Same kernels and results as ``fwd``; the state between row blocks lives in one
    rolling row per channel and state pair instead of the checkpoint buffer (a
    quarter of all h values), so evaluation needs a fraction of the memory.
    """
    return _lib.native().fwd_only(u, delta, A, B, C, D_, delta_bias_, bool(delta_softplus), bool(out_float), A_decay_)


def param_grad_layout(dim, dstate, has_D, has_bias, has_decay):
    """Offsets of the per-channel parameter gradients inside one flat fp32 buffer.

    ``[dA (dim*dstate) | dD (dim) | ddelta_bias (dim) | dA_decay (1)]`` with absent
    parts omitted.  These are the only outputs that sum over the batch, so a
    batch-sharded job all-reduces exactly this buffer (see ``cs2d.parallel``).
    Returns ``(total, {name: (offset, numel)})``.
    """
    parts, off = {}, 0
    for name, n, on in (("dA", dim * dstate, True), ("dD", dim, has_D), ("ddelta_bias", dim, has_bias),
                        ("dA_decay", 1, has_decay)):
        if on:
            parts[name] = (off, n)
            off += n
    return off, parts


def bwd(u, delta, A, B, C, D_, delta_bias_, dout, x_, x_v_, delta_softplus, A_decay_=None, x_sd_=None,
        param_grads=None, deterministic=None):
    """Selective nd scan backward.

    Returns ``[du, ddelta, dA, dB, dC, dD, ddelta_bias, dA_decay]`` with ``None``
    for the gradients of absent optional inputs.

    ``param_grads`` (not part of the reference signature) may be a zero-filled
    flat fp32 CUDA tensor of ``param_grad_layout(...)[0]`` elements; dA, dD,
    ddelta_bias and dA_decay are then views into it, so that one collective can
    reduce them across ranks without packing copies.

    ``deterministic`` (default: ``torch.are_deterministic_algorithms_enabled()``)
    selects the backward without floating-point atomics (``cs2d_bwd_det``):
    bit-identical gradients from run to run, for rows of at most 256 columns.  Where the forward did not know
    (``fwd`` outside of that mode) it may run the forward again for the checkpoints it reads.
    """
    return _lib.native().bwd(u, delta, A, B, C, D_, delta_bias_, dout, x_v_, bool(delta_softplus), A_decay_, param_grads,
                             deterministic)


class SelectiveScan2D(torch.autograd.Function):
    """The operator as a Function: ``SelectiveScan2D.apply(u, delta, A, B, C, D, delta_bias, delta_softplus, out_float,
    A_decay)``.  The autograd node itself is native (``csrc/cs2d_torch.cpp``)."""

    @staticmethod
    def apply(u, delta, A, B, C, D=None, delta_bias=None, delta_softplus=False, out_float=False, A_decay=None):
        return selective_scan_2d(u, delta, A, B, C, D, delta_bias, delta_softplus, out_float, A_decay)


def selective_scan_2d(u, delta, A, B, C, D=None, delta_bias=None, delta_softplus=False, out_float=False,
                      A_decay=None):
    """Differentiable 2D-CrossScan selective scan (one scan orientation; see ``fwd``), through a native autograd node.

    When nothing can ask for a gradient (``torch.no_grad()`` or no input requires one) the
    forward keeps no saved state (``fwd_only``).
    """
    return _lib.native().scan(u, delta, A, B, C, D, delta_bias, bool(delta_softplus), bool(out_float), A_decay)
