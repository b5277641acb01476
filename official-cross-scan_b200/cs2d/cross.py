"""Four-corner CrossScan with trainable direction-fusion weights.

The reference extension scans one orientation only (top-left origin, rows
down, columns right; an in-source TODO notes that per-group scan orders are
not implemented, ``selective_scan_fwd_kernel_oflex.cuh:140``) and expects its
caller to fold the K = 4 corner directions into the channel dimension as
``n_groups = K`` groups of flipped copies.  That caller is not part of the
reference.  This module is that caller:

    y[b, d, r, c] = sum_k w[k, d] * y_k[b, d, r, c]

where ``y_k`` is the scan of direction k (0: rows down / columns right, 1: rows
down / columns left, 2: rows up / columns right, 3: rows up / columns left)
over ``u[b, d]`` with the direction's own ``delta[b, k*D+d]``, ``A[k*D+d]``,
``B[b, k]``, ``C[b, k]``, ``D[k*D+d]``, ``delta_bias[k*D+d]``; every tensor is in
image coordinates.

All four directions run in ONE kernel launch each way.  The kernels apply the
flips as index maps while they stage tiles and write results, the K directions
read the same ``u`` (and, in the backward, the same ``dy``), and the weighted sum
over the directions happens inside the kernels as well (``cs2d_dirs.merge_w``):
the directions' CTAs add ``w*y_k`` (forward) and ``w*du_k`` (backward) onto one
fp32 image each, the other gradients are scaled by ``w`` and ``dw`` is
accumulated.  Nothing is flipped, replicated or kept per direction in memory;
rows wider than 256 columns run as column tiles like the plain operator.

Two forms of the merge.  By default the four directions of a channel tile are four
CTAs that add with fp32 atomics (the last bit of ``y`` / ``du`` depends on their
order).  With ``deterministic=True`` one CTA owns the channel tile for all K
directions and walks them one after the other, so it alone writes its part of the
merged images - stored by the first direction, read-modify-written by the others
in a fixed order: no atomics, no zero fills, bit-identical ``y`` and ``du`` from run
to run, at a quarter of the CTAs (measured 2.2 times slower on 56x56 and 128x128
maps, much slower when batch x channel tiles cannot fill the GPU).
"""
from __future__ import annotations

import torch

from . import _lib


def _masks(K):
    rows = sum(1 << k for k in range(K) if k % 4 in (2, 3))
    cols = sum(1 << k for k in range(K) if k % 4 in (1, 3))
    return rows, cols


def _check_shapes(u, delta, A, B, w):
    d, K = u.size(1), B.size(1)
    if delta.size(1) != K * d or A.size(0) != K * d or tuple(w.shape) != (K, d):
        raise RuntimeError("expected delta (b, K*D, h, w), A (K*D, n), w (K, D)")


def _dir_forward(u, delta, A, B, C, w, D, delta_bias, delta_softplus, keep_state=True, A_decay=None,
                 deterministic=False):
    """One launch for all directions, merged in the kernel: returns y (b, d, h, w) fp32 and the saved state
    (``None`` when ``keep_state`` is false: the forward then only holds one rolling row of state)."""
    return _lib.native().cross_fwd(u, delta, A, B, C, w, D, delta_bias, bool(delta_softplus), keep_state, A_decay,
                                   bool(deterministic))


def _dir_backward(u, delta, A, B, C, w, D, delta_bias, dy, saved, delta_softplus, A_decay=None, deterministic=False):
    """dy: gradient of the merged image (b, d, h, w), input dtype or fp32, shared by the directions."""
    return tuple(_lib.native().cross_bwd(u, delta, A, B, C, w, D, delta_bias, dy, saved, bool(delta_softplus), A_decay,
                                         bool(deterministic)))


class CrossScan2D(torch.autograd.Function):
    """The operator as a Function: ``CrossScan2D.apply(u, delta, A, B, C, w, D, delta_bias, delta_softplus,
    A_decay, deterministic)``.  The autograd node itself is native (``csrc/cs2d_torch.cpp``)."""

    @staticmethod
    def apply(u, delta, A, B, C, w, D=None, delta_bias=None, delta_softplus=True, A_decay=None, deterministic=False):
        return cross_scan_2d(u, delta, A, B, C, w, D, delta_bias, delta_softplus, A_decay, bool(deterministic))


def cross_scan_2d(u, delta, A, B, C, w, D=None, delta_bias=None, delta_softplus=True, A_decay=None,
                  deterministic=None):
    """Differentiable four-corner CrossScan; see the module docstring for shapes.  ``A_decay`` (a positive
    float32 tensor of one element) scales every state transition, as in the plain operator; its gradient
    follows the reference's formula (the row-scan term is left out there).  ``deterministic`` (default:
    ``torch.are_deterministic_algorithms_enabled()``) selects the form of the merge whose ``y`` and ``du``
    come out with the same bits on every run (one CTA walks all directions); it is slower."""
    return _lib.native().cross(u, delta, A, B, C, w, D, delta_bias, bool(delta_softplus), A_decay, deterministic)
