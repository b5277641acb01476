"""Sizes of the buffers between the calls: those of the kernels that run, without places for states and channels that do not
exist.  The built-in scratch array of ``cs2d_bwd_noalloc`` serves every problem whose
adjoint rows fit it in the tile kernels' layout, whichever kernels run: those that keep a row per warp take as many CTAs as
the array has rows for."""
import ctypes

import pytest
import torch

from conftest import TOL, check_close
import cs2d
from cs2d import _lib, ops
from cs2d.synthetic import make_inputs


def _problem(batch, groups, d, n, h, w, dtype=_lib.BF16):
    p = _lib.Problem()
    p.batch, p.dim, p.nrows, p.ncols, p.dstate, p.n_groups, p.delta_dim = batch, groups * d, h, w, n, groups, groups * d
    p.io_dtype, p.out_dtype, p.delta_softplus = dtype, dtype, 1
    for k in ("u", "delta", "A", "B", "C"):
        setattr(p, k, 16)  # never dereferenced: sizing only
    return p


SIZES = ("cs2d_saved_bytes", "cs2d_bwd_scratch_bytes", "cs2d_fwd_only_scratch_bytes")


def _sizes(p, dirs=None):
    """(for this set of directions, for every set) of each buffer"""
    o = ctypes.byref(dirs) if dirs is not None else None
    return [(getattr(_lib.lib(), n + "_dir")(ctypes.byref(p), o), getattr(_lib.lib(), n)(ctypes.byref(p))) for n in SIZES]


CORNERS = _lib.Dirs(0b1100, 0b1010, 3, 0, 16, None)
SERIAL = _lib.Dirs(0b1100, 0b1010, 3, _lib.DIRS_SERIAL, 16, None)


@pytest.mark.parametrize("n,w", [(1, 7), (1, 56), (1, 200), (2, 28), (3, 56), (16, 56), (16, 336)])
@pytest.mark.parametrize("d", [7, 8, 192])
def test_one_set_of_directions_needs_no_more_than_every_set(d, n, w):
    for dirs in (None, CORNERS, SERIAL):
        for exact, every in _sizes(_problem(2, 4, d, n, 20, w), dirs):
            assert 0 < exact <= every


def test_saved_state_of_the_kernels_that_run():
    pixels = 8 * 64 * 8 * 100 * 100
    exact, every = _sizes(_problem(8, 64, 8, 1, 100, 100))[0]
    assert exact == 8 * 64 * 4 * 25 * 128 * 8          # streaming: channel pairs x row blocks x padded columns
    assert every < 4.5 * pixels                        # pair-walk (corner directions): 3.5 bytes per channel and pixel, of five pairs for four
    exact, _ = _sizes(_problem(32, 4, 192, 2, 28, 28))[0]
    bc = 32 * 4 * 7 * 4 * 32 * 8 * 8                   # B and C of 8 state slots, in blocks of 32 pixels
    assert exact == bc + (6 * 4 + 7 * 3) * 4 * (32 * 4 * 96 * 3) * 16   # rows and columns of two states, and a place for the other six


def test_scratch_of_the_kernels_that_run():
    assert _sizes(_problem(128, 4, 192, 1, 56, 56))[1][0] == 16        # streaming: the adjoint row stays on the chip
    assert _sizes(_problem(32, 4, 192, 16, 56, 56, _lib.F32))[1][0] == 148 * 3 * 4 * 7 * 2048   # block-walk: 2 KB per warp and 8 columns


TILE = _lib.Dirs(0, 0, 0, _lib.DIRS_TILE_STATE, None, None)


@pytest.mark.parametrize("d,n,h,w", [(192, 16, 56, 56), (40, 16, 14, 14), (192, 4, 28, 28), (8, 2, 3, 5), (192, 1, 7, 7), (192, 1, 56, 56), (4, 16, 9, 9)])
def test_state_of_the_deterministic_backward(d, n, h, w):
    """It has another size wherever it is another state, and the scratch then has no room for a second forward's."""
    L, p = _lib.lib(), _problem(2, 4, d, n, h, w)
    state, tile = _sizes(p)[0][0], _sizes(p, TILE)[0][0]
    det = [L.cs2d_bwd_det_scratch_bytes_dir(ctypes.byref(p), o) for o in (None, ctypes.byref(TILE))]
    remade = d >= 8 and (n > 1 or w == 7)
    assert 0 < det[1] <= det[0] <= L.cs2d_bwd_det_scratch_bytes(ctypes.byref(p))
    assert (state != tile) == remade and (det[0] > det[1]) == remade


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 2, 16, 16, 9, 14), (1, 2, 14, 16, 13, 56), (2, 1, 9, 4, 11, 30), (1, 2, 10, 16, 6, 100), (2, 2, 33, 1, 9, 7)], ids=str)
def test_deterministic_step_runs_one_forward(shape):
    """The forward of a deterministic step writes the checkpoints that its backward reads: the launches of the backward and
    its sums only, the bits of the backward that makes them again, and a state that the other backward takes as well."""
    d = {k: v.cuda() for k, v in make_inputs(*shape, dtype=torch.float32, seed=3).items() if v is not None}
    names = ("u", "delta", "A", "B", "C", "D", "delta_bias")
    a = [d[k] for k in names]
    o = cs2d.fwd(*a, True, False, None)
    remade = cs2d.bwd(*a, d["dout"], o[1], o[2], True, None, o[3], deterministic=True)
    leaves = [t.clone().requires_grad_(True) for t in a]
    torch.use_deterministic_algorithms(True)
    try:
        y = cs2d.selective_scan_2d(*leaves, True)
        before = cs2d.launch_count()
        grads = torch.autograd.grad(y, leaves, d["dout"])
        assert cs2d.launch_count() - before == 6       # the backward, and the sums of dB, dC, dA, dD, ddelta_bias
        od = cs2d.fwd(*a, True, False, None)
        pair = cs2d.bwd(*a, d["dout"], od[1], od[2], True, None, od[3])
    finally:
        torch.use_deterministic_algorithms(False)
    assert od[2].numel() != o[2].numel()
    for g, p, r in zip(grads, pair, remade):
        assert torch.equal(g, r) and torch.equal(p, r)
    rtol, atol = TOL["float32"]
    check_close("out", y.detach().cpu().numpy(), o[0].cpu().numpy(), rtol, atol)
    mixed = cs2d.bwd(*a, d["dout"], od[1], od[2], True, None, od[3], deterministic=False)
    for k, x, r in zip(names, mixed, remade):
        check_close("d" + k, x.cpu().numpy(), r.cpu().numpy(), rtol, atol * 10)   # two orders of summation
    assert cs2d.device_status() == 0


def test_fake_saved_state_has_the_size_of_the_real_one():
    from torch._subclasses.fake_tensor import FakeTensorMode
    import cs2d.library  # noqa: F401
    with FakeTensorMode():
        e = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device="cuda")
        A = torch.empty(96, 1, device="cuda")
        for softplus in (True, False):      # pair-walk, streaming
            _, saved = torch.ops.cs2d.scan_fwd(e(2, 96, 7, 7), e(2, 96, 7, 7), A, e(2, 2, 1, 7, 7), e(2, 2, 1, 7, 7), None, None,
                                               softplus, False, None)
            p = _problem(2, 2, 48, 1, 7, 7)
            p.delta_softplus = softplus
            assert saved.numel() * 4 == _lib.lib().cs2d_saved_bytes_dir(ctypes.byref(p), None)


# (batch, groups, channels, states, rows, columns): at most 32 MiB of rows of 8 bytes per channel, state pair and column
FITS = [(170, 4, 192, 2, 28, 28), (42, 4, 192, 3, 56, 56), (10, 4, 192, 16, 56, 56), (56, 4, 9, 16, 5, 250), (500, 4, 8, 1, 5, 250)]


@pytest.mark.skipif(torch.cuda.is_available(), reason="the call has to stop at the missing device")
@pytest.mark.parametrize("shape", FITS, ids=str)
def test_noalloc_takes_what_fits_the_tile_layout(shape):
    one = ctypes.c_void_p(16)
    rc = _lib.lib().cs2d_bwd_noalloc(ctypes.byref(_problem(*shape)), one, 1, 1, 1, one, one, one, one, one, one, None, None, None, None)
    assert rc == -3, _lib.last_error()   # past the size check: there is no device to run on


@pytest.mark.gpu
@pytest.mark.parametrize("shape", FITS[3:], ids=str)
def test_noalloc_with_fewer_ctas(shape):
    """More rows than the array holds at once: same images as with a scratch buffer of the caller's."""
    d = {k: v.cuda() for k, v in make_inputs(*shape, dtype=torch.float32, seed=11).items() if v is not None}
    a = (d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"])
    o = cs2d.fwd(*a, True, False, None)
    ref = cs2d.bwd(*a, d["dout"], o[1], o[2], True, None, o[3])
    p = ops._problem(*a, None, True, torch.float32, "test")
    z = lambda t: torch.zeros_like(t, dtype=torch.float32)
    got = [torch.empty_like(d["u"]), torch.empty_like(d["u"]), z(d["A"]), z(d["B"]), z(d["C"]), z(d["D"]), z(d["delta_bias"])]
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = _lib.lib().cs2d_bwd_noalloc(ctypes.byref(p), vp(d["dout"]), *d["dout"].stride()[:3], vp(o[2]), *map(vp, got), None,
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, _lib.last_error()
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    rtol, atol = TOL["float32"]
    for name, x, y in zip(("dA", "dB", "dC", "dD", "ddelta_bias"), got[2:], ref[2:]):
        check_close(name, x.cpu().numpy(), y.cpu().numpy(), rtol, atol * 10)   # sums with atomics, in another order
    assert cs2d.device_status() == 0
