"""Sizes of the buffers between the calls.  The built-in scratch array of ``cs2d_bwd_noalloc`` serves every problem whose
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
