"""The pair-walk kernels (a single state per channel) against the float64 oracle: images of one block and less, ragged in both
directions, one to four row workers per CTA, odd and partial channel tiles, every size of piece that rows allow, fp32
results and gradients of 16-bit inputs, strided and misaligned views, the corner directions with their merge, and the
deterministic backward, which makes other kernels' checkpoints again."""
import ctypes

import pytest
import torch

from conftest import TOL, check_close
import cs2d
from cs2d.synthetic import make_inputs
from oracle import cs2d_oracle as O

pytestmark = pytest.mark.gpu
NAMES = ("du", "ddelta", "dA", "dB", "dC", "dD", "ddelta_bias")

# batch, groups, channels, states, rows, columns
CASES = [
    ((1, 1, 8, 1, 1, 1), torch.float32, {}),            # a single pixel
    ((1, 2, 9, 1, 4, 4), torch.float32, {}),            # one band; an odd number of channels
    ((2, 1, 64, 1, 5, 9), torch.bfloat16, {}),          # a full warp of channels; odd rows (element by element)
    ((1, 1, 65, 1, 8, 8), torch.float16, {}),           # one channel more; one group of eight columns
    ((2, 2, 130, 1, 7, 7), torch.bfloat16, {}),
    ((3, 1, 40, 1, 14, 14), torch.bfloat16, {}),        # pieces of four bytes
    ((1, 1, 24, 1, 6, 12), torch.float16, {}),          # eight
    ((1, 2, 24, 1, 13, 22), torch.bfloat16, {}),        # two blocks per band; a short last band
    ((1, 1, 12, 1, 33, 45), torch.float16, {"with_D": False}),
    ((2, 8, 10, 1, 9, 300), torch.bfloat16, {"with_bias": False}),
    ((4, 4, 8, 1, 5, 131), torch.float32, {}),
    ((60, 1, 1300, 1, 3, 5), torch.float32, {}),        # more warps than the GPU holds at once
    # One orientation, 16-bit: with few warps' worth of channels most of the shapes above run on the streaming kernels
    ((150, 1, 64, 1, 5, 9), torch.bfloat16, {}),        # a full warp of channels; odd rows (element by element)
    ((75, 1, 65, 1, 5, 13), torch.float16, {}),         # a channel more than a warp holds
    ((150, 1, 40, 1, 6, 14), torch.bfloat16, {}),       # pieces of four bytes
    ((150, 1, 24, 1, 6, 12), torch.float16, {}),        # eight
    ((150, 2, 9, 1, 5, 22), torch.bfloat16, {}),        # two blocks per band; a short last band
    # copied in 16-byte chunks
    ((150, 1, 66, 1, 7, 14), torch.bfloat16, {}),       # planes and bands in the middle of chunks; a short last band
    ((150, 1, 66, 1, 7, 16), torch.float16, {}),        # (16 columns of one orientation: the streaming kernels; chunks of them below, flipped)
    ((75, 2, 65, 1, 6, 8), torch.float32, {}),          # 128 bytes exactly
    ((40, 4, 9, 1, 6, 136), torch.bfloat16, {}),        # whole chunks per row, half a block at the end of a row
    ((5, 4, 70, 1, 7, 132), torch.float32, {}),
    ((150, 1, 64, 1, 3, 43), torch.float16, {"with_D": False}),
    ((150, 1, 11, 1, 9, 19), torch.float32, {"with_bias": False}),
    ((40, 4, 8, 1, 5, 131), torch.float32, {}),         # wider than the streaming kernels' rows
]


def _dev(inp):
    return {k: (v.cuda() if v is not None else None) for k, v in inp.items()}


def _oracle(inp):
    f = {k: (v.float() if v is not None else None) for k, v in inp.items()}
    a = (f["u"], f["delta"], f["A"], f["B"], f["C"], f["D"], f["delta_bias"])
    return O.fwd(*a, True), O.bwd(*a, f["dout"], True)


def _check(out, g, inp, dtype):
    yo, go = _oracle(inp)
    rtol, atol = TOL[str(dtype)[6:]]
    check_close("out", out.float().cpu().numpy(), yo, rtol, atol)
    for name, t in zip(NAMES, g):
        if go[name] is None:
            assert t is None, name
            continue
        check_close(name, t.float().cpu().numpy(), go[name], rtol, atol)
    assert cs2d.device_status() == 0


@pytest.mark.parametrize("det", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("shape,dtype,kw", CASES, ids=[f"{s}-{str(d)[6:]}" for s, d, _ in CASES])
def test_pair_walk_against_oracle(shape, dtype, kw, det):
    if det and shape[-1] > 128:
        pytest.skip("no deterministic backward for these rows")
    inp = make_inputs(*shape, dtype=dtype, seed=12, **kw)
    d = _dev(inp)
    args = (d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"])
    out, x, xv, xsd = cs2d.fwd(*args, True, False, None)
    g = cs2d.bwd(*args, d["dout"], x, xv, True, None, xsd, deterministic=det)
    assert torch.equal(cs2d.fwd_only(*args, True, False, None), out)
    _check(out, g, inp, dtype)


@pytest.mark.parametrize("w,batch", [(14, 2), (22, 2), (23, 2), (14, 75), (22, 150), (23, 75)])
def test_fp32_results_of_16_bit_views(w, batch):
    """fp32 results and gradients; u, delta and dout are views whose rows are not contiguous and start at odd elements.  (The
    small batches run on the streaming kernels.)"""
    inp = make_inputs(batch, 2, 20, 1, 9 if batch == 2 else 5, w, dtype=torch.bfloat16, seed=3)
    d = _dev(inp)

    def view(t, left):
        wide = torch.zeros(*t.shape[:-1], w + 4, dtype=t.dtype, device="cuda")
        wide[..., left:left + w] = t
        return wide[..., left:left + w]

    args = (view(d["u"], 1), view(d["delta"], 2), d["A"], view(d["B"], 3), d["C"], d["D"], d["delta_bias"])
    out, x, xv, xsd = cs2d.fwd(*args, True, True, None)
    assert out.dtype == torch.float32
    _check(out, cs2d.bwd(*args, view(d["dout"].float(), 1), x, xv, True, None, xsd), inp, torch.bfloat16)
    _check(out, cs2d.bwd(*args, view(d["dout"], 3), x, xv, True, None, xsd), inp, torch.bfloat16)


@pytest.mark.parametrize("shape,dtype", [((1, 4, 9, 1, 6, 20), torch.float32), ((2, 4, 66, 1, 7, 7), torch.bfloat16),
                                         ((1, 4, 12, 1, 10, 14), torch.float16), ((3, 4, 8, 1, 28, 56), torch.bfloat16),
                                         ((4, 4, 10, 1, 11, 100), torch.float32), ((10, 4, 30, 1, 5, 100), torch.float32), ((40, 4, 8, 1, 5, 130), torch.bfloat16),
                                         ((1, 4, 10, 1, 6, 21), torch.bfloat16),
                                         ((1, 4, 10, 1, 9, 7), torch.float32), ((4, 4, 14, 1, 9, 9), torch.bfloat16)])
def test_corner_directions_and_merge(shape, dtype):
    b, K, d, n, h, w = shape
    inp = make_inputs(*shape, dtype=dtype, seed=2)
    gen = torch.Generator().manual_seed(9)
    host = dict(u=torch.randn(b, d, h, w, generator=gen).to(dtype), delta=inp["delta"], A=inp["A"], B=inp["B"], C=inp["C"],
                w=torch.rand(K, d, generator=gen) + 0.1, D=inp["D"], delta_bias=inp["delta_bias"])
    dy = torch.randn(b, d, h, w, generator=gen).to(dtype)
    dev = {k: v.cuda().requires_grad_(True) for k, v in host.items()}
    y = cs2d.cross_scan_2d(*dev.values(), True)
    y.backward(dy.cuda())
    with torch.no_grad():
        torch.testing.assert_close(cs2d.cross_scan_2d(*dev.values(), True), y, rtol=1e-2, atol=1e-5)
    ref = {k: v.double().requires_grad_(True) for k, v in host.items()}
    yo = O.cross_fwd_torch(*ref.values(), True)
    yo.backward(dy.double())
    rtol, atol = (1e-4, 1e-5) if dtype == torch.float32 else (2e-2, 1e-3)
    check_close("y", y.detach().float().cpu().numpy(), yo.detach().numpy(), rtol, atol)
    for k in host:
        check_close("d" + k, dev[k].grad.float().cpu().numpy(), ref[k].grad.numpy(), rtol, atol)
    assert cs2d.device_status() == 0


def _placed(shape, dtype, off, pad=0, row_pad=0, fill=None):
    """A tensor `off` elements into its buffer, whose channels and rows end `pad` and `row_pad` elements before the next; and the rest of
    that buffer, as a check that nothing is written there."""
    b, c, h, w = shape
    hs = w + row_pad
    ds = h * hs + pad
    buf = torch.full((off + b * c * ds + 16,), 7.0, dtype=dtype, device="cuda")
    t = buf.as_strided(shape, (c * ds, ds, hs, 1), off)
    if fill is not None:
        t.copy_(fill)
    return t, buf


def _untouched(t, buf):
    seen = torch.zeros_like(buf, dtype=torch.bool)
    seen.as_strided(t.shape, t.stride(), t.storage_offset()).fill_(True)
    return bool((buf[~seen] == 7.0).all())


def _c_abi(d, dtype, flip=(False, False), at=0, pad=0, row_pad=0):
    """Forward, evaluation forward and backward through the C ABI with results at `at` elements into their buffers (`out`: with
    `pad` and `row_pad` too); every group is walked from the bottom (flip[0]) or from the right (flip[1])."""
    p = cs2d.ops._problem(d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"], None, True, dtype, "test")
    L, every = cs2d._lib.lib(), (1 << p.n_groups) - 1
    dirs = cs2d._lib.Dirs(every * flip[0], every * flip[1], 0, 0, None, None)
    ref, o, st = ctypes.byref(p), ctypes.byref(dirs), torch.cuda.current_stream().cuda_stream
    saved, scratch, rolling = (torch.empty(f(ref, o), dtype=torch.uint8, device="cuda") for f in (
        L.cs2d_saved_bytes_dir, L.cs2d_bwd_scratch_bytes_dir, L.cs2d_fwd_only_scratch_bytes_dir))
    shape, dout = tuple(d["u"].shape), d["dout"]
    out, out2 = (_placed(shape, dtype, at, pad, row_pad) for _ in range(2))
    du, ddelta = (_placed(shape, dtype, at) for _ in range(2))
    sums = [torch.zeros(s, device="cuda") for s in (d["A"].shape, d["B"].shape, d["C"].shape, p.dim, p.dim)]
    assert L.cs2d_fwd_dir(ref, o, out[0].data_ptr(), *out[0].stride()[:3], saved.data_ptr(), st) == 0
    assert L.cs2d_fwd_only(ref, o, out2[0].data_ptr(), *out2[0].stride()[:3], rolling.data_ptr(), st) == 0
    assert L.cs2d_bwd_dir(ref, o, dout.data_ptr(), *dout.stride()[:3], saved.data_ptr(), scratch.data_ptr(), du[0].data_ptr(), ddelta[0].data_ptr(),
                          *[t.data_ptr() for t in sums], None, st) == 0
    assert torch.equal(out[0], out2[0])
    for r in (out, out2, du, ddelta):
        assert _untouched(*r)
    return out[0], (du[0], ddelta[0], *sums)


def _check_flipped(out, g, inp, dtype, flip):
    """Walked from another corner: what the oracle gives for the mirrored images, mirrored."""
    dims = [i for i, f in zip((-2, -1), flip) if f]
    image = ("u", "delta", "B", "C", "dout")
    m = lambda t: t.flip(dims)
    _check(m(out), [m(t) if i in (0, 1, 3, 4) else t for i, t in enumerate(g)], {k: m(v) if k in image and dims else v for k, v in inp.items()}, dtype)


# blocks of whole chunks, linear and by rows; linear ones that start at every fourth byte, in both directions and in the forward alone; fp32; the
# last: element by element.  (A flip, where one orientation alone would run on the streaming kernels.)
PLACES = [((2, 1, 66, 1, 7, 8), torch.bfloat16, (False, False)), ((150, 1, 66, 1, 8, 14), torch.bfloat16, (False, False)),
          ((150, 1, 66, 1, 7, 14), torch.bfloat16, (False, False)), ((3, 1, 66, 1, 7, 16), torch.float16, (True, False)),
          ((3, 2, 65, 1, 6, 8), torch.float32, (False, False)), ((3, 1, 65, 1, 6, 6), torch.float32, (False, True)),
          ((3, 4, 9, 1, 6, 64), torch.bfloat16, (False, True)), ((2, 2, 70, 1, 7, 20), torch.float32, (True, True)),
          ((3, 1, 66, 1, 5, 9), torch.bfloat16, (False, True))]


@pytest.mark.parametrize("at,pad,row_pad", [(1, 0, 0), (2, 0, 0), (4, 0, 0), (0, 1, 0), (0, 2, 0), (3, 3, 1), (0, 0, 2)])
@pytest.mark.parametrize("shape,dtype,flip", PLACES, ids=[f"{s}-{str(t)[6:]}" for s, t, _ in PLACES])
def test_results_at_any_address(shape, dtype, flip, at, pad, row_pad):
    """The inputs allow 16-byte chunks, the results, which a caller of the C ABI places, start at any element."""
    inp = make_inputs(*shape, dtype=dtype, seed=at + 2)
    out, g = _c_abi(_dev(inp), dtype, flip, at, pad, row_pad)
    _check_flipped(out, g, inp, dtype, flip)


@pytest.mark.parametrize("at", [(2, 0, 0), (0, 4, 4), (6, 2, 1), (1, 3, 2)], ids=str)
@pytest.mark.parametrize("flip", [(False, False), (True, False), (False, True)], ids=["", "rows", "columns"])
@pytest.mark.parametrize("shape,dtype", [((150, 1, 65, 1, 14, 14), torch.bfloat16), ((150, 2, 33, 1, 7, 14), torch.float16), ((150, 1, 66, 1, 8, 8), torch.bfloat16),
                                         ((75, 1, 65, 1, 7, 8), torch.float16), ((75, 1, 66, 1, 7, 6), torch.float32)], ids=str)
def test_inputs_at_any_address(shape, dtype, flip, at):
    """u, delta and dout start elements into their buffers, as a view's do: the 16-byte chunks that a linear block touches begin before it, and
    what the copies without a source name (channels that a warp has too many, rows below the image) is a multiple of 16 all the same."""
    inp = make_inputs(*shape, dtype=dtype, seed=sum(at))
    d = _dev(inp)
    for name, n in zip(("u", "delta", "dout"), at):
        d[name] = _placed(d[name].shape, dtype, n, fill=d[name])[0]
    out, g = _c_abi(d, dtype, flip)
    _check_flipped(out, g, inp, dtype, flip)
