"""The pair-walk kernels (a single state per channel) against the float64 oracle: images of one block and less, ragged in both
directions, one to four row workers per CTA, odd and partial channel tiles, every size of piece that rows allow, fp32
results and gradients of 16-bit inputs, strided and misaligned views, the corner directions with their merge, and the
deterministic backward, which makes other kernels' checkpoints again."""
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
    ((150, 1, 66, 1, 7, 16), torch.float16, {}),        # 64 of 128 bytes of a short band missing: the chunks that remain are whole
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
