"""The block-walk kernels (two or more states, at least eight channels per group) against the float64 oracle: images of
one block and less, ragged in both directions, one to eight row workers per CTA, odd channel counts (a slot with one live
half), every number of state slots, delta shared by channels (the addresses of neighbouring channels coincide), fp32
results of 16-bit inputs, rows that do and do not allow groups of four, state decay, and the deterministic
backward, which makes the tile kernels' checkpoints again."""
import ctypes
import os
import subprocess

import pytest
import torch

from conftest import ROOT, TOL, check_close
import cs2d
from cs2d.synthetic import make_inputs
from oracle import cs2d_oracle as O

pytestmark = pytest.mark.gpu
NAMES = ("du", "ddelta", "dA", "dB", "dC", "dD", "ddelta_bias", "dA_decay")

CASES = [
    ((1, 1, 8, 3, 1, 1), torch.float32, {}),           # a single pixel
    ((1, 2, 9, 16, 4, 8), torch.float32, {}),          # exactly one block; an odd number of channels
    ((2, 1, 8, 8, 5, 9), torch.float32, {}),           # one row and one column more than a block
    ((2, 2, 13, 2, 6, 12), torch.bfloat16, {}),         # two states; half a block at the end of a row
    ((1, 1, 11, 9, 40, 7), torch.float32, {}),         # one block per row: the row of h stays in registers or waits for the workers
    ((3, 1, 10, 16, 9, 33), torch.bfloat16, {}),       # 5 blocks per row, two row workers with a short last pass
    ((1, 2, 12, 5, 27, 70), torch.float16, {}),        # 9 blocks per row, four row workers
    ((1, 1, 9, 16, 61, 21), torch.bfloat16, {}),       # 16 rows of 3 blocks, eight row workers: none starts before the one before it
    ((1, 1, 12, 6, 35, 130), torch.float32, {}),       # 9 rows, eight row workers: one of them has two
    ((1, 1, 16, 16, 16, 64), torch.float32, {"delta_dim": 4}),
    ((2, 1, 8, 7, 13, 20), torch.float32, {"a_decay": 0.9, "with_bias": False}),
    ((1, 4, 8, 16, 12, 300), torch.float32, {"with_D": False}),   # wider than a tile launch
    ((40, 1, 34, 16, 6, 10), torch.float32, {}),       # more warps than the GPU holds at once
]


def _dev(inp):
    return {k: (v.cuda() if v is not None else None) for k, v in inp.items()}


def _oracle(inp, softplus=True):
    f = {k: (v.float() if v is not None else None) for k, v in inp.items()}
    a = (f["u"], f["delta"], f["A"], f["B"], f["C"], f["D"], f["delta_bias"])
    return O.fwd(*a, softplus, f["A_decay"]), O.bwd(*a, f["dout"], softplus, f["A_decay"])


@pytest.mark.parametrize("det", [False, True], ids=["atomic", "deterministic"])
@pytest.mark.parametrize("shape,dtype,kw", CASES, ids=[f"{s}-{str(d)[6:]}" for s, d, _ in CASES])
def test_block_walk_against_oracle(shape, dtype, kw, det):
    if det and (shape[-1] > 256 or (shape[-1] > 64 and shape[3] <= 8)):
        pytest.skip("no deterministic backward for these rows")
    inp = make_inputs(*shape, dtype=dtype, seed=12, **kw)
    d = _dev(inp)
    args = (d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"])
    out, x, xv, xsd = cs2d.fwd(*args, True, False, d["A_decay"])
    g = cs2d.bwd(*args, d["dout"], x, xv, True, d["A_decay"], xsd, deterministic=det)
    assert torch.equal(cs2d.fwd_only(*args, True, False, d["A_decay"]), out)
    yo, go = _oracle(inp)
    rtol, atol = TOL[str(dtype)[6:]]
    check_close("out", out.float().cpu().numpy(), yo, rtol, atol)
    for name, t in zip(NAMES, g):
        ref = go["dA_decay_ref" if name == "dA_decay" else name]
        if ref is None:
            assert t is None, name
            continue
        check_close(name, t.float().cpu().numpy(), ref, rtol, atol)
    assert cs2d.device_status() == 0


@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 13, 15, 17])
@pytest.mark.parametrize("n", [3, 16])
def test_every_number_of_columns_in_the_last_block(n, w):
    """Forward and backward leave out the pairs of columns that a row's last block does not have."""
    inp = make_inputs(2, 1, 9, n, 9, w, dtype=torch.float32, seed=w)
    d = _dev(inp)
    args = (d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"])
    out, x, xv, xsd = cs2d.fwd(*args, True, False, None)
    g = cs2d.bwd(*args, d["dout"], x, xv, True, None, xsd)
    assert torch.equal(cs2d.fwd_only(*args, True, False, None), out)
    yo, go = _oracle(inp)
    check_close("out", out.cpu().numpy(), yo, *TOL["float32"])
    for name, t in zip(NAMES[:7], g):
        check_close(name, t.cpu().numpy(), go[name], *TOL["float32"])
    assert cs2d.device_status() == 0


def test_fp32_results_of_strided_16bit_inputs_without_softplus():
    inp = make_inputs(2, 2, 10, 6, 11, 19, dtype=torch.bfloat16, seed=5, with_bias=False)
    inp["delta"] = (inp["delta"].float().abs() * 0.1).to(torch.bfloat16)
    d = _dev(inp)
    big = torch.zeros(2, 30, 11, 24, dtype=torch.bfloat16, device="cuda")
    big[:, 7:27, :, 3:22] = d["u"]
    d["u"] = big[:, 7:27, :, 3:22]              # channels and columns of a larger tensor
    d["B"] = d["B"].transpose(0, 1).contiguous().transpose(0, 1)
    args = (d["u"], d["delta"], d["A"], d["B"], d["C"], d["D"], d["delta_bias"])
    o = cs2d.fwd(*args, False, True, None)
    assert o[0].dtype == torch.float32
    g = cs2d.bwd(*args, d["dout"].float(), o[1], o[2], False, None, o[3])
    yo, go = _oracle(inp, softplus=False)
    check_close("out", o[0].cpu().numpy(), yo, 1e-4, 1e-5)   # fp32 output: arithmetic error only
    for name, t in zip(NAMES, g):
        if t is not None:
            check_close(name, t.float().cpu().numpy(), go[name], 2e-2, 1e-3)


@pytest.mark.parametrize("shape,dtype", [((1, 4, 9, 16, 10, 21), torch.float32), ((2, 4, 8, 4, 19, 44), torch.bfloat16)])
def test_four_corner_merge(shape, dtype):
    b, K, dd, n, h, w = shape
    inp = make_inputs(b, K, dd, n, h, w, dtype=dtype, seed=2)
    gen = torch.Generator().manual_seed(9)
    host = dict(u=torch.randn(b, dd, h, w, generator=gen).to(dtype), delta=inp["delta"], A=inp["A"], B=inp["B"], C=inp["C"],
                w=torch.rand(K, dd, generator=gen) - 0.3, D=inp["D"], delta_bias=inp["delta_bias"])
    dy = torch.randn(b, dd, h, w, generator=gen).to(dtype)
    dev = {k: v.cuda().requires_grad_(True) for k, v in host.items()}
    y = cs2d.cross_scan_2d(*dev.values(), True)
    y.backward(dy.cuda())
    ref = {k: v.double().requires_grad_(True) for k, v in host.items()}
    yo = O.cross_fwd_torch(*ref.values(), True)
    yo.backward(dy.double())
    rtol, atol = TOL[str(dtype)[6:]]
    check_close("y", y.detach().float().cpu().numpy(), yo.detach().numpy(), rtol, atol)
    for k in host:
        check_close("d" + k, dev[k].grad.float().cpu().numpy(), ref[k].grad.numpy(), rtol, atol)
    assert cs2d.device_status() == 0


@pytest.mark.parametrize("n,batch", [(16, 250), (4, 200)])
def test_parameters_change_with_the_item(n, batch):
    """A warp goes through several items (a group's slots of channels) whose D and merge weights differ, the last of a group with a single
    channel: dw and dD are sums with the item's own.  (u, B, C and dy positive: no sum cancels.)"""
    K, dd, h, w = 4, 17, 3, 3
    inp = make_inputs(batch, K, dd, n, h, w, dtype=torch.float32, seed=n)
    gen = torch.Generator().manual_seed(n)
    host = dict(u=torch.rand(batch, dd, h, w, generator=gen) + 0.1, delta=inp["delta"], A=inp["A"], B=inp["B"].abs(), C=inp["C"].abs(),
                w=torch.rand(K, dd, generator=gen) + 0.1, D=torch.rand(K * dd, generator=gen) + 0.1, delta_bias=inp["delta_bias"])
    dy = torch.rand(batch, dd, h, w, generator=gen) + 0.1
    dev = {k: v.cuda().requires_grad_(True) for k, v in host.items()}
    cs2d.cross_scan_2d(*dev.values(), True).backward(dy.cuda())
    ref = {k: v.double().requires_grad_(True) for k, v in host.items()}
    O.cross_fwd_torch(*ref.values(), True).backward(dy.double())
    for k in ("w", "D"):
        check_close("d" + k, dev[k].grad.cpu().numpy(), ref[k].grad.numpy(), *TOL["float32"])
    assert cs2d.device_status() == 0


ROW_WAIT = r"""
#include "cs2d_blk.cuh"
using namespace cs2d;
// Two row workers, three blocks per row.  Worker 1 waits for a block of worker 0 that is never counted, worker 0 for one of worker 1's.
__global__ void row_wait_kernel(int *status, int *got) {
    __shared__ int count[BK_MAXRW];
    const int warp = threadIdx.x >> 5;
    RowSeq rs;
    rs.init(count, warp, 2, 3);
    __syncthreads();
    const bool ok = warp ? rs.wait(3, 1000) : rs.wait(6);
    if (!ok) rs.abandon(status);
    if ((threadIdx.x & 31) == 0) got[warp] = ok;
}
extern "C" int row_wait(int *status, int *got, void *stream) {
    row_wait_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(status, got);
    return cudaGetLastError();
}
"""


def test_a_wait_that_runs_out_ends_with_a_status(tmp_path):
    """The wait of a row worker, with a small number of polls: it gives up, says so, and lets the worker behind it go on."""
    src, so = tmp_path / "row_wait.cu", tmp_path / "row_wait.so"
    src.write_text(ROW_WAIT)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(ROOT, "official-cross-scan_b200", "csrc"), "-o", so, src], check=True)
    status, got = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((2,), -1, dtype=torch.int32, device="cuda")
    f = ctypes.CDLL(str(so)).row_wait
    assert f(ctypes.c_void_p(status.data_ptr()), ctypes.c_void_p(got.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert got.tolist() == [1, 0]
    assert status.item() == 4


def _places(t, how, n):
    """The same values `n` elements into a buffer, or in rows that are `n` elements longer than the image is wide."""
    if how == "offset":
        buf = torch.zeros(t.numel() + n, dtype=t.dtype, device=t.device)
        v = buf[n:].view(t.shape)
    else:
        v = torch.zeros(*t.shape[:-1], t.shape[-1] + n, dtype=t.dtype, device=t.device)[..., :t.shape[-1]]
    v.copy_(t)
    return v


@pytest.mark.parametrize("dtype,out_float", [(torch.float32, False), (torch.bfloat16, False), (torch.float16, True)], ids=["fp32", "bf16", "fp16-fp32"])
@pytest.mark.parametrize("how,n", [("offset", 1), ("offset", 2), ("offset", 4), ("pitch", 1), ("pitch", 2), ("pitch", 4)])
@pytest.mark.parametrize("W,N", [(16, 5), (20, 12), (9, 16)])
def test_backward_copies_of_every_width(W, N, how, n, dtype, out_float):
    """The inputs are copied 16, 8, 4 bytes or a shifted word at a time, as their addresses and strides allow: the
    gradients are those of contiguous inputs.  dB, dC and the parameters' gradients are sums in another order (fp32 atomics)."""
    inp = _dev(make_inputs(2, 2, 9, N, 11, W, dtype=dtype, seed=5))
    dout = inp["dout"].float() if out_float else inp["dout"]
    rest = (inp["A"], inp["B"], inp["C"], inp["D"], inp["delta_bias"])
    def grads(u, delta, g):
        _, x, xv, xsd = cs2d.fwd(u, delta, *rest, True, out_float, None)
        return cs2d.bwd(u, delta, *rest, g, x, xv, True, None, xsd)
    ref = grads(inp["u"], inp["delta"], dout)
    got = grads(_places(inp["u"], how, n), _places(inp["delta"], how, n), _places(dout, how, n))
    for name, a, b in zip(NAMES, ref, got):
        if name in ("du", "ddelta"):
            assert torch.equal(a, b), name
        elif a is not None:
            check_close(name, b.float().cpu().numpy(), a.float().cpu().numpy(), *TOL[str(dtype)[6:]])
