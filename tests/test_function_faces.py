"""The two operators as autograd Functions, and the C ABI's problem from Python: one set of checks, one autograd node each."""
import pytest
import torch

import cs2d
from cs2d import _lib, ops
from cs2d.synthetic import make_inputs


def test_functions_have_no_node_of_their_own():
    for f in (cs2d.SelectiveScan2D, cs2d.CrossScan2D):
        assert issubclass(f, torch.autograd.Function) and "backward" not in vars(f)


def test_problem_makes_the_operators_checks():
    u, A, B = torch.zeros(1, 4, 8, 8), torch.zeros(4, 2), torch.zeros(1, 2, 2, 8, 8)
    with pytest.raises(RuntimeError, match="u must be a CUDA tensor"):
        ops._problem(u, u, A, B, B, None, None, None, True, torch.float32, "here")
    with pytest.raises(RuntimeError, match="here not implemented for input type"):
        ops._problem(u.double(), u, A, B, B, None, None, None, True, torch.float32, "here")


@pytest.mark.gpu
def test_apply_and_problem():
    d = {k: v.cuda() for k, v in make_inputs(2, 4, 6, 5, 7, 9, seed=1).items() if v is not None}
    a = [d[k] for k in ("u", "delta", "A", "B", "C", "D", "delta_bias")]
    p = ops._problem(*a, None, True, torch.float32, "test")
    assert (p.batch, p.dim, p.nrows, p.ncols, p.dstate, p.n_groups, p.delta_dim) == (2, 24, 7, 9, 5, 4, 24)
    assert (p.io_dtype, p.out_dtype, p.delta_softplus, p.A_decay) == (_lib.F32, _lib.F32, 1, None)
    assert (p.B, p.B_bs, p.B_gs, p.B_ns, p.B_hs) == (d["B"].data_ptr(), *d["B"].stride()[:4])
    with pytest.raises(RuntimeError, match="n_groups channels"):
        ops._problem(*a, None, True, torch.float32, "test", shared_u_dim=25)
    a[0].requires_grad_(True)
    y, y2 = cs2d.SelectiveScan2D.apply(*a, True), cs2d.selective_scan_2d(*a, True)
    assert torch.equal(y, y2) and y.requires_grad
    g, g2 = (torch.autograd.grad(x, a[0], d["dout"])[0] for x in (y, y2))
    assert torch.equal(g, g2)
