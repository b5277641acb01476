"""Nothing that a kernel reads is left over from whoever used the memory before: saved states, scratch and rolling rows full of
NaN give the results of any other memory.  Shapes with lanes that have no channel, no state or no column, in each kernel family."""
import pytest
import torch

import cs2d
from cs2d.synthetic import make_inputs

pytestmark = pytest.mark.gpu


def _poison():
    """The blocks that the next allocations get hold NaN."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = [torch.full((1 << k,), float("nan"), device="cuda") for k in (8, 10, 12, 14, 16, 18, 20, 22, 24) for _ in range(6)]
    torch.cuda.synchronize()
    del held


@pytest.mark.parametrize("shape", [(2, 4, 9, 16, 13, 56), (1, 2, 11, 3, 18, 21), (2, 1, 8, 7, 9, 4), (1, 2, 10, 16, 9, 10), (1, 2, 13, 2, 22, 100), (2, 2, 65, 1, 14, 7),
                                   (1, 2, 9, 1, 13, 200), (2, 2, 5, 1, 14, 30), (2, 2, 5, 12, 9, 30), (1, 1, 3, 4, 9, 300)], ids=str)
@pytest.mark.parametrize("cross", [False, True], ids=["scan", "corners"])
def test_memory_full_of_nan(shape, cross):
    b, K, d, n, h, w = shape
    t = {k: v.cuda() for k, v in make_inputs(*shape, seed=5).items() if v is not None}
    a = [t[k] for k in ("u", "delta", "A", "B", "C", "D", "delta_bias")]
    dy = t["dout"]
    if cross:
        a[0], dy = a[0][:, :d].contiguous(), dy[:, :d].contiguous()
        a.insert(5, torch.rand(K, d, device="cuda"))
    leaves = [x.clone().requires_grad_(True) for x in a]
    op = cs2d.cross_scan_2d if cross else cs2d.selective_scan_2d

    def run():
        y = op(*leaves, True)
        with torch.no_grad():
            return [y, op(*leaves, True), *torch.autograd.grad(y, leaves, dy)]

    clean = run()
    _poison()
    for x, ref in zip(run(), clean):
        assert torch.isfinite(x).all()
        torch.testing.assert_close(x, ref, rtol=1e-3, atol=1e-4)   # sums with atomics, in another order
    assert cs2d.device_status() == 0
