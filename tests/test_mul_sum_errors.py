"""aggregate_mul_sumAN with as many corrupt codes as its lists hold and more, in
either column, against the C restatement: sum and both error vectors; columns of
unequal lengths and off a 16-byte boundary."""
import numpy as np
import pytest

from bats import encoded_col
from cases import assert_same, run_case

from ahead_b200.model import RESINT, RESSHORT, RESTINY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f1,f2", [(0, 0), (4096, 4096), (4097, 0), (0, 4097), (5, 4097), (9000, 20_000)])
@pytest.mark.parametrize("t2", [RESTINY, RESSHORT])
@pytest.mark.parametrize("shift", [0, 1])
def test_flips(f1, f2, t2, shift):
    from ahead_b200.gpu import GpuOps, err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    rng = np.random.default_rng(f1 + f2 + t2)
    n = 300_007
    a, b = encoded_col(RESINT, rng.integers(0, 1 << 20, n)), encoded_col(t2, rng.integers(0, 200, n - 4))
    for c, f in ((a, f1), (b, f2)):
        at = rng.choice(n - 4, f, replace=False)
        c.tail.data[at] ^= c.tail.data.dtype.type(1) << c.tail.data.dtype.type(c.tail.data.dtype.itemsize * 8 - 1)
    g = GpuOps(0)

    def dev(c):  # on the device, `shift` rows into a longer column
        d = to_device(c)
        if shift:
            w = d.tail.data.numel() // c.count
            longer = g.torch.zeros(d.tail.data.numel() + shift * w, dtype=g.torch.uint8, device="cuda")
            longer[shift * w:] = d.tail.data
            g.torch.cuda.synchronize()
            d.tail.data = longer[shift * w:]
        return d
    c = dict(op="aggregate_mul_sum_an", args=[a, b], kwargs={})
    assert_same(run_case(g, c, dev, to_host, err_to_host), run_case(Oracle("port"), c), "aggregate_mul_sum_an")
    g.close()
