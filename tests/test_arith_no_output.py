"""arithmeticAN without an output column: the error vectors alone, and no store
through the null pointer; with and without error vectors of the caller's."""
import ctypes

import numpy as np
import pytest

from bats import encoded_col

from ahead_b200.model import MUL, OK, RESBIGINT, RESINT, RESTINY, CBat, CErrVec, ainv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 8_191, 300_001])
@pytest.mark.parametrize("flips", [0, 9, 5_000])
def test_errors_only(n, flips):
    import torch
    import ahead_b200.gpu as mirror
    rng = np.random.default_rng(n + flips)
    g = mirror.GpuOps(0)
    a, b = encoded_col(RESINT, rng.integers(0, 1 << 20, n)), encoded_col(RESTINY, rng.integers(1, 50, n))
    a.tail.data[rng.choice(n, min(flips, n), replace=False)] ^= np.uint64(1 << 63)
    da, db = mirror.to_device(a), mirror.to_device(b)
    ca, cb, out, errs = mirror._in_bat(da), mirror._in_bat(db), CBat(), (CErrVec * 4)()
    bufs = [torch.zeros(8_192 * 8, dtype=torch.uint8, device="cuda") for _ in range(4)]
    for e, buf in zip(errs, bufs):
        e.data, e.capacity = buf.data_ptr(), 8_192
    torch.cuda.synchronize()
    for given in (errs, None):
        rc = g.lib.ahead_gpu_arithmetic_an(g.ctx, MUL, RESBIGINT, ctypes.byref(ca), ctypes.byref(cb),
                                           ctypes.c_uint64(65117), ctypes.c_uint64(ainv(65117, 64)),
                                           ctypes.c_uint64(16089), ctypes.byref(out), given)
        assert rc == OK and out.count == n
    want = np.nonzero(a.tail.data * np.uint64(ainv(a.tail.A, 64)) > np.uint64(a.tail.unenc_max))[0]
    assert errs[1].count == len(want) and errs[3].count == 0
    got = bufs[1].cpu().numpy().view(np.uint64)[: len(want)]
    assert np.array_equal(got, want.astype(np.uint64) * np.uint64(16089))
    g.close()
