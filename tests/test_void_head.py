"""A positional matchjoinAN of a list with a virtual head whose struct names the
list's own codes as the head's data (a caller's output struct, used again): the
head is seqbase + row all the same."""
import ctypes

import numpy as np
import pytest

from bats import encoded_col, oid_list

from ahead_b200.model import OK, RESINT, RESOID, WIDTH, Bat, CBat, CErrVec, void_col

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 8_193, 20_000])
def test_virtual_head_with_data(n):
    import torch
    import ahead_b200.gpu as mirror
    g = mirror.GpuOps(0)
    oids = oid_list(np.arange(n)[::-1].copy())
    a = mirror.to_device(Bat(void_col(7), oids.tail, n))
    b = mirror.to_device(encoded_col(RESINT, np.arange(n) + 5))
    ca, cb, out, errs = mirror._in_bat(a), mirror._in_bat(b), CBat(), (CErrVec * 4)()
    ca.head.data = ca.tail.data
    assert a.tail.type == RESOID
    head = torch.empty(n * 8, dtype=torch.uint8, device="cuda")
    tail = torch.empty(n * 8, dtype=torch.uint8, device="cuda")
    out.head.data, out.tail.data = head.data_ptr(), tail.data_ptr()
    torch.cuda.synchronize()
    rc = g.lib.ahead_gpu_matchjoin_an(g.ctx, ctypes.byref(ca), ctypes.byref(cb), 0, ctypes.c_uint64(0),
                                      ctypes.c_uint64(0), ctypes.c_uint64(0), ctypes.c_uint64(0),
                                      ctypes.c_uint64(16089), ctypes.byref(out), ctypes.c_uint64(n), errs)
    assert rc == OK and out.count == n
    w = WIDTH[out.head.type]
    got = head[: n * w].cpu().numpy().view({4: np.uint32, 8: np.uint64}[w])
    assert np.array_equal(got, np.arange(7, 7 + n))
    codes = tail.cpu().numpy().view(np.uint64)
    assert np.array_equal(codes, (np.arange(n)[::-1] + 5).astype(np.uint64) * np.uint64(b.tail.A))
    g.close()
