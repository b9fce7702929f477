"""The output function a caller set on a context is still set after the star join
composed in C++ has run there with one of its own."""
import ctypes

import numpy as np
import pytest

from bats import encoded_col

from ahead_b200.model import GE, OK, RESINT, CBat

pytestmark = pytest.mark.gpu


def test_plain_starjoin_keeps_the_callers_function():
    import torch
    import ahead_b200.gpu as mirror
    from ahead_b200.ssb import generate_device
    from ahead_b200.ssb_programs import program_query
    from ahead_b200.starjoin import StarJoinEngine
    g = mirror.GpuOps(0)
    # (columns above 16 MB of output, so that the star join's selections allocate theirs)
    ds = generate_device(dict(fact=2_200_000, date=2556, customer=3_000, part=2_000, supplier=200), seed=1)
    eng = StarJoinEngine(g, ds)
    bufs = []

    @mirror._OUTPUT_FN
    def take(user, column, nbytes):
        bufs.append(torch.empty(nbytes, dtype=torch.uint8, device="cuda"))
        return bufs[-1].data_ptr()

    g.lib.ahead_ctx_set_output_fn(g.ctx, take, None)
    eng.plain(program_query("q11"))
    assert not bufs  # the star join's columns are its own
    n = 5_000
    b = mirror.to_device(encoded_col(RESINT, np.arange(n)))
    out, cin = CBat(), mirror._in_bat(b)
    rc = g.lib.ahead_gpu_select_an(g.ctx, ctypes.byref(cin), GE, ctypes.c_uint64(100 * b.tail.A), 0,
                                   ctypes.c_uint64(0), 0, ctypes.c_uint64(16089), ctypes.byref(out),
                                   ctypes.c_uint64(mirror._SIZED), None)
    assert rc == OK and out.count == n - 100 and len(bufs) == 1 and out.head.data == bufs[0].data_ptr()
    assert np.array_equal(bufs[0].cpu().numpy().view(np.uint64), np.arange(100, n, dtype=np.uint64) * np.uint64(65117))
    g.lib.ahead_ctx_set_output_fn(g.ctx, None, None)
    eng.close()
    g.close()
