"""Calls whose first choice of form wants more scratch than the device has left
take the form that needs less: nearly all device memory is held while they run
on a context without an arena, and the results equal those of the same call
with memory to spare."""
import pytest

from ahead_b200.model import RESBIGINT, RESINT, RESOID, Bat, Col, an_meta, void_col

pytestmark = pytest.mark.gpu

LEFT = 120 << 20  # bytes of device memory left to the call
A = 65117


def col(t, values):
    import torch
    m = an_meta(t, A)
    return Col(t, (values * A).view(torch.uint8).reshape(-1), A, m["Ainv"], m["unenc_max"], 0)


def corrupt(c, rows):
    c.data.view(-1, 8)[rows, 7] ^= 0x80


def same(a, b):
    import torch
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(same(x, y) for x, y in zip(a, b))
    if isinstance(a, Bat):
        return a.count == b.count and same(a.head, b.head) and same(a.tail, b.tail)
    if isinstance(a, Col):
        return a.type == b.type and same(a.data, b.data)
    if isinstance(a, torch.Tensor):
        return torch.equal(a, b)
    return a == b if not hasattr(a, "values") else a.present == b.present and same(a.values, b.values)


def with_little_left(call):
    """call(ops) with memory to spare, twice (the second's buffers stay with
    torch for the third), then on a new context with LEFT bytes left."""
    import torch
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)
    want = call(g)
    call(g)
    g.close()
    g = GpuOps(0)
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - LEFT, dtype=torch.uint8, device="cuda")
    try:
        got = call(g)
    finally:
        del held
        torch.cuda.empty_cache()
        g.close()
    assert same(got, want)


@pytest.fixture(autouse=True)
def clean():
    import gc
    import torch
    gc.collect()
    torch.cuda.empty_cache()
    yield
    gc.collect()
    torch.cuda.empty_cache()


def test_check_and_decode():  # gaps closed in place: 134 MB; the compaction: 20
    import torch
    n = 1 << 27
    c = col(RESBIGINT, torch.arange(n, device="cuda") % 1000)
    corrupt(c, torch.tensor([5, 77_000, n - 1]))
    torch.cuda.synchronize()
    with_little_left(lambda g: g.check_and_decode_an(Bat(void_col(0), c, n)))


def test_positional_join():  # the same: 134 MB, 20
    import torch
    n, m = 1 << 26, 1 << 20
    oids = col(RESOID, torch.arange(n, device="cuda") * 7 % m)
    corrupt(oids, torch.tensor([0, 4_000_000]))
    value = col(RESBIGINT, torch.arange(m, device="cuda"))
    torch.cuda.synchronize()
    with_little_left(lambda g: g.matchjoin_an(Bat(oids, oids, n), Bat(void_col(0), value, m)))


def test_hash_join():  # the bitmap's values: 134 MB; the hash table and the probe's slots: 75
    import torch
    n, m = 1 << 24, 7
    probe = col(RESINT, torch.arange(n, device="cuda") * 11 % 4_000)
    keys, oids = col(RESINT, torch.arange(m, device="cuda") * 500), col(RESOID, torch.arange(m, device="cuda"))
    corrupt(probe, torch.tensor([9, n - 2]))
    torch.cuda.synchronize()
    with_little_left(lambda g: g.hashjoin_an(Bat(void_col(0), probe, n), Bat(keys, oids, m)))
