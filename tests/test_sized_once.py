"""Joins whose output columns the call allocates itself run once, also where the
inputs need another form (keys out of order, repeated or wide join keys), and
equal the C restatement."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import HASH_LEFT, HASH_RIGHT, INT, OID, RESINT, Bat, Col, void_col

pytestmark = pytest.mark.gpu


class Counted:
    """The library with its operator calls counted."""

    def __init__(self, lib):
        self.lib, self.calls = lib, []

    def __getattr__(self, name):
        if name.startswith("ahead_gpu_"):
            self.calls.append(name)
        return getattr(self.lib, name)


@pytest.fixture
def gpu(monkeypatch):
    import ahead_b200.gpu as mirror
    monkeypatch.setattr(mirror, "_SIZED_BYTES", 0)
    g = mirror.GpuOps(0)
    g.lib = Counted(g.lib)
    yield g
    g.lib = g.lib.lib
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    del gpu.lib.calls[:]
    got = run_case(gpu, c, to_device, to_host, err_to_host)
    assert gpu.lib.calls == ["ahead_gpu_" + op]
    assert_same(got, run_case(Oracle("port"), c), op)


@pytest.mark.parametrize("n1,n2", [(1, 3), (40, 300), (9_000, 700)])
def test_merge_out_of_order(gpu, n1, n2):
    rng = np.random.default_rng(n1)
    k1 = rng.permutation(n1).astype(np.uint64)
    k2 = rng.choice(2 * max(n1, n2), n2, replace=False).astype(np.uint64)
    k2[0] = k2[-1]  # a repeated key, too
    a, b = oid_list(k1), oid_list(k2)
    value = encoded_col(RESINT, rng.integers(0, 1 << 20, n2)).tail
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n1), Bat(b.tail, value, n2))
    p, q = Col(OID, k1.astype(np.uint32)), Col(OID, k2.astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n1), Bat(q, Col(INT, rng.integers(0, 99, n2).astype(np.uint32)), n2))
    same = oid_list(np.full(n1, 7, np.uint64))  # every key the same: the shorter input's length is kept
    other = oid_list(np.full(n2, 7, np.uint64))
    check(gpu, "matchjoin_an", Bat(same.tail, same.tail, n1), Bat(other.tail, other.tail, n2))


@pytest.mark.parametrize("why", ["repeated key", "all repeated", "wide range", "corrupt key"])
@pytest.mark.parametrize("n", [30, 9_000, 70_001])
def test_hashjoin_through_the_table(gpu, why, n):
    """Keys that the bitmap form does not take."""
    rng = np.random.default_rng(n)
    m = 2_000
    keys = np.sort(rng.choice(5_000, m, replace=False)).astype(np.uint64) + 100
    if why == "repeated key":
        keys[7] = keys[8]
    elif why == "all repeated":
        keys[:] = keys[rng.integers(0, 9, m)]
    elif why == "wide range":
        keys[-1] = 1 << 31
    k = encoded_col(RESINT, keys)
    if why == "corrupt key":
        k.tail.data[5] ^= np.uint64(1 << 50)
    build = Bat(k.tail, oid_list(rng.permutation(m)).tail, m)
    probe = encoded_col(RESINT, rng.integers(0, 6_000, n, dtype=np.uint64))
    probe.tail.data[rng.integers(0, n, 9)] ^= np.uint64(1 << 40)
    kw = dict(reenc_head=1, ah1r=65117, ah1invr=0x3E36D3BC8D9BC5F5)
    check(gpu, "hashjoin_an", probe, build, side=HASH_RIGHT, **kw)
    check(gpu, "hashjoin_an", build.reverse(), probe.reverse(), side=HASH_LEFT, **kw)
    p = Bat(void_col(2), Col(INT, rng.integers(0, 6_000, n).astype(np.uint32)), n)
    q = Bat(Col(INT, keys.astype(np.uint32)), Col(OID, np.arange(m, dtype=np.uint32)), m)
    check(gpu, "hashjoin", p, q, side=HASH_RIGHT)
