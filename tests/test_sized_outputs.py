"""Output columns allocated once the call knows its count (what the Python
mirror asks for where an output may be large) against the C restatement, at
small sizes: selections, joins and merges, with corrupt rows, nothing kept,
everything kept, and the calls that cannot be sized (repeated keys, unordered
inputs), which run again with the count they reported."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits, oid_list
from cases import assert_same, run_case

from ahead_b200.model import (AND, EQ, GE, HASH_LEFT, HASH_RIGHT, INT, LE, OID, RESINT, RESOID, RESSHORT, RESTINY,
                              SHORTINT, TINYINT, Bat, Col, void_col)

pytestmark = pytest.mark.gpu
AR, ARI = 65117, 0x3E36D3BC8D9BC5F5


@pytest.fixture
def gpu(monkeypatch):
    import ahead_b200.gpu as mirror
    monkeypatch.setattr(mirror, "_SIZED_BYTES", 0)
    g = mirror.GpuOps(0)
    yield g
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    assert_same(run_case(gpu, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), op)


@pytest.mark.parametrize("n", [0, 1, 300, 9_000, 70_001, (1 << 23) + 77])
def test_select(gpu, n):
    rng = np.random.default_rng(n)
    for t in (RESTINY, RESSHORT, RESINT):
        b = encoded_col(t, rng.integers(0, 200, n), seqbase=5)
        flip_bits(b.tail.data, min(n, 20), rng)
        A = b.tail.A
        check(gpu, "select_an", b, GE, 20 * A, LE, 60 * A, AND)
        if n < 10_000:
            check(gpu, "select_an", b, GE, 0)
            check(gpu, "select_an", b, EQ, 250 * A)
    check(gpu, "select", Bat(void_col(3), Col(TINYINT, rng.integers(0, 256, n).astype(np.uint8)), n), GE, 10, LE, 99)


@pytest.mark.parametrize("side", [HASH_RIGHT, HASH_LEFT])
@pytest.mark.parametrize("repeated", [False, True])
@pytest.mark.parametrize("n", [200, 20_001])
def test_hashjoin(gpu, side, repeated, n):
    rng = np.random.default_rng(n)
    keys = np.sort(rng.choice(5_000, 2_000, replace=False)).astype(np.uint64) + 100
    if repeated:
        keys[7] = keys[8]
    k = encoded_col(RESINT, keys)
    build = Bat(k.tail, oid_list(rng.permutation(2_000)).tail, 2_000)
    probe = encoded_col(RESINT, rng.integers(0, 6_000, n, dtype=np.uint64))
    flip_bits(probe.tail.data, 9, rng)
    kw = dict(reenc_head=1, ah1r=AR, ah1invr=ARI, side=side)
    if side == HASH_RIGHT:
        check(gpu, "hashjoin_an", probe, build, **kw)
        none = encoded_col(RESINT, rng.integers(6_000, 9_000, n, dtype=np.uint64))
        check(gpu, "hashjoin_an", none, build, **kw)
    else:
        check(gpu, "hashjoin_an", build.reverse(), probe.reverse(), **kw)
    p = Bat(void_col(2), Col(INT, rng.integers(0, 6_000, n).astype(np.uint32)), n)
    q = Bat(Col(INT, keys.astype(np.uint32)), Col(OID, np.arange(2_000, dtype=np.uint32)), 2_000)
    check(gpu, "hashjoin", p, q, side=HASH_RIGHT)


@pytest.mark.parametrize("n1,n2", [(0, 5), (40, 30), (9_000, 4_000), (70_000, 60_000)])
@pytest.mark.parametrize("ordered", [True, False])
def test_merge(gpu, n1, n2, ordered):
    rng = np.random.default_rng(n1)
    k1 = np.sort(rng.choice(150_000, n1, replace=False)).astype(np.uint64)
    k2 = np.sort(rng.choice(150_000, n2, replace=False)).astype(np.uint64)
    if not ordered:
        if n1 > 9_000:
            return  # (the replayed loop is one thread)
        k2[-1] = 0
    a, b = oid_list(k1), oid_list(k2)
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n1), Bat(b.tail, b.tail, n2))
    heads = oid_list(rng.integers(0, 1 << 20, n1)).tail
    heads.unenc_max = 0  # every head reads as corrupt
    check(gpu, "matchjoin_an", Bat(heads, a.tail, n1), Bat(b.tail, b.tail, n2))
    p, q = Col(OID, k1.astype(np.uint32)), Col(OID, k2.astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n1), Bat(q, q, n2))
