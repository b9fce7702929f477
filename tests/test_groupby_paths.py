"""The group-by's first-row table against the C restatement where it can go
wrong: around the seed block's 4,096 rows, the 4,096 groups one block ranks,
the table's key limit (2^16 words for small inputs; keys at it take the hash
table), corrupt codes in every column, past the 4,096 listed, and odd heads."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits
from cases import assert_same, run_case

from ahead_b200.model import (INT, OID, RESINT, RESOID, RESSHORT, RESTINY, SHORTINT, NP_DTYPE, WIDTH, Bat, Col,
                              an_meta, void_col)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)
    yield g
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    assert_same(run_case(gpu, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), op)


def _groups(rng, n, count, lo=0):
    """n values over `count` different ones, each present, in random order."""
    v = rng.integers(0, count, n)
    v[rng.permutation(n)[:count]] = np.arange(count)
    return (v + lo).astype(np.uint64)


def _gids(v, A=65117):
    m = an_meta(RESOID, A)
    return Bat(void_col(0), Col(RESOID, v.astype(np.uint64) * np.uint64(A), A, m["Ainv"], m["unenc_max"], 0), len(v))


@pytest.mark.parametrize("n,count,lo", [(1, 1, 0), (5, 3, 1992), (4095, 7, 0), (4096, 4096, 0), (4097, 40, 1992),
                                        (4099, 4097, 0), (20_003, 4096, 61_440), (20_003, 4097, 0),
                                        (50_001, 16_000, 49_000)])
@pytest.mark.parametrize("flips", [0, 3])
def test_unary(gpu, n, count, lo, flips):
    rng = np.random.default_rng(n + count)
    b = encoded_col(RESSHORT, _groups(rng, n, count, lo), seqbase=11)
    flip_bits(b.tail.data, min(flips, n), rng)
    check(gpu, "groupby_an", b)
    v = _groups(rng, n, count, lo)
    check(gpu, "groupby", Bat(void_col(3), Col(SHORTINT, v.astype(np.uint16)), n))


@pytest.mark.parametrize("t", [RESTINY, RESINT])
def test_unary_types_and_heads(gpu, t):
    rng = np.random.default_rng(t)
    n = 9_001
    b = encoded_col(t, _groups(rng, n, 200))
    flip_bits(b.tail.data, 5, rng)
    m = an_meta(RESOID)
    heads = (rng.integers(0, 1 << 20, n).astype(np.uint64) * np.uint64(m["A"]))
    flip_bits(heads, 4, rng)
    check(gpu, "groupby_an", Bat(Col(RESOID, heads, m["A"], m["Ainv"], m["unenc_max"], 0), b.tail, n))
    check(gpu, "groupby_an", Bat(Col(OID, rng.integers(0, 1 << 30, n).astype(np.uint32)), b.tail, n))
    check(gpu, "groupby", Bat(void_col(0), Col(t, b.tail.data), n))  # the raw codes: mostly past the table


@pytest.mark.parametrize("n,first,second,lo,aoid", [
    (280, 7, 40, 0, 65117), (12_001, 7, 40, 0, 65117), (30_001, 40, 7, 1992, 65117),  # 1998 * 40 + 39: past 2^16
    (4_097, 64, 64, 0, 65117), (65_539, 65, 64, 0, 65117), (70_003, 256, 256, 0, 1), (40_001, 300, 250, 0, 65117)])
@pytest.mark.parametrize("flips", [0, 4])
def test_binary(gpu, n, first, second, lo, aoid, flips):
    rng = np.random.default_rng(n + second)
    g = _gids(_groups(rng, n, first))
    b = encoded_col(RESSHORT, _groups(rng, n, second, lo))
    flip_bits(b.tail.data, flips, rng)
    flip_bits(g.tail.data, flips, rng)
    check(gpu, "groupby2_an", b, g, first, aoid=aoid, aoidinv=pow(aoid, -1, 1 << 64))
    check(gpu, "groupby2", Bat(void_col(0), Col(SHORTINT, _groups(rng, n, second, lo).astype(np.uint16)), n),
          Bat(void_col(0), Col(OID, _groups(rng, n, first).astype(np.uint32)), n), first)


def test_binary_codes_wider_than_an_oid(gpu):
    """Group codes at or above 2^32 (a large A): the dictionary's oid_t keeps
    only the first row's upper half."""
    rng = np.random.default_rng(3)
    n, A = 9_000, (1 << 31) + 1
    b = encoded_col(RESSHORT, _groups(rng, n, 30))
    check(gpu, "groupby2_an", b, _gids(_groups(rng, n, 5)), 5, aoid=A, aoidinv=pow(A, -1, 1 << 64))


@pytest.mark.parametrize("bad", [4096, 4097, 6000])
def test_many_corrupt_codes(gpu, bad):
    """A corrupt code whose decoded value still fits the table: the lists and,
    past 4,096 entries, the compaction."""
    rng = np.random.default_rng(bad)
    n = 12_345
    b = encoded_col(RESTINY, _groups(rng, n, 100))
    flip_bits(b.tail.data, bad, rng)
    check(gpu, "groupby_an", b)
    g = _gids(_groups(rng, n, 5))
    g.tail.unenc_max = 1  # most group ids read as corrupt, and stay small
    check(gpu, "groupby2_an", encoded_col(RESSHORT, _groups(rng, n, 50)), g, 5)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_unaligned_columns(gpu, offset):
    rng = np.random.default_rng(offset)
    n = 8_500
    for t, u in ((RESSHORT, None), (RESINT, None), (INT, INT)):
        b = encoded_col(RESSHORT if t == RESSHORT else RESINT, _groups(rng, n, 60))
        if u is not None:
            col = Col(INT, _groups(rng, n, 60).astype(np.uint32))
            check(gpu, "groupby", Bat(void_col(0), Col(INT, col.data[offset:]), n - offset))
            continue
        c = b.tail
        check(gpu, "groupby_an", Bat(void_col(0), Col(c.type, c.data[offset:], c.A, c.Ainv, c.unenc_max), n - offset))
