"""Operators that write every row in place and close the gaps of the few rows
they drop (checkAndDecodeAN, the positional matchjoinAN and fetchjoinAN, their
unencoded twins) against the C restatement: no, one, a few, 512, 2,048 and more
dropped rows; at both ends, next to each other, and around the chunks of 2,048
and 4,096 rows the gaps are closed in; both kinds of dropped row; every width."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits, oid_list
from cases import assert_same, run_case

from ahead_b200.model import (INT, OID, RESBIGINT, RESINT, RESOID, RESSHORT, RESTINY, SHORTINT, NP_DTYPE, WIDTH, Bat,
                              Col, an_meta, void_col)

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


def corrupt(arr, rows):
    """The highest bit of each row's code: always detected."""
    arr[rows] ^= arr.dtype.type(1) << arr.dtype.type(arr.dtype.itemsize * 8 - 1)


def places(rng, n, how):
    return {"none": [], "first": [0], "last": [n - 1], "ends": [0, 1, 2, n - 2, n - 1],
            "chunks": [r for c in range(0, n, 2048) for r in (c - 1, c, c + 1) if 0 <= r < n],
            "run": list(range(2040, 2055)) + list(range(4090, 4105)),
            "512": rng.choice(n, 512, replace=False), "2048": rng.choice(n, 2048, replace=False),
            "2049": rng.choice(n, 2049, replace=False), "block": list(range(5000, 5000 + 2048))}[how]


HOWS = ["none", "first", "last", "ends", "chunks", "run", "512", "2048", "2049", "block"]


@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT, RESBIGINT])
@pytest.mark.parametrize("how", HOWS)
def test_decode(gpu, t, how):
    rng = np.random.default_rng(t)
    n = 30_003
    b = encoded_col(t, rng.integers(0, 200, n), A=65117 if t == RESBIGINT else None)
    corrupt(b.tail.data, places(rng, n, how))
    check(gpu, "check_and_decode_an", b)


@pytest.mark.parametrize("n", [1, 3, 15, 17, 4095, 4096, 4097, 1_000_003])
def test_decode_lengths(gpu, n):
    rng = np.random.default_rng(n)
    for t in (RESTINY, RESSHORT, RESINT):
        b = encoded_col(t, rng.integers(0, 200, n))
        flip_bits(b.tail.data, min(n, 7), rng)
        check(gpu, "check_and_decode_an", b)


def _list(rng, n, size):
    return oid_list(np.sort(rng.choice(size, n, replace=size < n)))


@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT])
@pytest.mark.parametrize("how", HOWS)
def test_positional(gpu, t, how):
    rng = np.random.default_rng(t + 1)
    n, size = 20_011, 61_000
    col = encoded_col(t, rng.integers(0, 200, size))
    o = _list(rng, n, size)
    oids = o.tail.data // np.uint64(65117)
    rows = np.array(places(rng, n, how), dtype=np.int64)
    corrupt(col.tail.data, oids[rows[: len(rows) // 2]].astype(np.int64))  # half: corrupt values
    for r in rows[len(rows) // 2:]:                                        # half: OIDs past the column
        o.tail.data[r] = np.uint64(size + int(r)) * np.uint64(65117)
    check(gpu, "matchjoin_an", Bat(o.tail, o.tail, n), col)  # a mirrored list
    heads = oid_list(rng.integers(0, 1 << 24, n)).tail
    flip_bits(heads.data, 5, rng)
    check(gpu, "matchjoin_an", Bat(heads, o.tail, n), col)
    check(gpu, "matchjoin_an", Bat(Col(RESOID, heads.data, heads.A, heads.Ainv, 0, 0), o.tail, n), col)
    A2 = {RESTINY: 29, RESSHORT: 7785, RESINT: 16089}[t]
    inv = pow(A2, -1, 1 << (8 * WIDTH[t]))
    check(gpu, "matchjoin_an", Bat(heads, o.tail, n), col, reenc=1, ah1r=16089, ah1invr=pow(16089, -1, 1 << 64),
          at2r=A2, at2invr=inv)
    check(gpu, "fetchjoin_an", o, col)
    check(gpu, "fetchjoin_an", o, col, reenc=1, atr=A2, atrinv=inv)


@pytest.mark.parametrize("how", HOWS)
def test_unencoded_positional(gpu, how):
    rng = np.random.default_rng(5)
    n, size = 20_011, 61_000
    oids = np.sort(rng.choice(size, n, replace=False)).astype(np.uint32)
    oids[places(rng, n, how)] = 70_000
    col = Bat(void_col(0), Col(SHORTINT, rng.integers(0, 60_000, size).astype(np.uint16)), size)
    lst = Bat(Col(OID, rng.integers(0, 1 << 30, n).astype(np.uint32)), Col(OID, oids), n)
    check(gpu, "matchjoin", lst, col)
    check(gpu, "fetchjoin", Bat(void_col(0), lst.tail, n), col)


def test_positional_into_one_row(gpu):
    rng = np.random.default_rng(8)
    o = oid_list(rng.integers(0, 3, 9_000))
    check(gpu, "matchjoin_an", Bat(o.tail, o.tail, 9_000), encoded_col(RESINT, [5]))
    check(gpu, "matchjoin_an", Bat(o.tail, o.tail, 9_000), encoded_col(RESINT, []))
