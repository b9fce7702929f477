"""The merge matchjoin's tiles (256 rows of the first input against a stretch of
the second) against the C restatement: lengths around a tile and around one
block's 32 tiles, stretches that are empty, long or all of the second input,
key ranges far wider than the inputs, corrupt values, and keys out of order
(which replay the loop)."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits, oid_list
from cases import assert_same, run_case

from ahead_b200.model import (INT, OID, RESINT, RESOID, SHORTINT, Bat, Col, an_meta, void_col)

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


def keys(rng, n, lo, hi):
    return np.sort(rng.choice(hi - lo, n, replace=False)).astype(np.uint64) + np.uint64(lo)


SHAPES = [(1, 1, 0, 3, 0, 3), (255, 400, 0, 600, 0, 600), (256, 256, 0, 256, 0, 256), (257, 3, 0, 900, 0, 900),
          (8_192, 5_000, 0, 20_000, 0, 20_000), (8_193, 9_000, 0, 20_000, 0, 20_000),
          (20_000, 300, 0, 30_000, 29_000, 30_000),    # nearly every stretch is empty
          (300, 20_000, 29_000, 30_000, 0, 30_000),    # one long stretch ahead of the first tile
          (5_000, 5_000, 0, 10_000, 10_000, 20_000),   # nothing in common
          (5_000, 5_000, 10_000, 20_000, 0, 10_000),
          (9_000, 700, 0, 5_000_000, 0, 5_000_000)]


@pytest.mark.parametrize("n1,n2,lo1,hi1,lo2,hi2", SHAPES)
def test_encoded(gpu, n1, n2, lo1, hi1, lo2, hi2):
    rng = np.random.default_rng(n1 + n2)
    k1, k2 = keys(rng, n1, lo1, hi1), keys(rng, n2, lo2, hi2)
    k2[: min(n1, n2) // 2] = k2[: min(n1, n2) // 2]
    a, b = oid_list(k1), oid_list(k2)
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n1), Bat(b.tail, b.tail, n2))  # two selections, mirrored
    col = encoded_col(RESINT, rng.integers(0, 1 << 20, n2))
    other = oid_list(rng.integers(0, 1 << 20, n1)).tail
    check(gpu, "matchjoin_an", Bat(other, a.tail, n1), Bat(b.tail, col.tail, n2))
    flip_bits(col.tail.data, min(n2, 5), rng)
    flip_bits(other.data, min(n1, 5), rng)
    check(gpu, "matchjoin_an", Bat(other, a.tail, n1), Bat(b.tail, col.tail, n2))
    check(gpu, "matchjoin_an", Bat(other, a.tail, n1), Bat(b.tail, col.tail, n2), reenc=1, ah1r=16089,
          ah1invr=pow(16089, -1, 1 << 64), at2r=16089, at2invr=pow(16089, -1, 1 << 64))
    # a void list of the first input's rows against OIDs among them
    key = encoded_col(RESINT, rng.integers(0, 1 << 20, n1))
    rows = oid_list(keys(rng, max(1, n1 // 3), 0, n1))
    check(gpu, "matchjoin_an", Bat(key.tail, void_col(0), n1), Bat(rows.tail, rows.tail, rows.count))


@pytest.mark.parametrize("n1,n2,lo1,hi1,lo2,hi2", SHAPES)
def test_plain(gpu, n1, n2, lo1, hi1, lo2, hi2):
    rng = np.random.default_rng(n1)
    k1, k2 = keys(rng, n1, lo1, hi1).astype(np.uint32), keys(rng, n2, lo2, hi2).astype(np.uint32)
    a, b = Col(OID, k1), Col(OID, k2)
    check(gpu, "matchjoin", Bat(a, a, n1), Bat(b, b, n2))
    check(gpu, "matchjoin", Bat(Col(SHORTINT, rng.integers(0, 9, n1).astype(np.uint16)), a, n1),
          Bat(b, Col(INT, rng.integers(0, 1 << 30, n2).astype(np.uint32)), n2))
    key = Bat(Col(INT, rng.integers(0, 1 << 30, n1).astype(np.uint32)), void_col(0), n1)
    rows = Col(OID, keys(rng, max(1, n1 // 3), 0, n1).astype(np.uint32))
    check(gpu, "matchjoin", key, Bat(rows, rows, len(rows.data)))


@pytest.mark.parametrize("n", [2, 300, 9_000])
@pytest.mark.parametrize("where", ["first input", "second input", "a tie"])
def test_out_of_order(gpu, n, where):
    rng = np.random.default_rng(n)
    k1, k2 = keys(rng, n, 0, 3 * n), keys(rng, n, 0, 3 * n)
    (k1 if where != "second input" else k2)[n - 1] = 0 if where != "a tie" else k1[n - 2]
    a, b = oid_list(k1), oid_list(k2)
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n), Bat(b.tail, b.tail, n))
    p, q = Col(OID, k1.astype(np.uint32)), Col(OID, k2.astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n), Bat(q, q, n))


def test_corrupt_keys_in_order(gpu):
    """Keys whose largest value makes most of them read as corrupt: the loop's
    error positions, from the ordered form."""
    rng = np.random.default_rng(4)
    k1, k2 = keys(rng, 5_000, 0, 20_000), keys(rng, 4_000, 0, 20_000)
    for umax in (0, 10_000):
        a, b = oid_list(k1), oid_list(k2)
        a.tail.unenc_max = b.tail.unenc_max = umax
        check(gpu, "matchjoin_an", Bat(a.tail, a.tail, 5_000), Bat(b.tail, b.tail, 4_000))
