"""Group-bys through the hash table, whose insert pass takes the columns' checks
along, against the C restatement: a wide key among the seed rows, behind them and
in the last row; no, a few and too many corrupt codes for a list; one row a
thread and, from 2^22 rows on, four; and the key that marks empty slots."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits, oid_list
from cases import assert_same, run_case

from ahead_b200.model import INT, OID, RESINT, RESOID, Bat, Col, an_meta, void_col

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


def keys(rng, n, how):
    v = rng.integers(0, 50, n).astype(np.uint64)
    if how == "all":
        return v * np.uint64(80_003_001)
    if how == "many":
        return rng.integers(0, n, n).astype(np.uint64) + np.uint64(1 << 30)
    v[{"seed": min(7, n - 1), "behind": min(5_000, n - 1), "last": n - 1}[how]] = 1 << 31
    return v


@pytest.mark.parametrize("n", [1, 4_096, 4_097, 20_003])
@pytest.mark.parametrize("how", ["all", "many", "seed", "behind", "last"])
@pytest.mark.parametrize("flips", [0, 9, 6_000])
def test_wide(gpu, n, how, flips):
    rng = np.random.default_rng(n + flips)
    v = keys(rng, n, how)
    b = encoded_col(RESINT, v, seqbase=3)
    flip_bits(b.tail.data, min(flips, n), rng)
    check(gpu, "groupby_an", b)
    grp = oid_list(rng.integers(0, 5, n))
    flip_bits(grp.tail.data, min(flips, n), rng)
    check(gpu, "groupby2_an", b, grp, 5)
    heads = oid_list(rng.integers(0, 1 << 20, n)).tail
    flip_bits(heads.data, min(flips, n), rng)
    check(gpu, "groupby_an", Bat(heads, b.tail, n))
    plain = Bat(void_col(1), Col(INT, v.astype(np.uint32)), n)
    check(gpu, "groupby", plain)
    check(gpu, "groupby2", plain, Bat(void_col(0), Col(OID, rng.integers(0, 5, n).astype(np.uint32)), n), 5)


@pytest.mark.parametrize("n", [(1 << 22) - 1, 1 << 22, (1 << 22) + 2_500_001])
def test_four_rows_a_thread(gpu, n):
    rng = np.random.default_rng(n)
    b = encoded_col(RESINT, rng.integers(0, 60_000, n).astype(np.uint64) * np.uint64(70_001))
    flip_bits(b.tail.data, 20, rng)
    check(gpu, "groupby_an", b)
    grp = oid_list(rng.integers(0, 5, n))
    flip_bits(grp.tail.data, 20, rng)
    check(gpu, "groupby2_an", b, grp, 5)
    check(gpu, "groupby", Bat(void_col(1), Col(INT, rng.integers(0, 1 << 32, n).astype(np.uint32)), n))


def test_the_empty_mark_as_a_key(gpu):
    rng = np.random.default_rng(1)
    n = 9_000
    raw = rng.integers(0, 40, n).astype(np.uint64) * np.uint64(1 << 40)
    raw[rng.integers(0, n, 200)] = np.uint64(0xFFFFFFFFFFFFFFFF)
    m = an_meta(RESOID)
    check(gpu, "groupby", Bat(void_col(0), Col(RESOID, raw, m["A"], m["Ainv"], m["unenc_max"], 0), n))
