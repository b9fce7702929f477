"""arithmeticAN and the grouped sums in one pass against the C restatement:
lengths around a pair, a thread's and the grid's rows; every pair of operand
widths; operands that are not aligned to a pair; no, a few, 4,096 and 4,097
corrupt codes; group counts around the shared-memory copies and beyond them,
and corrupt group ids."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import (ADD, BIGINT, DIV, INT, MUL, OID, RESBIGINT, RESINT, RESSHORT, RESTINY, SUB, Bat, Col, ainv,
                              void_col)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)
    yield g
    g.close()


def check(gpu, op, *args, shift=0):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle

    def dev(b):  # on the device, `shift` rows into a longer column
        d = to_device(b)
        if shift and d.tail.data is not None:
            w = d.tail.data.numel() // b.count
            longer = gpu.torch.zeros(d.tail.data.numel() + shift * w, dtype=gpu.torch.uint8, device="cuda")
            longer[shift * w:] = d.tail.data
            d.tail.data = longer[shift * w:]
        return d
    c = dict(op=op, args=list(args), kwargs={})
    assert_same(run_case(gpu, c, dev, to_host, err_to_host), run_case(Oracle("port"), c), op)


def corrupt(b, rows):
    t = b.tail.data
    t[rows] ^= t.dtype.type(1) << t.dtype.type(t.dtype.itemsize * 8 - 1)


HIGH = {RESTINY: 200, RESSHORT: 50_000, RESINT: 10_000_000, RESBIGINT: 1 << 40}


def column(rng, t, n, flips, lo=0):
    b = encoded_col(t, rng.integers(lo, HIGH[t], n), A=65117 if t == RESBIGINT else None)
    corrupt(b, rng.choice(n, min(flips, n), replace=False))
    return b


@pytest.mark.parametrize("t1", [RESTINY, RESSHORT, RESINT])
@pytest.mark.parametrize("t2", [RESTINY, RESSHORT, RESINT])
@pytest.mark.parametrize("shift", [0, 1])
def test_arithmetic(gpu, t1, t2, shift):
    rng = np.random.default_rng(t1 * 16 + t2)
    for n in (1, 2, 3, 7, 8, 9, 2047, 2049, 100_001):
        a, b = column(rng, t1, n, 3), column(rng, t2, n, 2, lo=1)
        for op, rt in ((ADD, RESINT), (SUB, RESBIGINT), (MUL, RESBIGINT), (DIV, RESBIGINT)):
            check(gpu, "arithmetic_an", op, rt, a, b, 65117, ainv(65117, 64), shift=shift)


@pytest.mark.parametrize("f1,f2", [(0, 0), (4096, 0), (4097, 1), (1, 4097), (5000, 5000)])
def test_arithmetic_flips(gpu, f1, f2):
    rng = np.random.default_rng(f1 + f2)
    n = 148 * 16 * 256 * 8 + 2_005  # (a second round of the grid's loop)
    a, b = column(rng, RESINT, n, f1), column(rng, RESTINY, n, f2)
    check(gpu, "arithmetic_an", MUL, RESBIGINT, a, b, 65117, ainv(65117, 64))


def groups(rng, n, ngroups, flips):
    b = oid_list(rng.integers(0, ngroups, n, dtype=np.uint64))
    corrupt(b, rng.choice(n, min(flips, n), replace=False))
    return b


@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT, RESBIGINT])
@pytest.mark.parametrize("ngroups", [1, 2, 7, 33, 128, 129, 280, 2048, 2049, 4096, 4097, 60_000])
def test_grouped_sum(gpu, t, ngroups):
    rng = np.random.default_rng(ngroups + t)
    for n, shift in ((1, 0), (2, 0), (9, 1), (4_097, 0), (200_003, 1)):
        check(gpu, "aggregate_sum_grouped_an", column(rng, t, n, 3), groups(rng, n, ngroups, 2), ngroups, shift=shift)


@pytest.mark.parametrize("f1,f2", [(0, 0), (4096, 4096), (4097, 0), (0, 4097), (9000, 9000)])
def test_grouped_sum_flips(gpu, f1, f2):
    rng = np.random.default_rng(f1 + 3 * f2)
    n = 148 * 6 * 256 * 16 + 4_099
    check(gpu, "aggregate_sum_grouped_an", column(rng, RESBIGINT, n, f1), groups(rng, n, 280, f2), 280)


@pytest.mark.parametrize("ngroups", [1, 40, 4096, 4097])
@pytest.mark.parametrize("shift", [0, 1])
def test_plain_grouped_sum(gpu, ngroups, shift):
    rng = np.random.default_rng(ngroups)
    for n in (1, 2, 8_193, 300_001):
        a = Bat(void_col(0), Col(INT, rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)), n)
        g = Bat(void_col(0), Col(OID, rng.integers(0, ngroups, n, dtype=np.uint64).astype(np.uint32)), n)
        check(gpu, "aggregate_sum_grouped", a, g, ngroups, BIGINT, shift=shift)
