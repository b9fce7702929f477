"""The compaction's tile sizes against the C restatement where they change: a
short tile (256 rows; 512 of one-byte codes), what one block takes (32 short
tiles), the first length in long tiles (2^23 rows), one row to either side of
each, columns that start off a 16-byte boundary, and no, all and few rows kept."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits
from cases import assert_same, run_case

from ahead_b200.model import (AND, EQ, GE, GT, INT, LE, LT, OR, RESINT, RESOID, RESSHORT, RESTINY, SHORTINT, TINYINT,
                              NP_DTYPE, WIDTH, Bat, Col, an_meta, void_col)

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


def device_view(gpu, b, offset):
    """The BAT without its first `offset` rows, as a view into the device column."""
    from ahead_b200.gpu import to_device
    d = to_device(b)
    w = WIDTH[b.tail.type]
    t = d.tail
    t = Col(t.type, t.data[offset * w:], t.A, t.Ainv, t.unenc_max, t.seqbase)
    return Bat(d.head, t, b.count - offset)


@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 8191, 8192, 8193, 8449, (1 << 23) - 1, 1 << 23, (1 << 23) + 1025])
def test_select_an(gpu, t, n):
    rng = np.random.default_rng(n)
    b = encoded_col(t, rng.integers(0, 200, n), seqbase=5)
    flip_bits(b.tail.data, min(n // 4, 40), rng)
    A = b.tail.A
    check(gpu, "select_an", b, GE, 20 * A, LE, 60 * A, AND)
    if n < 10_000:
        check(gpu, "select_an", b, GE, 0)                      # every row
        check(gpu, "select_an", b, EQ, 250 * A)                # none
        check(gpu, "select_an", b, LT, 3 * A, GT, 190 * A, OR)


@pytest.mark.parametrize("n", [511, 512, 513, 16383, 16384, 16385, (1 << 23) + 7])
def test_select_bytes(gpu, n):
    rng = np.random.default_rng(n)
    b = Bat(void_col(3), Col(TINYINT, rng.integers(0, 256, n).astype(np.uint8)), n)
    check(gpu, "select", b, GE, 10, LE, 99, AND)


@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT])
@pytest.mark.parametrize("offset", [1, 3])
@pytest.mark.parametrize("n", [300, 20_000, (1 << 23) + 300])
def test_unaligned_select(gpu, t, offset, n):
    from ahead_b200.gpu import err_to_host, to_host
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n + offset)
    b = encoded_col(t, rng.integers(0, 200, n))
    flip_bits(b.tail.data, 20, rng)
    A = b.tail.A
    out, err = gpu.select_an(device_view(gpu, b, offset), GE, 20 * A, LE, 60 * A, AND)
    c = b.tail
    h = Bat(b.head, Col(c.type, c.data[offset:], c.A, c.Ainv, c.unenc_max, c.seqbase), n - offset)
    exp, eerr = Oracle("port").select_an(h, GE, 20 * A, LE, 60 * A, AND)
    assert_same([to_host(out), err_to_host(err)], [exp, eerr], "unaligned selectAN")


@pytest.mark.parametrize("n", [257, 9_000, 300_001, (1 << 23) + 5])
def test_several_streams(gpu, n):
    """checkAndDecodeAN with an encoded head: three streams, the sparse ones in a few tiles."""
    rng = np.random.default_rng(n)
    m = an_meta(RESOID)
    heads = np.arange(n, dtype=np.uint64) * np.uint64(m["A"])
    b = encoded_col(RESSHORT, rng.integers(0, 60_000, n))
    flip_bits(heads, 30, rng)
    flip_bits(b.tail.data, 30, rng)
    check(gpu, "check_and_decode_an", Bat(Col(RESOID, heads, m["A"], m["Ainv"], m["unenc_max"], 0), b.tail, n))
