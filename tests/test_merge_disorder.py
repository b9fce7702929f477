"""The merge matchjoin on keys out of order, which replays the loop, against the
C restatement: disorder where a tile of 256 rows starts and inside a tile's
stretch of the second input, by a corrupt code or by the list's own order, in
either input, with mirrored and separate value columns, below and above one
block's 32 tiles, with output columns given and allocated by the call."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import INT, OID, RESINT, Bat, Col

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[False, True], ids=["given", "sized"])
def gpu(request, monkeypatch):
    import ahead_b200.gpu as mirror
    if request.param:
        monkeypatch.setattr(mirror, "_SIZED_BYTES", 0)
    g = mirror.GpuOps(0)
    yield g
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    assert_same(run_case(gpu, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), op)


def disorder(how, k1, k2, rng):
    n = len(k1)
    if " row " in how:  # one key far above the rest
        which, row = how.split(" row ")
        (k1 if which == "first" else k2)[min(int(row), n - 1)] = 1 << 30
    elif how == "first descending":
        k1[:] = k1[::-1].copy()
    elif how == "first shuffled":
        rng.shuffle(k1)
    elif how == "second descending":
        k2[:] = k2[::-1].copy()
    elif how == "second shuffled":
        rng.shuffle(k2)
    elif how == "second swapped":
        for r in range(10, n - 1, 97):
            k2[[r, r + 1]] = k2[[r + 1, r]]


HOWS = ["first row 0", "first row 255", "first row 256", "first row 512", "first row 8192", "second row 0",
        "second row 256", "second row 700", "first descending", "first shuffled", "second descending",
        "second shuffled", "second swapped"]


@pytest.mark.parametrize("n", [300, 1024, 9_000])
@pytest.mark.parametrize("how", HOWS)
def test_disorder(gpu, n, how):
    rng = np.random.default_rng(n)
    k1 = np.sort(rng.choice(2 * n, n, replace=False)).astype(np.uint64)
    k2 = np.sort(rng.choice(2 * n, n, replace=False)).astype(np.uint64)
    disorder(how, k1, k2, rng)
    a, b = oid_list(k1), oid_list(k2)
    value = encoded_col(RESINT, rng.integers(0, 1 << 20, n)).tail
    other = oid_list(rng.integers(0, 1 << 20, n)).tail
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n), Bat(b.tail, b.tail, n))
    check(gpu, "matchjoin_an", Bat(other, a.tail, n), Bat(b.tail, value, n))
    p, q = Col(OID, k1.astype(np.uint32)), Col(OID, k2.astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n), Bat(q, q, n))
    plain = Col(INT, rng.integers(0, 1 << 30, n).astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n), Bat(q, plain, n))


@pytest.mark.parametrize("n", [300, 1024, 9_000])
@pytest.mark.parametrize("row", [0, 255, 256, 512, 8_192])
@pytest.mark.parametrize("bit", [0, 40, 63])
def test_flipped_code(gpu, n, row, bit):
    """One flipped bit of an OID code."""
    rng = np.random.default_rng(bit)
    for which in (0, 1):
        lists = [oid_list(np.sort(rng.choice(2 * n, n, replace=False))) for _ in range(2)]
        lists[which].tail.data[min(row, n - 1)] ^= np.uint64(1) << np.uint64(bit)
        a, b = lists
        value = encoded_col(RESINT, rng.integers(0, 1 << 20, n)).tail
        check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n), Bat(b.tail, b.tail, n))
        check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n), Bat(b.tail, value, n))
