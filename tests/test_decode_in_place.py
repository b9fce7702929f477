"""checkAndDecodeAN from 2^22 rows on decodes every row in place and closes the
gaps of the corrupt ones, 1- and 2-byte values by 32-bit words: the lengths
around that line and around the chunks (8,192 and 16,384 rows), with corrupt
rows at both ends, alone, adjacent, at chunk edges, and more than the list
holds; against the arithmetic itself."""
import numpy as np
import pytest

from bats import encoded_col

from ahead_b200.model import NP_DTYPE, RESBIGINT, RESINT, RESSHORT, RESTINY, UNENCODED_TYPE, WIDTH

pytestmark = pytest.mark.gpu

N = 1 << 22


@pytest.fixture(scope="module")
def gpu():
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)
    yield g
    g.close()


def rows_of(how, n, rng):
    return np.array({"none": [], "first": [0], "last": [n - 1], "two": [1, 2], "odd": [5, 6, 9, 8191, 8193],
                     "edges": [r for c in range(8192, n, 8192 * 9) for r in (c - 1, c, c + 1) if r < n],
                     "ends": [0, 1, 2, n - 3, n - 2, n - 1],
                     "512": np.sort(rng.choice(n, 512, replace=False)),
                     "513": np.sort(rng.choice(n, 513, replace=False)),
                     "many": np.sort(rng.choice(n, 2048, replace=False)),
                     "too many": np.sort(rng.choice(n, 2049, replace=False))}[how], np.int64)


@pytest.mark.parametrize("n", [N - 1, N, N + 1, N + 8191, N + 16385])
@pytest.mark.parametrize("how", ["none", "first", "last", "two", "odd", "edges", "ends", "512", "513", "many", "too many"])
@pytest.mark.parametrize("t", [RESTINY, RESSHORT, RESINT, RESBIGINT])
def test_decode(gpu, t, how, n):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    if t == RESBIGINT and n not in (N - 1, N + 1):
        pytest.skip("eight-byte values take the row path: two lengths do")
    rng = np.random.default_rng(n)
    bad = rows_of(how, n, rng)
    ut = UNENCODED_TYPE[t]
    v = rng.integers(0, 200, n)
    b = encoded_col(t, v, A=65117 if t == RESBIGINT else None)
    code = b.tail.data
    code[bad] ^= code.dtype.type(1) << code.dtype.type(code.dtype.itemsize * 8 - 1)  # (always detected)
    out, _, err = gpu.check_and_decode_an(to_device(b), aoid=16089)
    got = to_host(out)
    keep = np.ones(n, bool)
    keep[bad] = False
    assert got.tail.type == ut and got.count == n - len(bad)
    assert np.array_equal(got.tail.data, v[keep].astype(NP_DTYPE[WIDTH[ut]]))
    e = err_to_host(err)
    assert np.array_equal(np.asarray(e.values, np.uint64), bad.astype(np.uint64) * np.uint64(16089))
