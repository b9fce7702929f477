"""Calls whose scratch is nearly all of the context's arena, against the C
restatement: dropped rows whose gaps take the arena up to its end together with
heads of which too many are corrupt for a list."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import RESINT, Bat

pytestmark = pytest.mark.gpu


@pytest.fixture
def gpu():
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)  # (its arena starts at 64 MiB)
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


@pytest.mark.parametrize("drops", [256, 697, 698, 715, 716])
def test_dropped_rows_and_corrupt_heads(gpu, drops):
    """12M rows of 16 bytes in 64 MiB: 5,860 chunks' edges of up to 715 rows fit,
    from 698 on without room for the check of the heads."""
    rng = np.random.default_rng(drops)
    n = 12_000_000
    heads = oid_list(np.arange(n)).tail
    oids = oid_list(rng.integers(0, 1 << 20, n)).tail
    corrupt(heads.data, rng.choice(n, 5_000, replace=False))
    corrupt(oids.data, rng.choice(n, drops, replace=False))
    check(gpu, "matchjoin_an", Bat(heads, oids, n), encoded_col(RESINT, rng.integers(0, 1 << 20, 1 << 20)))
