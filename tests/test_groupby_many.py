"""Group-bys through the first-row table whose first 4,096 rows open more than 1,024
groups, so that new groups past 4,096 are counted by the compaction, against the C
restatement: counts of groups around 4,096, the first rows all new or nearly so."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import INT, OID, RESINT, Bat, Col, void_col

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4_096, 4_100, 30_003])
@pytest.mark.parametrize("seed_groups", [1_024, 1_025, 4_096])
@pytest.mark.parametrize("more", [0, 1, 2_900, 3_071, 3_072, 20_000])
def test_many_groups(n, seed_groups, more):
    from ahead_b200.gpu import GpuOps, err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n + seed_groups + more)
    v = rng.integers(0, seed_groups, n)
    v[:seed_groups] = rng.permutation(seed_groups)  # the first 4,096 rows open exactly these
    if n > 4_096:
        rest = rng.integers(0, seed_groups + more, n - 4_096)
        new = np.arange(seed_groups, seed_groups + min(more, n - 4_096))
        rest[rng.permutation(n - 4_096)[: len(new)]] = new
        v[4_096:] = rest
    g = GpuOps(0)
    tail = encoded_col(RESINT, v)
    tail.tail.data[[7, n - 1]] ^= np.uint64(1)  # (reported, and small groups of their own)
    plain = Bat(void_col(0), Col(INT, v.astype(np.uint32)), n)
    two = rng.integers(0, 2, n)
    for op, args in (("groupby_an", [tail]), ("groupby", [plain]), ("groupby2_an", [tail, oid_list(two), 2]),
                     ("groupby2", [plain, Bat(void_col(0), Col(OID, two.astype(np.uint32)), n), 2])):
        c = dict(op=op, args=args, kwargs={})
        assert_same(run_case(g, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), op)
    g.close()
