"""Hash joins whose table has 2^20 slots and more, where the scan of the slots'
counts takes a second launch, against the C restatement: build keys that repeat,
around the size at which the table doubles."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import HASH_LEFT, HASH_RIGHT, RESINT, Bat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 19) - 1, 1 << 19, (1 << 19) + 1, 1_100_003])
@pytest.mark.parametrize("side", [HASH_RIGHT, HASH_LEFT])
def test_repeated_keys(nb, side):
    from ahead_b200.gpu import GpuOps, err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    rng = np.random.default_rng(nb)
    g = GpuOps(0)
    build = rng.integers(0, nb, nb)  # (a third of the range does not occur, a quarter repeats)
    probe = encoded_col(RESINT, rng.integers(0, nb, 5_003))
    keys = encoded_col(RESINT, build)
    if side == HASH_RIGHT:
        args = [probe, Bat(keys.tail, oid_list(np.arange(nb)).tail, nb)]
    else:
        args = [keys, Bat(probe.tail, oid_list(np.arange(5_003)).tail, 5_003)]
    c = dict(op="hashjoin_an", args=args, kwargs=dict(side=side))
    assert_same(run_case(g, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), "hashjoin_an")
    g.close()
