"""Scans of 2^20 counts and more, which take a second launch: hash joins whose table
has as many slots, against the C restatement (build keys that repeat, around the
size at which the table doubles), and a join of 2^28 rows and more with a bitmap,
whose rows and error positions are computed with torch."""
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


@pytest.mark.parametrize("n", [(1 << 28) - 256, (1 << 28) + 777])
def test_many_tiles(n):
    import torch
    from ahead_b200.gpu import GpuOps
    from ahead_b200.model import RESOID, Col, an_meta, void_col
    g = GpuOps(0)
    m = an_meta(RESINT, None)
    v = torch.arange(n, device="cuda", dtype=torch.int64)
    v = v * 7919 % 1_000_003
    keep = v % 1000 == 1
    codes = v * m["A"]
    bad = torch.tensor([0, 4_095, 100_000_000, n - 1], device="cuda")
    codes[bad] ^= 1 << 62
    keep[bad] = False
    del v
    probe = Bat(void_col(0), Col(RESINT, codes.view(torch.uint8), m["A"], m["Ainv"], m["unenc_max"], 0), n)
    k = torch.arange(1001, device="cuda", dtype=torch.int64) * 1000 + 1
    mo = an_meta(RESOID, None)
    dim = Bat(Col(RESINT, (k * m["A"]).view(torch.uint8), m["A"], m["Ainv"], m["unenc_max"], 0),
              Col(RESOID, (torch.arange(1001, device="cuda") * mo["A"]).view(torch.uint8), mo["A"], mo["Ainv"],
                  mo["unenc_max"], 0), 1001)
    torch.cuda.synchronize()
    out, errs = g.hashjoin_an(probe, dim)
    want = torch.nonzero(keep).flatten()
    # (a flipped bit moves the decoded key, cut to 32 bits, by an even number: such a row may still join)
    head = out.head.data.view({4: torch.int32, 8: torch.int64}[out.head.data.numel() // out.count]).to(torch.int64)
    scale = 1 if int(head[-1]) < n else 65117
    mine = ~torch.isin(head // scale, bad)
    assert torch.equal((head // scale)[mine], want)
    e = errs[1].values.view(torch.int64)
    assert torch.equal(e, bad * 16089)
    g.close()
