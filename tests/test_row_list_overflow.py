"""The per-row strategy's row lists when the third filter keeps nearly every
listed row, so that its list overflows and the per-row pass takes the one before
it: the estimates expect uniform attribute values, and here nearly all rows hold
one value.  With and without corrupt codes in the columns the filters read."""
import pytest

pytestmark = pytest.mark.gpu

N = 14_000_003  # half of it, and the lists' chunk ends, stay below what is listed


def one_value(bat, value):
    """Every row of a dimension attribute but the first eight holds `value`."""
    import torch
    from ahead_b200.model import WIDTH
    w = WIDTH[bat.tail.type]
    code = (value * bat.tail.A) & ((1 << (8 * w)) - 1)
    raw = torch.tensor(list(code.to_bytes(w, "little")), dtype=torch.uint8, device=bat.tail.data.device)
    bat.tail.data.view(-1, w)[8:] = raw


@pytest.mark.parametrize("columns", [(), ("partkey",), ("custkey", "suppkey", "partkey", "revenue")])
def test_third_list_overflows(columns):
    import torch
    from ahead_b200.gpu import GpuOps, err_to_host, to_host
    from ahead_b200.pipelines import starjoin_continuous
    from ahead_b200.ssb import flip_device, generate_device
    from ahead_b200.ssb_programs import program_query
    from ahead_b200.starjoin import StarJoinEngine
    from test_programs import _fused_equal
    g = GpuOps(0)
    ds = generate_device(dict(fact=N, date=2556, customer=300_000, part=200_000, supplier=20_000), seed=3)
    for dim, attr in (("customer", "region"), ("supplier", "region"), ("part", "mfgr")):
        one_value(ds.tables[dim][attr], 1)
    if columns:
        flip_device(ds, 300 * len(columns), 11, columns=columns)
    torch.cuda.synchronize()
    eng = StarJoinEngine(g, ds)
    q = program_query("q41")
    for r in eng.run([q]) + eng.run([q]):
        _fused_equal(r, ds, q, starjoin_continuous(g, ds, q), to_host, err_to_host)
    eng.close()
    g.close()
