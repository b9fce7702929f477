"""The row lists of the per-row strategy (from 2^21 rows on) against the same
queries composed operator by operator: lengths around that line and around the
512-row steps, maps that fit shared memory, that share it and that are folded
(3M and 8M customers), a third filter (from 2^19 listed rows on), batches of
several queries, and corrupt codes in every fact column."""
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 21


def run_all(n, sizes, batches, flips=300, strategy=None):
    from ahead_b200.gpu import GpuOps, err_to_host, to_host
    from ahead_b200.pipelines import starjoin_continuous
    from ahead_b200.ssb import generate_device
    from ahead_b200.ssb_programs import program_query
    from ahead_b200.starjoin import StarJoinEngine
    from test_programs import _fused_equal
    g = GpuOps(0)
    ds = generate_device(dict(fact=n, date=2556, **sizes), seed=n % 97, flips=flips, flip_seed=n % 89)
    eng = StarJoinEngine(g, ds)
    for names in batches:
        qs = [program_query(x, fact_rows=r) if r else program_query(x) for x, r in names]
        for r, q in zip(eng.run(qs), qs):
            _fused_equal(r, ds, q, starjoin_continuous(g, ds, q), to_host, err_to_host)
    eng.close()
    g.close()


SMALL = dict(customer=30_000, part=200_000, supplier=2_000)
ONE = [[(x, 0)] for x in ("q11", "q13", "q21", "q22", "q31", "q33", "q41", "q43")]


@pytest.mark.parametrize("n", [N - 1, N, N + 1, N + 511, N + 513, 3_000_017])
def test_lengths(n):
    run_all(n, SMALL, ONE)


@pytest.mark.parametrize("sizes", [dict(customer=3_000_000, part=1_400_000, supplier=200_000),
                                   dict(customer=8_000_000, part=200_000, supplier=2_000),
                                   dict(customer=1_000_000, part=2_000_000, supplier=900_000)])
def test_maps_that_share_or_are_folded(sizes):
    run_all(2_500_003, sizes, ONE)


def test_batches_and_prefixes():
    run_all(3_000_001, SMALL, [[("q12", 0), ("q13", 2_600_000)], [("q32", 0), ("q33", 0), ("q34", 2_999_999)],
                               [("q21", 2_200_000), ("q22", 0)], [("q41", 0), ("q42", 2_500_001)]])


@pytest.mark.parametrize("flips", [0, 300, 40_000])
def test_third_filter(flips):
    run_all(14_000_003, dict(customer=3_000_000, part=200_000, supplier=20_000), [[("q41", 0)], [("q41", 0), ("q42", 0)]],
            flips)
