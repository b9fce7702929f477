"""Joins whose output columns the call allocates itself run once, also where the
inputs need another form (keys out of order), and against the C restatement."""
import numpy as np
import pytest

from bats import encoded_col, oid_list
from cases import assert_same, run_case

from ahead_b200.model import INT, OID, RESINT, Bat, Col

pytestmark = pytest.mark.gpu


class Counted:
    """The library with its operator calls counted."""

    def __init__(self, lib):
        self.lib, self.calls = lib, []

    def __getattr__(self, name):
        if name.startswith("ahead_gpu_"):
            self.calls.append(name)
        return getattr(self.lib, name)


@pytest.fixture
def gpu(monkeypatch):
    import ahead_b200.gpu as mirror
    monkeypatch.setattr(mirror, "_SIZED_BYTES", 0)
    g = mirror.GpuOps(0)
    g.lib = Counted(g.lib)
    yield g
    g.lib = g.lib.lib
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    del gpu.lib.calls[:]
    got = run_case(gpu, c, to_device, to_host, err_to_host)
    assert gpu.lib.calls == ["ahead_gpu_" + op]
    assert_same(got, run_case(Oracle("port"), c), op)


@pytest.mark.parametrize("n1,n2", [(1, 3), (40, 300), (9_000, 700)])
def test_merge_out_of_order(gpu, n1, n2):
    rng = np.random.default_rng(n1)
    k1 = rng.permutation(n1).astype(np.uint64)
    k2 = rng.choice(2 * max(n1, n2), n2, replace=False).astype(np.uint64)
    k2[0] = k2[-1]  # a repeated key, too
    a, b = oid_list(k1), oid_list(k2)
    value = encoded_col(RESINT, rng.integers(0, 1 << 20, n2)).tail
    check(gpu, "matchjoin_an", Bat(a.tail, a.tail, n1), Bat(b.tail, value, n2))
    p, q = Col(OID, k1.astype(np.uint32)), Col(OID, k2.astype(np.uint32))
    check(gpu, "matchjoin", Bat(p, p, n1), Bat(q, Col(INT, rng.integers(0, 99, n2).astype(np.uint32)), n2))
    same = oid_list(np.full(n1, 7, np.uint64))  # every key the same: the shorter input's length is kept
    other = oid_list(np.full(n2, 7, np.uint64))
    check(gpu, "matchjoin_an", Bat(same.tail, same.tail, n1), Bat(other.tail, other.tail, n2))
