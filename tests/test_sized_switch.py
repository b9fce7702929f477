"""The size from which output columns are allocated by the call is read when the
call is made: with it at 0 every such operator asks for its columns."""
import numpy as np
import pytest

from bats import encoded_col, oid_list

from ahead_b200.model import GE, INT, OID, RESBIGINT, RESINT, Bat, Col, void_col

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [0, 1 << 28])
def test_switch(monkeypatch, size):
    import ahead_b200.gpu as mirror
    monkeypatch.setattr(mirror, "_SIZED_BYTES", size)
    g = mirror.GpuOps(0)
    asked = []
    set_sized = g._set_sized
    monkeypatch.setattr(g, "_set_sized", lambda out: (asked.append(out), set_sized(out)))
    n = 1000
    code = mirror.to_device(encoded_col(RESINT, np.arange(n)))
    big = mirror.to_device(encoded_col(RESBIGINT, np.arange(n), A=65117))
    plain = mirror.to_device(Bat(void_col(0), Col(INT, np.arange(n, dtype=np.uint32)), n))
    oids = mirror.to_device(oid_list(np.arange(n)))
    keys = Bat(code.tail, oids.tail, n)
    poid = mirror.to_device(Bat(Col(OID, np.arange(n, dtype=np.uint32)), Col(OID, np.arange(n, dtype=np.uint32)), n))
    calls = [lambda: g.select_an(code, GE, 0)[0], lambda: g.select(plain, GE, 0),
             lambda: g.check_and_decode_an(big)[0], lambda: g.hashjoin_an(code, keys)[0],
             lambda: g.hashjoin(plain, Bat(plain.tail, poid.tail, n)),
             lambda: g.matchjoin_an(Bat(oids.tail, oids.tail, n), Bat(oids.tail, oids.tail, n))[0],
             lambda: g.matchjoin(poid, poid)]
    for k, call in enumerate(calls):
        assert call().count == n, k
        assert len(asked) == (k + 1 if size == 0 else 0), k
    g.close()
