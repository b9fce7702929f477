"""The direct (bitmap) hash join against the C restatement where it can go
wrong: key ranges at and past its limit and past the shared-memory bitmap,
repeated and corrupt build keys (the hash table), corrupt probe keys that
decode into the range, heads whose every row reads as corrupt, probe lengths
around one block's tiles, both hash sides, and the unencoded twin."""
import numpy as np
import pytest

from bats import encoded_col, flip_bits, oid_list
from cases import assert_same, run_case

from ahead_b200.model import (HASH_LEFT, HASH_RIGHT, INT, OID, RESINT, RESOID, RESSHORT, RESTINY, SHORTINT, TINYINT,
                              Bat, Col, an_meta, void_col)

pytestmark = pytest.mark.gpu
AR, ARI = 65117, 0x3E36D3BC8D9BC5F5


@pytest.fixture(scope="module")
def gpu():
    from ahead_b200.gpu import GpuOps
    g = GpuOps(0)
    yield g
    g.close()


def check(gpu, op, *args, **kw):
    from ahead_b200.gpu import err_to_host, to_device, to_host
    from oracle.oracle import Oracle
    c = dict(op=op, args=list(args), kwargs=kw)
    assert_same(run_case(gpu, c, to_device, to_host, err_to_host), run_case(Oracle("port"), c), op)


def _build(rng, t, keys, flips=0):
    """(key column, resoid) of the given keys, as a key -> OID map."""
    k = encoded_col(t, keys)
    flip_bits(k.tail.data, flips, rng)
    o = oid_list(rng.permutation(1 << 20)[: len(keys)])
    return Bat(k.tail, o.tail, k.count)


@pytest.mark.parametrize("side", [HASH_RIGHT, HASH_LEFT])
@pytest.mark.parametrize("nb,span,np_", [
    (1, 1, 1), (40, 40, 255), (2_556, 61_000, 8_192), (2_556, 61_000, 8_193), (1_000, 1_040_000, 300),
    (5, 1 << 21, 400),                       # past the limit of a small join: the hash table
    (30_000, 1_638_400, 50_001), (30_000, 1_638_401, 50_001), (30_000, 2_400_000, 50_001)])
@pytest.mark.parametrize("flips", [0, 20])
def test_key_ranges(gpu, side, nb, span, np_, flips):
    rng = np.random.default_rng(nb + np_)
    keys = np.sort(rng.choice(span, nb, replace=False)).astype(np.uint64)
    keys[0], keys[-1] = 0, span - 1
    build = _build(rng, RESINT, keys + 7)
    probe = encoded_col(RESINT, rng.integers(0, span + 20, np_, dtype=np.uint64), seqbase=3)
    probe.tail.data[: np_ // 2] = rng.choice(build.head.data, np_ // 2)
    flip_bits(probe.tail.data, min(flips, np_), rng)
    if side == HASH_RIGHT:
        check(gpu, "hashjoin_an", probe, build, side=side)
        check(gpu, "hashjoin_an", probe, build, reenc_head=1, ah1r=AR, ah1invr=ARI, reenc_tail=1, at2r=AR,
              at2invr=ARI, side=side)
    else:  # the build on the left: (resoid, key) x (key, void)
        check(gpu, "hashjoin_an", build.reverse(), probe.reverse(), side=side)
        check(gpu, "hashjoin_an", build.reverse(), probe.reverse(), reenc_head=1, ah1r=AR, ah1invr=ARI, side=side)


@pytest.mark.parametrize("t,hi", [(RESTINY, 256), (RESSHORT, 65_536), (RESINT, 1 << 32)])
@pytest.mark.parametrize("how", ["unique", "repeated", "corrupt", "all corrupt"])
def test_build_keys(gpu, t, hi, how):
    rng = np.random.default_rng(t)
    nb = min(hi, 4_500)
    keys = np.arange(nb, dtype=np.uint64)
    if how == "repeated":
        keys[nb // 2] = keys[3]
    build = _build(rng, t, keys, flips=6 if how == "corrupt" else 0)
    if how == "all corrupt":
        build.head.unenc_max = 0  # every key but 0 reads as corrupt, and joins all the same
        build.tail.unenc_max = 0
    probe = encoded_col(t, rng.integers(0, min(hi, 9_000), 20_001, dtype=np.uint64))
    flip_bits(probe.tail.data, 200, rng)
    check(gpu, "hashjoin_an", probe, build, reenc_head=1, ah1r=AR, ah1invr=ARI)


@pytest.mark.parametrize("n", [200, 9_000, 70_001])
@pytest.mark.parametrize("umax", [0, None])
def test_encoded_heads(gpu, n, umax):
    """A probe side with resoid heads: valid ones with flips, or (as re-encoded
    heads are) with a largest value of 0."""
    rng = np.random.default_rng(n)
    build = _build(rng, RESINT, np.arange(500, dtype=np.uint64) * 3)
    probe = encoded_col(RESINT, rng.integers(0, 1_600, n, dtype=np.uint64))
    heads = oid_list(rng.integers(0, 1 << 24, n)).tail
    flip_bits(heads.data, 9, rng)
    if umax is not None:
        heads.unenc_max = umax
    check(gpu, "hashjoin_an", Bat(heads, probe.tail, n), build)


@pytest.mark.parametrize("t,dt,hi", [(TINYINT, np.uint8, 256), (SHORTINT, np.uint16, 60_000),
                                     (INT, np.uint32, 1 << 21)])
@pytest.mark.parametrize("side", [HASH_RIGHT, HASH_LEFT])
@pytest.mark.parametrize("repeated", [False, True])
def test_unencoded(gpu, t, dt, hi, side, repeated):
    rng = np.random.default_rng(hi)
    nb = min(hi, 3_000)
    keys = rng.choice(hi, nb, replace=False).astype(dt)  # in any order
    if repeated:
        keys[5] = keys[9]
    build = Bat(Col(t, keys), Col(OID, rng.integers(0, 1 << 31, nb).astype(np.uint32)), nb)
    n = 40_001
    probe = Bat(void_col(9), Col(t, rng.integers(0, hi, n).astype(dt)), n)
    probe.tail.data[::3] = rng.choice(keys, len(probe.tail.data[::3]))
    if side == HASH_RIGHT:
        check(gpu, "hashjoin", probe, build, side=side)
    else:
        check(gpu, "hashjoin", build.reverse(), probe.reverse(), side=side)
