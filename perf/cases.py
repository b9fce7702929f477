"""The work a program over this library has it do, as measurable cases.

A program over the library calls the AN operators on columns in device memory
(`GpuOps`), composes them into the SSB query programs (`ssb_programs`), or
answers batches of star queries on the fused engine (`StarJoinEngine`).  The
cases take each of these through its public entry points, from a dimension
table of 2,556 rows to a fact table of 600,000,000: the selection, the decode
and encode of a column, the joins, the grouped aggregation, the string
operators of the dimension attributes, two whole programs, and the fused
batches.  Every output is whole numbers (AN codes, OIDs, sums modulo 2^64,
error positions) or string bytes, so there is nothing to compare in 64 bits.

Sizes are the schema's at scale factors 1, 10 and 100 (6M, 60M and 600M fact
rows; 30K, 300K and 3M customers).  The columns hold the values the schema
generator draws, and a few seeded bit flips where the operator reports them.
"""
import math

import numpy as np
import torch

from ahead_b200 import ssb, ssb_programs
from ahead_b200.gpu import GpuOps
from ahead_b200.model import (AND, EQ, GE, LE, MUL, RESBIGINT, RESINT, RESOID, RESSHORT, RESTINY, WIDTH,
                              A_RESOID_MAX, Bat, Col, ainv, an_meta, void_col)
from ahead_b200.pipelines import AR, AR_INV, select_sum_an
from ahead_b200.starjoin import StarJoinEngine

TYPES = {"restiny": RESTINY, "resshort": RESSHORT, "resint": RESINT}
# the values a column of each code type holds here: discounts, dictionary codes, prices
VALUES = {"restiny": (0, 51), "resshort": (0, 10_000), "resint": (90_000, 11_000_001)}
PLACEMENTS = ssb_programs.PLACEMENTS
PROGRAMS = ("q11", "q12", "q13", "q21", "q22", "q23", "q31", "q32", "q33", "q34", "q41", "q42", "q43")
AMERICA = ssb.REGION_NAMES.index("AMERICA")


def listed():
    return [
        # A predicate on a dimension attribute (d_year over the date table):
        # every program makes several such calls; launches and latency count.
        {"name": "select_dim", "kind": "select", "rows": 2_556, "type": "resshort", "share": 0.15, "flips": 0},
        # The largest selection: a 32-bit coded fact column at scale factor 100.
        {"name": "select_600m", "kind": "select", "rows": 600_000_000, "type": "resshort", "share": 0.2,
         "flips": 10},
        # The single-column path: select, positional fetch, check and decode, sum.
        {"name": "select_sum_6m", "kind": "select_sum", "rows": 6_000_000, "flips": 10},
        # Early detection decodes each column once before the query; an odd count.
        {"name": "decode_60m", "kind": "decode", "rows": 59_999_999, "type": "resint", "flips": 60},
        # The first join of a program: the whole foreign-key column against a
        # dimension's filtered key -> OID map (part, two of five manufacturers).
        {"name": "probe_60m", "kind": "probe", "rows": 60_000_000, "share": 0.4, "flips": 60},
        # Every later join and measure: a column fetched at a fifth of its rows.
        {"name": "fetch_60m", "kind": "fetch", "rows": 60_000_000, "type": "resint", "share": 0.2, "joined": False,
         "flips": 60},
        # The end of a grouped program: the product of the measures, the groups
        # by year and category in order of first occurrence, their sums.
        {"name": "group_12m", "kind": "group", "rows": 12_000_000, "first": 7, "second": 40},
        # String attributes of the largest dimension: a predicate on the region,
        # the nation's slots fetched and grouped.
        {"name": "strings_3m", "kind": "strings", "rows": 3_000_000},
        # A whole program with early detection: decode, then unencoded operators.
        {"name": "program_q11_60m", "kind": "program", "rows": 60_000_000, "program": "q11", "placement": "early"},
        # A whole program with continuous detection: four joins, two measures, two groups.
        {"name": "program_q41_6m", "kind": "program", "rows": 6_000_000, "program": "q41", "placement": "continuous"},
        # The serving workload: 64 random star queries over 600M rows in one batch.
        {"name": "star_batch_600m", "kind": "star", "rows": 600_000_000, "queries": 64, "program": "", "flips": 1000},
        # One of the programs as a single fused query over the same table.
        {"name": "star_q21_600m", "kind": "star", "rows": 600_000_000, "queries": 1, "program": "q21", "flips": 1000},
    ]


def draw(rng):
    def rows(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    kind = rng.choice(("select", "select", "select_sum", "decode", "encode", "probe", "fetch", "group", "strings",
                       "program", "program", "star", "star"))
    typ = rng.choice(("restiny", "resshort", "resint"))
    share = round(math.exp(rng.uniform(math.log(0.001), math.log(0.9))), 4)
    flips = rng.choice((0, 3, 30, 300))
    if kind == "select":
        return {"kind": kind, "rows": rows(2_556, 300_000_000), "type": typ, "share": share, "flips": flips}
    if kind == "select_sum":
        return {"kind": kind, "rows": rows(10_000, 60_000_000), "flips": flips}
    if kind in ("decode", "encode"):
        return {"kind": kind, "rows": rows(2_556, 150_000_000), "type": typ, "flips": flips if kind == "decode" else 0}
    if kind == "probe":
        return {"kind": kind, "rows": rows(10_000, 60_000_000), "share": share, "flips": flips}
    if kind == "fetch":
        return {"kind": kind, "rows": rows(10_000, 60_000_000), "type": rng.choice(("resshort", "resint")),
                "share": share, "joined": rng.random() < 0.5, "flips": flips}
    if kind == "group":
        first, second = rng.choice((7, 25, 400)), rng.choice((40, 250, 1600))
        return {"kind": kind, "rows": rows(2 * first * second, 12_000_000), "first": first, "second": second}
    if kind == "strings":
        return {"kind": kind, "rows": rows(10_000, 3_000_000)}
    if kind == "program":
        # (below a few million rows the narrowest programs select no row at all)
        return {"kind": kind, "rows": rows(3_000_000, 60_000_000), "program": rng.choice(PROGRAMS),
                "placement": rng.choice(PLACEMENTS)}
    one = rng.random() < 0.5
    return {"kind": kind, "rows": rows(1_000_000, 60_000_000), "queries": 1 if one else rng.randint(2, 64),
            "program": rng.choice(PROGRAMS) if one else "", "flips": 100}


# ------------------------------------------------------------------ inputs
_ops = None


def ops():
    """The process's library context, as a program keeps one."""
    global _ops
    if _ops is None:
        _ops = GpuOps(0)
    return _ops


def dims_of(rows):
    """Dimension sizes of a fact table of `rows` rows (SSB's scaling)."""
    sf = rows / 6_000_000
    return {"fact": rows, "date": 2556, "customer": max(1_000, int(30_000 * sf)),
            "supplier": max(200, int(2_000 * sf)), "part": 200_000 * (1 + int(math.log2(max(sf, 1))))}


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def narrow(v, width):
    """The low `width` bytes of 64-bit values, as a byte tensor."""
    b = v.view(torch.uint8).view(-1, 8)
    return (b if width == 8 else b[:, :width].contiguous()).reshape(-1)


def an_bat(t, v, A=None):
    """The (void, t) BAT of values `v` (consumed)."""
    m = an_meta(t, A)
    n = v.numel()
    data = narrow(v.mul_(m["A"]), WIDTH[t])
    return Bat(void_col(0), Col(t, data, m["A"], m["Ainv"], m["unenc_max"], 0), n)


def distinct(g, n, k):
    """`k` different numbers below n, in random order."""
    if 4 * k >= n:
        return torch.randperm(n, generator=g, device="cuda")[:k]
    some = torch.unique(ints(g, 0, n, 2 * k + 16))
    return some[torch.randperm(some.numel(), generator=g, device="cuda")[:k]]


def exactly(g, n, k):
    """A mask over n rows with exactly `k` of them set, each row as likely."""
    mask = torch.rand(n, generator=g, device="cuda") < k / n
    for value in (False, True):  # the few that are too many, or missing
        off = (int(mask.sum()) - k) * (1 if not value else -1)
        if off > 0:
            rows = torch.nonzero(mask != value).view(-1)
            mask[rows[distinct(g, rows.numel(), off)]] = value
    return mask


def flip(bat, rows, bits):
    """One flipped bit in each of `rows` of a BAT's tail."""
    w = WIDTH[bat.tail.type]
    bat.tail.data[rows * w + bits // 8] ^= (1 << (bits % 8)).to(torch.uint8)
    return bat


def oids(rows, unenc_max):
    """AN-coded OIDs as an operator's output head carries them."""
    return Col(RESOID, rows.mul(A_RESOID_MAX).view(torch.uint8).view(-1), A_RESOID_MAX, ainv(A_RESOID_MAX, 64),
               unenc_max, 0)


def selectable(g, case, t, span, interval, A=None):
    """A column over values span[0]..span[1]-1, exactly the case's share of
    its rows inside `interval` (both ends included), with bit flips on both
    kinds of rows: a code inside stays inside (its lowest bit), one outside
    stays outside (its highest)."""
    n, (lo, hi) = case["rows"], interval
    inside = exactly(g, n, max(1, round(case["share"] * n)))
    v = ints(g, span[0], span[1] - (hi - lo + 1), n)
    v += (v >= lo) * (hi - lo + 1)
    v = torch.where(inside, ints(g, lo, hi + 1, n), v)
    half = case["flips"] // 2
    deep, out = torch.nonzero(inside & (v > lo) & (v < hi)).view(-1), torch.nonzero(~inside).view(-1)
    deep, out = (r[distinct(g, r.numel(), min(k, r.numel() // 8))] for r, k in ((deep, half),
                                                                               (out, case["flips"] - half)))
    del inside
    bat = an_bat(t, v, A)
    flip(bat, deep, torch.zeros_like(deep))
    return flip(bat, out, torch.full_like(out, 8 * WIDTH[t] - 1))


def prepare(case, seed):
    kind, rows = case["kind"], case["rows"]
    g = generator(seed)
    s = {"kind": kind, "g": ops()}
    if kind == "select":  # an interval of about that share of the values, somewhere inside
        lo, hi = VALUES[case["type"]]
        width = max(1, round(case["share"] * (hi - lo)))
        first = lo + seed % (hi - lo - width + 1)
        s["lo"], s["hi"] = first, first + width - 1
        s["col"] = selectable(g, case, TYPES[case["type"]], (lo, hi), (s["lo"], s["hi"]))
    elif kind == "select_sum":
        s["col"] = selectable(g, dict(case, share=0.2), RESSHORT, (0, 10_000), (1_000, 2_999), A=233)
    elif kind == "decode":
        t = TYPES[case["type"]]
        s["col"] = an_bat(t, ints(g, *VALUES[case["type"]], rows))
        bad = distinct(g, rows, case["flips"])
        flip(s["col"], bad, ints(g, 0, 8 * WIDTH[t], bad.numel()))
    elif kind == "encode":
        t = ssb.UNENC[TYPES[case["type"]]]
        s["col"] = Bat(void_col(0), Col(t, narrow(ints(g, *VALUES[case["type"]], rows), WIDTH[t])), rows)
        s["A"] = an_meta(TYPES[case["type"]])["A"]
    elif kind == "probe":
        keys = dims_of(rows)["part"]
        mask = exactly(g, keys, max(1, round(case["share"] * keys)))
        kept, dropped = torch.nonzero(mask).view(-1), torch.nonzero(~mask).view(-1)
        hit = exactly(g, rows, max(1, round(case["share"] * rows)))
        v = torch.where(hit, kept[ints(g, 0, kept.numel(), rows)], dropped[ints(g, 0, dropped.numel(), rows)])
        s["fk"] = an_bat(RESINT, v + 1)  # partkey is the row's number + 1
        missed = torch.nonzero(~hit).view(-1)
        bad = missed[distinct(g, missed.numel(), case["flips"])]
        flip(s["fk"], bad, ints(g, 0, 64, bad.numel()))
        s["map"] = Bat(an_bat(RESINT, kept + 1).tail, oids(kept, an_meta(RESOID)["unenc_max"]), kept.numel())
    elif kind == "fetch":
        t = TYPES[case["type"]]
        s["col"] = an_bat(t, ints(g, *VALUES[case["type"]], rows))
        mask = exactly(g, rows, max(1, round(case["share"] * rows)))
        at, rest = torch.nonzero(mask).view(-1), torch.nonzero(~mask).view(-1)
        for r in (at, rest):  # corrupt values among the fetched rows and among the others
            bad = r[distinct(g, r.numel(), min(case["flips"] // 2, r.numel() // 8))]
            flip(s["col"], bad, ints(g, 0, 8 * WIDTH[t], bad.numel()))
        # a join's re-encoded head keeps the void column's largest value, 0
        head = oids(at, 0 if case["joined"] else an_meta(RESOID)["unenc_max"])
        s["list"] = Bat(head, head, at.numel())
    elif kind == "group":
        count = case["first"] * case["second"]
        s["price"] = an_bat(RESINT, ints(g, 90_000, 11_000_001, rows))
        s["discount"] = an_bat(RESTINY, ints(g, 0, 11, rows))
        pair = ints(g, 0, count, rows)
        pair[distinct(g, rows, count)] = torch.arange(count, device="cuda")  # each group occurs
        s["first"] = an_bat(RESSHORT, pair // case["second"])
        s["second"] = an_bat(RESSHORT, pair % case["second"])
    elif kind == "strings":
        america = exactly(g, rows, rows // 5)
        region = ints(g, 0, 4, rows)
        region = torch.where(america, AMERICA, region + (region >= AMERICA))
        for attr, codes, count in (("region", region, 5), ("nation", region * 8 + ints(g, 0, 8, rows), 40)):
            names = np.zeros((count, ssb.STRING_WIDTH[attr]), np.uint8)
            for k in range(count):
                name = ssb.string_of(attr, k).encode()
                names[k, : len(name)] = np.frombuffer(name, np.uint8)
            s[attr] = torch.from_numpy(names).cuda()[codes].view(-1)
        m = an_meta(RESOID)
        s["groups"] = Bat(void_col(0), Col(RESOID, narrow(ints(g, 0, 7, rows // 5).mul_(m["A"]), 8), m["A"],
                                           m["Ainv"], m["unenc_max"], 0), rows // 5)
    elif kind == "program":
        # clean columns: under flips some programs end in the reference's size mismatch
        schema = ssb.generate_device(dims_of(rows), seed=seed)
        s["program"], s["placement"] = getattr(ssb_programs, case["program"]), case["placement"]
        s["schema"] = schema
        s["plain"] = ssb.decoded_device(schema) if case["placement"] == "normal" else None
        # where the program keeps its results: up to 4,096 groups, the error positions
        s["groups"] = torch.zeros(6, 4096, dtype=torch.int64, device="cuda")
        s["errors"] = torch.zeros(3 * rows, dtype=torch.int64, device="cuda")
    else:
        s["schema"] = ssb.generate_device(dims_of(rows), seed=seed, flips=case["flips"], flip_seed=seed + 1)
        s["engine"] = StarJoinEngine(s["g"], s["schema"])
        if case["program"]:
            s["queries"] = [ssb_programs.program_query(case["program"])]
        else:
            rng = np.random.default_rng(seed)
            sizes = [n for n in (1_000_000, 6_000_000, 60_000_000) if n < rows] + [rows]
            s["queries"] = [ssb.random_query(rng, fact_sizes=sizes) for _ in range(case["queries"])]
            s["queries"][0].fact_rows = rows
        # where the program keeps its results: sums, group keys, error positions
        s["kept"] = [np.zeros(k << 20, np.uint64) for k in (1, 3, 1)]
    torch.cuda.synchronize()
    return s


# -------------------------------------------------------------------- passes
def column(bat, which="tail"):
    """A BAT's column as it is in device memory (None for a void one)."""
    c = getattr(bat, which)
    w = WIDTH[c.type]
    dtype = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[w]
    return None if c.data is None else c.data[: bat.count * w].view(dtype)


def positions(e):
    return e.values.view(torch.int64) if e.present and e.values is not None else None


def word(x):
    return np.array([x], np.uint64).view(np.int64)


def run(s):
    g, kind = s["g"], s["kind"]
    if kind == "select":
        A = s["col"].tail.A
        out, err = g.select_an(s["col"], GE, s["lo"] * A, LE, s["hi"] * A, AND)
        return [column(out, "head"), positions(err)]
    if kind == "select_sum":
        r = select_sum_an(g, s["col"], 1_000, 3_000)
        return [column(r.oids, "head"), word(r.total), positions(r.select_errors)] + \
            [positions(e) for e in r.fetch_errors + r.decode_errors]
    if kind == "decode":
        out, _, err = g.check_and_decode_an(s["col"])
        return [column(out), positions(err)]
    if kind == "encode":
        return [column(g.encode_an(s["col"], s["A"]))]
    if kind == "probe":
        out, errs = g.hashjoin_an(s["fk"], s["map"], reenc_head=1, ah1r=AR, ah1invr=AR_INV)
        return [column(out, "head"), column(out)] + [positions(e) for e in errs]
    if kind == "fetch":
        out, errs = g.matchjoin_an(s["list"], s["col"])
        return [column(out, "head"), column(out)] + [positions(e) for e in errs]
    if kind == "group":
        vals, errs = g.arithmetic_an(MUL, RESBIGINT, s["price"], s["discount"], AR, AR_INV)
        gids, firsts, e1 = g.groupby_an(s["first"])
        gids, firsts, e2 = g.groupby2_an(s["second"], gids, firsts.count)
        sums, e3 = g.aggregate_sum_grouped_an(vals, gids, firsts.count)
        return [column(vals), column(gids), column(firsts), column(sums)] + \
            [positions(e) for e in errs + e1 + e2 + e3]
    if kind == "strings":
        wr, wn = ssb.STRING_WIDTH["region"], ssb.STRING_WIDTH["nation"]
        kept = g.select_str_an(s["region"], wr, 0, EQ, b"AMERICA")
        n = kept.data.numel() // 8
        slots, errs = g.fetchjoin_str_an(Bat(void_col(0), kept, n), s["nation"], wn)
        gids, firsts, e2 = g.groupby2_str_an(slots.view(-1), wn, s["groups"], 7)
        return [kept.data.view(torch.int64), slots, column(gids), column(firsts)] + [positions(e) for e in errs + e2]
    if kind == "program":
        r = s["program"](g, s["schema"], s["placement"], s["plain"])
        out = [] if r.total is None else [word(r.total % (1 << 64))]
        groups = [r.years, r.nations, r.snations, r.profits] + [r.extra[k] for k in sorted(r.extra)]
        for k, b in enumerate(b for b in groups if b is not None):
            s["groups"][k, : b.count].copy_(column(b))
        at = 0
        for e in r.errors:
            p = positions(e)
            if p is not None and p.numel():
                s["errors"][at: at + p.numel()].copy_(p)
                at += p.numel()
        return out + [s["groups"], s["errors"]]
    rs = s["engine"].run(s["queries"], graph=True)
    none = np.zeros(0, np.uint64)
    totals = np.array([r.total or 0 for r in rs], np.uint64)
    sums = [none if r.sums is None else r.sums for r in rs]
    keys = [none] + [k for r in rs for k in r.keys]
    errs = [r.fact_errors[c] for r in rs for c in ssb.FACT_COLS]
    counts = np.array([r.status for r in rs] + [len(x) for x in sums] + [len(x) for x in errs], np.int64)
    for kept, parts in zip(s["kept"], (sums, keys, errs)):
        np.concatenate(parts, out=kept[: sum(map(len, parts))])
    return [totals.view(np.int64), counts] + [kept.view(np.int64) for kept in s["kept"]]


# ---------------------------------------------------------------------- work
def work(case):
    """Each column read once, each result written once; for positional reads
    of a share of a column, that share."""
    kind, n = case["kind"], case["rows"]
    w = WIDTH[TYPES[case["type"]]] if "type" in case else 0
    if kind == "select":
        b = n * w + case["share"] * n * 8
    elif kind == "select_sum":
        b = n * 4 + 0.2 * n * 8
    elif kind in ("decode", "encode"):
        b = n * w + n * (w // 2)
    elif kind == "probe":
        b = n * 8 + dims_of(n)["part"] * case["share"] * 16 + case["share"] * n * 16
    elif kind == "fetch":
        b = case["share"] * n * (8 + w + 8 + w)
    elif kind == "group":
        b = n * (8 + 2 + 4 + 4) + n * (8 + 8)
    elif kind == "strings":
        b = n * 13 + 0.2 * n * (8 + 16 + 16 + 8 + 8)
    elif kind == "program":
        # early detection decodes every column the program reads (Q1.x: quantity,
        # discount, date key, price; the others: three or four foreign keys and
        # one or two measures); the rest read the first column whole and the
        # others where rows survive
        q1, early = case["program"].startswith("q1"), case["placement"] == "early"
        b = n * ((20 if q1 else 32 if case["program"] < "q4" else 48) if early else 6 if q1 else 12)
    elif case["program"]:
        b = n * (4 if case["program"].startswith("q1") else 8) + 0.1 * n * 24
    else:
        b = n * 42
    return {"bytes": float(b), "flops": 0.0}
