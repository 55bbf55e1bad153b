"""The calls whose time matters: what a program that joins, partitions and filters on the GPU makes of them.

Every case is one call (or one plan replay) through the package's public entry points on inputs that
are already on the device, at the sizes of the benchmark's workloads and of the batched and served
ranges: a few thousand rows to 64M, unique and duplicated build keys, NULLs, one and two key columns,
every layout that the build chooses by itself (small, larger than L2, 128-bit slots, grouped).

A relation has no row order and the entry points promise none, so the output columns come back as
``Rows``: reading a column gives its rows in canonical order. A program that goes on with the result
reads the tensors as they were written, so ``run`` itself puts nothing in order.
"""
from __future__ import annotations

import ctypes
import functools
import math

import torch

from sirius_b200 import _lib as L
from sirius_b200 import batch as B
from sirius_b200 import join as J

DEV = "cuda"
TYPES = {"i4": torch.int32, "i8": torch.int64, "f4": torch.float32, "f8": torch.float64}
WIDTH = {"i4": 4, "i8": 8, "f4": 4, "f8": 8}
KINDS = {"left": L.SJ_JOIN_LEFT, "semi": L.SJ_JOIN_SEMI, "anti": L.SJ_JOIN_ANTI, "mark": L.SJ_JOIN_MARK,
         "full": L.SJ_JOIN_FULL}
MILLION = 1 << 20


def listed():
    """flow: probe (INNER probe and gather of a resident table), left / semi / anti / mark / full (the other
    join types on it), join (build, probe and gather in one call), batch, partition, filter. key: i4, i8 (unique
    in a sparse range of 2^40), wide (any int64, so 128-bit slots), zipf (duplicated on both sides), two (two
    int32 columns). hit: share of the probe rows whose key is in the build. nulls: share of NULL probe keys.
    pp / bp: payload columns of the probe and the build side. attach: the table holds the build payloads.
    native: the C entry point with its arguments made once, as a native operator calls it."""
    return [
        # a dimension of a thousand rows against one small batch: launches and latency, nothing else
        _case("probe_tiny", "probe", "i4", 1_000, 10_000, 0.83, "i4", "i4", native=True),
        # the benchmark's small workload: the table and the probe sit in L2
        _case("probe_small", "probe", "i4", 100_000, 1_000_000, 0.91, "i4", "i4", native=True),
        # a lookup request against a resident table of a lookup service, of an odd size, called from Python
        _case("probe_served", "probe", "wide", 4 * MILLION, 1_234_567, 0.7, "", "i8"),
        # the benchmark's headline: a foreign-key join whose table is larger than L2
        _case("probe_large", "probe", "i8", 16 * MILLION, 64 * MILLION, 1.0, "i8", "i8,f8"),
        # the benchmark's skewed many-to-many join: duplicated build keys, hot keys, NULL probe keys
        _case("probe_skewed", "probe", "zipf", 8 * MILLION, 32 * MILLION, 0.5, "", "i4", nulls=0.05, native=True),
        # two-column keys, row ids only: what an operator that gathers by itself asks for
        _case("probe_two_keys", "probe", "two", 8 * MILLION, 32 * MILLION, 1.0, "", "", attach=False),
        # an outer join of an ordinary fact table: absent and NULL keys, a nullable result column
        _case("left_outer", "left", "i8", 3_000_001, 12_345_678, 0.7, "i8", "f8", nulls=0.03),
        # EXISTS over the large table: only the rows that match, with a payload
        _case("semi_large", "semi", "i8", 16 * MILLION, 64 * MILLION, 0.7, "i8", ""),
        # a join whose both sides are new each time: the build is part of the call, payloads stay the caller's
        _case("join_once", "join", "i8", 2 * MILLION, 10_000_019, 0.9, "i8", "i8", attach=False),
        # many partition pairs joined by one plan, replayed with new contents in the same buffers
        dict(name="batch_pairs", flow="batch", key="i4", joins=64, low=1_000, high=1_000_000),
        # both sides of a join that is split over workers go through this one
        dict(name="partition_large", flow="partition", key="i8", probe=64 * MILLION, pp="i8", parts=64, nulls=0.0),
        # the scan of the probe side tests the join's dynamic filter before the join
        dict(name="filter_scan", flow="filter", key="i8", build=16 * MILLION, probe=64 * MILLION, hit=0.5, bits=16,
             nulls=0.0),
    ]


def _case(name, flow, key, build, probe, hit, pp, bp, attach=True, nulls=0.0, native=False):
    return dict(name=name, flow=flow, key=key, build=build, probe=probe, hit=hit, pp=pp, bp=bp, attach=attach,
                nulls=nulls, native=native)


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    flow = rng.choice(["probe"] * 5 + ["left", "semi", "anti", "mark", "full", "join", "join", "batch", "partition",
                                       "filter"])
    nulls = rng.choice([0.0, 0.0, 0.02, 0.1])
    if flow == "batch":
        high = _log(rng, 20_000, 1_000_000)
        return dict(flow=flow, key=rng.choice(["i4", "i8"]), joins=rng.randint(3, 64), low=1_000, high=high)
    probe = _log(rng, 10_000, 64 * MILLION)
    if flow == "partition":
        return dict(flow=flow, key=rng.choice(["i4", "i8"]), probe=probe, pp=rng.choice(["", "i4", "i8"]),
                    parts=1 << rng.randint(1, 8), nulls=nulls)
    build = min(_log(rng, 1_000, 16 * MILLION), max(1_000, probe // rng.choice([1, 3, 10])))
    if flow == "filter":
        return dict(flow=flow, key=rng.choice(["i4", "i8"]), build=build, probe=probe, hit=rng.uniform(0.1, 1.0),
                    bits=rng.choice([8, 16]), nulls=nulls)
    key = rng.choice(["i4", "i8", "i8", "wide"] + (["zipf", "two"] if flow in ("probe", "join") else []))
    if key == "zipf" or flow == "full":  # several output rows for each probe row, or three passes
        probe, build = min(probe, 24 * MILLION), min(build, 6 * MILLION)
    hit = 0.5 if key == "zipf" else round(rng.uniform(0.3, 1.0), 3)
    pp = rng.choice(["", "i4", "i8", "f8", "i8,i4"])
    bp = rng.choice(["", "i4", "i8", "f8", "i8,f8", "i8,i8,f4"])
    case = _case("", flow, key, build, probe, hit, pp, bp, flow not in ("join", "full") and rng.random() < 0.6, nulls,
                 flow == "probe" and rng.random() < 0.5)
    del case["name"]
    return case


# ---- inputs -------------------------------------------------------------------------------------------------

def _permuted(index, half, salt):
    """A bijection of [0, 2^(2 half)) on int64 tensors (four Feistel rounds): distinct, scattered keys."""
    mask = (1 << half) - 1
    left, right = (index >> half) & mask, index & mask
    for r in range(4):
        f = right * (0x9E3779B97F4A7C1 + 2 * r) + (salt * 7919 + r)
        f = (f ^ (f >> 29)) * 0x2545F4914F6CDD1
        left, right = right, left ^ ((f >> 17) & mask)
    return (left << half) | right


BUILD_POWER, PROBE_POWER = 1.1, 0.8  # of the duplicated keys' Zipf distributions


def _shares(domain, power, device):
    return torch.arange(1, domain + 1, dtype=torch.float64, device=device).pow(-power)


def _ranks(n, domain, power, gen):
    """n ranks in [0, domain), rank k with probability proportional to (k + 1)^-power."""
    cdf = _shares(domain, power, DEV).cumsum(0)
    u = torch.rand(n, dtype=torch.float64, device=DEV, generator=gen) * cdf[-1]
    return torch.searchsorted(cdf, u, right=True).clamp_(max=domain - 1)


def _value_of(rank, values):
    """The value that the probe's rank stands for: every other one is absent from the build, and the probe's hot
    keys are not the build's."""
    return torch.where(rank % 2 == 0, (rank // 2 * 40_503 + values // 3) % values, values + rank)


@functools.lru_cache(maxsize=16)
def _pairs(nb, n):
    """About how many pairs of rows the duplicated keys make."""
    values = max(1, nb // 8)
    b, p = _shares(values, BUILD_POWER, "cpu"), _shares(2 * values, PROBE_POWER, "cpu")
    at = _value_of(torch.arange(0, 2 * values, 2), values)
    return float((p[::2] * b[at]).sum() / p.sum() / b.sum()) * nb * n


def _length(case):
    """Rows that the outputs have room for."""
    if case["key"] == "zipf":
        return int(1.25 * _pairs(case["build"], case["probe"])) + 10_000
    return case["probe"] + (case["build"] if case["flow"] == "full" else 0)


def _column(kind, n, gen):
    if kind[0] == "f":
        return torch.rand(n, dtype=TYPES[kind], device=DEV, generator=gen) * 1000
    high = (1 << 31) - 1 if kind == "i4" else 1 << 62
    return torch.randint(-high, high, (n,), dtype=TYPES[kind], device=DEV, generator=gen)


def _columns(kinds, n, gen):
    return [_column(k, n, gen) for k in kinds.split(",") if k]


def _words(valid):
    """bool per row -> bitmask words."""
    padded = torch.zeros((valid.numel() + 31) // 32 * 32, dtype=torch.int64, device=DEV)
    padded[:valid.numel()] = valid
    words = (padded.view(-1, 32) << torch.arange(32, device=DEV)).sum(1)
    return torch.where(words >= 1 << 31, words - (1 << 32), words).to(torch.int32)


def _bits(words, n):
    return ((words[:, None] >> torch.arange(32, dtype=torch.int32, device=words.device)) & 1).view(-1)[:n].bool()


def _generator(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return gen


def _sides(case, seed):
    """(build keys, probe keys, valid probe rows or None, probe payloads, build payloads); keys are one tensor
    or, for two-column keys, a list of two."""
    gen = _generator(seed)
    nb, n, salt = case["build"], case["probe"], seed % 65_521
    key = case["key"]
    span = max(nb, int(nb / case["hit"]))  # the build's keys are the first nb of `span` values
    if key == "zipf":
        values = max(1, nb // 8)
        build = _permuted(_ranks(nb, values, BUILD_POWER, gen), 20, salt)
        probe = _permuted(_value_of(_ranks(n, 2 * values, PROBE_POWER, gen), values), 20, salt)
    else:
        of_probe = torch.randint(0, span, (n,), device=DEV, generator=gen)
        if key == "i4":
            build = torch.randperm(nb, device=DEV, generator=gen).int()
            probe = of_probe.int()
        elif key == "two":
            both = torch.randperm(nb, device=DEV, generator=gen)
            build = [(both // 4096).int(), (both % 4096).int()]
            probe = [(of_probe // 4096).int(), (of_probe % 4096).int()]
        else:
            half = 32 if key == "wide" else 20
            build = _permuted(torch.arange(nb, device=DEV), half, salt)
            probe = _permuted(of_probe, half, salt)
    valid = torch.rand(n, device=DEV, generator=gen) >= case["nulls"] if case["nulls"] else None
    return build, probe, valid, _columns(case.get("pp", ""), n, gen), _columns(case.get("bp", ""), nb, gen)


def _batch_sides(case, seed):
    """Build sizes log-uniform in [low, high]; ten probe rows for each build row, over 1.2 times its keys."""
    gen = _generator(seed)
    sizes = torch.exp(torch.rand(case["joins"], dtype=torch.float64, device=DEV, generator=_generator(case["joins"]))
                      * math.log(case["high"] / case["low"]) + math.log(case["low"])).long().tolist()
    kind = TYPES[case["key"]]
    return [(torch.randperm(m, device=DEV, generator=gen).to(kind),
             torch.randint(0, m + m // 5 + 1, (10 * m,), device=DEV, generator=gen).to(kind),
             _column("i4", m, gen), _column("i4", 10 * m, gen)) for m in sizes]


# ---- states and passes ----------------------------------------------------------------------------------------

class Rows(dict):
    """The output columns of a call, by name; reading one gives its rows in canonical order (by the columns that
    `order` names), values and validity of NULLs included, and zeros up to `length` rows. `count`: rows written, a
    number or the device's word."""

    def __init__(self, columns, count, length, order, validity=None):
        super().__init__(columns)
        for name in validity or {}:
            self[name + "_valid"] = validity[name]
        self._count, self._length, self._by, self._validity, self._order = count, length, order, validity or {}, None

    def __getitem__(self, name):
        n = min(int(self._count), self._length)
        if self._order is None:
            self._order = torch.arange(n, device=DEV)
            for by in reversed(self._by):
                key = by[:n] if isinstance(by, torch.Tensor) else super().__getitem__(by)[:n]
                self._order = self._order[torch.sort(key[self._order], stable=True).indices]
        raw = super().__getitem__(name)
        if name.endswith("_valid"):
            return _padded(_bits(raw, n)[self._order], self._length)
        rows = raw[:n][self._order]
        if name in self._validity:
            rows = rows.masked_fill(~_bits(self._validity[name], n)[self._order], 0)
        return _padded(rows, self._length)


def _padded(rows, length):
    return torch.cat([rows[:length], torch.zeros(max(0, length - rows.numel()), dtype=rows.dtype, device=rows.device)])


def _rows(out, count, length):
    columns, validity = {"probe_row": out.probe_rid}, {}
    if out.build_rid is not None:
        columns["build_row"] = out.build_rid
    for side, cols, words in (("probe", out.probe_payload, out.probe_payload_validity),
                              ("build", out.build_payload, out.build_payload_validity)):
        for c, (col, w) in enumerate(zip(cols, words)):
            columns["%s%d" % (side, c)] = col
            if w is not None:
                validity["%s%d" % (side, c)] = w
    return {"count": count, "rows": Rows(columns, count, length,
                                         [k for k in ("probe_row", "build_row") if k in columns], validity)}


def prepare(case, seed):
    flow = case["flow"]
    if flow == "batch":
        specs = [B.BatchJoinSpec(bk, pk, bp, pp) for bk, pk, bp, pp in _batch_sides(case, seed)]
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        return dict(flow=flow, specs=specs, plan=B.BatchPlan(specs, stream=stream), stream=stream)
    if flow == "partition":
        key = "i4" if case["key"] == "i4" else "i8"
        gen = _generator(seed)
        keys = _column(key, case["probe"], gen)
        words = _words(torch.rand(case["probe"], device=DEV, generator=gen) >= case["nulls"]) if case["nulls"] else None
        return dict(flow=flow, keys=[(keys, words)] if case["nulls"] else keys, parts=case["parts"],
                    columns=[keys] + _columns(case["pp"], case["probe"], gen))
    build, probe, valid, pp, bp = _sides(case, seed)
    words = _words(valid) if valid is not None else None
    state = dict(flow=flow, build=build, probe=probe, words=words, pp=pp, bp=bp, attach=case.get("attach", False),
                 length=_length(case))
    if isinstance(probe, list):  # (tensor, validity) for each of the key columns
        state["probe"], state["words"] = [(probe[0], words), (probe[1], None)], None
    if flow == "filter":
        state["filter"] = J.BloomFilter(build, bits_per_key=case["bits"])
    elif flow != "join":
        state["table"] = J.HashTable(build, attach=bp if state["attach"] else ())
    if flow == "probe":
        state["out"] = J.allocate_output(state["length"], pp, bp)
        state["d_count"] = torch.zeros(1, dtype=torch.int64, device=DEV)
        if case["native"]:
            state["call"] = _native_probe(state)
    return state


def _native_probe(state):
    """sj_probe_gather with its arguments made once."""
    table, out, lib = state["table"], state["out"], L.load()
    keys, n_keys, _ = J._keys(state["probe"], state["words"])
    pin = J._cols([J.make_column(c) for c in state["pp"]])
    bin_ = None if state["attach"] else J._cols([J.make_column(c) for c in state["bp"]])
    pout = J._cols([J._mut(t, None) for t in out.probe_payload], L.SjMutColumn)
    bout = J._cols([J._mut(t, None) for t in out.build_payload], L.SjMutColumn)
    args = (table.handle, keys, n_keys, pin, len(state["pp"]), bin_, len(state["bp"]), out.probe_rid.data_ptr(),
            out.build_rid.data_ptr(), pout, bout, out.probe_rid.numel(), None,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), state["d_count"].data_ptr())
    return lambda: L.check(lib.sj_probe_gather(*args), "sj_probe_gather")


def run(state):
    flow = state["flow"]
    if flow == "batch":
        with torch.cuda.stream(state["stream"]):
            state["plan"].replay(state["stream"])
            counts, error = state["plan"].counts()
        return {"counts": counts, "error": error, "rows": _BatchRows(state["specs"], counts)}
    if flow == "partition":
        columns, _, offsets = J.hash_partition(state["keys"], state["columns"], state["parts"])
        named = {"column%d" % c: t for c, t in enumerate(columns)}
        return {"offsets": offsets, "rows": _PartitionRows(named, offsets)}
    if flow == "filter":
        mask, valid = state["filter"].contains(state["probe"], state["words"])
        return {"mask": mask, "valid": valid}
    if flow == "join":
        out = J.inner_join(state["build"], state["probe"], None, state["words"], state["pp"], state["bp"])
        return _rows(out, out.count, state["length"])
    table = state["table"]
    build_payload = () if state["attach"] else state["bp"]
    if flow == "probe":
        if "call" in state:
            state["call"]()
        else:
            table.probe_gather(state["probe"], state["words"], state["pp"], build_payload, attached=state["attach"],
                               out=state["out"], d_count=state["d_count"], sync=False)
        return _rows(state["out"], state["d_count"], state["length"])
    out = table.probe_join(KINDS[flow], state["probe"], state["words"], state["pp"],
                           build_payload if flow in ("left", "full") else (),
                           attached=state["attach"] and flow == "left")
    if flow == "mark":
        return {"mark": out.mark, "valid": out.mark_validity}
    return _rows(out, out.count, state["length"])


class _BatchRows(dict):
    """The rows of all joins of a batch, one join after the other, each in canonical order."""

    def __init__(self, specs, counts):
        super().__init__(probe_row=[s.out.probe_rid for s in specs], build_row=[s.out.build_rid for s in specs],
                         probe0=[s.out.probe_payload for s in specs], build0=[s.out.build_payload for s in specs])
        self._counts, self._joins = counts, None

    def __getitem__(self, name):
        if self._joins is None:
            named = [dict(zip(self.keys(), columns)) for columns in zip(*self.values())]
            self._joins = [Rows(c, n, c["probe_row"].numel(), ["probe_row", "build_row"])
                           for c, n in zip(named, self._counts.tolist())]
        return torch.cat([rows[name] for rows in self._joins])


class _PartitionRows(Rows):
    """Rows ordered by partition, then by their columns."""

    def __init__(self, columns, offsets):
        n = next(iter(columns.values())).numel()
        super().__init__(columns, n, n, sorted(columns))
        self._offsets = offsets

    def __getitem__(self, name):
        if self._order is None:
            place = torch.arange(int(self._count), device=DEV)
            self._by = [torch.searchsorted(self._offsets[1:-1].contiguous(), place, right=True)] + self._by
        return super().__getitem__(name)


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def _row_bytes(kinds):
    return sum(WIDTH[k] for k in kinds.split(",") if k)


def work(case):
    """Inputs read once, outputs written once; flops: one comparison of a key for each probe row."""
    flow = case["flow"]
    if flow == "batch":
        mean = (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        rows, width = 10 * mean * case["joins"], WIDTH[case["key"]]
        return {"bytes": rows * (width + 4 + 16 / 1.2) + mean * case["joins"] * (width + 4), "flops": rows}
    n = case["probe"]
    width = 4 if case["key"] == "i4" else 8
    null_bits = n / 8 if case["nulls"] else 0
    if flow == "partition":
        return {"bytes": 2 * n * (width + _row_bytes(case["pp"])) + 8 * case["parts"] + null_bits, "flops": n}
    nb = case["build"]
    hits = n * min(1.0, nb / max(nb, int(nb / case["hit"]))) * (1 - case["nulls"])
    if flow == "filter":
        return {"bytes": n * (width + 1) + nb * case["bits"] / 8 + 2 * null_bits, "flops": n}
    probe_row, build_row = _row_bytes(case["pp"]), _row_bytes(case["bp"])
    read = n * width + null_bits
    if flow == "mark":
        return {"bytes": read + n + n / 8 + nb * width, "flops": n}
    if flow in ("semi", "anti"):
        rows = hits if flow == "semi" else n - hits
        return {"bytes": read + nb * width + rows * (4 + 2 * probe_row), "flops": n}
    rows = _pairs(nb, n) * (1 - case["nulls"]) if case["key"] == "zipf" else n if flow in ("left", "full") else hits
    each = 8 + probe_row + build_row + (0.125 * len([k for k in case["bp"].split(",") if k]) if flow == "left" else 0)
    read += n * probe_row + nb * build_row + (nb * width if flow in ("join", "full") else 0)
    return {"bytes": read + rows * each, "flops": n}


# ---- the same in plain torch ------------------------------------------------------------------------------------

def _matches(build, probe, valid):
    """(probe rows, build rows) of all pairs with equal keys, in canonical order."""
    if isinstance(build, list):
        build = build[0].long() * (1 << 32) + build[1].long()
        probe = probe[0].long() * (1 << 32) + probe[1].long()
    keys, rows = torch.sort(build, stable=True)
    first, last = torch.searchsorted(keys, probe), torch.searchsorted(keys, probe, right=True)
    times = last - first
    if valid is not None:
        times = times * valid
    probe_rows = torch.repeat_interleave(torch.arange(probe.numel(), device=DEV), times)
    ends = times.cumsum(0)
    within = torch.arange(probe_rows.numel(), device=DEV) - (ends - times)[probe_rows]
    return probe_rows, rows[first[probe_rows] + within], times


def _wide(column):
    return column.double() if column.is_floating_point() else column


def _exact_inner(build, probe, valid, pp, bp, length):
    probe_rows, build_rows, _ = _matches(build, probe, valid)
    rows = {"probe_row": probe_rows, "build_row": build_rows}
    rows.update({"probe%d" % c: _wide(t[probe_rows]) for c, t in enumerate(pp)})
    rows.update({"build%d" % c: _wide(t[build_rows]) for c, t in enumerate(bp)})
    return {"count": probe_rows.numel(), "rows": {k: _padded(t, length) for k, t in rows.items()}}


def exact(case, seed):
    flow = case["flow"]
    if flow in ("partition", "filter"):
        return None  # whole numbers of the package's own hash functions
    if flow == "batch":
        every = [_exact_inner(bk, pk, None, [pp], [bp], pk.numel()) for bk, pk, bp, pp in _batch_sides(case, seed)]
        return {"counts": torch.tensor([e["count"] for e in every]), "error": torch.zeros(1, dtype=torch.int32),
                "rows": {k: torch.cat([e["rows"][k] for e in every]) for k in every[0]["rows"]}}
    build, probe, valid, pp, bp = _sides(case, seed)
    if flow in ("probe", "join"):
        return _exact_inner(build, probe, valid, pp, bp, _length(case))
    probe_rows, build_rows, times = _matches(build, probe, valid)
    if flow == "mark":
        found = times > 0
        known = found if valid is None else found | valid
        return {"mark": found, "valid": _words(known if valid is not None else torch.ones_like(found))}
    if flow in ("semi", "anti"):
        kept = torch.nonzero((times > 0) if flow == "semi" else (times == 0)).view(-1)
        rows = {"probe_row": kept}
        rows.update({"probe%d" % c: _wide(t[kept]) for c, t in enumerate(pp)})
        return {"count": kept.numel(), "rows": {k: _padded(t, _length(case)) for k, t in rows.items()}}
    # every probe row; for a full join the unmatched build rows too, which canonical order puts first
    none = -(1 << 31)
    alone = torch.nonzero(times == 0).view(-1)
    p, b = torch.cat([probe_rows, alone]), torch.cat([build_rows, torch.full_like(alone, none)])
    if flow == "full":
        seen = torch.zeros(case["build"], dtype=torch.bool, device=DEV)
        seen[build_rows] = True
        left = torch.nonzero(~seen).view(-1)
        p, b = torch.cat([p, torch.full_like(left, none)]), torch.cat([b, left])
    order = torch.sort(b, stable=True).indices
    order = order[torch.sort(p[order], stable=True).indices]
    p, b = p[order], b[order]
    rows = {"probe_row": p, "build_row": b}
    for side, index, columns in (("probe", p, pp), ("build", b, bp)):
        for c, t in enumerate(columns):
            rows["%s%d" % (side, c)] = _wide(t[index.clamp(min=0)]).masked_fill(index < 0, 0)
            if side == "build" or flow == "full":
                rows["%s%d_valid" % (side, c)] = index >= 0
    return {"count": p.numel(), "rows": {k: _padded(t, _length(case)) for k, t in rows.items()}}
