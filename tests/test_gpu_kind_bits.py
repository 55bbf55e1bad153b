"""SEMI / ANTI / MARK / LEFT: row counts at the edges of words (32), units (32 and 128 rows), CTAs (1024) and select
CTAs (8192 rows); capacities that cut the output; tables that are looked up in partition order (unique, duplicated
and NULL build keys, int32 and wide slots, few and many keys in the build's range); allocators that refuse the
scratch, budgets that hold a part of it, and a capture."""
import ctypes

import numpy as np
import pytest
import torch

from jhelp import dev_t, dev_valid
from oracle import oracle as O
from sirius_b200 import _lib as L
from sirius_b200 import join as J

pytestmark = pytest.mark.gpu


def _check(cuda, bk, pk, pv, pp, capacity=None, **kw):
    dpk, dpv = dev_t(pk, cuda), None if pv is None else dev_valid(O.pack_validity(pv), cuda)
    valid = np.ones(len(pk), bool) if pv is None else pv
    hit = np.isin(pk, bk) & valid
    with J.HashTable(dev_t(bk, cuda), attach=[dev_t(bk, cuda)], **kw) as t:
        for kind, keep in ((L.SJ_JOIN_SEMI, hit), (L.SJ_JOIN_ANTI, ~hit)):
            out = t.probe_join(kind, dpk, dpv, [dev_t(c, cuda) for c in pp], capacity=capacity)
            rid = out.probe_rid[:out.count].cpu().numpy()
            assert np.array_equal(np.sort(rid), np.nonzero(keep)[0])
            for c, got in zip(pp, out.probe_payload):
                assert np.array_equal(got[:out.count].cpu().numpy(), c[rid])
        m = t.probe_join(L.SJ_JOIN_MARK, dpk, dpv)
        assert np.array_equal(m.mark.cpu().numpy().astype(bool), hit)
        words = m.mark_validity.cpu().numpy().view(np.uint32)
        assert np.array_equal(O.unpack_validity(words, len(words) * 32)[:len(pk)], hit | valid)
        assert not O.unpack_validity(words, len(words) * 32)[len(pk):].any()
        out = t.probe_join(L.SJ_JOIN_LEFT, dpk, dpv, [dev_t(c, cuda) for c in pp], attached=True)
        rid, brid = out.probe_rid[:out.count].cpu().numpy(), out.build_rid[:out.count].cpu().numpy()
        assert np.array_equal(np.sort(rid), np.arange(len(pk)))
        assert np.array_equal(brid != -2**31, hit[rid])
        assert np.array_equal(bk[brid[hit[rid]]], pk[rid[hit[rid]]])
        for c, got in zip(pp, out.probe_payload):
            assert np.array_equal(got[:out.count].cpu().numpy(), c[rid])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 1023, 1025, 8191, 8192, 8193, 100_001,
                               (16 << 20) - 1, 16 << 20, (16 << 20) + 8193])
@pytest.mark.parametrize("types", [(), (np.int64,), (np.int8, np.int32), (np.float32, np.int16)])
def test_row_count_edges(cuda, n, types):
    rng = np.random.default_rng(n + len(types))
    bk = rng.permutation(5000)[:1500].astype(np.int64)
    pk = rng.integers(0, 5000, n).astype(np.int64)
    pv = rng.random(n) > 0.2 if n % 2 else None
    _check(cuda, bk, pk, pv, [rng.integers(0, 100, n).astype(t) for t in types], capacity=n)


def _bits(words, n):
    return ((words[:, None] >> torch.arange(32, device=words.device, dtype=torch.int32)) & 1).view(-1)[:n].bool()


def _ordered(cuda, dtype, n, far, dup=False, bnull=False, nulls=0.0, seed=3, **kw):
    """A build whose slots take 256 MB, and a probe of n rows: (build, its validity or None, probe, its validity,
    match per row), `far` of the probe's keys outside the build's range. All on the GPU."""
    g = torch.Generator(device=cuda)
    g.manual_seed(seed)
    nb = (1_700_003 if kw.get("force_wide") else 3_400_003) * (3 if bnull else 2) // 2
    bk = torch.randperm(3 * nb, device=cuda, generator=g)[:nb].to(dtype)
    if dup:  # most keys twice
        bk[nb // 2:] = bk[: nb - nb // 2].clone()
    bv = torch.rand(nb, device=cuda, generator=g) > 0.3 if bnull else None
    pk = torch.randint(0, 3 * nb, (n,), device=cuda, generator=g)
    pv = torch.rand(n, device=cuda, generator=g) >= nulls
    there = torch.zeros(3 * nb, dtype=torch.bool, device=cuda)
    there[(bk if bv is None else bk[bv]).long()] = True
    out = torch.rand(n, device=cuda, generator=g) < far
    hit = there[pk] & ~out & pv
    pk = torch.where(out, torch.where(pk % 2 == 0, -1 - pk, 3 * nb + pk), pk).to(dtype)
    return bk, bv, pk, pv, hit


def _words(valid):
    n = valid.numel()
    padded = torch.zeros((n + 31) // 32 * 32, dtype=torch.int64, device=valid.device)
    padded[:n] = valid
    return (padded.view(-1, 32) << torch.arange(32, device=valid.device)).sum(1).to(torch.int32)


ORDERED_ROWS = 33_600_019


@pytest.mark.parametrize("dtype,wide", [(torch.int32, False), (torch.int64, False), (torch.int64, True)])
@pytest.mark.parametrize("far,dup,bnull", [(0.0, False, False), (0.1, True, False), (0.1, False, True), (0.9, False, False)])
def test_lookup_in_partition_order(cuda, dtype, wide, far, dup, bnull):
    """256 MB of slots, and a probe that touches each sector four times. Where few keys lie in the build's range the
    device goes back to the lookup in place. NULL build keys make every unmatched row of a MARK NULL."""
    kw = dict(force_wide=wide, load_factor=0.2)
    bk, bv, pk, pv, hit = _ordered(cuda, dtype, ORDERED_ROWS, far, dup, bnull, 0.03, **kw)
    n, pw = pk.numel(), _words(pv)
    pay = torch.randint(0, 100, (n,), device=cuda).to(torch.int16)
    layout = L.SJ_LAYOUT_GROUPED if dup else L.SJ_LAYOUT_DISTINCT
    with J.HashTable(bk, None if bv is None else _words(bv), layout=layout, **kw) as t:
        info = t.info()
        assert info.layout == layout and info.partition_bits > 0
        assert info.num_slots * (16 if wide else 8) >= 256 << 20
        L.timing_collect()
        L.timing_enable(True)
        try:
            for kind, keep in ((L.SJ_JOIN_SEMI, hit), (L.SJ_JOIN_ANTI, ~hit)):
                out = t.probe_join(kind, pk, pw, [pay])
                rid = out.probe_rid[:out.count].long()
                assert torch.equal(torch.sort(rid).values, torch.nonzero(keep).view(-1))
                assert torch.equal(out.probe_payload[0][:out.count], pay[rid])
            m = t.probe_join(L.SJ_JOIN_MARK, pk, pw)
        finally:
            L.timing_enable(False)
        names = [name for name, _ in L.timing_collect()]
        assert names.count("find_units") == 3, names
    assert torch.equal(m.mark.bool(), hit)
    assert torch.equal(_bits(m.mark_validity, n), hit | (pv if bv is None else torch.zeros_like(hit)))


@pytest.mark.parametrize("far", [0.0, 0.9])
@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI])
@pytest.mark.parametrize("capacity", [0, 1, 1000, 5_000_033])
def test_capacity_cuts_rows_found_in_partition_order(cuda, far, kind, capacity):
    bk, _, pk, _, hit = _ordered(cuda, torch.int64, ORDERED_ROWS, far, seed=4)
    pay = torch.arange(pk.numel(), dtype=torch.int64, device=cuda)
    with J.HashTable(bk, load_factor=0.2) as t:
        _check_cut(cuda, t, kind, pk, pay, None, capacity)


def _check_cut(cuda, t, kind, pk, pay, pay_valid, capacity):
    """The rows up to the capacity are right, none twice, the count is of all, and nothing is written behind."""
    guard, n = 4096, pk.numel()
    full = t.probe_join(kind, pk, None, [pay])
    want = full.probe_rid[:full.count].long()
    keep = torch.zeros(n, dtype=torch.bool, device=cuda)
    keep[want] = True
    rid = torch.full((capacity + guard,), -7, dtype=torch.int32, device=cuda)
    got = torch.full((capacity + guard,), -7, dtype=pay.dtype, device=cuda)
    words = torch.full(((capacity + 31) // 32 + guard,), 0x55555555, dtype=torch.int32, device=cuda)
    dc = torch.zeros(1, dtype=torch.int64, device=cuda)
    keys, nk, _ = J._keys(pk)
    pin = J._cols([J.make_column(pay, pay_valid)])
    pout = J._cols([J._mut(got, words)], L.SjMutColumn)
    L.check(L.load().sj_probe_join(t.handle, kind, keys, nk, pin, 1, None, 0, rid.data_ptr(), None, pout, None, capacity,
                                   None, None, None, None, dc.data_ptr()), "sj_probe_join")
    torch.cuda.synchronize()
    assert int(dc.item()) == full.count
    m = min(capacity, full.count)
    r = rid[:m].long()
    assert bool(keep[r].all()) and torch.unique(r).numel() == m
    assert torch.equal(got[:m], pay[r])
    assert bool((rid[m:] == -7).all()) and bool((got[m:] == -7).all())
    if pay_valid is not None:
        assert torch.equal(_bits(words, m), _bits(pay_valid, n)[r])
        assert bool((words[(capacity + 31) // 32:] == 0x55555555).all())


@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI])
@pytest.mark.parametrize("capacity", [0, 1, 31, 33, 1000, 20_001, 60_000])
@pytest.mark.parametrize("nullable", [False, True])
def test_capacity_cuts_rows_found_in_place(cuda, kind, capacity, nullable):
    rng = np.random.default_rng(capacity)
    bk = dev_t(rng.permutation(40_000)[:20_000].astype(np.int64), cuda)
    pk = dev_t(rng.integers(-5000, 45_000, 50_021).astype(np.int64), cuda)
    pay = dev_t(rng.integers(0, 100, 50_021).astype(np.int8), cuda)
    pw = dev_valid(O.pack_validity(rng.random(50_021) > 0.4), cuda) if nullable else None
    with J.HashTable(bk) as t:
        _check_cut(cuda, t, kind, pk, pay, pw, capacity)


@pytest.mark.parametrize("capacity", [1, 700, 30_000])
@pytest.mark.parametrize("layout", [L.SJ_LAYOUT_DISTINCT, L.SJ_LAYOUT_GROUPED])
@pytest.mark.parametrize("pbits", [-1, 3])
def test_left_whose_inner_rows_overflow(cuda, capacity, layout, pbits):
    """The count is of all rows, those written are INNER rows, and nothing is written behind the capacity."""
    rng = np.random.default_rng(6)
    bk = rng.permutation(60_000)[:40_000].astype(np.int64)
    pk = rng.integers(0, 60_000, 70_003).astype(np.int64)
    with J.HashTable(dev_t(bk, cuda), layout=layout, partition_bits=pbits) as t:
        rid = torch.full((2, capacity + 512), -7, dtype=torch.int32, device=cuda)
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        keys, nk, _ = J._keys(dev_t(pk, cuda))
        L.check(L.load().sj_probe_join(t.handle, L.SJ_JOIN_LEFT, keys, nk, None, 0, None, 0, rid[0].data_ptr(),
                                       rid[1].data_ptr(), None, None, capacity, None, None, None, None, dc.data_ptr()),
                "sj_probe_join")
        torch.cuda.synchronize()
    assert int(dc.item()) == len(pk)
    p, b = rid[:, :capacity].cpu().numpy()
    assert len(np.unique(p)) == capacity and np.array_equal(bk[b], pk[p])
    assert bool((rid[:, capacity:] == -7).all())


@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI, L.SJ_JOIN_MARK])
def test_captured_join_asks_for_no_scratch(cuda, kind):
    """A graph keeps no memory of the caller's allocator: the captured call, which would be looked up in partition
    order, allocates nothing, and its replays see new probe keys."""
    bk, _, pk, _, hit = _ordered(cuda, torch.int64, ORDERED_ROWS, 0.0, seed=5)
    n = pk.numel()
    rid = torch.empty(n, dtype=torch.int32, device=cuda)
    mark = torch.empty(n, dtype=torch.uint8, device=cuda)
    words = torch.empty((n + 31) // 32, dtype=torch.int32, device=cuda)
    dc = torch.zeros(1, dtype=torch.int64, device=cuda)
    col, nk, _ = J._keys(pk)
    with J.HashTable(bk, load_factor=0.2) as t:
        def call(stream, alloc=None):
            return L.load().sj_probe_join(t.handle, kind, col, nk, None, 0, None, 0, rid.data_ptr(), None, None, None, n,
                                          mark.data_ptr(), words.data_ptr(), alloc, stream, dc.data_ptr())
        call(torch.cuda.current_stream().cuda_stream)  # kernels loaded before the capture
        torch.cuda.synchronize()
        budget = Budget(cuda)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            st = call(torch.cuda.current_stream().cuda_stream, ctypes.byref(budget.c))
        assert st == L.SJ_OK and budget.peak == 0
        for flip in (False, True):
            if flip:
                pk.copy_(torch.flip(pk, [0]))
                hit = torch.flip(hit, [0])
            g.replay()
            torch.cuda.synchronize()
            if kind == L.SJ_JOIN_MARK:
                assert torch.equal(mark.bool(), hit)
            else:
                m = int(dc.item())
                keep = hit if kind == L.SJ_JOIN_SEMI else ~hit
                assert torch.equal(torch.sort(rid[:m].long()).values, torch.nonzero(keep).view(-1))
        del g


@pytest.mark.parametrize("n", [33, 1025, 300_001])
@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI, L.SJ_JOIN_MARK])
def test_validity_at_odd_bit_offsets(cuda, kind, n):
    """Slices of columns: key and payload bitmasks that do not start at a word, mark bytes that do not start at four."""
    rng = np.random.default_rng(n)
    bk, pk = rng.permutation(4000)[:2000].astype(np.int32), rng.integers(-500, 4500, n).astype(np.int32)
    pv, av = rng.random(n) > 0.2, rng.random(n) > 0.4
    hit = np.isin(pk, bk) & pv
    pay = dev_t(rng.integers(0, 100, n).astype(np.int16), cuda)

    def words(v, offset):
        return dev_valid(O.pack_validity(np.concatenate([rng.random(offset) > 0.5, v])), cuda)
    kw, aw = words(pv, 37), words(av, 5)
    dpk = dev_t(pk, cuda)
    keys = J._cols([J.make_column(dpk, kw, 37)])
    pin = J._cols([J.make_column(pay, aw, 5)])
    rid = torch.empty(n, dtype=torch.int32, device=cuda)
    out, ow = torch.empty_like(pay), torch.empty((n + 31) // 32, dtype=torch.int32, device=cuda)
    mark, mw = torch.empty(n + 3, dtype=torch.uint8, device=cuda)[3:], torch.empty_like(ow)
    dc = torch.zeros(1, dtype=torch.int64, device=cuda)
    with J.HashTable(dev_t(bk, cuda)) as t:
        L.check(L.load().sj_probe_join(t.handle, kind, keys, 1, pin, 1, None, 0, rid.data_ptr(), None,
                                       J._cols([J._mut(out, ow)], L.SjMutColumn), None, n, mark.data_ptr(),
                                       mw.data_ptr(), None, None, dc.data_ptr()), "sj_probe_join")
        torch.cuda.synchronize()
    if kind == L.SJ_JOIN_MARK:
        assert np.array_equal(mark.cpu().numpy().astype(bool), hit)
        assert np.array_equal(_bits(mw, n).cpu().numpy(), hit | pv)
        return
    m = int(dc.item())
    r = rid[:m].cpu().numpy()
    assert np.array_equal(np.sort(r), np.nonzero(hit if kind == L.SJ_JOIN_SEMI else ~hit)[0])
    assert np.array_equal(out[:m].cpu().numpy(), pay.cpu().numpy()[r])
    assert np.array_equal(_bits(ow, m).cpu().numpy(), av[r])


@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI])
def test_nulls_equal_and_null_build_keys_in_place(cuda, kind):
    """NULL probe keys match the NULL group, if the build has one (MARK compares NULLs as unequal)."""
    rng = np.random.default_rng(1)
    n = 450_003  # units of 128 rows
    bk, pk = rng.integers(0, 3000, 2000).astype(np.int64), rng.integers(0, 6000, n).astype(np.int64)
    pv = rng.random(n) > 0.2
    for bv in (rng.random(2000) > 0.1, np.ones(2000, bool)):
        hit = np.where(pv, np.isin(pk, bk[bv]), not bv.all())
        with J.HashTable(dev_t(bk, cuda), dev_valid(O.pack_validity(bv), cuda), null_equality=L.SJ_NULLS_EQUAL) as t:
            out = t.probe_join(kind, dev_t(pk, cuda), dev_valid(O.pack_validity(pv), cuda))
        got = np.sort(out.probe_rid[:out.count].cpu().numpy())
        assert np.array_equal(got, np.nonzero(hit if kind == L.SJ_JOIN_SEMI else ~hit)[0])


class Budget:
    """An allocator over torch tensors that refuses what would take more than `limit` bytes at a time."""

    def __init__(self, cuda, limit=1 << 62):
        self.limit, self.live, self.peak, held = limit, 0, 0, {}

        def alloc(ctx, size, stream):
            if self.live + size > self.limit:
                return None
            t = torch.empty(max(1, size), dtype=torch.uint8, device=cuda)
            held[t.data_ptr()] = (t, size)
            self.live += size
            self.peak = max(self.peak, self.live)
            return t.data_ptr()

        def free(ctx, p, size, stream):
            self.live -= held.pop(p)[1]
        self._calls = L.SjAlloc._fields_[1][1](alloc), L.SjAlloc._fields_[2][1](free)
        self.c = L.SjAlloc(None, *self._calls)


def _join_under(budget, t, kind, pk, n_out, rids=True):
    """(status, count, probe row ids, build row ids) of a join whose scratch comes from `budget`."""
    rid = [torch.empty(max(1, n_out), dtype=torch.int32, device=pk.device) for _ in range(2)]
    dc = torch.zeros(1, dtype=torch.int64, device=pk.device)
    keys, nk, _ = J._keys(pk)
    p = [r.data_ptr() if rids else None for r in rid]
    st = L.load().sj_probe_join(t.handle, kind, keys, nk, None, 0, None, 0, *p, None, None, n_out, None, None,
                                ctypes.byref(budget.c), None, dc.data_ptr())
    torch.cuda.synchronize()
    return st, int(dc.item()), rid[0], rid[1]


@pytest.mark.parametrize("kind", [L.SJ_JOIN_LEFT, L.SJ_JOIN_FULL])
@pytest.mark.parametrize("layout", [L.SJ_LAYOUT_DISTINCT, L.SJ_LAYOUT_GROUPED])
@pytest.mark.parametrize("pbits", [-1, 3])
def test_outer_joins_need_no_more_than_the_larger_of_their_parts(cuda, kind, layout, pbits):
    """The match bits are not worth a refusal: with room for the INNER probe's scratch or the bits, not both."""
    rng = np.random.default_rng(2)
    bk = rng.permutation(300_000)[:200_000].astype(np.int64)
    pk = dev_t(rng.integers(0, 300_000, 1_000_000).astype(np.int64), cuda)
    bits = 1_000_000 // 8
    with J.HashTable(dev_t(bk, cuda), layout=layout, partition_bits=pbits) as t:
        inner = Budget(cuda)
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        out = torch.empty(1_000_000, dtype=torch.int32, device=cuda)
        keys, nk, _ = J._keys(pk)
        L.check(L.load().sj_probe_gather(t.handle, keys, nk, None, 0, None, 0, out.data_ptr(), None, None, None,
                                         1_000_000, ctypes.byref(inner.c), None, dc.data_ptr()), "sj_probe_gather")
        torch.cuda.synchronize()
        n_out = 1_000_000 + (200_000 if kind == L.SJ_JOIN_FULL else 0)
        st, want, p, b = _join_under(Budget(cuda), t, kind, pk, n_out)
        assert st == L.SJ_OK and want == 1_000_000 + (
            200_000 - len(np.intersect1d(bk, pk.cpu().numpy())) if kind == L.SJ_JOIN_FULL else 0)
        rows = O.canonical(p[:want].cpu().numpy(), b[:want].cpu().numpy())
        # the two counters of the call, and for FULL its flag bytes (one per slot) and build-row bits
        later = (int(t.info().num_slots) + 1 + 200_000 // 8 + 64 if kind == L.SJ_JOIN_FULL else 0)
        budget = Budget(cuda, 16 + max(inner.peak, bits + later))
        st, got, p, b = _join_under(budget, t, kind, pk, n_out)
        assert st == L.SJ_OK, (st, L.load().sj_last_error())
        assert got == want
        for x, y in zip(rows, O.canonical(p[:got].cpu().numpy(), b[:got].cpu().numpy())):
            assert np.array_equal(x, y)
        # no row ids wanted: no bits are needed either
        st, got, _, _ = _join_under(Budget(cuda, 16 + max(inner.peak, later)), t, kind, pk, n_out, rids=False)
        assert st == L.SJ_OK and got == want


@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI, L.SJ_JOIN_MARK])
@pytest.mark.parametrize("room", [0, ORDERED_ROWS // 8 + 64])
def test_refused_scratch_takes_the_pass_without(cuda, kind, room):
    """An allocator that refuses everything after the build, or all but the bits: the join still runs, with the same
    rows."""
    bk, _, pk, _, _ = _ordered(cuda, torch.int64, ORDERED_ROWS, 0.0, seed=8)
    with J.HashTable(bk, load_factor=0.2) as t:
        want = t.probe_join(kind, pk)
        n = pk.numel()
        rid = torch.empty(n, dtype=torch.int32, device=cuda)
        mark = torch.empty(n, dtype=torch.uint8, device=cuda)
        words = torch.empty((n + 31) // 32, dtype=torch.int32, device=cuda)
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        keys, nk, _ = J._keys(pk)
        budget = Budget(cuda, room)
        st = L.load().sj_probe_join(t.handle, kind, keys, nk, None, 0, None, 0, rid.data_ptr(), None, None, None, n,
                                    mark.data_ptr(), words.data_ptr(), ctypes.byref(budget.c), None, dc.data_ptr())
        torch.cuda.synchronize()
        assert st == L.SJ_OK and budget.live == 0
        if kind == L.SJ_JOIN_MARK:
            assert torch.equal(mark, want.mark) and torch.equal(words, want.mark_validity)
        else:
            assert int(dc.item()) == want.count
            assert torch.equal(rid[:want.count].sort().values, want.probe_rid[:want.count].sort().values)


@pytest.mark.parametrize("kind", [L.SJ_JOIN_SEMI, L.SJ_JOIN_ANTI, L.SJ_JOIN_MARK])
def test_composite_keys_need_scratch(cuda, kind):
    """The packed key column is scratch of every kind: refused, the call says so."""
    k = [dev_t(np.arange(5000, dtype=np.int32) // m, cuda) for m in (1, 7)]
    with J.HashTable(k) as t:
        rid = torch.empty(5000, dtype=torch.int32, device=cuda)
        mark = torch.empty(5000, dtype=torch.uint8, device=cuda)
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        keys, nk, _ = J._keys(k)
        for limit, want in ((-1, L.SJ_ERR_OOM), (1 << 20, L.SJ_OK)):
            st = L.load().sj_probe_join(t.handle, kind, keys, nk, None, 0, None, 0, rid.data_ptr(), None, None, None, 5000,
                                        mark.data_ptr(), None, ctypes.byref(Budget(cuda, limit).c), None, dc.data_ptr())
            torch.cuda.synchronize()
            assert st == want
