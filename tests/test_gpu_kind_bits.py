"""SEMI / ANTI / MARK / LEFT by match bits: row counts at the edges of words (32), units (128), select CTAs (8192
rows) and of the sizes that take two passes; a table that is looked up in partition order, with NULL keys and int32
and wide slots; an allocator that refuses the bits."""
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


@pytest.mark.parametrize("dtype,wide", [(np.int32, False), (np.int64, False), (np.int64, True)])
@pytest.mark.parametrize("far", [0.0, 0.4])
def test_lookup_in_partition_order(cuda, dtype, wide, far):
    """More than 64 MB of slots, and a probe that touches each sector twice or more; `far` of the rows' keys lie
    outside the build's range, on both sides, and take no part in the partition."""
    rng = np.random.default_rng(3)
    nb = (2 << 20) + 5 if wide else (5 << 20)
    bk = rng.permutation(3 * nb)[:nb].astype(dtype)
    n = 16_800_019
    pk = rng.integers(0, 3 * nb, n).astype(dtype)
    pk = np.where(rng.random(n) < far, np.where(pk % 2, -1 - pk, 3 * nb + pk), pk).astype(dtype)
    _check(cuda, bk, pk, rng.random(n) > 0.03, [rng.integers(0, 100, n).astype(np.int32)], force_wide=wide, load_factor=0.4)


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
def test_refused_scratch_takes_the_pass_without(cuda, kind):
    """An allocator that refuses everything after the build: the join still runs, with the same rows."""
    rng = np.random.default_rng(8)
    bk = dev_t(rng.permutation(40_000)[:20_000].astype(np.int64), cuda)
    pk = dev_t(rng.integers(0, 40_000, 17_000_001).astype(np.int64), cuda)
    with J.HashTable(bk) as t:
        want = t.probe_join(kind, pk)
        A, F = L.SjAlloc._fields_[1][1], L.SjAlloc._fields_[2][1]
        refuse = L.SjAlloc(None, A(lambda ctx, size, s: None), F(lambda ctx, p, size, s: None))
        n = pk.numel()
        rid = torch.empty(n, dtype=torch.int32, device=cuda)
        mark = torch.empty(n, dtype=torch.uint8, device=cuda)
        words = torch.empty((n + 31) // 32, dtype=torch.int32, device=cuda)
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        keys, nk, _ = J._keys(pk)
        st = L.load().sj_probe_join(t.handle, kind, keys, nk, None, 0, None, 0, rid.data_ptr(), None, None, None, n,
                                    mark.data_ptr(), words.data_ptr(), ctypes.byref(refuse), None, dc.data_ptr())
        torch.cuda.synchronize()
        assert st == L.SJ_OK
        if kind == L.SJ_JOIN_MARK:
            assert torch.equal(mark, want.mark) and torch.equal(words, want.mark_validity)
        else:
            assert int(dc.item()) == want.count
            assert torch.equal(rid[:want.count].sort().values, want.probe_rid[:want.count].sort().values)
