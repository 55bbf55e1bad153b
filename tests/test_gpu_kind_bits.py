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
def test_lookup_in_partition_order(cuda, dtype, wide):
    """More than 64 MB of slots, and a probe that touches each sector twice or more."""
    rng = np.random.default_rng(3)
    nb = (2 << 20) + 5 if wide else (5 << 20)
    bk = rng.permutation(3 * nb)[:nb].astype(dtype)
    n = 16_800_019
    pk = rng.integers(0, 3 * nb, n).astype(dtype)
    _check(cuda, bk, pk, rng.random(n) > 0.03, [rng.integers(0, 100, n).astype(np.int32)], force_wide=wide, load_factor=0.4)


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
