"""The unit probe at the edges of its units and CTAs: row counts around 32, 128, 256 and 1024 rows and around the
switch from 32-row to 128-row units, tile-local partitions around their 4096-row tiles, buckets that overflow
(load factor 0.97), all hits, no hits, NULL probe keys at an odd bit offset, tables without a valid key, and keys
whose slot image is all ones."""
import numpy as np
import pytest
import torch

from jhelp import assert_same_rows, dev_t, dev_valid, oracle_join
from oracle import oracle as O
from sirius_b200 import _lib as L
from sirius_b200 import datagen as D
from sirius_b200 import join as J

pytestmark = pytest.mark.gpu


def _join(cuda, bk, pk, bp, pp, pv=None, bv=None, attach=True, **kw):
    with J.HashTable(dev_t(bk, cuda), dev_valid(bv, cuda), attach=[dev_t(c, cuda) for c in bp] if attach else (), **kw) as t:
        out = t.probe_gather(dev_t(pk, cuda), dev_valid(pv, cuda), [dev_t(c, cuda) for c in pp],
                             () if attach else [dev_t(c, cuda) for c in bp], attached=attach).trimmed()
    got = [x.cpu().numpy() for x in [out.probe_rid, out.build_rid] + out.probe_payload + out.build_payload]
    assert_same_rows(got, oracle_join(D.JoinInput("units", bk, pk, bp, pp, bv, pv)))
    return len(got[0])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025, 399_999, 400_000,
                               400_001, 401_025])
@pytest.mark.parametrize("dtype,bp_types", [(np.int32, (np.int32,)), (np.int64, (np.int64, np.float64)),
                                            (np.int64, (np.int32, np.int64))])
def test_unit_edges(cuda, n, dtype, bp_types):
    rng = np.random.default_rng(n)
    nb = max(1, n // 7)
    bk = rng.permutation(4 * nb)[:nb].astype(dtype)
    pk = rng.integers(0, 4 * nb, n).astype(dtype)
    pv = O.pack_validity(rng.random(n) > 0.1) if n % 2 else None
    bp = [rng.integers(0, 1 << 30, nb).astype(t) for t in bp_types]
    pp = [rng.integers(0, 1 << 30, n).astype(np.int64)]
    _join(cuda, bk, pk, bp, pp, pv, attach=n % 3 != 0)


@pytest.mark.parametrize("n", [65_536, 16 * 4096 - 1, 16 * 4096 + 1, 300_007])
@pytest.mark.parametrize("pbits", [1, 4, 5, 6, 8, 10])
@pytest.mark.parametrize("wide", [False, True])
def test_partition_runs(cuda, n, pbits, wide):
    """From 64 partitions on a unit joins the runs of 2, 8 or 32 tiles, of which there may be fewer. The share is small
    enough for the probe to take as many partitions as the table has."""
    rng = np.random.default_rng(n + pbits)
    nb = 40_000 if pbits < 5 else 40_000 << pbits - 4  # at least 1 MB of slots and records for each partition
    bk = (rng.permutation(3 * nb)[:nb]).astype(np.int64)
    pk = rng.integers(0, 3 * nb, n).astype(np.int64)
    pk[: n // 3] = bk[0]  # one hot key: long runs of one partition
    pv = O.pack_validity(rng.random(n) > 0.05)
    bp = [rng.integers(0, 1 << 40, nb).astype(np.int64)]
    _join(cuda, bk, pk, bp, [], pv, partition_bits=pbits, force_wide=wide, probe_partition_mb=1)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("far", [0.4, 1.0])
def test_partition_runs_without_keys_outside_the_range(cuda, dtype, full, far):
    """The partition drops what lies outside the build's key range, the type's ends among it; with a build that holds
    both ends of the type nothing lies outside."""
    rng = np.random.default_rng(9)
    info, nb, n = np.iinfo(dtype), 30_000, 200_003
    bk = (rng.permutation(3 * nb)[:nb] - nb).astype(dtype)
    if full:
        bk[:2] = info.min, info.max
    pk = rng.integers(-nb, 2 * nb, n).astype(dtype)
    ends = np.array([info.min, info.min + 1, bk.min() - (not full), bk.max() + (not full), info.max - 1, info.max])
    pk = np.where(rng.random(n) < far, rng.choice(ends.astype(dtype), n), pk)
    pv = O.pack_validity(rng.random(n) > 0.05)
    rows = _join(cuda, bk, pk, [rng.integers(0, 9, nb).astype(np.int64)], [rng.integers(0, 9, n).astype(np.int32)], pv,
                 partition_bits=4)
    assert (rows > 0) == (full or far < 1)
    with J.HashTable(dev_t(bk, cuda), partition_bits=4) as t:
        left = t.probe_join(L.SJ_JOIN_LEFT, dev_t(pk, cuda), dev_valid(pv, cuda))
    prid, brid = left.probe_rid[:left.count].cpu().numpy(), left.build_rid[:left.count].cpu().numpy()
    assert np.array_equal(np.sort(prid), np.arange(n)) and (brid >= 0).sum() == rows
    assert np.array_equal(bk[brid[brid >= 0]], pk[prid[brid >= 0]])


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("hits", [0.0, 1.0])
def test_full_buckets(cuda, wide, hits):
    rng = np.random.default_rng(5)
    nb = 127_000  # of 131,072 slots
    bk = rng.permutation(1 << 20)[:nb].astype(np.int64) * 2
    pk = rng.choice(bk, 500_000) + (0 if hits else 1)
    rows = _join(cuda, bk, pk, [rng.integers(0, 9, nb).astype(np.int64)], [], load_factor=0.97, force_wide=wide)
    assert rows == (len(pk) if hits else 0)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("wide", [False, True])
def test_no_valid_build_key(cuda, dtype, wide):
    """Every slot is EMPTY (all ones): no key may match it, whatever its bits."""
    nb = 50_000
    info = np.iinfo(dtype)
    pk = np.concatenate([np.arange(-70_000, 70_000), [info.min, info.max, -1, 0]]).astype(dtype)
    assert _join(cuda, np.arange(nb, dtype=dtype), pk, [], [], bv=O.pack_validity(np.zeros(nb, bool)), force_wide=wide) == 0


def test_keys_near_the_empty_image(cuda):
    """Keys that fill the packed key field up to one below all ones, and probes above and below the range."""
    nb = 1 << 16
    top = (1 << 48) - 2  # 16 row-id bits: the key field's largest live value
    bk = np.concatenate([np.arange(nb - 1), [top]]).astype(np.int64) - 5
    pk = np.concatenate([bk[-9:], bk[:9], [top - 4, top - 3, top + (1 << 48), -6, -1 << 62, (1 << 62) + 3]]).astype(np.int64)
    pk = np.tile(pk, 30_000)
    assert _join(cuda, bk, pk, [], []) == 18 * 30_000
