"""GROUPED probes at the edges of the expand's 256-output tiles, 8-tile runs and 32-entry staging: groups of one row,
of about 32, 256 and 2048 rows and one of 300,000, every row a match or few, NULL keys equal, and capacities that
cut a tile. Record shapes with compile-time write-out (one 4- or 8-byte payload) and without."""
import numpy as np
import pytest
import torch

from jhelp import assert_same_rows, dev_t, dev_valid, oracle_join
from oracle import oracle as O
from sirius_b200 import _lib as L
from sirius_b200 import datagen as D
from sirius_b200 import join as J

pytestmark = pytest.mark.gpu


def _run(cuda, sizes, n_probe, types, seed, capacity=None, null_frac=0.0, absent=0.0, nulls_equal=False, build_nulls=0):
    rng = np.random.default_rng(seed)
    keys = rng.permutation(4 * len(sizes))[: len(sizes)].astype(np.int64)
    bk = np.repeat(keys, sizes)
    bk = bk[rng.permutation(len(bk))]
    bv = None
    if build_nulls:
        valid = np.ones(len(bk), bool)
        valid[rng.permutation(len(bk))[:build_nulls]] = False
        bv = O.pack_validity(valid)
    pk = np.where(rng.random(n_probe) < absent, -5, rng.choice(keys, n_probe)).astype(np.int64)
    pv = O.pack_validity(rng.random(n_probe) >= null_frac) if null_frac else None
    bp = [rng.integers(0, 1 << 30, len(bk)).astype(t) for t in types]
    inp = D.JoinInput("expand", bk, pk, bp, [], bv, pv)
    rule = L.SJ_NULLS_EQUAL if nulls_equal else L.SJ_NULLS_UNEQUAL
    with J.HashTable(dev_t(bk, cuda), dev_valid(bv, cuda), attach=[dev_t(c, cuda) for c in bp],
                     layout=L.SJ_LAYOUT_GROUPED, null_equality=rule) as t:
        out = J.allocate_output(capacity, (), [dev_t(c, cuda) for c in bp]) if capacity else None
        dc = torch.zeros(1, dtype=torch.int64, device=cuda)
        total = int(t.count(dev_t(pk, cuda), dev_valid(pv, cuda)).item())
        out = t.probe_gather(dev_t(pk, cuda), dev_valid(pv, cuda), attached=True, out=out, d_count=dc, sync=False)
    torch.cuda.synchronize()
    exp = oracle_join(inp, nulls_equal)
    assert int(dc.item()) == total == len(exp[0])
    n = min(total, capacity or total)
    got = [x[:n].cpu().numpy() for x in [out.probe_rid, out.build_rid] + out.build_payload]
    if n == total:
        assert_same_rows(got, exp)
        return
    pairs = set(zip(exp[0].tolist(), exp[1].tolist()))  # a prefix of the rows, in no order: each one right, none twice
    assert len({(p, b) for p, b in zip(got[0].tolist(), got[1].tolist())} & pairs) == n
    for c, g in zip(bp, got[2:]):
        assert np.array_equal(g, c[got[1]])


SIZES = {"ones": lambda r: np.ones(3000, int), "small": lambda r: r.integers(1, 12, 2000),
         "warp": lambda r: r.integers(31, 34, 300), "tile": lambda r: r.integers(255, 258, 40),
         "run": lambda r: np.array([2047, 2048, 2049, 1]), "mixed": lambda r: np.r_[300_000, r.integers(1, 5, 500), 256, 512]}


@pytest.mark.parametrize("sizes", sorted(SIZES))
@pytest.mark.parametrize("types", [(np.int32,), (np.float64,), (), (np.int16, np.int64)])
@pytest.mark.parametrize("n_probe,absent,null_frac", [(1, 0.0, 0.0), (33, 0.0, 0.0), (129, 0.3, 0.0), (1025, 0.9, 0.2)])
def test_group_sizes(cuda, sizes, types, n_probe, absent, null_frac):
    s = SIZES[sizes](np.random.default_rng(1))
    if sizes == "mixed":
        n_probe = min(n_probe, 33)
    _run(cuda, s, n_probe, types, n_probe, None, null_frac, absent)


@pytest.mark.parametrize("nulls_equal", [False, True])
@pytest.mark.parametrize("types", [(np.int32,), (), (np.int16, np.int64)])
@pytest.mark.parametrize("build_nulls,n_probe", [(1, 1), (33, 129), (257, 1025), (2500, 40)])
def test_null_group(cuda, nulls_equal, types, build_nulls, n_probe):
    """NULL keys on both sides: the NULL group is matched like any other when NULLs are equal, else by nothing."""
    _run(cuda, SIZES["ones"](None), n_probe, types, build_nulls, None, 0.3, 0.2, nulls_equal, build_nulls)


@pytest.mark.parametrize("nulls_equal", [False, True])
def test_build_without_null_rows(cuda, nulls_equal):
    """NULL probe keys, and no NULL group to match."""
    _run(cuda, SIZES["small"](np.random.default_rng(3)), 1025, (np.int32,), 11, None, 0.4, 0.0, nulls_equal)


@pytest.mark.parametrize("capacity", [1, 31, 255, 256, 257, 2047, 2049, 5000])
def test_capacity_cuts_a_tile(cuda, capacity):
    _run(cuda, SIZES["small"](np.random.default_rng(2)), 1500, (np.int32,), 7, capacity)


def test_no_outputs_is_a_count(cuda):
    """Row ids and payloads all left out, any capacity: the matches are counted and nothing is expanded."""
    rng = np.random.default_rng(4)
    bk, pk = rng.integers(0, 500, 20_000), rng.integers(0, 1000, 30_000)
    dk, dc = dev_t(pk, cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
    keys, nk, _ = J._keys(dk)
    with J.HashTable(dev_t(bk, cuda), layout=L.SJ_LAYOUT_GROUPED) as t:
        L.timing_collect()
        L.timing_enable(True)
        try:
            L.check(L.load().sj_probe_gather(t.handle, keys, nk, None, 0, None, 0, None, None, None, None, 1 << 62, None,
                                             None, dc.data_ptr()), "sj_probe_gather")
            torch.cuda.synchronize()
            names = [name for name, _ in L.timing_collect()]
        finally:
            L.timing_enable(False)
    assert int(dc.item()) == int(np.bincount(bk, minlength=1000)[pk].sum())
    assert "expand" not in names and names, names
