"""The partition operator's column scatter at the edges of its 4096-row tiles: row counts around a tile and
around one chunk per CTA, the key column first, last and absent among 0..8 columns of every width, NULLs,
columns that do not start on a row pair's alignment, no rows,
and threads with different part counts (their shared memory differs)."""
import threading

import numpy as np
import pytest
import torch

from jhelp import dev_t
from oracle import oracle as O
from sirius_b200 import join as J

pytestmark = pytest.mark.gpu

WIDTHS = [np.int8, np.int16, np.int32, np.int64, np.float32, np.float64]


@pytest.mark.parametrize("n", [0, 1, 2, 4095, 4096, 4097, 8193, 296 * 4, 296 * 4096 + 5, 1_300_001])
@pytest.mark.parametrize("key_at,n_cols,shift", [(0, 1, 0), (2, 4, 1), (-1, 7, 0), (-1, 0, 1)])
def test_column_scatter_edges(cuda, n, key_at, n_cols, shift):
    rng = np.random.default_rng(n + 10 * n_cols)
    P = 1 << int(rng.integers(0, 11))
    ktype = [np.int32, np.int64][n_cols % 2]
    keys = rng.integers(-2**31, 2**31 - 1, n).astype(ktype)

    def put(a):  # `shift` elements into a larger buffer
        return dev_t(np.concatenate([np.zeros(shift, a.dtype), a]), cuda)[shift:]
    dkeys = put(keys)
    host = [rng.integers(0, 100, n).astype(WIDTHS[(c + n_cols) % 6]) for c in range(n_cols)]
    valid = [rng.random(n) > 0.4 if c % 3 == 2 else None for c in range(n_cols)]
    cols = [(put(a), None if v is None else dev_t(O.pack_validity(v).view(np.int32), cuda))
            for a, v in zip(host, valid)]
    rid = np.arange(n, dtype=np.int32)
    host.append(rid)
    valid.append(None)
    cols.append((dev_t(rid, cuda), None))
    if key_at >= 0:
        host[key_at], valid[key_at], cols[key_at] = keys, None, (dkeys, None)
    outs, vouts, off = J.hash_partition(dkeys, cols, P)
    off = off.cpu().numpy()
    part = O.partition_ids([keys], [None], P)
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(part, minlength=P))]))
    at = outs[n_cols if key_at != n_cols else 0].cpu().numpy() if n_cols else outs[0].cpu().numpy()
    assert np.array_equal(np.sort(at), rid)
    assert np.all(np.diff(part[at]) >= 0)
    for o, vo, h, v in zip(outs, vouts, host, valid):
        assert np.array_equal(o.cpu().numpy(), h[at])
        if v is not None:
            assert np.array_equal(O.unpack_validity(vo.cpu().numpy().view(np.uint32), n), v[at])


@pytest.mark.parametrize("null_keys", [False, True])
def test_threads_with_different_part_counts(cuda, null_keys):
    n = 20_000
    keys = torch.arange(n, dtype=torch.int64, device=cuda)
    key = [(keys, torch.full(((n + 31) // 32,), -1, dtype=torch.int32, device=cuda))] if null_keys else keys
    errors, streams = [], [torch.cuda.Stream(device=cuda) for _ in range(3)]
    torch.cuda.synchronize()

    def work(parts, stream):
        try:
            with torch.cuda.stream(stream):
                for _ in range(400):
                    off = J.hash_partition(key, [keys], parts, stream=stream)[2]
                assert int(off[-1].item()) == n
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=a) for a in zip((1024, 2, 64), streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
