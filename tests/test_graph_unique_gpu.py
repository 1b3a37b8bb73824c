"""Distinct edges by hashing (graph_unique.cu) in graph builds of 2^20 edges and
more, against the sorted path on the same graph: sizes on both sides of its
line, repeats of one edge far beyond a bucket's set, a star, self loops only,
and edges made to fall into one bucket (which go back to the sort)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 1 << 20


def _reference(u, v, n):
    """Degree-ordered strictly lower CSR in numpy."""
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    key = np.unique((lo * n + hi)[lo != hi])
    a, b = key // n, key % n
    deg = np.bincount(a, minlength=n) + np.bincount(b, minlength=n)
    label = np.empty(n, np.int64)
    label[np.lexsort((np.arange(n), -deg))] = np.arange(n)
    x, y = label[a], label[b]
    row, col = np.maximum(x, y), np.minimum(x, y)
    order = np.lexsort((col, row))
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(np.bincount(row, minlength=n))
    return off, col[order]


def _mix(k):
    k = k * np.uint64(0x9E3779B97F4A7C15)
    k ^= k >> np.uint64(32)
    return k * np.uint64(0xD6E8FEB86659FD93)


def _edges(kind, m, n, rng):
    if kind == "random":
        return rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "repeats":  # two edges many times over, both ways round, and a few others
        u, v = np.full(m, 5), np.full(m, 9)
        u[: m // 2], v[: m // 2] = 9, 5
        u[::3], v[::3] = 1, 2
        u[::1001], v[::1001] = rng.integers(0, n, u[::1001].size), rng.integers(0, n, u[::1001].size)
        return u, v
    if kind == "star":
        return np.full(m, 7), np.arange(m) % n
    if kind == "loops":
        return np.arange(m) % n, np.arange(m) % n
    # one bucket: keys whose hash has the top ten bits zero
    with np.errstate(over="ignore"):
        lo = rng.integers(0, n - 1, 40_000_000)
        hi = lo + 1 + rng.integers(0, 1 << 20, lo.size) % (n - 1 - lo)
        s = int(n - 1).bit_length()
        key = (lo.astype(np.uint64) << np.uint64(s)) | hi.astype(np.uint64)
        pick = np.flatnonzero(_mix(key) >> np.uint64(54) == 0)
    assert pick.size > 20_000
    pick = np.resize(pick, m)
    return lo[pick], hi[pick]


@pytest.mark.parametrize("kind,m,n", [("random", M - 1, 50_000), ("random", M, 50_000), ("random", M + 8191, 1 << 18),
                                      ("random", 5 * M + 17, 1 << 12), ("repeats", M + 5, 3_000), ("star", M + 1, 1 << 19),
                                      ("loops", M, 1_000), ("one bucket", M + 3, 1 << 20)])
def test_build_matches_numpy(cuda, bale, kind, m, n):
    import torch

    u, v = _edges(kind, m, n, np.random.default_rng(m + n))
    off, col = bale.graph_build_dev(torch.from_numpy(u.astype(np.int64)).to(cuda),
                                    torch.from_numpy(v.astype(np.int64)).to(cuda), n)
    want_off, want_col = _reference(u.astype(np.int64), v.astype(np.int64), n)
    np.testing.assert_array_equal(off.cpu().numpy(), want_off)
    np.testing.assert_array_equal(col.cpu().numpy(), want_col)


def test_out_of_range_endpoint_is_still_an_error(cuda, bale):
    import torch

    u = torch.zeros(M + 9, dtype=torch.int64, device=cuda)
    v = torch.ones_like(u)
    v[M] = 40
    with pytest.raises(bale.BaleError, match="outside"):
        bale.graph_build_dev(u, v, 40)
