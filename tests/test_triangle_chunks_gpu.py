"""The wedge path's scan and fill split the nonzeros into equal chunks (256
and more) whatever the rows' lengths: against the oracle with totals at the
edges of a chunk and of a block's chunks, rows that span many chunks, long
stretches of empty rows inside a chunk, unused nonzeros around the matrix, and
labels on both sides of the shared-memory counters' limit of 8192."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def wedge(bale):
    bale.tune_set("tri.mode", 2)
    yield
    bale.tune_set("tri.mode", -1)


def _matrix(n, lengths, rng):
    """Row i (of those given a length) gets that many random columns below i."""
    off = np.zeros(n + 1, np.int64)
    rows = {}
    for i, d in lengths:
        rows[i] = np.sort(rng.choice(min(i, 40_000), min(d, i), replace=False))
        off[i + 1] = rows[i].size
    off = np.cumsum(off)
    return off, np.concatenate([rows[i].astype(np.int64) for i in sorted(rows)])


def _check(bale, oracle, off, col):
    cnt, sr, _ = bale.triangle_agi(bale.SparseMatrix(off, col))
    deg = np.diff(off)
    p = np.arange(col.size) - np.repeat(off[:-1], deg)
    assert cnt == oracle.triangle_agi(off, col)[0]
    assert sr == int(p[deg[col] > 0].sum())  # a probe per column before j, where row j has any


@pytest.mark.parametrize("total", [1, 255, 256, 257, 4095, 4096, 4097, 8193])
def test_chunk_edges(cuda, bale, oracle, wedge, total):
    rng = np.random.default_rng(total)
    n, left, lengths = 600, total, []
    for i in range(1, n):
        d = min(left, int(rng.integers(0, min(i, 40) + 1)))
        if i == n - 1:
            d = left
        if d:
            lengths.append((i, d))
        left -= min(d, i)
    off, col = _matrix(n, lengths, rng)
    _check(bale, oracle, off, col)


@pytest.mark.parametrize("gap", [1, 31, 32, 33, 64, 1000, 40_000])
def test_empty_stretches_and_long_rows(cuda, bale, oracle, wedge, gap):
    rng = np.random.default_rng(gap)
    lengths = [(i, 3) for i in range(5, 60)]
    i = 9_000
    for d in (5, 700, 2, 9_000, 40, 8_192, 1, 300):
        lengths.append((i, d))
        i += gap + 1
    lengths += [(i + 3 * t, 20) for t in range(200)]
    off, col = _matrix(i + 700 + gap, lengths, rng)
    _check(bale, oracle, off, col)


@pytest.mark.parametrize("before,after", [(1, 0), (300, 0), (0, 5_000), (5_000, 700)])
def test_nonzeros_outside_every_row_are_not_read(cuda, bale, oracle, wedge, before, after):
    import torch

    rng = np.random.default_rng(before + after)
    off, col = _matrix(900, [(i, 12) for i in range(20, 900, 2)], rng)
    want = oracle.triangle_agi(off, col)[0]
    wide = np.concatenate([np.full(before, -7), col, np.full(after, 1 << 40)]).astype(np.int64)
    count, bad = torch.zeros(1, dtype=torch.int64, device=cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
    bale.triangle_dev(torch.from_numpy(off + before).to(cuda), torch.from_numpy(wide).to(cuda), count, bad=bad)
    assert int(bad.item()) == 0 and int(count.item()) == want


@pytest.mark.parametrize("what", ["outside", "backward", "order at a chunk's edge", "column at a chunk's edge"])
def test_malformed_matrices_count_nothing(cuda, bale, wedge, what):
    import torch

    rng = np.random.default_rng(3)
    off, col = _matrix(3_000, [(2_999, 2_600), (2_000, 1_500)], rng)
    if what == "outside":
        off[2_500] = col.size + 9
    elif what == "backward":
        off[1:2_000:2] = col.size
    elif what.startswith("order"):
        col[256] = col[255]
    else:
        col[1_024] = 2_001
    count, bad = torch.zeros(1, dtype=torch.int64, device=cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
    bale.triangle_dev(torch.from_numpy(off).to(cuda), torch.from_numpy(col).to(cuda), count, bad=bad)
    assert int(bad.item()) > 0 and int(count.item()) == 0


@pytest.mark.parametrize("n", [31, 32, 33, 4_096, 32_766, 32_767, 32_768, 32_769, 33_100, 65_600, 70_000])
def test_rows_around_the_low_labels(cuda, bale, oracle, wedge, n):
    """Rows and columns at both sides of 2^15 (near and far rows, low columns
    and the list's, rows read in 16 bits), hubs with many prefixes, short far
    rows beside long ones, and more other columns than the list holds."""
    rng = np.random.default_rng(n)
    edge = np.unique(np.clip(np.concatenate([np.arange(0, 40), np.arange(32_740, 32_800), np.arange(65_520, 65_560),
                                             rng.integers(0, n, 300)]), 0, n - 1))
    rows, off = [], np.zeros(n + 1, np.int64)
    for i in range(n):
        if i in (n - 1, n - 2, n - 3):  # long rows, all of whose columns are neighbours
            r = edge[edge < i]
            r = np.union1d(r, np.arange(max(0, i - 300), i))
        elif i % 3 == 0 or i > n - 400:
            below = edge[edge < i]
            r = np.sort(rng.choice(below, min(below.size, int(rng.integers(0, 90))), replace=False))
        else:
            r = np.zeros(0, np.int64)
        rows.append(r.astype(np.int64))
        off[i + 1] = off[i] + r.size
    _check(bale, oracle, off, np.concatenate(rows))


@pytest.mark.parametrize("many", [3, 40, 200])
def test_high_labels_that_share_a_code(cuda, bale, oracle, wedge, many):
    """Columns from 2^15 on that are equal in their last 14 bits: neighbours of
    one row (as many as the list holds and more), of another row only, or both."""
    rng = np.random.default_rng(many)
    base = np.sort(rng.choice(np.arange(32_767, 40_000), many, replace=False))
    labels = np.unique(np.concatenate([base + 16_384 * k for k in range(4)]))
    low = np.arange(100, 170)
    n = 100_600
    off, rows = np.zeros(n + 1, np.int64), []
    for i in range(n):
        if i >= n - 60 or (i in labels and i % 3 == 0):
            below = labels[labels < i]
            r = np.union1d(low, rng.choice(below, int(rng.integers(below.size // 2, below.size + 1)), replace=False)) \
                if below.size else low
            if i >= n - 60:
                r = np.union1d(r, np.arange(n - 60, i))
        else:
            r = np.zeros(0, np.int64)
        rows.append(np.asarray(r, np.int64))
        off[i + 1] = off[i] + rows[-1].size
    _check(bale, oracle, off, np.concatenate(rows))
