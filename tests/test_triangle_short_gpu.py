"""The hybrid's short-row kernel (tri_hybrid.cu) against the oracle: row
lengths around its limit of 63, columns that share a place of the row's table
(equal low 9 bits), neighbours long enough to be searched, empty rows, rows
that are not a multiple of its groups of eight, and malformed rows."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(rows):
    off = np.zeros(len(rows) + 1, np.int64)
    off[1:] = np.cumsum([len(r) for r in rows])
    return off, np.concatenate([np.asarray(r, np.int64) for r in rows]) if off[-1] else np.zeros(0, np.int64)


def _random_rows(n, lengths, rng, stride=1):
    rows = []
    for i in range(n):
        top = i // stride if stride > 1 else i
        d = min(top, int(lengths[i]))
        rows.append(np.sort(rng.choice(top, d, replace=False)) * stride if d else np.zeros(0, np.int64))
    return rows


@pytest.fixture
def hybrid(bale):
    bale.tune_set("tri.mode", 1)
    yield
    bale.tune_set("tri.mode", -1)


def _graph(kind, rng):
    if kind == "mixed":  # lengths across the limit: short, heavy and empty rows in one group
        n = 3_003
        return _random_rows(n, rng.choice([0, 1, 2, 7, 8, 9, 31, 33, 62, 63, 64, 65, 100], n), rng)
    if kind == "shared":  # every column a multiple of 512: all on one place
        return _random_rows(513 * 40, np.where(np.arange(513 * 40) % 512 < 3, 12, 0), rng, 512)
    if kind == "pairs":  # clusters of columns 512 apart
        base = _random_rows(4_001, np.full(4_001, 6), rng)
        return [np.array(sorted({c for v in r for c in (v, v + 512) if c < i}), np.int64) for i, r in enumerate(base)]
    # one long row of 900 columns, neighbour of many short rows at a small position
    n = 6_000
    rows = _random_rows(1_000, np.full(1_000, 5), rng)
    rows.append(np.arange(50, 950))
    for i in range(1_001, n):
        rows.append(np.array(sorted({int(rng.integers(0, 1_000)), int(rng.integers(0, 1_000)), 1_000}), np.int64))
    return rows


@pytest.mark.parametrize("kind", ["mixed", "shared", "pairs", "long_neighbour"])
def test_short_rows_match_oracle(cuda, bale, oracle, hybrid, kind):
    off, col = _csr(_graph(kind, np.random.default_rng(5)))
    cnt, sr, _ = bale.triangle_agi(bale.SparseMatrix(off, col))
    assert cnt == oracle.triangle_agi(off, col)[0]
    # the tally: per nonzero after a row's first, the cheaper of streaming row j
    # and searching the q columns before it
    deg = np.diff(off)
    q = np.arange(col.size) - np.repeat(off[:-1], deg)
    want = 0
    for k in range(col.size):
        if q[k]:
            d = int(deg[col[k]])
            want += int(q[k]) if q[k] * (d + 1).bit_length() < d else d
    heavy = deg >= 64  # their neighbours are always streamed
    hk = np.repeat(heavy, deg) & (q > 0)
    for k in np.flatnonzero(hk):
        d = int(deg[col[k]])
        if q[k] * (d + 1).bit_length() < d:
            want += d - int(q[k])
    assert sr == want


def test_malformed_short_rows_are_counted_not_followed(cuda, bale, hybrid):
    import torch

    rng = np.random.default_rng(6)
    off, col = _csr(_random_rows(2_000, np.full(2_000, 10), rng))
    for what in ("column", "order", "negative", "offset", "backward"):
        o, c = off.copy(), col.copy()
        k = int(off[700])
        if what == "column":
            c[k + 3] = 700
        elif what == "order":
            c[k + 3], c[k + 4] = c[k + 4], c[k + 3]
        elif what == "negative":
            c[k] = -4
        elif what == "offset":
            o[700] = col.size + 50
        else:  # alternating: every other row seems to hold most of the matrix
            o[1:-1:2] = col.size
        count, bad = torch.zeros(1, dtype=torch.int64, device=cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
        bale.triangle_dev(torch.from_numpy(o).to(cuda), torch.from_numpy(c).to(cuda), count, bad=bad)
        assert int(bad.item()) > 0, what
