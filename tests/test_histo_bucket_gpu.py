"""The histogram by shared-memory buckets (histo_bucket.cu) against numpy's
exact counts: chunk edges (12288 updates), bucket edges, partial buckets and
chunks, skew, out-of-range updates, and the launcher's choice of it."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK, BUCKET = 12288, 18432


@pytest.fixture
def forced(bale):
    bale.tune_set("histo.mode", 4)
    yield
    bale.tune_set("histo.mode", -1)


def _indices(dist, n, tsize, seed):
    rng = np.random.default_rng(seed)
    if dist == "uniform":
        return rng.integers(0, tsize, n)
    if dist == "one":  # every update on the last counter
        return np.full(n, tsize - 1, np.int64)
    if dist == "sorted":  # each chunk in one or two buckets
        return np.sort(rng.integers(0, tsize, n))
    hot = rng.integers(0, tsize, n)  # half on one counter
    hot[rng.random(n) < 0.5] = tsize // 3
    return hot


@pytest.mark.parametrize("shift", [0, 16])
@pytest.mark.parametrize("n,tsize", [
    (1, 1), (CHUNK - 1, 8191), (CHUNK, 8192), (CHUNK + 1, 8193), (8 * CHUNK, BUCKET), (9 * CHUNK + 7, BUCKET + 1),
    (3 * CHUNK + 1, 456 * 8192), (100_003, 456 * BUCKET + 1), (700_001, 4094 * BUCKET), (1_500_001, 999_983)])
def test_sizes_around_chunks_and_buckets(cuda, bale, forced, n, tsize, shift):
    import torch

    idx = _indices("uniform", n, tsize, n + shift)
    idx[n // 2:: 977] = tsize  # first value out of range
    idx[n // 3:: 1013] = -1
    idx[-1] = tsize - 1
    ok = (idx >= 0) & (idx < tsize)
    start = np.arange(tsize, dtype=np.int64) % 7
    counts, bad = torch.from_numpy(start.copy()).to(cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
    index = torch.from_numpy(bale.pack_index(idx) if shift else idx).to(cuda)
    for _ in range(2):  # adds on both calls, the second on a used workspace
        bale.histo_dev(counts, index, shift=shift, bad=bad)
    np.testing.assert_array_equal(counts.cpu().numpy(), start + 2 * np.bincount(idx[ok], minlength=tsize))
    assert int(bad.item()) == 2 * int((~ok).sum())


@pytest.mark.parametrize("dist", ["one", "sorted", "hot"])
@pytest.mark.parametrize("n,tsize", [(40 * CHUNK + 11, 60_000), (200 * CHUNK, 5_000_000)])
def test_skewed_updates(cuda, bale, forced, dist, n, tsize):
    import torch

    idx = _indices(dist, n, tsize, 3)
    counts = torch.zeros(tsize, dtype=torch.int64, device=cuda)
    bale.histo_dev(counts, torch.from_numpy(idx).to(cuda))
    np.testing.assert_array_equal(counts.cpu().numpy(), np.bincount(idx, minlength=tsize))


@pytest.mark.parametrize("n,tsize", [(8 << 20, 49_153), ((8 << 20) - 1, 1_000_000), (4 << 20, 14_000_000)])
def test_default_choice_captured_and_eager_agree(cuda, bale, n, tsize):
    """Sizes on both sides of the choice: an eager call, and a captured one
    (which takes no workspace) replayed, each add the same counts."""
    import torch

    g = torch.Generator(device=cuda).manual_seed(n)
    index = torch.randint(0, tsize, (n,), dtype=torch.int64, device=cuda, generator=g)
    want = torch.bincount(index, minlength=tsize)
    counts = torch.zeros(tsize, dtype=torch.int64, device=cuda)
    bale.histo_dev(counts, index)
    assert torch.equal(counts, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        bale.histo_dev(counts, index)
    for _ in range(2):
        graph.replay()
    assert torch.equal(counts, 3 * want)


def test_threads_and_streams_share_nothing(cuda, bale, forced):
    """Calls from several threads, on one stream and on ten (more than keep a
    workspace), interleaved: every table gets its own counts."""
    import torch

    jobs = []
    for k in range(10):
        idx = torch.from_numpy(_indices("uniform", 20 * CHUNK + k, 70_000 + k, k)).to(cuda)
        jobs.append((idx, torch.zeros(70_000 + k, dtype=torch.int64, device=cuda), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def work(k, own):
        idx, counts, stream = jobs[k]
        for _ in range(5):
            bale.histo_dev(counts, idx, stream=stream if own else jobs[0][2])

    for own in (True, False):
        threads = [threading.Thread(target=work, args=(k, own)) for k in range(10)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
    for k, (idx, counts, _) in enumerate(jobs):
        assert torch.equal(counts, 10 * torch.bincount(idx, minlength=70_000 + k)), k
