"""The region-partitioned gather of middling streams: the default's choice of
it on both sides of its line, its fixed segment order and its partial last
chunk, under capture, in place, from several threads, and without memory."""
from __future__ import annotations

import threading

import pytest

pytestmark = pytest.mark.gpu

TABLE = 1 << 25


def _case(cuda, n, tsize, seed, packed=False):
    import torch

    g = torch.Generator(device=cuda).manual_seed(seed)
    idx = torch.randint(0, tsize, (n,), dtype=torch.int64, device=cuda, generator=g)
    idx[5::100_003] = tsize + 3  # out of range: value 0, counted
    idx[7::100_003] = -1
    ok = (idx >= 0) & (idx < tsize)
    want = torch.where(ok, -(idx + 1), torch.zeros_like(idx))
    return (idx << 16 if packed else idx), want, int((~ok).sum().item())


def _table(cuda, tsize, odd):
    import torch

    t = torch.empty(tsize + 1, dtype=torch.int64, device=cuda)
    t = t[1:] if odd else t[:tsize]  # a table on an 8-byte boundary
    t.copy_(-(torch.arange(tsize, dtype=torch.int64, device=cuda) + 1))
    return t


@pytest.mark.parametrize("n,tsize,packed,odd", [
    (8 << 20, TABLE, False, False), ((8 << 20) + 2047, TABLE + 1, True, True), ((8 << 20) - 1, TABLE, False, True),
    ((8 << 20) + 1, TABLE - 1, True, False), (43_000_001, TABLE + 12_345, False, False)])
def test_default_choice_eager_captured_and_in_place(cuda, bale, n, tsize, packed, odd):
    import torch

    index, want, nbad = _case(cuda, n, tsize, n, packed)
    table, shift = _table(cuda, tsize, odd), 16 if packed else 0
    tgt, bad = torch.full_like(index, 9), torch.zeros(1, dtype=torch.int64, device=cuda)
    bale.ig_dev(tgt, index, table, shift=shift, bad=bad)
    assert torch.equal(tgt, want) and int(bad.item()) == nbad
    tgt.fill_(8)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # nothing may be allocated here
        bale.ig_dev(tgt, index, table, shift=shift, bad=bad)
    graph.replay()
    assert torch.equal(tgt, want) and int(bad.item()) == 2 * nbad
    bale.ig_dev(index, index, table, shift=shift)  # output over the requests
    assert torch.equal(index, want)


def test_threads_on_one_stream_and_on_their_own(cuda, bale):
    import torch

    table = _table(cuda, TABLE, False)
    jobs = [(*_case(cuda, (8 << 20) + 100 * k, TABLE, k)[:2], torch.cuda.Stream()) for k in range(4)]
    outs = [torch.zeros_like(j[0]) for j in jobs]
    torch.cuda.synchronize()
    for own in (True, False):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()

        def work(k):
            for _ in range(3):
                bale.ig_dev(outs[k], jobs[k][0], table, stream=jobs[k][2] if own else jobs[0][2])

        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        for k in range(4):
            assert torch.equal(outs[k], jobs[k][1]), (own, k)


def test_without_memory_for_a_workspace(cuda, bale):
    """Device memory filled to a few MiB: the call runs without a workspace."""
    import torch

    index, want, _ = _case(cuda, 9 << 20, TABLE, 1)
    table, tgt = _table(cuda, TABLE, False), torch.zeros_like(index)
    bale.release_buffers()
    torch.cuda.empty_cache()
    hold = []
    size = 1 << 36
    while size >= 1 << 24:
        try:
            hold.append(torch.empty(size, dtype=torch.uint8, device=cuda))
        except torch.OutOfMemoryError:
            size //= 2
    try:
        bale.ig_dev(tgt, index, table)
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert torch.equal(tgt, want)
