"""A plan's large histograms run by shared-memory buckets from the entry
points' sizes on, each with a workspace of its own: counts, out-of-range
updates and replays against numpy, beside instances just below the rule."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packed", [False, True])
def test_large_histograms_of_a_plan(cuda, bale, packed):
    import torch

    from bale_old_gb300 import batch

    sizes = [(1 << 23, 100_003), ((1 << 23) - 1, 100_003), ((1 << 23) + 4_097, 1_000_000),
             ((1 << 22) + 3, 14_000_001), ((1 << 22) - 1, 14_000_001), ((1 << 23) + 1, 49_153)]
    insts, checks = [], []
    for k, (n, t) in enumerate(sizes):
        idx = bale.gen_zipf(n, t, 1.1, 4, k) if k % 2 else bale.gen_uniform(n, t + 7, 30 + k)
        counts0 = bale.gen_uniform(t, 5, k)
        ok = idx < t
        d_idx = torch.from_numpy(bale.pack_index(idx) if packed else idx).to(cuda)
        d_cnt = torch.from_numpy(counts0).to(cuda)
        insts.append(batch.histo(d_cnt, d_idx, shift=16 if packed else 0))
        checks.append((d_cnt, counts0, np.bincount(idx[ok], minlength=t), int((~ok).sum())))
    b = batch.Batch(insts)
    for replay in (1, 2):
        b.run()
        torch.cuda.synchronize()
        for (d_cnt, counts0, add, _), (n, t) in zip(checks, sizes):
            assert np.array_equal(d_cnt.cpu().numpy(), counts0 + replay * add), (n, t, replay)
        assert [int(x) for x in b.bad()] == [c[3] for c in checks]
