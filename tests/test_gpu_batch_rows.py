"""Batches of at most one matrix per SM whose small matrices have a row past
the shared-memory engine's chunks (512 entries): taken together by the solo
engine (up to 1,024 entries, longer ones by the team), not one after the
other."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spoke(n, row, seed):
    """A path of n nodes whose first node has a row of exactly `row` entries
    (its diagonal among them)."""
    from parallelbatchrcm_b200 import gen
    i = np.arange(1, n)
    far = np.arange(2, row) * ((n - 1) // row)
    e = np.concatenate([np.stack([i - 1, i], 1), np.stack([np.zeros_like(far), far], 1)])
    p = np.random.default_rng(seed).permutation(n)[e]
    m = gen.from_edges(n, p[:, 0], p[:, 1])
    assert int(np.diff(m.row_ptr.astype(np.int64)).max()) == row
    return m


def _device(mats):
    import torch
    return [tuple(torch.from_numpy(a.view(np.int32)).cuda() for a in (m.row_ptr, m.col_idx))
            + (torch.empty(m.n, dtype=torch.int32, device="cuda"),) for m in mats]


@pytest.mark.parametrize("rows", [[513], [512, 513], [511, 512, 513, 600, 1023, 1024, 1025, 40],
                                  [513, 514, 1024, 1025, 1500]])
@pytest.mark.parametrize("form", ["host", "device"])
def test_rows_past_a_chunk(pbrcm, gpu_ctx, oracle_mod, rows, form):
    mats = [_spoke(3100 + 7 * k, r, k) for k, r in enumerate(rows)]
    d = _device(mats)
    for _ in range(2):  # the second call of the device form replays the captured batch
        if form == "host":
            perms, res = pbrcm.reorder_batch([(m.row_ptr, m.col_idx) for m in mats], ctx=gpu_ctx)
        else:
            res = pbrcm.reorder_batch_device(d, ctx=gpu_ctx)
            perms = [x[2].cpu().numpy().view(np.uint32) for x in d]
        for m, p, r in zip(mats, perms, res):
            ref = oracle_mod.full_reorder(m.row_ptr, m.col_idx, reverse=True)
            assert (r["status"], r["start_node"], r["peripheral_passes"]) == (0, ref["start"], ref["passes"])
            assert np.array_equal(p, ref["perm"])
            assert r["bandwidth"] == ref["bandwidth"] and r["profile"] == ref["profile"]


def test_many_in_one_launch(pbrcm, gpu_ctx):
    """64 matrices with a row of 600 entries take about as long as 64 with one
    of 500, not 64 reruns (a factor of 60 or more)."""
    import torch
    best = {}
    for row in (500, 600):
        d = _device([_spoke(3100 + k, row, k) for k in range(64)])
        pbrcm.reorder_batch_device(d, ctx=gpu_ctx)
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            pbrcm.reorder_batch_device(d, ctx=gpu_ctx)
            best[row] = min(best.get(row, 1e9), time.perf_counter() - t)
    assert best[600] < 8 * best[500], best
