"""Start search of thread-block-cluster teams (a batch whose every matrix goes
to one) against the oracle: searches that end on the third pass and ones that
go on, with and without ties, levels run by one CTA and by all."""
import os

import numpy as np
import pytest

from test_gpu_search import _cases, _same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[2, 4])
def cluster_ctx(request, pbrcm):
    env = {"PBRCM_BATCH_CLUSTER": str(request.param), "PBRCM_BATCH_CLUSTER_NNZ": "1", "PBRCM_BATCH_CLUSTERS": "64",
           "PBRCM_RESIDENT_GROUP": "0"}
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        ctx = pbrcm.Context(0)
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v
    yield ctx
    ctx.close()


def test_cluster_search(pbrcm, cluster_ctx, oracle_mod):
    from parallelbatchrcm_b200 import gen
    mats = [f() for f in _cases().values()]
    mats += [gen.rgg(n, kmin=4, kmax=12, seed=s) for n in (3000, 12000) for s in range(100, 110)]
    perms, res = pbrcm.reorder_batch([(m.row_ptr, m.col_idx) for m in mats], ctx=cluster_ctx)
    passes = set()
    for m, p, r in zip(mats, perms, res):
        _same(p, r, oracle_mod.full_reorder(m.row_ptr, m.col_idx, reverse=True))
        passes.add(r["peripheral_passes"])
    assert {2, 3, 4} <= passes
