"""Device calls right behind the work that makes their tensors: on torch's
default stream and on a stream of the caller's, while a long kernel still
runs there ahead of the last writes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gen(seed):
    from parallelbatchrcm_b200 import gen
    return gen.grid2d(131, 117, seed=seed)


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("default", [True, False])
@pytest.mark.parametrize("op", ["reorder", "batch", "permute", "connect"])
def test_inputs_still_being_written(pbrcm, gpu_ctx, oracle_mod, op, default):
    import torch
    old, new = _gen(1), _gen(2)
    perm = np.random.default_rng(3).permutation(new.n).astype(np.uint32)
    rp, ci, pm = _dev(old.row_ptr), _dev(old.col_idx), _dev(np.arange(new.n, dtype=np.uint32))
    src = [_dev(a) for a in (new.row_ptr, new.col_idx, perm)]
    out = torch.empty(new.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = torch.cuda.default_stream() if default else torch.cuda.Stream()
    with torch.cuda.stream(st):
        torch.cuda._sleep(50_000_000)  # about 25 ms
        for d, s in zip((rp, ci, pm), src):
            d.copy_(s)
        if op == "reorder":
            got = [pbrcm.reorder_device(rp, ci, out, ctx=gpu_ctx)[0]]
        elif op == "batch":
            pbrcm.reorder_batch_device([(rp, ci, out)], ctx=gpu_ctx)
            got = [out]
        elif op == "permute":
            got = pbrcm.permute_device(rp, ci, pm, ctx=gpu_ctx)[:2]
        else:
            got = pbrcm.connect_device(rp, ci, ctx=gpu_ctx)[:2]
    if op in ("reorder", "batch"):
        want = [oracle_mod.full_reorder(new.row_ptr, new.col_idx, reverse=True)["perm"]]
    elif op == "permute":
        want = oracle_mod.permute_csr(new.row_ptr, new.col_idx, perm)[:2]
    else:
        want = [new.row_ptr, new.col_idx]
    for g, w in zip(got, want):
        assert np.array_equal(_host(g), w)
