"""The device connectivity repair (pbrcm_connect_device, csrc/connect.cu)
against the oracle's restatement of prepareRCM (include/Graph.h:160-263):
the joined CSR must be identical entry for entry (integer work: exact)."""
import numpy as np
import pytest

from test_connect_cpu import random_pattern

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint32)


def _run(pbrcm, ctx, rp, ci, **kw):
    orp, oci, links = pbrcm.connect_device(_dev(rp), _dev(ci), ctx=ctx, **kw)
    return _host(orp), _host(oci), links


def _check(pbrcm, ctx, oracle_mod, rp, ci, **kw):
    arp, aci, links = _run(pbrcm, ctx, rp, ci, **kw)
    erp, eci, _ = oracle_mod.prepare_csr(rp, ci, check_sym=False)
    assert np.array_equal(arp, erp) and np.array_equal(aci, eci)
    assert links == (eci.shape[0] - ci.shape[0]) // 2
    return links


@pytest.mark.parametrize("seed", range(24))
def test_random_patterns_match_oracle(pbrcm, gpu_ctx, oracle_mod, seed):
    """Many small components, rows without the diagonal, empty rows (the
    first rows too, so that row 0 takes the (0, minn) link), duplicates."""
    rng = np.random.default_rng(100 + seed)
    n = int(rng.integers(2, 5000))
    rp, ci = random_pattern(rng, n, int(rng.integers(1, 2 * n)), diag_frac=rng.random(),
                            dup_frac=0.1 if seed % 2 else 0.0, empty_head=int(rng.integers(0, 4)) if seed % 3 == 0 else 0)
    if ci.shape[0] == 0:
        pytest.skip("no entries")
    _check(pbrcm, gpu_ctx, oracle_mod, rp, ci)


def test_connected_matrix_unchanged(pbrcm, gpu_ctx):
    from parallelbatchrcm_b200 import gen
    m = gen.grid3d(24, 20, 16, seed=5)
    arp, aci, links = _run(pbrcm, gpu_ctx, m.row_ptr, m.col_idx)
    assert links == 0 and np.array_equal(arp, m.row_ptr) and np.array_equal(aci, m.col_idx)


def test_sparse_rgg_1m_matches_oracle(pbrcm, gpu_ctx, oracle_mod):
    """A 1M-node random geometric graph of 1-3 nearest neighbours per point
    before the loader joins it (about 40k components), the generator's own
    join, and a reorder of the joined matrix against the oracle."""
    from parallelbatchrcm_b200 import gen
    m = gen.rgg(1_000_000, kmin=1, kmax=3, long_frac=0.0, connect=False)
    links = _check(pbrcm, gpu_ctx, oracle_mod, m.row_ptr, m.col_idx)
    assert links > 10_000
    j = gen.connect_components(m)
    arp, aci, _ = _run(pbrcm, gpu_ctx, m.row_ptr, m.col_idx)
    assert np.array_equal(arp, j.row_ptr) and np.array_equal(aci, j.col_idx)
    perm, res = pbrcm.reorder(arp, aci, reverse=True, ctx=gpu_ctx)
    eperm = oracle_mod.full_reorder(arp, aci)["perm"]
    assert np.array_equal(perm, eperm)


def test_forest_of_small_trees(pbrcm, gpu_ctx, oracle_mod):
    """2M nodes in ~1M components (a random forest with half the edges a
    tree needs): long union chains and a million links."""
    rng = np.random.default_rng(9)
    n = 2_000_000
    child = rng.permutation(n)[: n // 2]
    par = (child * rng.random(child.size)).astype(np.int64)  # an earlier node: a forest
    rp, ci = random_pattern(rng, n, 0, diag_frac=1.0)
    rows = np.concatenate([np.repeat(np.arange(n), np.diff(rp).astype(np.int64)), child, par]).astype(np.uint64)
    cols = np.concatenate([ci.astype(np.int64), par, child]).astype(np.uint64)
    key = np.unique((rows << np.uint64(32)) | cols)
    r = (key >> np.uint64(32)).astype(np.int64)
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    rp, ci = rp.astype(np.uint32), (key & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    assert _check(pbrcm, gpu_ctx, oracle_mod, rp, ci) > n // 4


def test_output_room_grows(pbrcm, gpu_ctx, oracle_mod):
    """With room for only the input's entries the wrapper sees the size the
    call reports and calls again."""
    rng = np.random.default_rng(4)
    rp, ci = random_pattern(rng, 3000, 1500, diag_frac=0.5)
    _check(pbrcm, gpu_ctx, oracle_mod, rp, ci, cap=ci.shape[0])


def test_rejects_bad_patterns(pbrcm, gpu_ctx):
    from parallelbatchrcm_b200 import PbrcmError
    # not symmetric: 0 -> 1 without 1 -> 0
    rp, ci = np.array([0, 2, 3], np.uint32), np.array([0, 1, 1], np.uint32)
    with pytest.raises(PbrcmError) as e:
        _run(pbrcm, gpu_ctx, rp, ci)
    assert e.value.status == 1
    # a row not sorted by column
    rp, ci = np.array([0, 2, 4], np.uint32), np.array([1, 0, 0, 1], np.uint32)
    with pytest.raises(PbrcmError) as e:
        _run(pbrcm, gpu_ctx, rp, ci)
    assert e.value.status == 1
    # a column past the matrix
    rp, ci = np.array([0, 1, 2], np.uint32), np.array([0, 7], np.uint32)
    with pytest.raises(PbrcmError) as e:
        _run(pbrcm, gpu_ctx, rp, ci)
    assert e.value.status == 1
    # no entry at all
    rp, ci = np.zeros(4, np.uint32), np.zeros(1, np.uint32)[:0]
    import torch
    with pytest.raises(PbrcmError) as e:
        pbrcm.connect_device(_dev(rp), torch.zeros(1, dtype=torch.int32, device="cuda")[:0], ctx=gpu_ctx)
    assert e.value.status == 7


def _band(n, width, first):
    """Chains of three rows (n rows in all), every row from `first` on with the
    diagonal and links inside its chain repeated to `width` entries."""
    rows = []
    for r in range(n):
        c = [x for x in range(r // 3 * 3, min(r // 3 * 3 + 3, n)) if abs(x - r) <= 1]
        rows.append(sorted(c + [r] * max(0, width - len(c))) if r >= first else c)
    rp = np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.uint32)
    return rp, np.concatenate(rows).astype(np.uint32)


@pytest.mark.parametrize("n", [31, 32, 33, 63, 64, 65, 257])
@pytest.mark.parametrize("width", [1, 15, 16, 17, 33])
def test_row_groups(pbrcm, gpu_ctx, oracle_mod, n, width):
    """Row counts around the 32 rows a warp takes and rows (of repeated
    diagonal entries) around the lengths its lanes take together."""
    _check(pbrcm, gpu_ctx, oracle_mod, *_band(n, width, n // 2))


@pytest.mark.parametrize("entry", [(3, 40), (40, 3), (0, 63), (63, 0)])
def test_one_sided_entry_rejected(pbrcm, gpu_ctx, entry):
    """An entry without its transpose, above and below the diagonal."""
    n = 64
    rows = [sorted({r, max(r - 1, 0), min(r + 1, n - 1)} | ({entry[1]} if r == entry[0] else set()))
            for r in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.uint32)
    with pytest.raises(pbrcm.PbrcmError):
        _run(pbrcm, gpu_ctx, rp, np.concatenate(rows).astype(np.uint32))


def _hubs_apart(sizes, at, seed):
    """Stars (hub rows of the given lengths, diagonal included) that are
    components of their own among single nodes; the hubs' labels begin at
    `at`, everything else is shuffled."""
    n = at + sum(sizes) + 40
    free = np.random.default_rng(seed).permutation(np.concatenate([np.arange(at), np.arange(at + len(sizes), n)]))
    rows, cols, used = [np.arange(n)], [np.arange(n)], 0
    for i, s in enumerate(sizes):
        leaves = free[used:used + s - 1]
        used += s - 1
        hub = np.full(s - 1, at + i)
        rows += [hub, leaves]
        cols += [leaves, hub]
    r, c = np.concatenate(rows), np.concatenate(cols)
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.uint32)
    return rp, c[o].astype(np.uint32)


@pytest.mark.parametrize("sizes", [[992], [993], [994], [1024], [1025], [1026], [1504, 2], [1536], [20000],
                                   [700, 700, 700, 3000, 50], [1100] * 70])
@pytest.mark.parametrize("at", [0, 31, 500])
def test_long_rows(pbrcm, gpu_ctx, oracle_mod, sizes, at):
    """Groups of 32 rows around the 1,024 entries up to which a warp takes them and
    far beyond, one and many, with links falling into them."""
    _check(pbrcm, gpu_ctx, oracle_mod, *_hubs_apart(sizes, at, len(sizes) + at))


def test_hub_row_is_shared_out(pbrcm, gpu_ctx):
    """A star takes about as long as a path of as many nodes (72 ms against
    0.3 when one warp takes the hub's row)."""
    import time
    import torch
    n, best = 1_000_000, {}
    i = torch.arange(1, n, device="cuda")
    for name, j in (("star", torch.zeros_like(i)), ("path", i - 1)):
        p = torch.randperm(n, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
        u, v = p[i], p[j]
        key = torch.sort(torch.cat([u * n + v, v * n + u])).values
        rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        rp[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
        rp, ci = rp.int(), (key % n).int()
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _, _, links = pbrcm.connect_device(rp, ci, ctx=gpu_ctx)
            best[name] = min(best.get(name, 1e9), time.perf_counter() - t)
        assert links == 0
    assert best["star"] < 10 * best["path"], best


def test_long_rows_one_sided(pbrcm, gpu_ctx):
    """An entry without its transpose in a long row, and in a short one beside
    long rows, is still refused."""
    rp, ci = _hubs_apart([5000], 31, 3)
    n = rp.size - 1
    rows = [ci[rp[r]:rp[r + 1]] for r in range(n)]
    single = next(r for r in range(n) if rows[r].size == 1 and r > 40)
    for r, c in ((31, single), (single, 31), (single, single - 1)):
        bad = [np.union1d(x, [c]).astype(np.uint32) if i == r else x for i, x in enumerate(rows)]
        brp = np.concatenate([[0], np.cumsum([x.size for x in bad])]).astype(np.uint32)
        with pytest.raises(pbrcm.PbrcmError):
            _run(pbrcm, gpu_ctx, brp, np.concatenate(bad))
