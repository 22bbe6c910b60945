"""Start-search passes that run unordered inside a level (batch and team
engines) against the oracle: where the next start is decided without the
order, where it is not (ties, a last level past the kept nodes, wide
stencils) and where the unordered pass's shapes have their edges (rows of 31 and 32 entries, 256
entries a warp, a visited bitmap in global memory)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relabel(n, edges, seed):
    p = np.random.default_rng(seed).permutation(n)
    e = p[np.asarray(edges, dtype=np.int64)]
    from parallelbatchrcm_b200 import gen
    return gen.from_edges(n, e[:, 0], e[:, 1])


def _broom(handle, leaves, linked, seed):
    """A path with `leaves` leaves at each end; linked: the first leaf of each
    end has a second link (to the second leaf), so that the minimal valence is
    shared by the others (or, with two leaves, by none alone)."""
    n = handle + 2 * leaves
    edges = [(i, i + 1) for i in range(handle - 1)]
    for end, base in ((0, handle), (handle - 1, handle + leaves)):
        edges += [(end, base + k) for k in range(leaves)]
        if linked and leaves > 1:
            edges.append((base, base + 1))
    return _relabel(n, edges, seed)


def _hubs(rows, seed):
    """Hub nodes with rows of exactly the given lengths (diagonal included)
    joined in a ring, every other node a leaf."""
    edges, n = [], len(rows)
    for i in range(len(rows)):
        edges.append((i, (i + 1) % len(rows)))
    for i, r in enumerate(rows):
        for _ in range(r - 3):  # diagonal and two ring links
            edges.append((i, n))
            n += 1
    return _relabel(n, edges, seed)


def _stencil(nx, ny, nz, reach, drop, seed):
    """A mesh of (2 reach + 1)-wide stencils (9- or 27-point for reach 1);
    drop: this share of the rows loses its links but a path, which takes the
    mean valence below the share of the largest that a wide stencil has."""
    i = np.arange(nx * ny * nz)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    rz = reach if nz > 1 else 0
    edges = [np.stack([i[:-1], i[1:]], 1)]
    keep = np.random.default_rng(seed).random(i.size) >= drop
    for dx in range(-reach, reach + 1):
        for dy in range(-reach, reach + 1):
            for dz in range(-rz, rz + 1):
                at = (x + dx, y + dy, z + dz)
                ok = np.all([(a >= 0) & (a < lim) for a, lim in zip(at, (nx, ny, nz))], axis=0)
                j = i + dx + dy * nx + dz * nx * ny
                ok &= j > i
                ok[ok] &= keep[i[ok]] & keep[j[ok]]
                edges.append(np.stack([i[ok], j[ok]], 1))
    return _relabel(i.size, np.concatenate(edges), seed)


def _cases():
    from parallelbatchrcm_b200 import gen
    out = {}
    for leaves in (1, 2, 3, 31, 32, 33):
        for linked in (False, True):
            out[f"broom_{leaves}_{int(linked)}"] = lambda a=leaves, b=linked: _broom(40, a, b, 10 * a + b)
    out["hubs_31_32_33"] = lambda: _hubs([31, 32, 33, 30, 40, 31, 32], 1)
    out["hubs_255_257"] = lambda: _hubs([255, 256, 257, 8, 9, 300, 600], 2)
    out["grid2d_61x59"] = lambda: gen.grid2d(61, 59, seed=3)
    out["grid3d_23x21x19"] = lambda: gen.grid3d(23, 21, 19, seed=4)
    out["rgg_9001"] = lambda: gen.rgg(9001, kmin=4, kmax=12, seed=6)
    out["rgg_700"] = lambda: gen.rgg(700, kmin=4, kmax=12, seed=8)
    out["grid2d_530x500"] = lambda: gen.grid2d(530, 500, seed=9)  # over 2^18 nodes
    for drop in (0.0, 0.1, 0.3):  # passes that begin in discovery order, or not
        out[f"stencil9_60x57_{drop}"] = lambda d=drop: _stencil(60, 57, 1, 1, d, 12)
        out[f"stencil27_31x29x30_{drop}"] = lambda d=drop: _stencil(31, 29, 30, 1, d, 13)
    out["stencil25_16x900"] = lambda: _stencil(16, 900, 1, 2, 0.0, 14)
    out["stencil27_9x8x7"] = lambda: _stencil(9, 8, 7, 1, 0.0, 15)
    out["random_30000"] = lambda: gen.erdos_renyi(30000, 14, seed=16)  # heavy levels
    out["random_60000"] = lambda: gen.erdos_renyi(60000, 40, seed=17)  # rows of 32 and more in them
    out["random_5000"] = lambda: gen.erdos_renyi(5000, 14, seed=11)
    return out


@pytest.fixture(scope="module")
def built(oracle_mod):
    cache = {}

    def get(name):
        if name not in cache:
            m = _cases()[name]()
            cache[name] = (m, oracle_mod.full_reorder(m.row_ptr, m.col_idx, reverse=True))
        return cache[name]
    return get


def _same(perm, res, ref):
    assert (res["start_node"], res["peripheral_passes"], res["eccentricity"]) == (
        ref["start"], ref["passes"], ref["ecc"])
    assert np.array_equal(perm, ref["perm"])
    assert res["bandwidth"] == ref["bandwidth"] and res["profile"] == ref["profile"]


@pytest.mark.parametrize("name", list(_cases()))
def test_team_search(pbrcm, gpu_ctx_team, built, name):
    m, ref = built(name)
    _same(*pbrcm.reorder(m.row_ptr, m.col_idx, ctx=gpu_ctx_team), ref)
    got = pbrcm.find_peripheral(m.row_ptr, m.col_idx, ctx=gpu_ctx_team)
    assert got == (ref["start"], ref["passes"], ref["ecc"])


@pytest.fixture(scope="module")
def solo_ctx(pbrcm, gpu_ctx):
    """A context whose batches keep every matrix on the solo kernel."""
    import os
    old = os.environ.get("PBRCM_RESIDENT_GROUP")
    os.environ["PBRCM_RESIDENT_GROUP"] = "0"
    try:
        ctx = pbrcm.Context(0)
    finally:
        if old is None:
            del os.environ["PBRCM_RESIDENT_GROUP"]
        else:
            os.environ["PBRCM_RESIDENT_GROUP"] = old
    yield ctx
    ctx.close()


@pytest.mark.parametrize("engine", ["default", "solo"])
@pytest.mark.parametrize("device", [False, True])
def test_batch_search(pbrcm, gpu_ctx, solo_ctx, built, engine, device):
    """A batch of fewer matrices than SMs, small ones (shared-memory engine by
    default) and big ones mixed, from host and from device buffers."""
    import torch
    ctx = gpu_ctx if engine == "default" else solo_ctx
    names = list(_cases())
    mats = [built(k)[0] for k in names]
    if device:
        d = [tuple(torch.from_numpy(a.view(np.int32)).cuda() for a in (m.row_ptr, m.col_idx))
             + (torch.empty(m.n, dtype=torch.int32, device="cuda"),) for m in mats]
        res = pbrcm.reorder_batch_device(d, ctx=ctx)
        perms = [x[2].cpu().numpy().view(np.uint32) for x in d]
    else:
        perms, res = pbrcm.reorder_batch([(m.row_ptr, m.col_idx) for m in mats], ctx=ctx)
    for k, p, r in zip(names, perms, res):
        _same(p, r, built(k)[1])


@pytest.mark.parametrize("name", list(_cases()))
def test_shared_memory_engine_search(pbrcm, gpu_ctx, built, name):
    """The single-matrix path's own choice (the shared-memory engine for all
    but the biggest)."""
    m, ref = built(name)
    _same(*pbrcm.reorder(m.row_ptr, m.col_idx, ctx=gpu_ctx), ref)


@pytest.mark.parametrize("keep", [1, 4, 40])
def test_kept_nodes_option(pbrcm, gpu_ctx, gpu_ctx_team, keep):
    """peripheral_nodes decides which of the last level's nodes count: the
    batch and the team (ordered and unordered passes mixed differently) agree
    with each other and with the shared-memory engine."""
    m = _cases()["rgg_700"]()
    one = pbrcm.reorder(m.row_ptr, m.col_idx, ctx=gpu_ctx, peripheral_nodes=keep)
    team = pbrcm.reorder(m.row_ptr, m.col_idx, ctx=gpu_ctx_team, peripheral_nodes=keep)
    perms, res = pbrcm.reorder_batch([(m.row_ptr, m.col_idx)], ctx=gpu_ctx, peripheral_nodes=keep)
    for perm, r in (team, (perms[0], res[0])):
        assert np.array_equal(perm, one[0])
        assert (r["start_node"], r["peripheral_passes"]) == (one[1]["start_node"], one[1]["peripheral_passes"])
