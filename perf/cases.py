"""The work a user has this library do, as measurable cases over its public
Python entry points: single reorders (host and device buffers), batches,
the serving session, P A P^T and the connectivity repair.

The matrices are seeded patterns of the kinds the repository generates
(parallelbatchrcm_b200/gen.py): 5-point and 7-point grids, random geometric
graphs with 0.1% random long edges, and random graphs, labels shuffled and
components joined by the loader's rule.  They are built here with torch on
the GPU, thousands of matrices at a time as one disjoint union, so that
making them costs little beside reordering them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import parallelbatchrcm_b200 as P

DEV = "cuda"
GROUP_ENTRIES = 60_000_000  # matrices are generated in unions of about this many entries


# ---------------------------------------------------------------------------
# Generators
# ---------------------------------------------------------------------------

def _excl(x: torch.Tensor) -> torch.Tensor:
    return torch.cumsum(x, 0) - x


def _ids(counts: torch.Tensor):
    """(segment, index inside the segment) of every element of a union."""
    seg = torch.repeat_interleave(torch.arange(counts.numel(), device=DEV), counts)
    return seg, torch.arange(seg.numel(), device=DEV) - _excl(counts)[seg]


def _grid_edges(dims):
    """Nearest-neighbour links of a union of nx x ny x nz grids."""
    d = torch.tensor(dims, device=DEV)
    count = d.prod(1)
    seg, i = _ids(count)
    g = torch.arange(seg.numel(), device=DEV)
    nx, ny, nz = d[seg, 0], d[seg, 1], d[seg, 2]
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    us, vs = [], []
    for ok, step in ((x + 1 < nx, 1), (y + 1 < ny, nx), (z + 1 < nz, nx * ny)):
        u = g[ok]
        us.append(u)
        vs.append(u + (step if isinstance(step, int) else step[ok]))
    return torch.cat(us), torch.cat(vs)


def _rgg_edges(ns, kmin, kmax, long_frac, gen):
    """A union of random geometric graphs: points uniform in the unit square,
    each joined to its k ~ U{kmin..kmax} nearest neighbours (searched in the
    3 x 3 cells around it), plus random long edges."""
    per_cell, cap = max(4, (kmax + 3) // 2), 3 * max(4, (kmax + 3) // 2)
    n = torch.tensor(ns, device=DEV)
    side = torch.clamp(torch.sqrt(n / per_cell).long(), min=1)
    cell0 = _excl(side * side)
    seg, _ = _ids(n)
    pts = torch.rand((seg.numel(), 2), device=DEV, generator=gen)
    s = side[seg]
    cx, cy = [(torch.minimum((pts[:, a] * s).long(), s - 1)) for a in (0, 1)]
    cell, order = torch.sort(cell0[seg] + cy * s + cx, stable=True)
    # the points renumbered in cell order (labels are shuffled later)
    pts, cx, cy = pts[order], cx[order], cy[order]
    ncell = int((side * side).sum())
    cnt = torch.bincount(cell, minlength=ncell)
    first = _excl(cnt)
    k = torch.randint(kmin, kmax + 1, (seg.numel(),), device=DEV, generator=gen)
    us, vs = [], []
    for a in range(0, seg.numel(), 400_000):
        b = min(a + 400_000, seg.numel())
        r = torch.arange(a, b, device=DEV)
        cand = []
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                x, y, w = cx[a:b] + dx, cy[a:b] + dy, s[a:b]
                ok = (x >= 0) & (x < w) & (y >= 0) & (y < w)
                c = torch.where(ok, cell0[seg[a:b]] + y * w + x, 0)
                j = torch.arange(cap, device=DEV)[None, :]
                at = first[c][:, None] + j
                cand.append(torch.where(ok[:, None] & (j < cnt[c][:, None]), at, -1))
        cand = torch.cat(cand, 1)
        d = pts[cand.clamp(min=0)] - pts[a:b, None, :]
        d = torch.where((cand >= 0) & (cand != r[:, None]), (d * d).sum(2), torch.inf)
        dist, idx = torch.topk(d, kmax, dim=1, largest=False)
        take = (torch.arange(kmax, device=DEV)[None, :] < k[a:b, None]) & torch.isfinite(dist)
        us.append(r[:, None].expand(-1, kmax)[take])
        vs.append(torch.gather(cand, 1, idx)[take])
    u, v = torch.cat(us), torch.cat(vs)
    nlong = int(round(long_frac * u.numel()))
    if nlong:
        sg = seg[torch.randint(0, seg.numel(), (nlong,), device=DEV, generator=gen)]
        ends = [_excl(n)[sg] + (torch.rand(nlong, device=DEV, generator=gen, dtype=torch.float64) * n[sg]).long()
                for _ in range(2)]
        u, v = torch.cat([u, ends[0]]), torch.cat([v, ends[1]])
    return u, v


def _random_edges(ns, deg, gen):
    n = torch.tensor(ns, device=DEV)
    seg, _ = _ids(n * deg // 2)
    return tuple(_excl(n)[seg] + (torch.rand(seg.numel(), device=DEV, generator=gen, dtype=torch.float64)
                                  * n[seg]).long() for _ in range(2))


def _join(n, u, v):
    """The links (m - 1, m) of the loader: m = the smallest node of each
    component that is not its matrix's first one (min-label propagation)."""
    total = int(n.sum())
    lab = torch.arange(total, device=DEV)
    while True:
        m = torch.minimum(lab[u], lab[v])
        new = lab.clone()
        new.scatter_reduce_(0, lab[u], m, "amin")
        new.scatter_reduce_(0, lab[v], m, "amin")
        new = new[new][new]
        if torch.equal(new, lab):
            break
        lab = new
    roots = torch.nonzero(lab == torch.arange(total, device=DEV)).flatten()
    roots = roots[~torch.isin(roots, _excl(n))]
    return torch.cat([u, roots - 1]), torch.cat([v, roots])


def _union(specs, gen, relabel, joined):
    """(row_ptr, col_idx) int32 CUDA tensors of matrices of one kind: links
    drawn from gen, labels from relabel."""
    kind = specs[0][0]
    if kind in ("grid2d", "grid3d"):
        n = torch.tensor([math.prod(s[1]) for s in specs], device=DEV)
        u, v = _grid_edges([s[1] for s in specs])
    elif kind == "rgg":
        n = torch.tensor([s[1][0] for s in specs], device=DEV)
        u, v = _rgg_edges([s[1][0] for s in specs], specs[0][1][1], specs[0][1][2], specs[0][1][3], gen)
    else:
        n = torch.tensor([s[1][0] for s in specs], device=DEV)
        u, v = _random_edges([s[1][0] for s in specs], specs[0][1][1], gen)
    total, base = int(n.sum()), _excl(n)
    seg, _ = _ids(n)
    # labels shuffled inside each matrix
    lot = torch.randint(0, 1 << 40, (total,), device=DEV, generator=relabel)
    label = torch.empty(total, dtype=torch.long, device=DEV)
    label[torch.argsort((seg << 40) | lot, stable=True)] = torch.arange(total, device=DEV)
    u, v = label[u], label[v]
    if joined and kind in ("rgg", "random"):
        u, v = _join(n, u, v)
    keep = u != v
    u, v = u[keep], v[keep]
    diag = torch.arange(total, device=DEV)
    key = torch.sort(torch.cat([(u << 32) | v, (v << 32) | u, (diag << 32) | diag])).values
    key = torch.unique_consecutive(key)
    rows = key >> 32
    rp = torch.zeros(total + 1, dtype=torch.long, device=DEV)
    torch.cumsum(torch.bincount(rows, minlength=total), 0, out=rp[1:])
    ci = ((key & 0xFFFFFFFF) - base[seg[rows]]).int()
    b = base.tolist() + [total]
    e = rp[torch.tensor(b, device=DEV)].tolist()
    return [((rp[b[i]:b[i + 1] + 1] - e[i]).int(), ci[e[i]:e[i + 1]].clone()) for i in range(len(specs))]


def _entries(spec):
    """About how many entries a spec's matrix has."""
    kind, d = spec
    if kind == "grid2d":
        return 5 * math.prod(d) - 2 * (d[0] + d[1])
    if kind == "grid3d":
        return 7 * math.prod(d) - 2 * (d[0] * d[1] + d[1] * d[2] + d[0] * d[2])
    if kind == "rgg":
        return int(d[0] * (1 + 1.25 * (d[1] + d[2]) / 2))
    return d[0] * (1 + d[1])


def _generator(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return gen


def _make(specs, seed, joined=True, fixed_links=False):
    """fixed_links: the unlabelled graph is the specs' own, the seed shuffles
    its labels (every seed then has the same number of entries)."""
    relabel = _generator(seed)
    gen = _generator(1) if fixed_links else relabel
    out = [None] * len(specs)
    for kind in ("grid2d", "grid3d", "rgg", "random"):
        group, size = [], 0
        for i in [i for i, s in enumerate(specs) if s[0] == kind] + [None]:
            if group and (i is None or size + _entries(specs[i]) > GROUP_ENTRIES):
                for j, m in zip(group, _union([specs[g] for g in group], gen, relabel, joined)):
                    out[j] = m
                group, size = [], 0
            if i is not None:
                group.append(i)
                size += _entries(specs[i])
    return out


def _spec(kind, n, kmin=6, kmax=14):
    if kind == "grid2d":
        a = max(2, round(math.sqrt(n)))
        return kind, (a, max(2, round(n / a)), 1)
    if kind == "grid3d":
        a = max(2, round(n ** (1 / 3)))
        b = max(2, round(math.sqrt(n / a)))
        return kind, (a, b, max(2, round(n / (a * b))))
    if kind == "rgg":
        return kind, (n, kmin, kmax, 0.001)
    return kind, (n, 14)


def _case_specs(case):
    """The matrices of a case; sizes are the case's own, log-uniform in
    [nmin, nmax] where it has many (40% 2-D grids, 30% 3-D grids, 30%
    geometric graphs, as the repository's mixed batch)."""
    if "nx" in case:
        return [(case["kind"], (case["nx"], case["ny"], case["nz"]))]
    if "count" not in case:
        if case["op"] == "connect":  # few neighbours a point: many components
            return [("rgg", (case["n"], 1, 3, 0.0))]
        return [_spec(case["kind"], case["n"])]
    c, lo, hi = case["count"], math.log(case["nmin"]), math.log(case["nmax"])
    sizes = [int(math.exp(lo + (hi - lo) * (i + 0.5) / c)) for i in range(c)]
    cycle = ("grid2d", "grid3d", "rgg", "grid2d", "grid3d", "rgg", "grid2d", "grid3d", "rgg", "grid2d")
    return [_spec(cycle[(7 * i) % 10], n, 4, 12) for i, n in enumerate(sizes)]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: one small mesh from host arrays (the repository's
        # 64 x 64 grid); fixed costs and copies count as much as the kernel
        {"name": "host_grid2d_64", "op": "host", "kind": "grid2d", "nx": 64, "ny": 64, "nz": 1},
        # an ordinary irregular matrix already on the GPU, an odd size
        {"name": "dev_rgg_20k", "op": "device", "kind": "rgg", "n": 20011},
        # a long, thin level structure: about 1,400 levels a pass
        {"name": "dev_grid2d_701x699", "op": "device", "kind": "grid2d", "nx": 701, "ny": 699, "nz": 1},
        # the repository's large single matrices: the 128^3 grid, the 1M-node
        # geometric graph, and a random graph of few, wide levels
        {"name": "dev_grid3d_128", "op": "device", "kind": "grid3d", "nx": 128, "ny": 128, "nz": 128},
        {"name": "dev_rgg_1m", "op": "device", "kind": "rgg", "n": 1000000},
        {"name": "dev_random_2m", "op": "device", "kind": "random", "n": 2000000},
        # a small batch of small matrices (blocks of a decomposed problem)
        {"name": "batch_small_96", "op": "batch_device", "count": 96, "nmin": 500, "nmax": 5000},
        # the headline batch: 4,096 mixed matrices resident on the GPU
        {"name": "batch_mixed_4096", "op": "batch_device", "count": 4096, "nmin": 500, "nmax": 200000},
        # a batch from pinned host buffers, copies included
        {"name": "batch_host_384", "op": "batch_host", "count": 384, "nmin": 500, "nmax": 200000},
        # serving: a burst of requests of mixed sizes from host arrays
        {"name": "serve_96", "op": "serve", "count": 96, "nmin": 1000, "nmax": 400000},
        # the reordered matrix with its values, and the loader's repair of a
        # pattern in many pieces
        {"name": "permute_f64_grid3d_128", "op": "permute", "kind": "grid3d", "nx": 128, "ny": 128, "nz": 128,
         "val_bytes": 8, "map": False},
        {"name": "connect_4m", "op": "connect", "n": 4000000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["host", "device", "device", "device", "device", "batch_device", "batch_device", "batch_host",
                     "serve", "permute", "connect"])
    if op in ("host", "device"):
        kind = rng.choice(["grid2d", "grid3d", "rgg", "random"])
        top = 500_000 if kind == "grid2d" or op == "host" else 2_000_000
        return {"op": op, "kind": kind, "n": _log(rng, 500, top), "reverse": rng.random() < 0.8,
                "bandwidth": rng.random() < 0.8, "given_start": rng.random() < 0.2}
    if op in ("batch_device", "batch_host"):
        nmin = _log(rng, 500, 5000)
        return {"op": op, "count": _log(rng, 8, 1500 if op == "batch_device" else 300), "nmin": nmin,
                "nmax": _log(rng, 2 * nmin, 200_000), "reverse": rng.random() < 0.8, "bandwidth": rng.random() < 0.8}
    if op == "serve":
        return {"op": op, "count": _log(rng, 8, 96), "nmin": 1000, "nmax": _log(rng, 3000, 400_000)}
    if op == "permute":
        return {"op": op, "kind": rng.choice(["grid2d", "grid3d", "rgg", "random"]), "n": _log(rng, 4000, 1_900_000),
                "val_bytes": rng.choice([0, 4, 8]), "map": rng.random() < 0.3}
    return {"op": op, "n": _log(rng, 50_000, 4_000_000)}


def _host(t: torch.Tensor) -> np.ndarray:
    return t.cpu().numpy().view(np.uint32)


def prepare(case, seed):
    op = case["op"]
    # (permute and connect return arrays as long as the matrix: the same for
    # every seed)
    mats = _make(_case_specs(case), seed, joined=op != "connect", fixed_links=op in ("permute", "connect"))
    st = {"op": op, "ctx": P.Context(torch.cuda.current_device()), "opts": {
        "reverse": case.get("reverse", True), "want_bandwidth": case.get("bandwidth", True)}}
    if op in ("host", "device") and case.get("given_start"):
        st["opts"]["start"] = seed % (mats[0][0].numel() - 1)
    if op == "host":
        st["mat"] = [_host(t) for t in mats[0]]
    elif op == "device":
        st["mat"] = mats[0]
        st["perm"] = torch.empty(mats[0][0].numel() - 1, dtype=torch.int32, device=DEV)
    elif op == "batch_device":
        # one permutation buffer, a slice for each matrix
        ns = [rp.numel() - 1 for rp, _ in mats]
        st["perm"] = torch.empty(sum(ns), dtype=torch.int32, device=DEV)
        st["batch"] = P.PreparedBatch([(rp, ci, p) for (rp, ci), p in zip(mats, torch.split(st["perm"], ns))],
                                      device=True)
    elif op == "batch_host":
        # pinned staging, each matrix's col_idx behind its row_ptr
        st["slab"] = torch.cat([t for m in mats for t in m]).cpu().pin_memory()
        flat, sizes = st["slab"].numpy().view(np.uint32), [t.numel() for m in mats for t in m]
        parts = np.split(flat, np.cumsum(sizes)[:-1])
        ns = [s - 1 for s in sizes[::2]]
        st["perm"] = torch.empty(sum(ns), dtype=torch.int32).pin_memory()
        perms = np.split(st["perm"].numpy().view(np.uint32), np.cumsum(ns)[:-1])
        st["batch"] = P.PreparedBatch(list(zip(parts[::2], parts[1::2])), perms)
    elif op == "serve":
        st["mats"] = [tuple(_host(t) for t in m) for m in mats]
        st["session"] = P.Session(st["ctx"], streams=96)
    elif op == "permute":
        st["mat"] = mats[0]
        st["perm"], _ = P.reorder_device(*mats[0], ctx=st["ctx"])
        vb = case["val_bytes"]
        st["vals"] = None if vb == 0 else torch.randn(mats[0][1].numel(), device=DEV, generator=_generator(seed),
                                                      dtype=torch.float64 if vb == 8 else torch.float32)
        st["map"] = case["map"]
    else:
        st["mat"] = mats[0]
    torch.cuda.synchronize()
    return st


def _fields(results):
    """The numbers a caller reads beside the permutations."""
    keys = ("status", "start_node", "peripheral_passes", "eccentricity", "levels", "placed", "bandwidth",
            "initial_bandwidth", "profile")
    return np.array([[int(r[k]) for k in keys] for r in results], dtype=np.int64)


def run(st):
    op, ctx = st["op"], st["ctx"]
    if op == "host":
        perm, res = P.reorder(*st["mat"], ctx=ctx, **st["opts"])
        return perm, _fields([res])
    if op == "device":
        perm, res = P.reorder_device(*st["mat"], st["perm"], ctx=ctx, **st["opts"])
        return perm, _fields([res])
    if op == "batch_device":
        return st["perm"], _fields(P.reorder_batch_device(st["batch"], ctx=ctx, **st["opts"]))
    if op == "batch_host":
        _, res = P.reorder_batch(st["batch"], ctx=ctx, **st["opts"])
        return st["perm"], _fields(res)
    if op == "serve":
        tickets = [st["session"].submit(rp, ci) for rp, ci in st["mats"]]
        st["session"].drain()
        done = [st["session"].poll(t) for t in tickets]
        return np.concatenate([p for p, _ in done]), _fields([r for _, r in done])
    if op == "permute":
        return tuple(x for x in P.permute_device(*st["mat"], st["perm"], st["vals"], want_map=st["map"], ctx=ctx)
                     if x is not None)
    return P.connect_device(*st["mat"], ctx=ctx)


def work(case):
    """Bytes of one pass: every input read once, every output written once."""
    specs = _case_specs(case)
    n = sum(math.prod(s[1]) if s[0] in ("grid2d", "grid3d") else s[1][0] for s in specs)
    nnz = sum(_entries(s) for s in specs)
    csr = 4 * (n + len(specs)) + 4 * nnz
    if case["op"] == "permute":
        vb = case["val_bytes"]
        return {"bytes": 2 * csr + 4 * n + (2 * vb + (4 if case["map"] else 0)) * nnz, "flops": 0}
    if case["op"] == "connect":
        return {"bytes": 2 * csr, "flops": 0}
    return {"bytes": csr + 4 * n, "flops": 0}
