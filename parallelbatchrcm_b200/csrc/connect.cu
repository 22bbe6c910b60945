// connect.cu -- the connectivity repair of the reference loader, on the device.
//
// prepareRCM (include/Graph.h:160-263) walks the matrix breadth-first from
// its first non-empty row `minn`; while nodes are left over it links the
// smallest unvisited node i to the largest visited node below i (or, with
// none below, to the smallest visited node above i), then walks on from i,
// and finally rebuilds the CSR sorted by (row, col) with both directions of
// every link added.  Every node below the smallest unvisited one has been
// visited by then, so the links depend on the components alone:
//   - a component whose smallest node m > 0 is not minn's gets (m - 1, m);
//   - the component {0} (row 0 empty, so minn > 0) gets (0, minn).
// An empty row is a component of its own.  (The reference never finishes on
// an empty row, which it queues without marking; the host loader of this
// library and this pass link it like any other component.)
//
// Passes (a warp takes 32 rows at a time and deals their entries out to its
// lanes, so that no entry searches row_ptr for its row; in the hook pass a
// lane has four entries' chains of dependent loads in flight; groups of 32 rows
// with more than 1,024 entries are cut into units of 512, in a second form of
// passes 2 and 4):
//   1. k_cc_init: parent[v] = min(v, first column of row v) (rows are sorted,
//      so that is the smallest neighbour) and minn; checks the row pointers
//      and lists the groups of 32 rows with more than 1,024 entries;
//      k_cc_flatten: every node under its root in that forest;
//   2. k_cc_hook: union-find over the entries (u, v), u < v, hooking the
//      larger root under the smaller with atomicCAS and halving paths on the
//      way up -- the minimum-label form of the ECL-CC algorithm (Jaiganesh and
//      Burtscher, HPDC 2018), so that each component's root is its smallest
//      node and "m is a component minimum" is parent[m] == m afterwards.  The
//      same pass checks each entry: column in range, row sorted, and the
//      pattern symmetric (the repair is defined on symmetric patterns): every
//      entry left of the diagonal has its transposed entry, and there are as
//      many distinct entries right of it, so those have theirs too -- half the
//      random searches of checking every entry.  The unions that are left are dealt
//      out to the lanes (each a chain of dependent loads; one after the other they
//      took 375 us of 15M entries, side by side 284);
//   3. k_connect_rowlen: row length plus the links of the row (at most two),
//      scanned into row_ptr_out (the scan kernels of permute.cu);
//   4. k_connect_copy: each entry shifted to its place in the output row, then
//      each link inserted at its sorted position.
#include <algorithm>
#include <cstdint>

#include <cuda_runtime.h>

#include "entries.h"
#include "kernels.h"
#include "types.h"

namespace pbrcm {

namespace {

constexpr int kThreads = 256;
constexpr int kInFlight = 4;  // entries a lane of the hook pass works on at once
// A tile of more than kBigTile entries is cut into units of kUnit that all warps
// take (a row has as many entries as its node has neighbours: the repair of a
// star of 2M nodes takes 72 ms with a tile to a warp, 0.29 so).
constexpr uint32_t kBigTile = 1024, kUnit = 512;

// counters[0] minn, [1] links, [2] check flags, [3] distinct entries left of
// the diagonal less those right of it, [4..5] the 64-bit head of the big tiles
constexpr uint32_t kFlagRange = 1, kFlagUnsorted = 2, kFlagAsym = 4, kFlagDepth = 8, kFlagBig = kConnectBig;

// Row v's entry range, clamped into [0, nnz] (a bad row_ptr must not send a
// kernel out of bounds before the call's verdict is read).
__device__ __forceinline__ void row_range(const uint32_t* __restrict__ rp, uint32_t v, uint32_t nnz, uint32_t& b,
                                          uint32_t& e)
{
    b = min(rp[v], nnz);
    e = min(max(rp[v + 1], b), nnz);
}

// The 32 rows from v0 on, one per lane (empty past n).
struct RowTile {
    uint32_t b, e;      // this lane's row
    uint32_t beg, end;  // entries of the tile
    __device__ __forceinline__ RowTile(const uint32_t* __restrict__ rp, uint32_t n, uint32_t nnz, uint32_t v0)
    {
        const uint32_t lane = threadIdx.x & 31u;
        const uint64_t v = (uint64_t)v0 + lane;
        b = e = min(rp[n], nnz);
        if (v < n)
            row_range(rp, (uint32_t)v, nnz, b, e);
        beg = __shfl_sync(kFull, b, 0);
        end = __shfl_sync(kFull, e, 31);
    }
    // The lane whose row holds entry k: the last with b <= k (by the whole
    // warp; k past the end names some lane).
    __device__ __forceinline__ uint32_t lane_of(uint32_t k) const
    {
        uint32_t l = 0;
#pragma unroll
        for (uint32_t d = 16; d > 0; d >>= 1)
            l = __shfl_sync(kFull, b, l + d) <= k ? l + d : l;
        return l;
    }
};

// The tiles of more than kBigTile entries (k_cc_init lists them): list[i] = {tile,
// units of the tiles before it}; *head = tiles << 32 | units.
struct BigTiles {
    uint2* list;
    uint32_t cap;  // all tiles
    unsigned long long* head;
};

// What a pass over entries works on: visit(v0, t, kb, ke) for entries [kb, ke) of
// the tile t from row v0 on -- every tile, or (BIG: there are big ones) every
// other tile, then the big ones' units.  Patterns with big tiles have kernels of
// their own, launched behind the verdict that there are any (launch_connect_big):
// with the units in the same kernels an ordinary pattern takes 2-11 % longer
// (other registers and spills; 1.2M nodes, 4.5M entries: the hook pass 114 us,
// 118-137 with them).
template <bool BIG, class Visit>
__device__ __forceinline__ void for_tiles(const uint32_t* __restrict__ rp, uint32_t n, uint32_t nnz, Visit visit)
{
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32 < n; w += nwarps) {
        const uint32_t v0 = (uint32_t)(w * 32);
        const RowTile t(rp, n, nnz, v0);
        if (!BIG || t.end - t.beg <= kBigTile)
            visit(v0, t, t.beg, t.end);
    }
}

template <class Visit>
__device__ __forceinline__ void for_units(const uint32_t* __restrict__ rp, uint32_t n, uint32_t nnz,
                                          const BigTiles& big, Visit visit)
{
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned long long head = __ldcg(big.head);
    const uint32_t tiles = min((uint32_t)(head >> 32), big.cap), units = tiles != 0 ? (uint32_t)head : 0u;
    for (uint64_t x = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < units; x += nwarps) {
        uint32_t lo = 0;  // the last listed tile that begins at or before unit x
        for (uint32_t len = tiles; len > 1;) {
            const uint32_t half = len / 2;
            if (big.list[lo + half].y <= x)
                lo += half;
            len -= half;
        }
        const uint2 at = big.list[lo];
        const RowTile t(rp, n, nnz, at.x * 32);
        const uint32_t all = t.end - t.beg, k = ((uint32_t)x - at.y) * kUnit;
        const uint32_t kb = k < all ? t.beg + k : t.end;
        visit(at.x * 32, t, kb, t.end - kb > kUnit ? kb + kUnit : t.end);
    }
}

// First index in ci[b, e) whose column is >= x (a sorted row).
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* __restrict__ ci, uint32_t b, uint32_t e, uint32_t x)
{
    while (b < e) {
        const uint32_t mid = b + (e - b) / 2;
        if (ci[mid] < x)
            b = mid + 1;
        else
            e = mid;
    }
    return b;
}

// Root of v.  Parents only ever point to smaller nodes of the same component,
// so x strictly decreases and the climb ends within v steps; each visited
// node is re-pointed to its grandparent (path halving).  Parent words are
// read through L2 (other threads hook roots concurrently); a halving store
// only ever replaces a non-root's parent by one of its ancestors, and roots
// change only by the atomicCAS in cc_unite, so no hook is lost.
__device__ __forceinline__ uint32_t cc_root(uint32_t* parent, uint32_t v)
{
    uint32_t x = v;
    uint32_t p = __ldcg(parent + x);
    while (p != x) {
        const uint32_t g = __ldcg(parent + p);
        if (g != p)
            parent[x] = g;
        x = g;
        p = __ldcg(parent + x);
    }
    return x;
}

// Joins the components of a and b: the larger root is hooked under the
// smaller.  A failed atomicCAS means that root was hooked meanwhile; the
// union climbs on from its new parent.  Every retry follows a successful hook
// by another thread, and there are at most n - 1 hooks, so the loop is
// bounded by the size of the graph; the explicit limit only guards that.
__device__ __forceinline__ bool cc_unite(uint32_t* parent, uint32_t a, uint32_t b, uint32_t limit)
{
    uint32_t ra = cc_root(parent, a), rb = cc_root(parent, b);
    for (uint32_t it = 0; ra != rb; ++it) {
        if (it > limit)
            return false;
        if (ra < rb) {
            const uint32_t t = ra;
            ra = rb;
            rb = t;
        }
        const uint32_t old = atomicCAS(parent + ra, ra, rb);
        if (old == ra)
            return true;
        ra = cc_root(parent, old);
        rb = cc_root(parent, rb);
    }
    return true;
}

__device__ __forceinline__ bool is_link_min(const uint32_t* __restrict__ parent, uint32_t n, uint32_t minn, uint32_t x)
{
    return x < n && minn < n && x != minn && __ldg(parent + x) == x;
}

// The links of row v in ascending column order; returns their count (0-2).
__device__ __forceinline__ int row_links(const uint32_t* __restrict__ parent, uint32_t n, uint32_t minn, uint32_t v,
                                         uint32_t e[2])
{
    uint32_t c[3];
    int k = 0;
    if (v == minn && minn > 0 && is_link_min(parent, n, minn, 0))
        c[k++] = 0;  // row minn takes (0, minn)
    if (is_link_min(parent, n, minn, v))
        c[k++] = v > 0 ? v - 1 : minn;  // v is a component's smallest node
    if (v + 1 < n && is_link_min(parent, n, minn, v + 1))
        c[k++] = v + 1;  // v + 1 is one, linked to v
    // at most two of the three hold (v == minn excludes the second); sort
    if (k == 2 && c[0] > c[1]) {
        const uint32_t t = c[0];
        c[0] = c[1];
        c[1] = t;
    }
    e[0] = k > 0 ? c[0] : 0;
    e[1] = k > 1 ? c[1] : 0;
    return k > 2 ? 2 : k;
}

__global__ void __launch_bounds__(kThreads, 8) k_cc_init(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                                                      uint32_t n, uint32_t nnz, uint32_t* __restrict__ parent,
                                                      uint32_t* counters, BigTiles big)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t first = kFull, flags = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint32_t v = (uint32_t)i;
        uint32_t b, e;
        const uint32_t b0 = rp[v], e0 = rp[v + 1];
        if (e0 < b0 || e0 > nnz || (v == 0 && b0 != 0) || (v == n - 1 && e0 != nnz))
            flags |= kFlagRange;
        row_range(rp, v, nnz, b, e);
        if ((v & 31u) == 0) {  // the tile's entries
            const uint32_t end = min(max(rp[min(i + 32, (uint64_t)n)], b), nnz);
            if (end - b > kBigTile) {
                const unsigned long long units = (end - b - 1) / kUnit + 1;
                const unsigned long long old = atomicAdd(big.head, 1ull << 32 | units);
                if ((uint32_t)(old >> 32) < big.cap)  // (bad row pointers may list more)
                    big.list[old >> 32] = make_uint2(v / 32u, (uint32_t)old);
                flags |= kFlagBig;
            }
        }
        uint32_t p = v;
        if (e > b) {
            first = min(first, v);
            const uint32_t c = ci[b];
            if (c < p)
                p = c;
        }
        parent[v] = p;
    }
    first = __reduce_min_sync(0xFFFFFFFFu, first);
    if ((threadIdx.x & 31) == 0 && first != kFull)
        atomicMin(counters, first);
    flags = __reduce_or_sync(0xFFFFFFFFu, flags);
    if ((threadIdx.x & 31) == 0 && flags)
        atomicOr(counters + 2, flags);
}

// parent[v] = root of v in the forest of first columns (k_cc_init), so that
// most entries of the hook pass find both ends under one root and the others
// start their climb at one.
__global__ void __launch_bounds__(kThreads) k_cc_flatten(uint32_t n, uint32_t* parent)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
        uint32_t p = __ldcg(parent + v);
        for (uint32_t g = __ldcg(parent + p); g != p; g = __ldcg(parent + p))
            p = g;
        parent[v] = p;
    }
}

// (PART 0: every tile, 1: all but the big ones, 2: the units)
template <int PART>
__device__ __forceinline__ void hook_entries(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                                             uint32_t n, uint32_t nnz, uint32_t* parent, uint32_t* counters,
                                             const BigTiles& big, uint2* list)
{
    constexpr int U = kInFlight;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t flags = 0, lower = 0;
    auto visit = [&](uint32_t v0, const RowTile& t, uint32_t kb, uint32_t ke) {
        for (EntrySteps<U> es(kb, ke); es.more(); es.next()) {
            uint32_t v[U], u[U], ub[U], ue[U];
#pragma unroll
            for (int i = 0; i < U; ++i) {
                uint32_t k;
                const bool in = es.entry(i, lane, k);
                const uint32_t l = t.lane_of(k);
                const uint32_t b = __shfl_sync(kFull, t.b, l), e = __shfl_sync(kFull, t.e, l);
                v[i] = v0 + l;
                u[i] = v[i];  // nothing to do
                if (in) {
                    if (k < b || k >= e) {  // only a bad row_ptr leaves k outside every row
                        flags |= kFlagRange;
                    } else {
                        const uint32_t c = ci[k], prev = k > b ? ci[k - 1] : kFull;
                        if (c >= n)
                            flags |= kFlagRange;
                        else if (c < v[i])
                            u[i] = c;
                        if (k > b && prev > c)
                            flags |= kFlagUnsorted;
                        if (prev != c)
                            lower += c < v[i] ? 1u : c > v[i] ? 0xFFFFFFFFu : 0u;
                    }
                }
            }
            // the neighbours' rows, and both ends' parents
            uint32_t pu[U], pv[U];
#pragma unroll
            for (int i = 0; i < U; ++i) {
                ub[i] = ue[i] = pu[i] = pv[i] = 0;
                if (u[i] != v[i]) {
                    row_range(rp, u[i], nnz, ub[i], ue[i]);
                    pu[i] = __ldcg(parent + u[i]);
                    pv[i] = __ldcg(parent + v[i]);
                }
            }
            // the transposed entry: four columns of each neighbour's row at a
            // time (rows are short), a longer row narrowed first
#pragma unroll
            for (int i = 0; i < U; ++i)
                while (ue[i] - ub[i] > 16) {
                    const uint32_t mid = ub[i] + (ue[i] - ub[i]) / 2;
                    if (ci[mid] <= v[i])
                        ub[i] = mid;
                    else
                        ue[i] = mid;
                }
            bool more = true;
            while (__any_sync(kFull, more)) {
                uint32_t x[U][4];
#pragma unroll
                for (int i = 0; i < U; ++i)
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        x[i][q] = ub[i] + q < ue[i] ? ci[ub[i] + q] : kFull;
                more = false;
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    // found: an empty range, with the row's end as a mark
                    if (x[i][0] == v[i] || x[i][1] == v[i] || x[i][2] == v[i] || x[i][3] == v[i])
                        ub[i] = ue[i] = kFull;
                    else if (ub[i] < ue[i])
                        ub[i] = min(ub[i] + 4, ue[i]);
                    more |= ub[i] < ue[i];
                }
            }
            // the pairs to join (two ends under one parent are one component
            // already), side by side
            uint32_t pairs = 0;
#pragma unroll
            for (int i = 0; i < U; ++i) {
                if (u[i] != v[i] && ub[i] != kFull)
                    flags |= kFlagAsym;
                const bool need = u[i] != v[i] && pu[i] != pv[i];
                const uint32_t bal = __ballot_sync(kFull, need);
                if (need)
                    list[pairs + __popc(bal & ((1u << lane) - 1u))] = make_uint2(pu[i], pv[i]);
                pairs += __popc(bal);
            }
            __syncwarp();
            for (uint32_t i = lane; i < pairs; i += 32) {
                const uint2 p = list[i];
                if (!cc_unite(parent, p.x, p.y, n))
                    flags |= kFlagDepth;
            }
            __syncwarp();
        }
    };
    if (PART == 2)
        for_units(rp, n, nnz, big, visit);
    else
        for_tiles<PART == 1>(rp, n, nnz, visit);
    flags = __reduce_or_sync(0xFFFFFFFFu, flags);
    lower = __reduce_add_sync(0xFFFFFFFFu, lower);
    if (lane == 0 && flags)
        atomicOr(counters + 2, flags);
    if (lane == 0 && lower)
        atomicAdd(counters + 3, lower);
}

__device__ __noinline__ void hook_units(const uint32_t* rp, const uint32_t* ci, uint32_t n, uint32_t nnz,
                                        uint32_t* parent, uint32_t* counters, BigTiles big, uint2* list)
{
    hook_entries<2>(rp, ci, n, nnz, parent, counters, big, list);
}

template <bool BIG>
__global__ void __launch_bounds__(kThreads, BIG ? 4 : 0) k_cc_hook(const uint32_t* __restrict__ rp,
                                                                   const uint32_t* __restrict__ ci, uint32_t n,
                                                                   uint32_t nnz, uint32_t* parent, uint32_t* counters,
                                                                   BigTiles big)
{
    // bad row pointers (k_cc_init): the tiles need not partition the entries; or big
    // tiles, for the other form of this pass
    if (__ldcg(counters + 2) & (BIG ? kFlagRange : kFlagRange | kFlagBig))
        return;
    __shared__ uint2 pair_list[kThreads / 32][32 * kInFlight];
    uint2* const list = pair_list[threadIdx.x >> 5];
    hook_entries<BIG ? 1 : 0>(rp, ci, n, nnz, parent, counters, big, list);
    if (BIG)
        hook_units(rp, ci, n, nnz, parent, counters, big, list);
}

// out_rp[v + 1] = length of row v + its links; counters[1] = number of links.
__global__ void __launch_bounds__(kThreads) k_connect_rowlen(const uint32_t* __restrict__ rp, uint32_t n, uint32_t nnz,
                                                             const uint32_t* __restrict__ parent,
                                                             uint32_t* counters, uint32_t* __restrict__ out_rp)
{
    const uint32_t minn = __ldcg(counters);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t links = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint32_t v = (uint32_t)i;
        uint32_t b, e, lk[2];
        row_range(rp, v, nnz, b, e);
        out_rp[v + 1] = (e - b) + (uint32_t)row_links(parent, n, minn, v, lk);
        links += is_link_min(parent, n, minn, v) ? 1u : 0u;
        if (v == 0)
            out_rp[0] = 0;
    }
    links = __reduce_add_sync(0xFFFFFFFFu, links);
    if ((threadIdx.x & 31) == 0 && links)
        atomicAdd(counters + 1, links);
}

// Entry k of row v goes to out_rp[v] + (k - rp[v]) + (links of v below its
// column); a link e_j goes to out_rp[v] + (entries of v below e_j) + j.
// Links never coincide with an entry (they join different components).
// Writes past `cap` are dropped (the host reports the size needed).
template <bool BIG>
__global__ void __launch_bounds__(kThreads) k_connect_copy(const uint32_t* __restrict__ rp,
                                                           const uint32_t* __restrict__ ci, uint32_t n, uint32_t nnz,
                                                           const uint32_t* __restrict__ parent,
                                                           const uint32_t* counters, const uint32_t* __restrict__ out_rp,
                                                           uint32_t* __restrict__ out_ci, uint64_t cap, BigTiles big)
{
    constexpr int U = 4;
    if (__ldcg(counters + 2) != 0)
        return;  // the call fails
    const uint32_t minn = __ldcg(counters);
    const uint32_t lane = threadIdx.x & 31u;
    auto visit = [&](uint32_t v0, const RowTile& t, uint32_t kb, uint32_t ke) {
        uint32_t ob = 0, lk[2] = {0, 0};
        int nl = 0;
        if (v0 + (uint64_t)lane < n) {
            ob = out_rp[v0 + lane];
            if (out_rp[v0 + lane + 1] - ob != t.e - t.b)
                nl = row_links(parent, n, minn, v0 + lane, lk);
        }
        const bool links = __any_sync(kFull, nl != 0);
        for (EntrySteps<U> es(kb, ke); es.more(); es.next()) {
            uint32_t c[U], l[U];
#pragma unroll
            for (int i = 0; i < U; ++i) {
                uint32_t k;
                const bool in = es.entry(i, lane, k);
                l[i] = t.lane_of(k);
                c[i] = in ? ci[k] : 0u;
            }
#pragma unroll
            for (int i = 0; i < U; ++i) {
                uint32_t k;
                const bool in = es.entry(i, lane, k);
                const uint32_t b = __shfl_sync(kFull, t.b, l[i]), e = __shfl_sync(kFull, t.e, l[i]);
                uint64_t at = (uint64_t)__shfl_sync(kFull, ob, l[i]) + (k - b);
                if (links) {
                    const int ln = __shfl_sync(kFull, nl, l[i]);
                    const uint32_t l0 = __shfl_sync(kFull, lk[0], l[i]), l1 = __shfl_sync(kFull, lk[1], l[i]);
                    at += (ln > 0 && l0 < c[i] ? 1 : 0) + (ln > 1 && l1 < c[i] ? 1 : 0);
                }
                if (in && k >= b && k < e && at < cap)
                    out_ci[at] = c[i];
            }
        }
        for (int j = 0; kb == t.beg && j < nl; ++j) {
            const uint64_t at = (uint64_t)ob + (lower_bound(ci, t.b, t.e, lk[j]) - t.b) + j;
            if (at < cap)
                out_ci[at] = lk[j];
        }
    };
    for_tiles<BIG>(rp, n, nnz, visit);
    if (BIG)
        for_units(rp, n, nnz, big, visit);
}

int row_blocks(uint32_t n, int sms)
{
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)n + kThreads - 1) / kThreads, (uint64_t)sms * 8));
}

BigTiles big_tiles(uint2* list, uint32_t n, uint32_t* counters)
{
    return BigTiles{list, connect_tiles_cap(n), reinterpret_cast<unsigned long long*>(counters + 4)};
}

}  // namespace

uint32_t connect_tiles_cap(uint32_t n) { return (uint32_t)(((uint64_t)n + 31) / 32); }

namespace {

// the unions of the entries and the passes behind them
template <bool BIG>
cudaError_t launch_entries(const uint32_t* rp, const uint32_t* ci, uint32_t n, uint32_t nnz, uint32_t* out_rp,
                           uint32_t* out_ci, uint64_t cap, uint32_t* parent, uint32_t* partials, uint32_t* counters,
                           const BigTiles& big, int sms, cudaStream_t st)
{
    // a warp per 32 rows, or per unit of a big tile
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)n + kThreads - 1) / kThreads +
                                                                         (BIG ? nnz / (kUnit * (kThreads / 32)) : 0),
                                                                     (uint64_t)sms * 16));
    if (nnz > 0)
        k_cc_hook<BIG><<<blocks, kThreads, 0, st>>>(rp, ci, n, nnz, parent, counters, big);
    k_connect_rowlen<<<row_blocks(n, sms), kThreads, 0, st>>>(rp, n, nnz, parent, counters, out_rp);
    const cudaError_t e = launch_scan(out_rp + 1, n, partials, st);
    if (e != cudaSuccess)
        return e;
    k_connect_copy<BIG><<<blocks, kThreads, 0, st>>>(rp, ci, n, nnz, parent, counters, out_rp, out_ci, cap, big);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_connect(const uint32_t* rp, const uint32_t* ci, uint32_t n, uint32_t nnz, uint32_t* out_rp,
                           uint32_t* out_ci, uint64_t cap, uint32_t* parent, uint32_t* partials, uint32_t* counters,
                           uint2* tiles, int sms, cudaStream_t st)
{
    const BigTiles big = big_tiles(tiles, n, counters);
    cudaError_t e = cudaMemsetAsync(counters, 0xFF, sizeof(uint32_t), st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(counters + 1, 0, 5 * sizeof(uint32_t), st);
    if (e != cudaSuccess)
        return e;
    k_cc_init<<<row_blocks(n, sms), kThreads, 0, st>>>(rp, ci, n, nnz, parent, counters, big);
    k_cc_flatten<<<row_blocks(n, sms), kThreads, 0, st>>>(n, parent);
    return launch_entries<false>(rp, ci, n, nnz, out_rp, out_ci, cap, parent, partials, counters, big, sms, st);
}

cudaError_t launch_connect_big(const uint32_t* rp, const uint32_t* ci, uint32_t n, uint32_t nnz, uint32_t* out_rp,
                               uint32_t* out_ci, uint64_t cap, uint32_t* parent, uint32_t* partials,
                               uint32_t* counters, uint2* tiles, int sms, cudaStream_t st)
{
    // (links were counted before any union)
    const cudaError_t e = cudaMemsetAsync(counters + 1, 0, 2 * sizeof(uint32_t), st);
    if (e != cudaSuccess)
        return e;
    return launch_entries<true>(rp, ci, n, nnz, out_rp, out_ci, cap, parent, partials, counters,
                                big_tiles(tiles, n, counters), sms, st);
}

}  // namespace pbrcm
