// solo.cuh -- the one-group engine of the batch kernels: the whole reorder of
// one matrix (start search, Cuthill-McKee pass, reverse, bandwidth) by one
// thread group, with the visited set in shared memory.
//
// What it computes is what engine.cuh computes (the serial stable order of
// src/rcm_cpu.cpp:57-104 from the start node of
// src/simple_peripheral.cpp:92-141, and the bandwidth of src/main.cpp:143-184);
// how differs, because a group that owns its matrix alone needs no claim
// protocol:
//
//   * the queue is walked in chunks of consecutive positions (at most B
//     parents and EMAX edges, never across a level boundary); a chunk's
//     children are the still-unvisited neighbours, each taken by the first
//     (parent, slot) that reaches it -- exactly the serial loop, since every
//     node an earlier chunk placed is already marked;
//   * visited is a bitmap in shared memory (n <= kSoloMaxN), so checking a
//     neighbour costs no global load and marking one no atomic in global
//     memory; a larger matrix keeps the bitmap in global memory (n / 8
//     bytes, L2-resident: one L2 round trip more per chunk); inside a chunk a
//     shared-memory hash keeps the first edge to a node (atomicMin of the
//     edge index);
//   * every entry's neighbour record -- its column and that column's row
//     start and valence -- is one 8-byte record of an edge table built once
//     per matrix (solo_build_edges, during the CSR check), so a chunk needs
//     one dependent global load per edge (coalesced along each row) instead
//     of a column load followed by a node-table load; the queue holds the
//     same 8-byte records (node and valence in one word, row start in the
//     other: n <= kSoloMaxNodes, valences < 4,096);
//   * the children of a chunk that is a whole level, if they fit one chunk,
//     stay in shared memory as the next chunk's parents.
//
// Per chunk: each edge's parent by a binary search of the parents' edge
// offsets, the edge records, the visited test and the dedup-table insert, a
// warp-ballot compaction in edge order, the rank of each parent's children
// by (valence, slot), the writes of the queue records and the permutation,
// and the visited marks -- four group barriers in the chunk and three where
// its parents are formed.
//
// Start-search passes whose order does not matter run as solo_level_pass
// instead: no dedup table, no ranks, the first test-and-set of a node's
// visited bit places it.
#pragma once

#include "engine.cuh"

namespace pbrcm {

constexpr uint32_t kSoloEmpty = 0xFFFFFFFFu;

// Shared memory of one solo group (B threads, EMAX edges per chunk).
template <int B, int EMAX>
struct SoloSmem {
    static constexpr int W = B / 32;
    static constexpr int H = 2 * EMAX;  // dedup table slots (power of two, > 2x a chunk's candidates)
    uint32_t vis[kSoloMaxN / 32];
    // parents of the chunk
    uint32_t pn[B], prs[B], pdeg[B];
    uint32_t soff[B + 1];
    uint32_t cs[B], cc[B];  // first compacted child / child count per parent (clear between chunks)
    // the dedup table: (node << kEdgeBits | chunk edge) of the first edge to
    // each unvisited node of the chunk; kSoloEmpty where free (clear between
    // chunks)
    uint32_t tab[H];
    uint32_t so_idx[EMAX];  // the children's ranked order: rank -> compacted index
    // the chunk's children in edge order: node, row start, and valence with
    // the parent's chunk index in the high bits (valence < 2^kParShift); in
    // an unordered pass (solo_level_pass) instead the entries of each warp's
    // rows and the queue records of the current and the next level (the
    // first CAP of each)
    static constexpr int CAP = EMAX / 4 < B ? EMAX / 4 : B;
    static_assert(2 * W * 32 * 8 + 16 * CAP <= 12 * EMAX, "the level pass fits the chunk's child arrays");
    union {
        struct {
            uint32_t ch_c[EMAX], ch_rs[EMAX], ch_dp[EMAX];
        };
        struct {
            uint2 lbuf[2][CAP];
            uint16_t ent[W][32 * 8];
        };
    };
    uint32_t wcnt[W], wdeg[W];
    uint32_t scanbuf[2][W];
    uint32_t tmp32[W + 1];
    unsigned long long tmp64[2 * W + 2];
    uint32_t m, Ec;
    uint32_t bcast[4];
    uint32_t lcnt[3];  // level pass: children of level L at [L % 3]
};

// Chunk edge indices take kEdgeBits bits below the node in a dedup word
// (nodes < 2^20, chunks of at most 2,048 edges: 31 bits).
constexpr uint32_t kEdgeBits = 11;
constexpr uint32_t kParShift = 20;  // ch_dp: valence in the low 20 bits, parent index above
constexpr uint32_t kDegMask = (1u << kParShift) - 1u;

// Edge and queue records of the solo engine: (node | valence << 20, row
// start).  A record word never equals kSoloEmpty (valences stay below 4,096).
constexpr uint32_t kRecNodeBits = 20;
constexpr uint32_t kRecNodeMask = (1u << kRecNodeBits) - 1u;
__device__ __forceinline__ uint2 solo_rec(uint32_t node, uint32_t deg, uint32_t rs)
{
    return make_uint2(node | (deg << kRecNodeBits), rs);
}
__device__ __forceinline__ uint32_t rec_node(uint2 r) { return r.x & kRecNodeMask; }
__device__ __forceinline__ uint32_t rec_deg(uint2 r) { return r.x >> kRecNodeBits; }

// Requests the lines of e2[rs .. rs + deg) into L2 (at most four 128-byte
// lines: the rows the engine chunks are short), without waiting.
__device__ __forceinline__ void prefetch_row(const uint2* e2, uint32_t rs, uint32_t deg)
{
    if (deg == 0)
        return;
    const uintptr_t a = reinterpret_cast<uintptr_t>(e2 + rs) & ~(uintptr_t)127;
    const uintptr_t z = reinterpret_cast<uintptr_t>(e2 + rs + deg - 1) & ~(uintptr_t)127;
    for (uintptr_t l = a; l <= z && l < a + 4 * 128; l += 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(l));
}

template <int B, int EMAX>
struct Solo {
    static constexpr int MAXEPT = EMAX / B;
    static_assert(EMAX % B == 0 && (EMAX & (EMAX - 1)) == 0, "EMAX: a power of two, a multiple of B");
    static_assert(EMAX <= (1 << kEdgeBits), "a chunk edge index fits the dedup word");
    SoloSmem<B, EMAX>& s;
    const MatrixView& M;
    const uint2* e2;
    uint2* q;  // the queue: rec[] of the matrix as 8-byte records
    uint32_t* gvis;  // visited bitmap in global memory (matrices over kSoloMaxN nodes), or nullptr
    // queue record of position pf_base + (group thread), loaded by the last
    // form() for the chunk after it (its latency hides behind that chunk);
    // pf_base == kUnvisited: none
    uint32_t pf_base = kUnvisited;
    uint2 pf = make_uint2(0u, 0u);
    bool pf_ok = false;  // this thread holds a record in pf

    __device__ __forceinline__ bool visited(uint32_t c) const
    {
        const uint32_t w = gvis ? __ldcg(gvis + (c >> 5)) : s.vis[c >> 5];
        return (w >> (c & 31)) & 1u;
    }
    __device__ __forceinline__ void mark(uint32_t c)
    {
        atomicOr(gvis ? gvis + (c >> 5) : &s.vis[c >> 5], 1u << (c & 31));
    }

    // Loads the next chunk's parents from the queue records rec[p .. pend):
    // the longest prefix of at most B parents with at most EMAX edges (every
    // row fits one chunk: the engine is only used when the largest valence
    // is at most EMAX).  Returns the number of parents.
    __device__ uint32_t form(uint32_t p, uint32_t pend)
    {
        const uint32_t t = gtid<B>();
        uint32_t deg = 0;
        const bool have = p + t < pend;
        if (have) {
            const uint2 r = p == pf_base ? pf : __ldcg(q + p + t);
            deg = rec_deg(r);
            s.pn[t] = rec_node(r);
            s.prs[t] = r.y;
            s.pdeg[t] = deg;
        }
        uint32_t total;
        const uint32_t excl = block_scan1<B>(deg, total, s.scanbuf[0]);
        const uint32_t incl = excl + deg;
        const int fits = have && incl <= (uint32_t)EMAX;
        const int m = gsync_count<B>(fits);
        if (fits)
            s.soff[t] = excl;
        if (m > 0 && t == (uint32_t)(m - 1)) {
            s.soff[m] = incl;
            s.m = (uint32_t)m;
            s.Ec = incl;
        }
        // the next chunk of this level starts where this one ends: load its
        // records now
        const uint32_t nb = p + (uint32_t)m;
        pf_base = kUnvisited;
        pf_ok = false;
        if (nb < pend) {
            pf_base = nb;
            if (nb + t < pend) {
                pf = __ldcg(q + nb + t);
                pf_ok = true;
            }
        }
        gsync<B>();
        return (uint32_t)m;
    }

    // next_peripheral_start (engine.cuh) over this queue's 8-byte records:
    // among the last min(outnodes, n-1) positions, those on the last level;
    // the last of minimal valence.  One thread.
    __device__ uint32_t next_start(uint32_t outnodes, uint32_t last_start) const
    {
        const uint32_t n = M.n;
        uint32_t lo = n - min(outnodes, n - 1);
        lo = max(lo, max(last_start, 1u));
        uint32_t best = 0, bestdeg = kUnvisited;
        for (uint32_t pos = lo; pos < n; ++pos) {
            const uint2 r = __ldcg(q + pos);
            if (rec_deg(r) <= bestdeg) {
                bestdeg = rec_deg(r);
                best = rec_node(r);
            }
        }
        return best;
    }

    // The Q ranked children of the last chunk become the parents of the next.
    __device__ void form_from_children(uint32_t Q)
    {
        const uint32_t t = gtid<B>();
        uint32_t deg = 0;
        if (t < Q) {
            const uint32_t x = s.so_idx[t];
            deg = s.ch_dp[x] & kDegMask;
            s.pn[t] = s.ch_c[x];
            s.prs[t] = s.ch_rs[x];
            s.pdeg[t] = deg;
        }
        uint32_t total;
        const uint32_t excl = block_scan1<B>(deg, total, s.scanbuf[1]);
        if (t < Q)
            s.soff[t] = excl;
        if (t == 0) {
            s.soff[Q] = total;
            s.m = Q;
            s.Ec = total;
        }
        gsync<B>();
    }

    // One chunk: finds the children of parents [0, m), ranks them (sorted:
    // by valence, stable; else slot order), writes their queue records at
    // positions P.. and, with write_perm, the permutation, and marks them
    // visited.  Returns the number of children; qdeg = their valences' sum.
    // Four group barriers.  Ends without one: the next form() has barriers
    // before anyone touches this chunk's shared buffers again (the caller
    // adds one where the next chunk reads the queue records this one
    // wrote).  Leaves the dedup table and the parent counters clear.
    __device__ uint32_t step(uint32_t P, bool sorted, bool write_perm, bool reverse, uint32_t& qdeg)
    {
        const uint32_t t = gtid<B>(), lane = t & 31u, w = t >> 5;
        const uint32_t m = s.m, Ec = s.Ec;
        // warp w owns edges [w * 32 * MAXEPT, ...); lane l takes e = base +
        // l + 32 r, so that a warp reads consecutive records of a row
        const uint32_t base = w * 32u * MAXEPT;
        uint2 v[MAXEPT];
        uint32_t par[MAXEPT], slot[MAXEPT];
        bool cand[MAXEPT];
        // each edge's parent (the last j < m with soff[j] <= e: a binary
        // search of fixed depth, the edges' searches side by side; a parent
        // of valence 0 owns no edge), then the edge's record
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            const uint32_t e = base + lane + 32u * r;
            uint32_t lo = 0;
#pragma unroll
            for (uint32_t d = (uint32_t)B / 2u; d > 0; d >>= 1) {
                const uint32_t mid = lo + d;
                if (mid < m && s.soff[mid] <= e)
                    lo = mid;
            }
            par[r] = lo;
            v[r] = make_uint2(kSoloEmpty, 0u);
            if (e < Ec) {
                const uint64_t idx = (uint64_t)s.prs[lo] + (e - s.soff[lo]);
                if (PB_CHECK(M.res, idx < M.nnz, 601))
                    v[r] = __ldcg(e2 + idx);
            }
        }
        // the next chunk's rows into L2 while these records are in flight
        // (its queue records came with the last form())
        if (pf_ok)
            prefetch_row(e2, pf.y, rec_deg(pf));
        // the visited test after all the records are in flight
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r)
            cand[r] = v[r].x != kSoloEmpty && PB_CHECK(M.res, rec_node(v[r]) < M.n, 602) && !visited(rec_node(v[r]));
        // first edge to each unvisited node: (node, edge) in one word, so
        // that the word's minimum under a fixed node is the first edge; the
        // node's slot by linear probing (at most EMAX distinct nodes in 2
        // EMAX slots: a free slot is always found)
        constexpr uint32_t mask = (uint32_t)SoloSmem<B, EMAX>::H - 1u;
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            slot[r] = 0;
            if (cand[r]) {
                const uint32_t c = rec_node(v[r]);
                const uint32_t key = (c << kEdgeBits) | (base + lane + 32u * r);
                uint32_t h = (c * 2654435761u) & mask;
                while (true) {
                    const uint32_t old = atomicCAS(&s.tab[h], kSoloEmpty, key);
                    if (old == kSoloEmpty)
                        break;
                    if ((old >> kEdgeBits) == c) {
                        atomicMin(&s.tab[h], key);
                        break;
                    }
                    h = (h + 1u) & mask;
                }
                slot[r] = h;
            }
        }
        gsync<B>();
        // the winners, compacted in edge order: per warp by ballot, then the
        // warps' counts
        uint32_t cnt = 0, posr[MAXEPT], dsum = 0;
        bool win[MAXEPT];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            win[r] = cand[r] && s.tab[slot[r]] == ((rec_node(v[r]) << kEdgeBits) | (base + lane + 32u * r));
            const uint32_t bal = __ballot_sync(kFull, win[r]);
            posr[r] = cnt + __popc(bal & ((1u << lane) - 1u));
            cnt += __popc(bal);
            dsum += win[r] ? rec_deg(v[r]) : 0u;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            dsum += __shfl_xor_sync(kFull, dsum, o);
        if (lane == 0) {
            s.wcnt[w] = cnt;
            s.wdeg[w] = dsum;
        }
        gsync<B>();
        uint32_t wbase = 0, Q = 0;
        qdeg = 0;
#pragma unroll
        for (int i = 0; i < SoloSmem<B, EMAX>::W; ++i) {
            const uint32_t c = s.wcnt[i];
            wbase += (uint32_t)i < w ? c : 0u;
            Q += c;
            qdeg += s.wdeg[i];
        }
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            if (win[r]) {
                const uint32_t x = wbase + posr[r];
                const uint32_t j = par[r];
                s.ch_c[x] = rec_node(v[r]);
                s.ch_rs[x] = v[r].y;
                s.ch_dp[x] = rec_deg(v[r]) | (j << kParShift);
                atomicAdd(&s.cc[j], 1u);
                atomicMin(&s.cs[j], x);
            }
        }
        gsync<B>();
        // rank inside each parent's run: (valence, position) when sorted
        for (uint32_t x = t; x < Q; x += B) {
            const uint32_t j = s.ch_dp[x] >> kParShift;
            const uint32_t st = s.cs[j], len = s.cc[j];
            uint32_t rank = x - st;
            if (sorted && len > 1) {
                const uint32_t dx = s.ch_dp[x] & kDegMask;
                rank = 0;
                for (uint32_t y = st; y < st + len; ++y) {
                    const uint32_t dy = s.ch_dp[y] & kDegMask;
                    rank += (dy < dx) || (dy == dx && y < x);
                }
            }
            s.so_idx[st + rank] = x;
        }
        gsync<B>();
        // place: queue records, the permutation, the visited marks
        for (uint32_t i = t; i < Q; i += B) {
            const uint32_t x = s.so_idx[i];
            const uint32_t pos = P + i;
            if (PB_CHECK(M.res, pos < M.n, 603)) {
                __stcg(q + pos, solo_rec(s.ch_c[x], s.ch_dp[x] & kDegMask, s.ch_rs[x]));
                if (write_perm)
                    M.perm[reverse ? M.n - 1 - pos : pos] = s.ch_c[x];
            }
            mark(s.ch_c[x]);
        }
        // the table slots and parent counters this chunk used, clear again
        // (their last readers are behind the barriers above)
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r)
            if (cand[r])
                s.tab[slot[r]] = kSoloEmpty;
        for (uint32_t j = t; j < m; j += B) {
            s.cs[j] = kSoloEmpty;
            s.cc[j] = 0;
        }
        return Q;
    }
};

// The per-edge neighbour records of a matrix (e2[k] = solo_rec(c, rp[c+1] -
// rp[c], rp[c]) for c = ci[k]) by one group, coalesced.  A column out of
// range gets an empty record (the CSR check reports it); a valence of 4,096
// or more does not fit a record, but such a matrix never reaches the solo
// engine (its rows exceed every chunk).
template <int B>
__device__ void solo_build_edges(const MatrixView& M, uint2* e2)
{
    bool bad = false;
#pragma unroll 8
    for (uint32_t k = gtid<B>(); k < M.nnz; k += B) {
        const uint32_t c = ld_ro(M.ci + k);
        uint2 r = make_uint2(kSoloEmpty, 0u);
        if (c < M.n) {
            const uint32_t a = ld_ro(M.rp + c), b = ld_ro(M.rp + c + 1);
            r = solo_rec(c, b - a, a);
        } else {
            bad = true;
        }
        __stcg(e2 + k, r);
    }
    // the CSR check's column test (validate_rows leaves it to this pass)
    if (bad)
        set_status(M.res, kErrArg, 200);
}

// One ordered BFS pass from `start` by one solo group.  Fills rec[0 ..
// placed); returns the level count and the first position of the last level.
template <int B, int EMAX>
__device__ void solo_pass(Solo<B, EMAX>& so, uint32_t start, bool sorted, bool write_perm, bool reverse,
                          uint32_t& placed, uint32_t& nlevels, uint32_t& last_start)
{
    SoloSmem<B, EMAX>& s = so.s;
    const MatrixView& M = so.M;
    const uint32_t t = gtid<B>();
    const uint32_t words = (M.n + 31u) / 32u;
    uint32_t* vis = so.gvis ? so.gvis : s.vis;
    for (uint32_t i = t; i < words; i += B)
        vis[i] = 0u;
    // the dedup table and the parent counters start clear (each chunk
    // leaves them so)
    for (uint32_t i = t; i < (uint32_t)SoloSmem<B, EMAX>::H; i += B)
        s.tab[i] = kSoloEmpty;
    s.cs[t] = kSoloEmpty;
    s.cc[t] = 0;
    gsync<B>();
    if (t == 0) {
        const uint32_t a = ld_ro(M.rp + start), b = ld_ro(M.rp + start + 1);
        __stcg(so.q, solo_rec(start, b - a, a));
        if (write_perm)
            M.perm[reverse ? M.n - 1 : 0] = start;
        so.mark(start);
    }
    gsync<B>();
    uint32_t head = 0, tail = 1, lvl_end = 1, L = 0, lstart = 0;
    bool carry = false;  // the chunk's parents are the last chunk's children, still in shared memory
    uint32_t q = 0;
    while (head < tail) {
        if (head == lvl_end) {
            L += 1;
            lstart = head;
            lvl_end = tail;
        }
        uint32_t m;
        if (carry) {
            so.form_from_children(q);
            m = q;
        } else {
            m = so.form(head, lvl_end);
        }
        // a whole level in one chunk whose children fit one chunk: they are
        // the next chunk's parents
        const bool whole_level = head + m == lvl_end && head + m == tail;
        uint32_t qdeg = 0;
        q = so.step(tail, sorted, write_perm, reverse, qdeg);
        head += m;
        tail += q;
        carry = whole_level && q > 0 && q <= (uint32_t)B && qdeg <= (uint32_t)EMAX;
        // a chunk that ends its level hands its children over through the
        // queue records it has just written (unless they stay in shared
        // memory): every thread's records must be in before the next chunk
        // reads them.  Otherwise the next chunk's parents were written by
        // earlier chunks, behind barriers already passed.
        if (head == lvl_end && !carry)
            gsync<B>();
        if (tail > M.n) {  // cannot happen on a valid run
            if (t == 0)
                set_status(M.res, kErrCheck, 604);
            break;
        }
    }
    placed = tail;
    nlevels = L + 1;
    last_start = lstart;
}

// Sets bits of *p under a predicate, without a branch around the atomic (eight
// in a row are in flight together); the old word, or all ones when off.
template <bool GV>
__device__ __forceinline__ uint32_t or_if(uint32_t* p, uint32_t v, bool on)
{
    uint32_t old = 0xFFFFFFFFu;
    if (GV)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p atom.global.or.b32 %0, [%1], %2;\n\t}"
                     : "+r"(old)
                     : "l"(__cvta_generic_to_global(p)), "r"(v), "r"((uint32_t)on)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
                     : "+r"(old)
                     : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v), "r"((uint32_t)on)
                     : "memory");
    return old;
}

// One breadth-first pass from `start`, unordered inside a level: what a
// start-search pass needs when its order does not matter (see solo_reorder).
// Test-and-set of the visited bit is the whole dedup, and the group meets
// once a level: each warp takes up to 32 parents at a time, as many as have
// 256 entries between them, deals their entries out to its lanes in order
// (entry e = lane + 32 u; ent[e] = parent lane << 5 | slot names its row), and
// appends the children it marked.  A row of more than kLevelRow entries goes
// alone.
// Returns the last level's records in s.lbuf[(nlevels - 1) & 1] (those past
// CAP in the queue).  GV: the visited bitmap is in global memory.
template <bool GV, int B, int EMAX>
__device__ void solo_level_pass(Solo<B, EMAX>& so, uint32_t start, uint32_t& placed, uint32_t& nlevels,
                                uint32_t& last_start)
{
    using S = SoloSmem<B, EMAX>;
    constexpr uint32_t CAP = (uint32_t)S::CAP;
    constexpr int U = 8;
    S& s = so.s;
    const MatrixView& M = so.M;
    const uint32_t n = M.n;
    const uint2* const e2 = so.e2;
    uint2* const q = so.q;
    uint32_t* const vis = GV ? so.gvis : s.vis;
    const uint32_t t = gtid<B>(), lane = t & 31u, w = t >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t words = (n + 31u) / 32u;
    for (uint32_t i = t; i < words; i += B)
        vis[i] = 0u;
    gsync<B>();
    if (t == 0) {
        const uint32_t a = ld_ro(M.rp + start), b = ld_ro(M.rp + start + 1);
        s.lbuf[0][0] = solo_rec(start, b - a, a);
        so.mark(start);
        s.lcnt[0] = 0;
        s.lcnt[1] = 0;
        s.lcnt[2] = 0;
    }
    gsync<B>();
    uint32_t head = 0, lvl_end = 1, L = 0, slot = 0;
    while (true) {
        const uint2* cur = s.lbuf[L & 1u];
        uint2* nxt = s.lbuf[(L & 1u) ^ 1u];
        const uint32_t width = lvl_end - head;
        // the warps' shares of the level: consecutive parents
        const uint32_t share = (width + B / 32 - 1) / (B / 32);
        const uint32_t bend = min(width, (w + 1) * share);
        for (uint32_t b = w * share; b < bend;) {
            const uint32_t i = b + lane;
            uint2 r = make_uint2(0u, 0u);
            if (i < bend)
                r = i < CAP ? cur[i] : __ldcg(q + head + i);
            const uint32_t deg = rec_deg(r);
            uint32_t x = deg;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                x += lane >= o ? y : 0u;
            }
            // the parents taken: the longest prefix of rows of at most kLevelRow
            // entries, 32 U between them; or one longer row
            const uint32_t bad = ~__ballot_sync(kFull, i < bend && deg <= kLevelRow && x <= 32u * U);
            const uint32_t m = bad ? (uint32_t)__ffs(bad) - 1u : 32u;
            const uint32_t took = max(m, 1u);
            const uint32_t soff = x - deg, shift = r.y - soff;
            const uint32_t E = __shfl_sync(kFull, x, (int)took - 1);
            __syncwarp();
            if (lane < m)
                for (uint32_t k = 0; k < deg; ++k)
                    s.ent[w][soff + k] = (uint16_t)lane;
            __syncwarp();
            for (uint32_t e0 = 0; e0 < E; e0 += 32u * U) {
                uint2 v[U];
                uint32_t cand = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t e = e0 + 32u * u + lane;
                    v[u] = make_uint2(0u, 0u);
                    if (e0 + 32u * u < E) {
                        const uint32_t j = m != 0 ? (uint32_t)s.ent[w][32u * u + lane] : 0u;
                        const uint32_t idx = __shfl_sync(kFull, shift, (int)j) + e;
                        const bool in = e < E && PB_CHECK(M.res, idx < M.nnz, 611);
                        v[u] = __ldcg(e2 + (in ? idx : 0u));
                        cand |= in ? 1u << u : 0u;
                    }
                }
                uint32_t old[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t c = rec_node(v[u]);
                    const uint32_t word = GV ? __ldcg(vis + (c >> 5)) : vis[c >> 5];
                    if ((word >> (c & 31u)) & 1u)
                        cand &= ~(1u << u);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t c = rec_node(v[u]), bit = 1u << (c & 31u);
                    old[u] = or_if<GV>(vis + (c >> 5), bit, (cand >> u) & 1u) & bit;
                }
                // the children this warp marked, behind those of the others
                uint32_t bal[U], tot = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    bal[u] = __ballot_sync(kFull, old[u] == 0u);
                    tot += __popc(bal[u]);
                }
                if (tot != 0) {
                    uint32_t at = 0;
                    if (lane == 0)
                        at = atomicAdd(&s.lcnt[slot], tot);
                    at = __shfl_sync(kFull, at, 0);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t p = at + __popc(bal[u] & lt);
                        if (old[u] == 0u) {
                            if (p < CAP)
                                nxt[p] = v[u];
                            else if (PB_CHECK(M.res, lvl_end + p < n, 612))
                                __stcg(q + lvl_end + p, v[u]);
                        }
                        at += __popc(bal[u]);
                    }
                }
            }
            b += took;
        }
        gsync<B>();
        const uint32_t cnt = s.lcnt[slot];
        slot = slot == 2 ? 0 : slot + 1;
        // the counter of the level after next: last read before this barrier
        if (t == 0)
            s.lcnt[slot == 2 ? 0 : slot + 1] = 0;
        if (cnt == 0)
            break;
        head = lvl_end;
        lvl_end += cnt;
        ++L;
    }
    gsync<B>();
    placed = lvl_end;
    nlevels = L + 1;
    last_start = head;
}

// Full reorder of one matrix by one solo group: start search
// (simple_peripheral.cpp:92-141), the sorted pass, reverse, bandwidth.
// e2: the matrix's edge records; inv: n words for the inverse permutation;
// gvis: ceil(n / 32) words for the visited bitmap when n > kSoloMaxN (else
// nullptr: the bitmap is in shared memory).
template <int B, int EMAX>
__device__ void solo_reorder(SoloSmem<B, EMAX>& s, const MatrixView& M, const uint2* e2, uint32_t* inv,
                             uint32_t* gvis, const Options& opt)
{
    const uint32_t t = gtid<B>();
    const uint32_t n = M.n;
    if (t == 0)
        M.res->t_begin = globaltimer();
    Solo<B, EMAX> so{s, M, e2, reinterpret_cast<uint2*>(M.rec), gvis};
    uint32_t start = opt.start;
    if (start != kUnvisited && start >= n) {
        if (t == 0)
            set_status(M.res, kErrArg, 2);
        return;
    }
    uint32_t passes = 0, ecc = 0, placed = 0, nlevels = 0, last_start = 0;
    bool searching = start == kUnvisited && n > 1;
    if (n == 1) {
        passes = start == kUnvisited ? 1 : 0;
        start = 0;
    } else if (searching) {
        start = n / 2;
    }
    uint32_t lastdist = 0;
    bool repeat = false;  // this pass repeats the last one in discovery order
    const uint32_t maxdeg = __ldcg(&M.res->maxdeg);
    bool fifo = long_rows(maxdeg) || wide_stencil(n, M.nnz, maxdeg);  // this search pass runs in discovery order at once
    while (true) {
        if (!searching && opt.mode == kModeStartOnly)
            break;
        if (searching && !repeat)
            ++passes;
        // a start-search pass has to deliver its level count and the next
        // start, and that start -- the last node of minimal valence among the
        // last outnodes discovered, on the last level
        // (simple_peripheral.cpp:118-127) -- does not depend on the order
        // when the last level has at most outnodes nodes and one of them
        // alone has the minimal valence: the search runs unordered and is
        // only repeated in order where that fails (never on 5- and 7-point
        // grids; a third of the passes of random geometric graphs; always on
        // wider stencils, which begin in order; a second pass after one that
        // needed it is ordered at once, and so is every one of a matrix with
        // long rows, see long_rows).  From the third pass on,
        // which usually confirms the eccentricity, the pass of a sparse
        // matrix is the sorted one itself: the result if it does (444 at once
        // of 100,000 nodes: 2-D grids 12.3 ms against 14.1 with a third
        // unordered pass, 3-D grids 15.3 / 16.6; but random geometric graphs
        // of 11 entries a row, whose third pass confirms less often and whose
        // sorted pass costs two unordered ones, 38.0 / 35.0).
        const bool sorted = !searching || (!repeat && passes >= 3 && opt.mode != kModeStartOnly && M.nnz <= 8ull * n);
        const bool ordered = !sorted && (repeat || fifo);
        if (sorted)
            solo_pass<B, EMAX>(so, start, true, true, opt.reverse != 0, placed, nlevels, last_start);
        else if (ordered)
            solo_pass<B, EMAX>(so, start, false, false, false, placed, nlevels, last_start);
        else if (so.gvis)
            solo_level_pass<true, B, EMAX>(so, start, placed, nlevels, last_start);
        else
            solo_level_pass<false, B, EMAX>(so, start, placed, nlevels, last_start);
        if (read_status(M.res) != 0)
            return;
        if (!searching)
            break;
        if (placed != n) {
            if (t == 0)
                set_status(M.res, kErrDisconnected, 0);
            return;
        }
        const uint32_t dist = nlevels - 1;
        if (dist == lastdist && !repeat) {
            ecc = dist;
            searching = false;
            if (sorted)
                break;  // confirmed by the sorted pass: the result
            continue;   // the sorted pass from the same start comes next
        }
        const uint32_t width = n - last_start;
        bool known = false;
        if (width <= min(opt.outnodes, n - 1) && width <= (uint32_t)SoloSmem<B, EMAX>::CAP) {
            if (t < 32) {
                uint32_t d = kUnvisited, v = 0, same = 0;
                for (uint32_t i = t; i < width; i += 32) {
                    const uint2 r = sorted || ordered ? __ldcg(so.q + last_start + i) : s.lbuf[(nlevels - 1) & 1u][i];
                    const uint32_t di = rec_deg(r);
                    same = di < d ? 1u : same + (di == d ? 1u : 0u);
                    if (di < d) {
                        d = di;
                        v = rec_node(r);
                    }
                }
                const uint32_t dm = __reduce_min_sync(kFull, d);
                const uint32_t count = __reduce_add_sync(kFull, d == dm ? same : 0u);
                v = __shfl_sync(kFull, v, __ffs(__ballot_sync(kFull, d == dm)) - 1);
                if (t == 0) {
                    s.bcast[0] = v;
                    s.bcast[1] = count;
                }
            }
            gsync<B>();
            known = s.bcast[1] == 1u;
        }
        gsync<B>();
        if (!known && !ordered) {
            repeat = true;
            continue;
        }
        if (ordered) {
            if (t == 0)
                s.bcast[0] = so.next_start(opt.outnodes, last_start);
            gsync<B>();
        }
        fifo = long_rows(maxdeg) || (!known && passes < 2);
        repeat = false;
        start = s.bcast[0];
        gsync<B>();
        lastdist = dist;
        if (passes > n) {
            if (t == 0)
                set_status(M.res, kErrCheck, 3);
            return;
        }
    }
    if (opt.mode == kModeStartOnly) {
        if (t == 0) {
            M.res->start = start;
            M.res->passes = passes;
            M.res->ecc = ecc;
            M.res->placed = n;
        }
        return;
    }
    if (placed != n) {
        if (t == 0) {
            set_status(M.res, kErrDisconnected, 1);
            M.res->placed = placed;
        }
        return;
    }
    if (opt.want_bw) {
        // the inverse permutation (four records in flight per thread)
        for (uint32_t pos = t; pos < n; pos += 4 * B) {
            uint2 r[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                r[u] = pos + u * B < n ? __ldcg(so.q + pos + u * B) : make_uint2(0u, 0u);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (pos + u * B < n)
                    inv[rec_node(r[u])] = pos + u * B;
        }
        gsync<B>();
        unsigned long long bw = 0, bw0 = 0, plo = 0, phi = 0;
        for (uint32_t i = t; i < n; i += B) {
            const uint32_t a = ld_ro(M.rp + i), e = ld_ro(M.rp + i + 1);
            if (a == e)
                continue;
            const uint32_t me = __ldcg(inv + i);
            uint32_t mnr = kUnvisited, mxr = 0, c0 = 0, c1 = 0;
            // the row's columns four at a time, then their positions (the
            // loads of a group side by side)
            for (uint32_t k = a; k < e; k += 4) {
                uint32_t c[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    c[u] = k + u < e ? ld_ro(M.ci + k + u) : kUnvisited;
                if (k == a)
                    c0 = c[0];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c[u] != kUnvisited) {
                        const uint32_t p = __ldcg(inv + c[u]);
                        mnr = min(mnr, p);
                        mxr = max(mxr, p);
                        c1 = c[u];
                    }
            }
            // computeBandwidth (main.cpp:143-184): max(row - min, max - row)
            const unsigned long long b1 = me >= mnr ? (unsigned long long)(me - mnr) : 0ull;
            const unsigned long long b2 = mxr >= me ? (unsigned long long)(mxr - me) : 0ull;
            bw = max(bw, max(b1, b2));
            plo += b1;
            phi += b2;
            // initial bandwidth: first / last stored column (main.cpp:114-129)
            const unsigned long long i0 = i >= c0 ? i - c0 : 0, i1 = c1 >= i ? c1 - i : 0;
            bw0 = max(bw0, max(i0, i1));
        }
        bw = block_reduce_max<B, unsigned long long>(bw, s.tmp64);
        bw0 = block_reduce_max<B, unsigned long long>(bw0, s.tmp64);
        block_reduce_sum2<B>(plo, phi, s.tmp64);
        if (t == 0) {
            M.res->bandwidth = bw;
            M.res->initial_bw = bw0;
            M.res->profile_lo = plo;
            M.res->profile_hi = phi;
        }
    }
    if (t == 0) {
        M.res->start = start;
        M.res->passes = passes;
        M.res->ecc = ecc;
        M.res->levels = nlevels;
        M.res->placed = placed;
        M.res->t_end = globaltimer();
    }
}

}  // namespace pbrcm
