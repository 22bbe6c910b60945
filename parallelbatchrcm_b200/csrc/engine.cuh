// engine.cuh -- device core of the B200 Cuthill-McKee engine (sm_100a).
//
// What it computes
//   The serial stable Cuthill-McKee order of the reference
//   (src/rcm_cpu.cpp:57-104): FIFO over positions; the parent at position i
//   appends its still-unvisited neighbours, stable-sorted by valence (row
//   length).  The reference's GPU_BATCH reaches it with a chain of
//   speculative batches (include/device/batchWorker.cuh); this engine reaches
//   it level by level, every CTA of a team working on one BFS level at a time.
//
// The claim key
//   Within one BFS pass the edges are numbered in queue order: edge (position
//   i, slot k) has id ebase(i) + k, where ebase(i) = sum of the valences at
//   positions < i.  Pass p owns the key range [p*kspan, p*kspan + nnz + 1]
//   (kspan = nnz + 2); edge id e maps to key base_p - 1 - e with
//   base_p = p*kspan + nnz + 1 (the start node takes base_p itself).  Every
//   frontier edge does atomicMax(node[child].claim, key).  Once a level's
//   claims are done, a node's claim is the key of the FIRST edge that reaches
//   it in queue order -- exactly the (parent, slot) that discovers it in the
//   serial algorithm, duplicate entries included -- so an edge is a child
//   edge iff node[col].claim == its key: a purely local test.  Keys of later
//   levels are smaller, so claiming for the next level never disturbs a node
//   already placed, and keys of a later pass are larger than every key of an
//   earlier one, so passes need no reset.  The key is an order-preserving
//   (parent position, slot) code; the reference's batch code
//   (batchId << 11 | offset, batchWorker.cuh:574-586) plays the same role for
//   its batches.
//
// One level (frontier = positions [a, b), edge ids [Ka, Kb))
//   collect: each CTA takes a contiguous range of parents, splits it into
//            chunks (<= B parents, <= EMAX edges), reads one node entry per
//            edge (claim + row start + valence in one 16-byte load), keeps
//            the child edges in (parent, slot) order and ranks every
//            parent's children by (valence, slot).
//   place:   children get positions b + (children of earlier parents) + rank
//            and edge bases Kb + (valences of earlier children): records to
//            rec[], the node to perm[].
//   claim:   the placed children claim their own edges for the next level.
//   A grid team publishes per-CTA (children, valence) totals with a
//   level-tagged all-gather, places, and meets at a barrier; while every
//   CTA's children fit a chunk each expands its own.  Levels with a small
//   frontier run on CTA 0 alone ("solo") with block barriers only; the
//   other CTAs park at a gate until CTA 0 hands a large level back.  Parents
//   with more than EMAX edges ("hubs") are collected and radix-sorted in
//   global scratch by one CTA.
//
// Start-search passes whose order does not matter (reorder_matrix) run as
// level_pass instead: a node's first claim of the pass places it.
//
// Every wait is bounded by %globaltimer and reports PBRCM_ERR_TIMEOUT.
// With PBRCM_CHECKS defined, every global index is range-checked and a
// failure records PBRCM_ERR_CHECK and skips the access.
#pragma once

#include <cstdint>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "search.h"
#include "types.h"

namespace pbrcm {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void st_release(unsigned int* p, unsigned int v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_ro(const uint32_t* p) { return __ldg(p); }

__device__ __forceinline__ uint4 ld_node(const NodeEntry* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

__device__ __forceinline__ uint32_t* claim_ptr(const MatrixView& M, uint32_t v) { return &M.node[v].claim; }

__device__ __forceinline__ void set_status(DevResult* r, uint32_t code, uint32_t where)
{
    if (atomicCAS(&r->status, 0u, code) == 0u)
        r->where = where;
}

__device__ __forceinline__ uint32_t read_status(const DevResult* r)
{
    return *reinterpret_cast<const volatile uint32_t*>(&r->status);
}

#ifdef PBRCM_CHECKS
#define PB_CHECK(res, cond, where) ((cond) ? true : (set_status((res), kErrCheck, (where)), false))
#else
#define PB_CHECK(res, cond, where) true
#endif

// ---------------------------------------------------------------------------
// Thread groups.  One engine instance runs on a group of B consecutive
// threads of a CTA: the whole CTA, or one of blockDim.x / B equal slices, so
// that one CTA can reorder several matrices at once.  Group g synchronises on
// named barrier 1 + g (barrier 0 stays the CTA-wide __syncthreads); every
// engine barrier is reached by all B threads of the group, never by a
// diverged subset.
// ---------------------------------------------------------------------------
template <int B>
__device__ __forceinline__ uint32_t gtid()
{
    static_assert(B >= 32 && B <= 1024 && (B & (B - 1)) == 0, "groups are a power-of-two number of warps");
    return threadIdx.x & (B - 1);
}

template <int B>
__device__ __forceinline__ uint32_t gbar_id()
{
    return 1u + threadIdx.x / B;
}

template <int B>
__device__ __forceinline__ void gsync()
{
    asm volatile("bar.sync %0, %1;" ::"r"(gbar_id<B>()), "n"(B) : "memory");
}

// Group barrier that also counts the threads whose predicate holds.
template <int B>
__device__ __forceinline__ int gsync_count(bool pred)
{
    int r;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.popc.u32 %0, %2, %3, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(gbar_id<B>()), "n"(B)
        : "memory");
    return r;
}

// Barrier of a group given at run time (id, threads).
__device__ __forceinline__ void gsync_n(uint32_t id, uint32_t nthr)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthr) : "memory");
}

// Block-wide exclusive scan of one value per thread (T = uint32_t or
// unsigned long long).  `tmp` holds B/32 + 1 entries.  Ends with a barrier,
// so `tmp` can be reused right away.
template <int B, typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T& total, T* tmp)
{
    constexpr int W = B / 32;
    const int lane = threadIdx.x & 31, w = gtid<B>() >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(kFull, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        tmp[w] = x;
    gsync<B>();
    if (w == 0) {
        T s = lane < W ? tmp[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(kFull, s, o);
            if (lane >= o)
                s += y;
        }
        if (lane < W)
            tmp[lane] = s;
    }
    gsync<B>();
    T r = (w ? tmp[w - 1] : T(0)) + x - v;
    total = tmp[W - 1];
    gsync<B>();
    return r;
}

// Block-wide exclusive scan with a single barrier.  `buf` (B/32 entries) must
// belong to this call site alone: it is read after the barrier and not
// cleared, so the next write to it must come after another block barrier.
template <int B>
__device__ __forceinline__ uint32_t block_scan1(uint32_t v, uint32_t& total, uint32_t* buf)
{
    constexpr int W = B / 32;
    const int lane = threadIdx.x & 31, w = gtid<B>() >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        buf[w] = x;
    gsync<B>();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const uint32_t b = buf[i];
        before += i < w ? b : 0u;
        all += b;
    }
    total = all;
    return before + x - v;
}

template <int B, typename T>
__device__ __forceinline__ T block_reduce_max(T v, T* tmp)
{
    constexpr int W = B / 32;
    const int lane = threadIdx.x & 31, w = gtid<B>() >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T y = __shfl_xor_sync(kFull, v, o);
        v = v > y ? v : y;
    }
    if (lane == 0)
        tmp[w] = v;
    gsync<B>();
    T r = tmp[0];
    for (int i = 1; i < W; ++i)
        r = r > tmp[i] ? r : tmp[i];
    gsync<B>();
    return r;
}

template <int B, typename T>
__device__ __forceinline__ T block_reduce_sum(T v, T* tmp)
{
    constexpr int W = B / 32;
    const int lane = threadIdx.x & 31, w = gtid<B>() >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0)
        tmp[w] = v;
    gsync<B>();
    T r = 0;
    for (int i = 0; i < W; ++i)
        r += tmp[i];
    gsync<B>();
    return r;
}

// Two sums at once (tmp holds 2 * (B/32) entries).
template <int B>
__device__ __forceinline__ void block_reduce_sum2(unsigned long long& a, unsigned long long& b,
                                                  unsigned long long* tmp)
{
    constexpr int W = B / 32;
    const int lane = threadIdx.x & 31, w = gtid<B>() >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(kFull, a, o);
        b += __shfl_xor_sync(kFull, b, o);
    }
    if (lane == 0) {
        tmp[w] = a;
        tmp[W + w] = b;
    }
    gsync<B>();
    unsigned long long ra = 0, rb = 0;
    for (int i = 0; i < W; ++i) {
        ra += tmp[i];
        rb += tmp[W + i];
    }
    a = ra;
    b = rb;
    gsync<B>();
}

// Level state of one pass, the same in every CTA of a team.
constexpr int kTeamShared = 15;  // group-shared ints a team needs (Team::sh)

struct LevelState {
    uint32_t a, b;     // frontier positions [a, b)
    uint32_t Ka, Kb;   // edge ids of the frontier [Ka, Kb)
    uint32_t L;        // level index of the frontier
    uint32_t last_start;
};

// ---------------------------------------------------------------------------
// Team: one CTA, or all CTAs of a cooperative launch (global-memory
// barriers, all-gather and gate, every wait bounded by wait_ns).
// ---------------------------------------------------------------------------
struct Team {
    static constexpr bool kGrid = true;
    GridSync* gs;        // nullptr for a one-CTA team
    unsigned int* flags; // one barrier flag word per CTA (+ phantom), zeroed per launch
    uint32_t size;       // CTAs in the team
    uint32_t rank;       // this CTA
    uint32_t expected;   // CTAs a barrier waits for (size + phantom)
    uint32_t target;     // barriers passed so far
    uint32_t mode;       // barrier implementation (see sync)
    uint32_t epoch;      // gate epochs seen
    uint32_t word = 0;   // barriers of unordered levels passed (level_wait)
    unsigned long long wait_ns;
    DevResult* res;
    // the thread group running this CTA's part (see gtid): its thread 0 is
    // tid == 0, its barrier is (bar, nthr); sh holds kTeamShared ints of
    // group-shared scratch, one slot per function so that one function's
    // result can still be read while the next one writes its own
    uint32_t tid, bar, nthr;
    int* sh;

    __device__ __forceinline__ void gbar() const { gsync_n(bar, nthr); }

    // Group-uniform "keep going?" after a group barrier.
    __device__ bool block_ok()
    {
        gbar();
        if (tid == 0)
            sh[0] = read_status(res) == 0;
        gbar();
        return sh[0] != 0;
    }

    // Team barrier, two implementations (Options::barrier):
    //  0  monotonic counter: one release-add per CTA on gs->count, thread 0
    //     acquire-polls until it reaches (barriers so far) x (team size);
    //  1  flag array: every CTA release-stores the barrier's sequence number
    //     into its own flag word; threads i < expected poll flag i with
    //     relaxed loads, then fence (acquire pattern).
    // Returns false if the team must stop (an error anywhere, or the wait
    // ran out).
    __device__ bool sync(uint32_t where)
    {
        if (gs == nullptr)
            return block_ok();
        target += 1;
        // this barrier's verdict, in one of two slots by parity (the next
        // barrier resets the other one, so no thread reading this one meets
        // the reset and no barrier is needed after the read)
        int& s_ok = sh[(target & 1u) ? 1 : 10];
        if (tid == 0)
            s_ok = 1;
        gbar();
        if (mode == 0) {
            if (tid == 0) {
                red_release_add(&gs->count, 1u);
                // the status read goes out with the polls, not after them:
                // an error posted before this CTA arrived is seen here, one
                // posted later at the next barrier or bounded wait (each
                // checks the status)
                const uint32_t st0 = read_status(res);
                const uint32_t goal = target * expected;
                unsigned long long t0 = 0;
                uint32_t spins = 0;
                while ((int)(ld_acquire(&gs->count) - goal) < 0) {
                    if ((++spins & 31u) == 0 && !wait_check(t0, where)) {
                        s_ok = 0;
                        break;
                    }
                    if (spins > 2048)
                        __nanosleep(128);
                }
                if (st0 != 0)
                    s_ok = 0;
            }
            gbar();
            return s_ok != 0;
        } else {
            if (tid == 0)
                st_release(flags + rank, target);
            for (uint32_t i = tid; i < expected; i += nthr) {
                unsigned long long t0 = 0;
                uint32_t spins = 0;
                while ((int)(*reinterpret_cast<volatile unsigned int*>(flags + i) - target) < 0) {
                    if ((++spins & 31u) == 0 && !wait_check(t0, where)) {
                        s_ok = 0;
                        break;
                    }
                    if (spins > 256)
                        __nanosleep(64);
                }
                __threadfence();
            }
        }
        gbar();
        const int ok = s_ok && read_status(res) == 0;
        gbar();
        return ok != 0;
    }

    // The barrier of an unordered level (level_pass), in two halves so that
    // work goes on in between: one 64-bit word gathers the arrivals, the
    // requests for a new split and the level's totals (fields of 8, 8, 24 and
    // 24 bits: at most 255 CTAs of at most EMAX nodes and entries each; more
    // than that comes with a request).  The words turn by threes in gs->word,
    // each cleared two barriers before its use.
    __device__ __forceinline__ void level_arrive(uint32_t cnt, uint32_t esum, bool ask)
    {
        if (tid == 0) {
            const unsigned long long v = 1ull << 56 | (unsigned long long)(ask ? 1u : 0u) << 48 |
                                         (unsigned long long)(ask ? 0u : esum) << 24 | (ask ? 0u : cnt);
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&gs->word[word % 3u]), "l"(v) : "memory");
        }
    }
    // keep: nobody asked for a new split.  False: the team must stop.
    __device__ bool level_wait(uint32_t where, uint32_t& all_cnt, uint32_t& all_esum, bool& keep)
    {
        int& s_ok = sh[(word & 1u) ? 1 : 10];
        gbar();
        if (tid == 0) {
            const uint32_t st0 = read_status(res);
            unsigned long long t0 = 0, got;
            uint32_t spins = 0;
            int ok = 1;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(got) : "l"(&gs->word[word % 3u]) : "memory");
                if ((uint32_t)(got >> 56) >= expected)
                    break;
                if ((++spins & 31u) == 0 && !wait_check(t0, where)) {
                    ok = 0;
                    break;
                }
                if (spins > 2048)
                    __nanosleep(128);
            }
            // the word after next: everyone is past its last use
            if (rank == 0)
                st_relaxed64(&gs->word[(word + 2u) % 3u], 0ull);
            sh[11] = (int)(uint32_t)((got >> 48) & 0xFFu);
            sh[12] = (int)(uint32_t)((got >> 24) & 0xFFFFFFu);
            sh[13] = (int)(uint32_t)(got & 0xFFFFFFu);
            s_ok = ok && st0 == 0;
        }
        gbar();
        ++word;
        keep = sh[11] == 0;
        all_esum = (uint32_t)sh[12];
        all_cnt = (uint32_t)sh[13];
        return s_ok != 0;
    }

    // Shared by every bounded wait: false once an error is posted or the
    // wait has run longer than wait_ns (then it posts PBRCM_ERR_TIMEOUT).
    __device__ __forceinline__ bool wait_check(unsigned long long& t0, uint32_t where)
    {
        if (read_status(res) != 0)
            return false;
        const unsigned long long now = globaltimer();
        if (t0 == 0) {
            t0 = now;
        } else if (now - t0 > wait_ns) {
            set_status(res, kErrTimeout, where);
            return false;
        }
        return true;
    }

    // Heartbeat of CTA 0's solo run (keeps the gate waiters' bound fresh).
    __device__ __forceinline__ void beat()
    {
        if (gs != nullptr && tid == 0)
            atomicAdd(&gs->heartbeat, 1u);
    }

    // Bounded wait at the gate for CTA 0 to hand a solo run back.  Thread 0
    // polls; the wait only runs out if CTA 0's heartbeat stops for wait_ns.
    __device__ bool gate_wait(LevelState& st)
    {
        int& s_ok = sh[2];
        int* s_st = sh + 3;  // 6 slots
        gbar();
        if (tid == 0) {
            int ok = 1;
            const uint32_t want = epoch + 1;
            unsigned long long t0 = globaltimer();
            uint32_t hb = *reinterpret_cast<volatile uint32_t*>(&gs->heartbeat);
            uint32_t spins = 0;
            while ((int)(ld_acquire(&gs->epoch) - want) < 0) {
                if ((++spins & 63u) == 0) {
                    if (read_status(res) != 0) {
                        ok = 0;
                        break;
                    }
                    const uint32_t h = *reinterpret_cast<volatile uint32_t*>(&gs->heartbeat);
                    const unsigned long long now = globaltimer();
                    if (h != hb) {
                        hb = h;
                        t0 = now;
                    } else if (now - t0 > wait_ns) {
                        set_status(res, kErrTimeout, 50);
                        ok = 0;
                        break;
                    }
                }
                if (spins > 1024)
                    __nanosleep(256);
            }
            if (ok)
                for (int i = 0; i < 6; ++i)
                    s_st[i] = (int)__ldcg(&gs->st[i]);
            s_ok = ok && read_status(res) == 0;
        }
        gbar();
        epoch += 1;
        if (s_ok) {
            st.a = s_st[0];
            st.b = s_st[1];
            st.Ka = s_st[2];
            st.Kb = s_st[3];
            st.L = s_st[4];
            st.last_start = s_st[5];
        }
        return s_ok != 0;
    }

    // CTA 0 publishes the state and opens the gate.  Returns whether the
    // team goes on (the waiters read the error status themselves).
    __device__ bool gate_open(const LevelState& st, bool ok)
    {
        gbar();
        if (tid == 0) {
            gs->st[0] = st.a;
            gs->st[1] = st.b;
            gs->st[2] = st.Ka;
            gs->st[3] = st.Kb;
            gs->st[4] = st.L;
            gs->st[5] = st.last_start;
            __threadfence();
            st_release(&gs->epoch, epoch + 1);
        }
        gbar();
        epoch += 1;
        return ok;
    }

    // Level all-gather, first half: this CTA's (children, edges), tagged
    // with the level's step number.
    __device__ __forceinline__ void ag_publish(uint32_t cnt, uint32_t esum, uint32_t step, unsigned long long* agg)
    {
        if (tid == 0) {
            st_relaxed64(agg + 2 * rank, ((unsigned long long)step << 32) | cnt);
            st_relaxed64(agg + 2 * rank + 1, ((unsigned long long)step << 32) | esum);
        }
    }

    // Second half: the sums over the CTAs before this one (pre) and over
    // all (all), children in the low and edges in the high 32 bits; over: a
    // CTA has more than B children or more than emax edges.
    template <int B>
    __device__ bool ag_collect(uint32_t step, const unsigned long long* agg, uint32_t emax, unsigned long long& pre,
                               unsigned long long& all, bool& over, unsigned long long* red)
    {
        int& s_ok = sh[9];
        int& s_over = sh[14];
        const uint32_t t = tid;
        pre = 0;
        all = 0;
        if (t == 0) {
            s_ok = 1;
            s_over = 0;
        }
        gbar();
        for (uint32_t i = t; i < size; i += B) {
            unsigned long long vc, ve;
            unsigned long long t0 = 0;
            uint32_t spins = 0;
            while (true) {
                vc = ld_relaxed64(agg + 2 * i);
                ve = ld_relaxed64(agg + 2 * i + 1);
                if ((uint32_t)(vc >> 32) == step && (uint32_t)(ve >> 32) == step)
                    break;
                if ((++spins & 31u) == 0 && !wait_check(t0, 4)) {
                    s_ok = 0;
                    break;
                }
                if (spins > 2048)
                    __nanosleep(128);
            }
            const unsigned long long v = ((ve & 0xFFFFFFFFull) << 32) | (vc & 0xFFFFFFFFull);
            all += v;
            if (i < rank)
                pre += v;
            if ((uint32_t)vc > (uint32_t)B || (uint32_t)ve > emax)
                s_over = 1;
        }
        block_reduce_sum2<B>(pre, all, red);
        over = s_over != 0;
        return s_ok != 0;
    }
};

// ---------------------------------------------------------------------------
// ClusterTeam: the CTAs of one thread-block cluster.  The hardware cluster
// barrier (release / acquire at cluster scope) replaces the global-memory
// barrier, and the all-gather and the gate hand-over read the peers' shared
// memory (DSMEM).  A hardware barrier has no time bound, so every CTA of the
// cluster must reach every barrier: the engine takes each "stop" decision
// uniformly (from flags all CTAs read after the same barrier) and returns
// only through such decisions.
// ---------------------------------------------------------------------------
struct ClusterShared {
    unsigned long long ag[2][2];  // all-gather words by barrier phase: children, edges
    uint32_t ok[2];               // "no error seen" flag at a barrier, by phase
    uint32_t st[6];               // CTA 0: level state handed over at the gate
    uint32_t job;                 // CTA 0: the job the cluster works on
    uint32_t all_ok;              // this CTA's AND of the peers' flags
    uint32_t job_ok;              // this CTA's verdict on the job (CSR arrived and valid, no hub)
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

struct ClusterTeam {
    static constexpr bool kGrid = false;
    ClusterShared* cs;  // this CTA's
    uint32_t size;      // CTAs in the cluster
    uint32_t rank;      // this CTA's rank in the cluster
    uint32_t phase;     // cluster barriers passed (slot parity)
    DevResult* res;
    // the CTA's thread group (a cluster team always spans whole CTAs) and
    // its group-shared scratch, as in Team
    uint32_t tid, bar, nthr;
    int* sh;

    __device__ __forceinline__ void gbar() const { gsync_n(bar, nthr); }

    __device__ __forceinline__ ClusterShared* peer(uint32_t r) const
    {
        return cooperative_groups::this_cluster().map_shared_rank(cs, r);
    }

    __device__ bool block_ok()
    {
        gbar();
        if (tid == 0)
            sh[0] = read_status(res) == 0;
        gbar();
        return sh[0] != 0;
    }

    // Cluster barrier; true iff no CTA had seen an error when it arrived.
    __device__ bool sync(uint32_t)
    {
        if (size == 1)
            return block_ok();
        const uint32_t ph = phase & 1u;
        gbar();
        if (tid == 0)
            cs->ok[ph] = read_status(res) == 0 ? 1u : 0u;
        cluster_arrive();
        cluster_wait();
        if (tid == 0) {
            uint32_t a = 1;
            for (uint32_t r = 0; r < size; ++r)
                a &= peer(r)->ok[ph];
            cs->all_ok = a;
        }
        gbar();
        ++phase;
        return cs->all_ok != 0;
    }

    __device__ __forceinline__ void beat() {}

    // Every CTA but 0: wait (hardware barrier) for CTA 0 to end its solo run,
    // then take its level state and its go / stop decision.
    __device__ bool gate_wait(LevelState& st)
    {
        const uint32_t ph = phase & 1u;
        gbar();
        cluster_arrive();
        cluster_wait();
        if (tid == 0) {
            const ClusterShared* p0 = peer(0);
            cs->st[0] = p0->st[0];
            cs->st[1] = p0->st[1];
            cs->st[2] = p0->st[2];
            cs->st[3] = p0->st[3];
            cs->st[4] = p0->st[4];
            cs->st[5] = p0->st[5];
            cs->all_ok = p0->ok[ph];
        }
        gbar();
        ++phase;
        st.a = cs->st[0];
        st.b = cs->st[1];
        st.Ka = cs->st[2];
        st.Kb = cs->st[3];
        st.L = cs->st[4];
        st.last_start = cs->st[5];
        return cs->all_ok != 0;
    }

    // CTA 0: hand the state over; the decision is CTA 0's alone.
    __device__ bool gate_open(const LevelState& st, bool ok)
    {
        const uint32_t ph = phase & 1u;
        gbar();
        if (tid == 0) {
            cs->st[0] = st.a;
            cs->st[1] = st.b;
            cs->st[2] = st.Ka;
            cs->st[3] = st.Kb;
            cs->st[4] = st.L;
            cs->st[5] = st.last_start;
            cs->ok[ph] = ok && read_status(res) == 0 ? 1u : 0u;
        }
        cluster_arrive();
        cluster_wait();
        ++phase;
        return cs->ok[ph] != 0;
    }

    // All-gather, first half: publish and arrive (the caller may work before
    // ag_collect waits).
    __device__ __forceinline__ void ag_publish(uint32_t cnt, uint32_t esum, uint32_t, unsigned long long*)
    {
        const uint32_t ph = phase & 1u;
        gbar();
        if (tid == 0) {
            cs->ag[ph][0] = cnt;
            cs->ag[ph][1] = esum;
            cs->ok[ph] = read_status(res) == 0 ? 1u : 0u;
        }
        cluster_arrive();
    }

    template <int B>
    __device__ bool ag_collect(uint32_t, const unsigned long long*, uint32_t emax, unsigned long long& pre,
                               unsigned long long& all, bool& over, unsigned long long* red)
    {
        const uint32_t ph = phase & 1u;
        cluster_wait();
        const uint32_t t = tid;
        pre = 0;
        all = 0;
        if (t == 0) {
            cs->all_ok = 1;
            sh[14] = 0;
        }
        gbar();
        for (uint32_t i = t; i < size; i += B) {
            const ClusterShared* pi = peer(i);
            if ((uint32_t)pi->ag[ph][0] > (uint32_t)B || (uint32_t)pi->ag[ph][1] > emax)
                sh[14] = 1;
            const unsigned long long v = (pi->ag[ph][1] << 32) | (pi->ag[ph][0] & 0xFFFFFFFFull);
            if (!pi->ok[ph])
                atomicAnd(&cs->all_ok, 0u);
            all += v;
            if (i < rank)
                pre += v;
        }
        block_reduce_sum2<B>(pre, all, red);
        over = sh[14] != 0;
        ++phase;
        return cs->all_ok != 0;
    }
};

// ---------------------------------------------------------------------------
// Shared memory of one thread group (one engine instance).
// ---------------------------------------------------------------------------
template <int B, int EMAX>
struct Smem {
    static constexpr int W = B / 32;
    static constexpr int PREMAX = 4 * EMAX;  // prefetched child adjacency
    // parents of the current chunk
    uint32_t pn[B], prs[B], pdeg[B], peb[B];
    uint32_t soff[B + 1];   // edge offset of parent j inside the chunk
    uint32_t cs[B], cc[B];  // first child index / child count of parent j
    // children of the current chunk (compacted in (parent, slot) order);
    // the hub radix sort reuses this space for its per-warp digit counts
    static_assert(4 * EMAX >= W * 256, "EMAX too small for the hub counters");
    union {
        struct {
            uint32_t ch_node[EMAX], ch_deg[EMAX], ch_rs[EMAX], ch_par[EMAX];
        };
        uint32_t hcnt[W * 256];
    };
    uint32_t so_idx[EMAX];       // ranked position -> compacted index
    uint32_t so_eoff[EMAX + 1];  // edge offset of the child at ranked position
    uint32_t pre[PREMAX];        // children's adjacency loaded ahead of the all-gather
    uint32_t tmp32[W + 1];
    unsigned long long tmp64[2 * W + 2];
    unsigned long long gat64[2 * W + 2];  // all-gather reduction (its own buffer)
    uint32_t scanbuf[5][W];               // one per block_scan1 call site
    uint32_t wq[EMAX / B][W];             // collect: child edges per (round, warp)
    uint32_t hist[256];
    // chunk scalars
    uint32_t m, Ec, Q, Qdeg, hub, npre;
    uint32_t bcast[8];
    int gsh[kTeamShared];  // the team's group-shared slots (Team::sh)
};

// Wires a team to the calling thread group (B threads) and its shared memory.
template <int B, int EMAX, class TeamT>
__device__ __forceinline__ void bind_group(TeamT& tm, Smem<B, EMAX>& s)
{
    tm.tid = gtid<B>();
    tm.bar = gbar_id<B>();
    tm.nthr = B;
    tm.sh = s.gsh;
}

// Counts of one collected unit (chunk or hub).
struct Agg {
    uint32_t cnt;   // children
    uint32_t esum;  // sum of their valences
};

// ---------------------------------------------------------------------------
// Chunk machinery
// ---------------------------------------------------------------------------
template <int B, int EMAX>
struct Chunk {
    static constexpr int MAXEPT = EMAX / B;
    static_assert(EMAX % B == 0, "EMAX must be a multiple of B");
    Smem<B, EMAX>& s;
    const MatrixView& M;
    uint32_t base;  // key of the pass: edge id e has key base - 1 - e
    // queue record of position pf_base + (group thread), loaded by the previous
    // form() for the chunk that follows it (its latency hides behind that
    // chunk's work); pf_base == kUnvisited: none
    uint32_t pf_base = kUnvisited;
    uint4 pf = make_uint4(0u, 0u, 0u, 0u);

    // Loads up to B parents starting at position p (< pend) and forms the
    // next chunk: the longest run with <= EMAX edges.  Sets s.m (0 = the
    // first parent is a hub; s.hub = 1 then) and s.Ec.  Returns the number of
    // parents consumed (the hub counts as 1).
    __device__ uint32_t form(uint32_t p, uint32_t pend)
    {
        const uint32_t t = gtid<B>();
        uint32_t deg = 0;
        const bool have = p + t < pend;
        if (have) {
            const uint32_t pos = p + t;
            if (PB_CHECK(M.res, pos < M.n, 101)) {
                const uint4 r = p == pf_base ? pf : __ldcg(reinterpret_cast<const uint4*>(M.rec) + pos);
                s.pn[t] = r.x;
                s.prs[t] = r.y;
                s.pdeg[t] = r.z;
                s.peb[t] = r.w;
                deg = r.z;
            }
        }
        s.cc[t] = 0;
        uint32_t total;
        const uint32_t excl = block_scan1<B>(deg, total, s.scanbuf[0]);
        const uint32_t incl = excl + deg;
        // incl is monotone in t, so the fitting parents are a prefix
        const int fits = have && incl <= (uint32_t)EMAX;
        const int m = gsync_count<B>(fits);
        if (fits)
            s.soff[t] = excl;
        if (m > 0 && t == (uint32_t)(m - 1))
            s.soff[m] = incl;
        if (t == 0) {
            s.m = (uint32_t)m;
            s.hub = (m == 0 && p < pend) ? 1u : 0u;
            if (m == 0)
                s.soff[0] = 0;
        }
        // the next chunk starts where this one ends: load its records now
        const uint32_t used = m > 0 ? (uint32_t)m : (p < pend ? 1u : 0u);
        const uint32_t nb = p + used;
        pf_base = kUnvisited;
        if (nb < pend) {
            pf_base = nb;
            if (nb + t < pend && PB_CHECK(M.res, nb + t < M.n, 109))
                pf = __ldcg(reinterpret_cast<const uint4*>(M.rec) + nb + t);
        }
        gsync<B>();
        if (t == 0)
            s.Ec = m > 0 ? s.soff[m] : 0;
        gsync<B>();
        return used;
    }

    // Makes the ranked children of the previous chunk (still in shared memory,
    // with their adjacency in s.pre) the parents of this one: no global load.
    // Needs Q <= B and Qdeg <= EMAX; K0prev is the edge base they were placed
    // with.
    __device__ void form_from_children(uint32_t K0prev)
    {
        const uint32_t t = gtid<B>();
        const uint32_t F = s.Q, E = s.Qdeg;
        if (t < F) {
            const uint32_t x = s.so_idx[t];
            s.pn[t] = s.ch_node[x];
            s.prs[t] = s.ch_rs[x];
            s.pdeg[t] = s.ch_deg[x];
            s.peb[t] = K0prev + s.so_eoff[t];
            s.soff[t] = s.so_eoff[t];
        }
        s.cc[t] = 0;
        if (t == 0) {
            s.soff[F] = E;
            s.m = F;
            s.Ec = E;
            s.hub = 0;
        }
        gsync<B>();
    }

    // Finds the child edges of the chunk, compacts them, ranks every
    // parent's children (sorted = by valence, stable; else slot order) and
    // computes the edge offsets of the ranked children.  BITS: vis holds a bit
    // per node placed by an earlier level (set here for the children): most
    // columns of a wide level are settled by it, without their node entry.
    template <bool BITS = false>
    __device__ Agg collect(bool sorted, bool from_pre = false, uint32_t* vis = nullptr)
    {
        const uint32_t t = gtid<B>(), lane = t & 31u, w = t >> 5;
        const uint32_t m = s.m, Ec = s.Ec;
        // thread t takes the edges e = t + B r: a warp loads consecutive
        // entries of the parents' rows (coalesced), and edge order is
        // (round r, warp, lane), the order the compaction below keeps
        uint32_t c[MAXEPT], jj[MAXEPT], key[MAXEPT], kk[MAXEPT];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            const uint32_t e = t + (uint32_t)B * r;
            c[r] = kUnvisited;
            jj[r] = 0;
            kk[r] = 1;
            if (e < Ec) {
                // the edge's parent: the last j < m with soff[j] <= e (a
                // parent of valence 0 owns no edge)
                uint32_t j = 0;
#pragma unroll
                for (uint32_t d = (uint32_t)B / 2u; d > 0; d >>= 1) {
                    const uint32_t mid = j + d;
                    if (mid < m && s.soff[mid] <= e)
                        j = mid;
                }
                const uint32_t k = e - s.soff[j];
                const uint32_t idx = s.prs[j] + k;
                jj[r] = j;
                kk[r] = k;
                key[r] = base - 1u - (s.peb[j] + k);
                if (from_pre)
                    c[r] = s.pre[e];  // the parents' adjacency, loaded when they were placed
                else if (PB_CHECK(M.res, idx < M.nnz, 102))
                    c[r] = ld_ro(M.ci + idx);
            }
        }
        if (BITS) {
            uint32_t word[MAXEPT];
#pragma unroll
            for (int r = 0; r < MAXEPT; ++r)
                word[r] = c[r] != kUnvisited && PB_CHECK(M.res, c[r] < M.n, 162) ? vis[c[r] >> 5] : kFull;
#pragma unroll
            for (int r = 0; r < MAXEPT; ++r)
                if ((word[r] >> (c[r] & 31u)) & 1u)
                    c[r] = kUnvisited;
        }
        uint4 nd[MAXEPT];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            nd[r] = make_uint4(0, 0, 0, 0);
            if (c[r] != kUnvisited && PB_CHECK(M.res, c[r] < M.n, 103))
                nd[r] = ld_node(M.node + c[r]);
        }
        // the child edges (claimed by this edge's key) compacted in edge
        // order: a ballot per warp and round, then the (round, warp) counts
        uint32_t pos[MAXEPT];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            if (!(c[r] != kUnvisited && c[r] < M.n && nd[r].x == key[r]))
                c[r] = kUnvisited;
            else if (BITS)
                atomicOr(vis + (c[r] >> 5), 1u << (c[r] & 31u));
            const uint32_t bal = __ballot_sync(kFull, c[r] != kUnvisited);
            pos[r] = __popc(bal & ((1u << lane) - 1u));
            if (lane == 0)
                s.wq[r][w] = __popc(bal);
        }
        gsync<B>();
        uint32_t Q = 0;
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
#pragma unroll
            for (int i = 0; i < Smem<B, EMAX>::W; ++i) {
                const uint32_t n_ = s.wq[r][i];
                pos[r] += (uint32_t)i < w ? n_ : 0u;
                Q += n_;
            }
            // the rounds before this one
            if (r + 1 < MAXEPT)
                pos[r + 1] += Q;
        }
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            const uint32_t e = t + (uint32_t)B * r;
            if (e < Ec) {
                const uint32_t q = pos[r];
                if (kk[r] == 0)
                    s.cs[jj[r]] = q;
                if (c[r] != kUnvisited && PB_CHECK(M.res, q < (uint32_t)EMAX, 104)) {
                    s.ch_node[q] = c[r];
                    s.ch_rs[q] = nd[r].y;
                    s.ch_deg[q] = nd[r].z;
                    s.ch_par[q] = jj[r];
                    atomicAdd(&s.cc[jj[r]], 1u);
                }
            }
        }
        gsync<B>();
        // rank every child inside its parent's run
        for (uint32_t x = t; x < Q; x += B) {
            const uint32_t jp = s.ch_par[x];
            const uint32_t st = s.cs[jp], len = s.cc[jp];
            uint32_t rank = x - st;
            if (sorted && len > 1) {
                const uint32_t dx = s.ch_deg[x];
                rank = 0;
                for (uint32_t y = st; y < st + len; ++y) {
                    const uint32_t dy = s.ch_deg[y];
                    rank += (dy < dx) || (dy == dx && y < x);
                }
            }
            s.so_idx[st + rank] = x;
        }
        gsync<B>();
        // edge offsets in ranked order (blocked exclusive scan)
        const uint32_t per = (Q + B - 1) / B;
        const uint32_t i0 = min(t * per, Q), i1 = min(i0 + per, Q);
        uint32_t loc = 0;
        for (uint32_t i = i0; i < i1; ++i)
            loc += s.ch_deg[s.so_idx[i]];
        uint32_t Qdeg;
        uint32_t off = block_scan1<B>(loc, Qdeg, s.scanbuf[2]);
        for (uint32_t i = i0; i < i1; ++i) {
            s.so_eoff[i] = off;
            off += s.ch_deg[s.so_idx[i]];
        }
        if (t == 0) {
            s.so_eoff[Q] = Qdeg;
            s.Q = Q;
            s.Qdeg = Qdeg;
            s.npre = 0;
        }
        gsync<B>();
        return Agg{Q, Qdeg};
    }

    // ---- unordered passes (level_pass) --------------------------------
    // A list of queue entries in shared memory (node, row start, valence):
    // two of EMAX entries, in the child arrays and in the room of the
    // prefetched adjacency.
    struct List {
        uint32_t *node, *rs, *deg;
    };
    __device__ __forceinline__ List list(uint32_t which) const
    {
        return which ? List{s.pre, s.pre + EMAX, s.pre + 2 * EMAX} : List{s.ch_node, s.ch_rs, s.ch_deg};
    }

    // The next chunk's parents from entries [p, F) of a list: the longest run
    // of at most B parents with at most EMAX edges.  Returns their number.
    __device__ uint32_t form_list(const List& P, uint32_t p, uint32_t F)
    {
        const uint32_t t = gtid<B>();
        const bool have = p + t < F;
        const uint32_t deg = have ? P.deg[p + t] : 0u;
        uint32_t total;
        const uint32_t excl = block_scan1<B>(deg, total, s.scanbuf[1]);
        uint32_t m = F - p;
        if (m > (uint32_t)B || total > (uint32_t)EMAX)  // the same in every thread
            m = (uint32_t)gsync_count<B>(have && excl + deg <= (uint32_t)EMAX);
        if (t < m) {
            s.prs[t] = P.rs[p + t];
            s.soff[t] = excl;
            if (t == m - 1) {
                s.soff[m] = excl + deg;
                s.m = m;
                s.Ec = excl + deg;
            }
        }
        gsync<B>();
        return m;
    }

    // The columns of the chunk's edges: thread t's are t + B r.
    __device__ __forceinline__ void load_cols(uint32_t c[MAXEPT]) const
    {
        const uint32_t t = gtid<B>();
        const uint32_t m = s.m, Ec = s.Ec;
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            const uint32_t e = t + (uint32_t)B * r;
            c[r] = kUnvisited;
            if (e < Ec) {
                uint32_t j = 0;
#pragma unroll
                for (uint32_t d = (uint32_t)B / 2u; d > 0; d >>= 1) {
                    const uint32_t mid = j + d;
                    if (mid < m && s.soff[mid] <= e)
                        j = mid;
                }
                const uint32_t idx = s.prs[j] + (e - s.soff[j]);
                if (PB_CHECK(M.res, idx < M.nnz, 152))
                    c[r] = ld_ro(M.ci + idx);
            }
        }
    }

    // The unordered form of collect: those of the chunk's columns that no
    // edge of this pass has claimed yet (claims below `first` are earlier
    // passes'), each new node once; its claim and its node entry come with
    // one round trip, side by side.  They go behind the C.cnt entries of
    // list `out`, which `flush` empties first when they do not fit.
    // counted(C) is called once their number is known, before they are
    // listed.
    template <typename Flush, typename Counted>
    __device__ void claim_list(uint32_t first, const uint32_t c[MAXEPT], const List& out, Agg& C, Flush flush,
                               Counted counted)
    {
        const uint32_t t = gtid<B>(), lane = t & 31u, w = t >> 5;
        uint32_t old[MAXEPT];
        uint4 nd[MAXEPT];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            old[r] = kUnvisited;
            nd[r] = make_uint4(0u, 0u, 0u, 0u);
            if (c[r] != kUnvisited && PB_CHECK(M.res, c[r] < M.n, 153)) {
                old[r] = atomicMax(&M.node[c[r]].claim, base);
                nd[r] = ld_node(M.node + c[r]);
            }
        }
        uint32_t pos[MAXEPT], dsum = 0;
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            const bool win = old[r] < first;
            const uint32_t bal = __ballot_sync(kFull, win);
            pos[r] = __popc(bal & ((1u << lane) - 1u));
            dsum += win ? nd[r].z : 0u;
            if (lane == 0)
                s.wq[r][w] = __popc(bal);
        }
        dsum = __reduce_add_sync(kFull, dsum);
        if (lane == 0)
            s.tmp32[w] = dsum;
        gsync<B>();
        uint32_t Q = 0, Qdeg = 0;
#pragma unroll
        for (int i = 0; i < Smem<B, EMAX>::W; ++i)
            Qdeg += s.tmp32[i];
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r) {
            pos[r] += Q;
#pragma unroll
            for (int i = 0; i < Smem<B, EMAX>::W; ++i) {
                const uint32_t n_ = s.wq[r][i];
                pos[r] += (uint32_t)i < w ? n_ : 0u;
                Q += n_;
            }
        }
        if (C.cnt + Q > (uint32_t)EMAX)
            flush();
        counted(Agg{C.cnt + Q, C.esum + Qdeg});
#pragma unroll
        for (int r = 0; r < MAXEPT; ++r)
            if (old[r] < first) {
                const uint32_t at = C.cnt + pos[r];
                out.node[at] = c[r];
                out.rs[at] = nd[r].y;
                out.deg[at] = nd[r].z;
            }
        C.cnt += Q;
        C.esum += Qdeg;
        gsync<B>();
    }

    template <typename Flush>
    __device__ __forceinline__ void collect_any(uint32_t first, const List& out, Agg& C, Flush flush)
    {
        uint32_t c[MAXEPT];
        load_cols(c);
        claim_list(first, c, out, C, flush, [](const Agg&) {});
    }

    // The share [p_beg, p_end) of a level too wide for one chunk a CTA: no
    // chunks, each warp works on its own (up to 32 parents with 32 U entries
    // between them at a time, a row of 32 or more entries alone), so that all
    // its loads are in flight together and nothing waits at a barrier.  The
    // node entry is read before the claim: on such levels most columns are
    // claimed already.  Children go behind the CTA's list `out` while there is
    // room, else straight to the queue (positions P0 + the level's counter).
    // A 1M-node geometric graph (levels of 2,300 entries a CTA, bound by the
    // latency of the gathers): 3.7 ms a call in chunks, 1.87 ms so.
    __device__ void claim_wide(uint32_t first, uint32_t p_beg, uint32_t p_end, const List& out, Agg& C, uint32_t P0,
                               unsigned long long* counter)
    {
        constexpr uint32_t W = B / 32;
        // entries a lane holds: 8, or what the warps' entry lists leave room
        // for in so_idx
        constexpr int U = 4 * EMAX / (W * 64) < 8 ? 4 * EMAX / (W * 64) : 8;
        const uint32_t t = gtid<B>(), lane = t & 31u, w = t >> 5;
        const uint32_t lt = (1u << lane) - 1u;
        uint16_t* const ent = reinterpret_cast<uint16_t*>(s.so_idx) + w * 32 * U;
        if (t == 0) {
            s.bcast[2] = 0;     // taken in `out`
            s.bcast[3] = EMAX;  // entries of `out` without a gap
            s.bcast[4] = 0;     // sum of their valences
        }
        gsync<B>();
        const uint32_t F = p_end - p_beg, share = (F + W - 1) / W;
        const uint32_t pe = p_beg + min(F, (w + 1) * share);
        for (uint32_t p = p_beg + min(F, w * share); p < pe;) {
            uint2 r = make_uint2(0u, 0u);  // row start, valence
            if (p + lane < pe && PB_CHECK(M.res, p + lane < M.n, 158)) {
                const uint4 q = __ldcg(reinterpret_cast<const uint4*>(M.rec) + p + lane);
                r = make_uint2(q.y, q.z);
            }
            uint32_t x = r.y;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                x += lane >= o ? y : 0u;
            }
            const uint32_t out_of = ~__ballot_sync(kFull, p + lane < pe && r.y < 32u && x <= 32u * U);
            const uint32_t m = out_of ? (uint32_t)__ffs(out_of) - 1u : 32u;
            const uint32_t took = max(m, 1u);
            const uint32_t soff = x - r.y, shift = r.x - soff;
            const uint32_t E = __shfl_sync(kFull, x, (int)took - 1);
            __syncwarp();
            if (lane < m)
                for (uint32_t k = 0; k < r.y; ++k)
                    ent[soff + k] = (uint16_t)lane;
            __syncwarp();
            for (uint32_t e0 = 0; e0 < E; e0 += 32u * U) {
                uint32_t c[U];
                uint4 nd[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t e = e0 + 32u * u + lane;
                    c[u] = kUnvisited;
                    if (e0 + 32u * u < E) {
                        const uint32_t j = m != 0 ? (uint32_t)ent[32u * u + lane] & 31u : 0u;
                        const uint32_t idx = __shfl_sync(kFull, shift, (int)j) + e;
                        if (e < E && PB_CHECK(M.res, idx < M.nnz, 159))
                            c[u] = ld_ro(M.ci + idx);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    nd[u] = make_uint4(kUnvisited, 0u, 0u, 0u);
                    if (c[u] != kUnvisited && PB_CHECK(M.res, c[u] < M.n, 160))
                        nd[u] = ld_node(M.node + c[u]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (nd[u].x < first)
                        nd[u].x = atomicMax(&M.node[c[u]].claim, base);
                uint32_t bal[U], q = 0, dsum = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    bal[u] = __ballot_sync(kFull, nd[u].x < first);
                    q += __popc(bal[u]);
                    dsum += nd[u].x < first ? nd[u].z : 0u;
                }
                if (q == 0)
                    continue;
                dsum = __reduce_add_sync(kFull, dsum);
                uint32_t at = 0;
                if (lane == 0)
                    at = atomicAdd(&s.bcast[2], q);
                at = __shfl_sync(kFull, at, 0);
                const bool listed = at + q <= (uint32_t)EMAX;
                if (lane == 0) {
                    if (listed) {
                        atomicAdd(&s.bcast[4], dsum);
                    } else {
                        atomicMin(&s.bcast[3], at);
                        at = P0 + (uint32_t)atomicAdd(counter, (unsigned long long)dsum << 32 | q);
                    }
                }
                at = __shfl_sync(kFull, at, 0);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t i = at + __popc(bal[u] & lt);
                    if (nd[u].x < first) {
                        if (listed) {
                            out.node[i] = c[u];
                            out.rs[i] = nd[u].y;
                            out.deg[i] = nd[u].z;
                        } else if (PB_CHECK(M.res, i < M.n, 161)) {
                            __stcg(reinterpret_cast<uint4*>(M.rec) + i, make_uint4(c[u], nd[u].y, nd[u].z, 0u));
                        }
                    }
                    at += __popc(bal[u]);
                }
            }
            p += took;
        }
        gsync<B>();
        C = Agg{min(s.bcast[2], s.bcast[3]), s.bcast[4]};
    }

    // Writes the first Q entries of a list to queue positions P0..
    __device__ void place_list(const List& P, uint32_t P0, uint32_t Q)
    {
        for (uint32_t i = gtid<B>(); i < Q; i += B)
            if (PB_CHECK(M.res, P0 + i < M.n, 154))
                __stcg(reinterpret_cast<uint4*>(M.rec) + P0 + i, make_uint4(P.node[i], P.rs[i], P.deg[i], 0u));
    }

    // The ranked child owning edge offset f: so_eoff[lo] <= f < so_eoff[lo+1].
    __device__ __forceinline__ uint32_t child_of(uint32_t f) const
    {
        uint32_t lo = 0, hi = s.Q;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s.so_eoff[mid] <= f)
                lo = mid;
            else
                hi = mid;
        }
        return lo;
    }

    // Walks the ranked children's edges in blocks of consecutive edge offsets
    // (one search per thread, then a forward walk), calling
    // fn(f, col_index) for each.
    template <typename Fn>
    __device__ __forceinline__ void for_child_edges(Fn fn) const
    {
        const uint32_t Qdeg = s.Qdeg;
        const uint32_t per = (Qdeg + B - 1) / B;
        const uint32_t f0 = gtid<B>() * per, f1 = min(f0 + per, Qdeg);
        if (f0 >= f1)
            return;
        uint32_t lo = child_of(f0);
        uint32_t beg = s.so_eoff[lo], nxt = s.so_eoff[lo + 1];
        uint32_t rs = s.ch_rs[s.so_idx[lo]];
        for (uint32_t f = f0; f < f1; ++f) {
            while (f >= nxt) {
                ++lo;
                beg = nxt;
                nxt = s.so_eoff[lo + 1];
                rs = s.ch_rs[s.so_idx[lo]];
            }
            fn(f, rs + (f - beg));
        }
    }

    // Loads the ranked children's adjacency into s.pre (when it fits) so that
    // the claims after the all-gather issue no dependent load.
    __device__ void prefetch()
    {
        const uint32_t Qdeg = s.Qdeg;
        if (Qdeg > (uint32_t)Smem<B, EMAX>::PREMAX)
            return;
        for_child_edges([&](uint32_t f, uint32_t idx) {
            s.pre[f] = PB_CHECK(M.res, idx < M.nnz, 108) ? ld_ro(M.ci + idx) : 0u;
        });
        gsync<B>();
        if (gtid<B>() == 0)
            s.npre = Qdeg;
        gsync<B>();
    }

    // Writes the ranked children of the chunk at positions P0.. and edge
    // bases K0.., then claims their edges for the next level.
    __device__ void place_and_claim(uint32_t P0, uint32_t K0, bool write_perm, bool reverse)
    {
        const uint32_t t = gtid<B>();
        const uint32_t Q = s.Q, Qdeg = s.Qdeg;
        const bool have_pre = s.npre == Qdeg && Qdeg > 0;
        for (uint32_t i = t; i < Q; i += B) {
            const uint32_t x = s.so_idx[i];
            const uint32_t pos = P0 + i;
            if (PB_CHECK(M.res, pos < M.n, 105)) {
                const uint4 r = make_uint4(s.ch_node[x], s.ch_rs[x], s.ch_deg[x], K0 + s.so_eoff[i]);
                __stcg(reinterpret_cast<uint4*>(M.rec) + pos, r);
                if (write_perm)
                    M.perm[reverse ? M.n - 1 - pos : pos] = r.x;
            }
        }
        const uint32_t kb = base - 1u - K0;
        if (have_pre) {
            for (uint32_t f = t; f < Qdeg; f += B) {
                const uint32_t d = s.pre[f];
                if (PB_CHECK(M.res, d < M.n, 107))
                    atomicMax(claim_ptr(M, d), kb - f);
            }
        } else {
            for_child_edges([&](uint32_t f, uint32_t idx) {
                if (PB_CHECK(M.res, idx < M.nnz, 106)) {
                    const uint32_t d = ld_ro(M.ci + idx);
                    if (PB_CHECK(M.res, d < M.n, 107))
                        atomicMax(claim_ptr(M, d), kb - f);
                }
            });
        }
    }

    // Writes the ranked children of the chunk to M.stage[at..]: node, row
    // start, valence and the child-edge offset eoff0 + so_eoff[i].
    __device__ void stage_children(uint32_t at, uint32_t eoff0)
    {
        const uint32_t Q = s.Q;
        for (uint32_t i = gtid<B>(); i < Q; i += B) {
            const uint32_t x = s.so_idx[i];
            if (PB_CHECK(M.res, (uint64_t)at + i < M.nnz, 130))
                __stcg(reinterpret_cast<uint4*>(M.stage) + at + i,
                       make_uint4(s.ch_node[x], s.ch_rs[x], s.ch_deg[x], eoff0 + s.so_eoff[i]));
        }
    }

    // Places the `count` children staged at M.stage[at..] (in order) at
    // positions P0.. with edge ids K0 + their child-edge offsets, and claims
    // their edges, in tiles of up to EMAX children.
    __device__ void place_staged(uint32_t at, uint32_t count, uint32_t P0, uint32_t K0, bool write_perm,
                                 bool reverse)
    {
        uint32_t done = 0, kdone = 0;
        while (done < count) {
            const uint32_t cnt = min((uint32_t)EMAX, count - done);
            for (uint32_t i = gtid<B>(); i < cnt; i += B) {
                uint4 r = make_uint4(0u, 0u, 0u, kdone);
                if (PB_CHECK(M.res, (uint64_t)at + done + i < M.nnz, 131))
                    r = __ldcg(reinterpret_cast<const uint4*>(M.stage) + at + done + i);
                s.ch_node[i] = r.x;
                s.ch_rs[i] = r.y;
                s.ch_deg[i] = r.z;
                s.so_idx[i] = i;
                s.so_eoff[i] = r.w - kdone;
                if (i == cnt - 1) {
                    s.so_eoff[cnt] = r.w + r.z - kdone;
                    s.Q = cnt;
                    s.Qdeg = r.w + r.z - kdone;
                    s.npre = 0;
                }
            }
            gsync<B>();
            const uint32_t qdeg = s.Qdeg;
            place_and_claim(P0 + done, K0 + kdone, write_perm, reverse);
            gsync<B>();
            done += cnt;
            kdone += qdeg;
        }
    }

    // ---- hubs: one parent with more than EMAX edges -----------------------
    // Scratch layout (4 arrays of nnz words): key0 | val0 | key1 | val1.  A
    // hub at level-relative edge offset r0 owns [r0, r0 + deg) of each.
    __device__ uint32_t* hk0() const { return M.hub; }
    __device__ uint32_t* hv0() const { return M.hub + M.nnz; }
    __device__ uint32_t* hk1() const { return M.hub + 2ull * M.nnz; }
    __device__ uint32_t* hv1() const { return M.hub + 3ull * M.nnz; }

    // Collects the hub's children (valence, slot) in slot order and sorts
    // them stably by valence (sorted == true) into key0/val0.  The counts
    // are also left in key1[r0], key1[r0+1] for a later placement.
    __device__ Agg hub_collect(uint32_t r0, bool sorted)
    {
        const uint32_t t = gtid<B>();
        const uint32_t rs = s.prs[0], D = s.pdeg[0], eb = s.peb[0];
        if (M.hub == nullptr) {
            set_status(M.res, kErrCheck, 120);
            return Agg{0, 0};
        }
        uint32_t Q = 0;
        unsigned long long Qdeg = 0;
        uint32_t maxkey = 0;
        constexpr uint32_t TILE = B * MAXEPT;
        for (uint32_t base0 = 0; base0 < D; base0 += TILE) {
            uint32_t nv = 0;
            uint32_t dg[MAXEPT];
            bool ok[MAXEPT];
#pragma unroll
            for (int r = 0; r < MAXEPT; ++r) {
                const uint32_t e = base0 + t * MAXEPT + r;
                ok[r] = false;
                if (e < D && PB_CHECK(M.res, rs + e < M.nnz, 121)) {
                    const uint32_t c = ld_ro(M.ci + rs + e);
                    if (PB_CHECK(M.res, c < M.n, 122)) {
                        const uint4 nd = ld_node(M.node + c);
                        if (nd.x == base - 1u - (eb + e)) {
                            dg[r] = nd.z;
                            ok[r] = true;
                            ++nv;
                        }
                    }
                }
            }
            uint32_t tot;
            uint32_t q = block_scan1<B>(nv, tot, s.scanbuf[3]);
            uint32_t lsum = 0, lmax = 0;
#pragma unroll
            for (int r = 0; r < MAXEPT; ++r) {
                if (ok[r]) {
                    const uint32_t w = r0 + Q + q;
                    if (PB_CHECK(M.res, w < M.nnz, 123)) {
                        hk0()[w] = dg[r];
                        hv0()[w] = base0 + t * MAXEPT + r;
                    }
                    lsum += dg[r];
                    lmax = max(lmax, dg[r]);
                    ++q;
                }
            }
            Qdeg += block_reduce_sum<B, unsigned long long>(lsum, s.tmp64);
            maxkey = max(maxkey, block_reduce_max<B, uint32_t>(lmax, s.tmp32));
            Q += tot;
        }
        if (sorted && Q > 1) {
            // stable LSD radix sort, 8-bit digits, an even number of passes
            // so that the result lands back in key0/val0
            uint32_t passes = 0;
            while (passes < 4 && (maxkey >> (8 * passes)) != 0)
                ++passes;
            if (passes == 0)
                passes = 1;
            passes += passes & 1;
            for (uint32_t ps = 0; ps < passes; ++ps) {
                uint32_t* sk = (ps & 1) ? hk1() : hk0();
                uint32_t* sv = (ps & 1) ? hv1() : hv0();
                uint32_t* dk = (ps & 1) ? hk0() : hk1();
                uint32_t* dv = (ps & 1) ? hv0() : hv1();
                radix_pass(sk + r0, sv + r0, dk + r0, dv + r0, Q, 8 * ps);
            }
        }
        if (t == 0) {
            __stcg(hk1() + r0, Q);
            __stcg(hk1() + r0 + 1, (uint32_t)Qdeg);
        }
        gsync<B>();
        return Agg{Q, (uint32_t)Qdeg};
    }

    // One stable counting pass on digit (key >> shift) & 255.
    __device__ void radix_pass(const uint32_t* sk, const uint32_t* sv, uint32_t* dk, uint32_t* dv, uint32_t Q,
                               uint32_t shift)
    {
        const uint32_t t = gtid<B>(), lane = t & 31, w = t >> 5;
        for (uint32_t d = t; d < 256; d += B)
            s.hist[d] = 0;
        gsync<B>();
        for (uint32_t i = t; i < Q; i += B)
            atomicAdd(&s.hist[(__ldcg(sk + i) >> shift) & 255u], 1u);
        gsync<B>();
        if (t == 0) {
            uint32_t run = 0;
            for (int d = 0; d < 256; ++d) {
                const uint32_t h = s.hist[d];
                s.hist[d] = run;
                run += h;
            }
        }
        gsync<B>();
        for (uint32_t base0 = 0; base0 < Q; base0 += B) {
            for (uint32_t i = t; i < (uint32_t)(Smem<B, EMAX>::W * 256); i += B)
                s.hcnt[i] = 0;
            gsync<B>();
            const uint32_t i = base0 + t;
            const bool act = i < Q;
            uint32_t key = 0, val = 0, dgt = 0;
            if (act) {
                key = __ldcg(sk + i);
                val = __ldcg(sv + i);
                dgt = (key >> shift) & 255u;
            }
            const uint32_t peers = __match_any_sync(kFull, act ? dgt : 256u + lane);
            const uint32_t below = peers & ((1u << lane) - 1u);
            const uint32_t rank_w = __popc(below);
            const bool leader = act && below == 0;
            if (leader)
                s.hcnt[w * 256 + dgt] = __popc(peers);
            gsync<B>();
            if (act) {
                uint32_t before = 0;
                for (uint32_t ww = 0; ww < w; ++ww)
                    before += s.hcnt[ww * 256 + dgt];
                const uint32_t dst = s.hist[dgt] + before + rank_w;
                dk[dst] = key;
                dv[dst] = val;
            }
            gsync<B>();
            for (uint32_t d = t; d < 256; d += B) {
                uint32_t add = 0;
                for (int ww = 0; ww < Smem<B, EMAX>::W; ++ww)
                    add += s.hcnt[ww * 256 + d];
                s.hist[d] += add;
            }
            gsync<B>();
        }
    }

    // Places the sorted hub children (count Q) at P0.. / K0.. in tiles of
    // EMAX, reusing the chunk arrays, and claims their edges.
    __device__ void hub_place_and_claim(uint32_t r0, uint32_t Q, uint32_t P0, uint32_t K0, bool write_perm,
                                        bool reverse)
    {
        const uint32_t t = gtid<B>();
        const uint32_t rs = s.prs[0];
        uint32_t done = 0, kdone = 0;
        while (done < Q) {
            const uint32_t cnt = min((uint32_t)EMAX, Q - done);
            uint32_t loc = 0;
            const uint32_t per = (cnt + B - 1) / B;
            const uint32_t i0 = min(t * per, cnt), i1 = min(i0 + per, cnt);
            for (uint32_t i = i0; i < i1; ++i) {
                const uint32_t slot = __ldcg(hv0() + r0 + done + i);
                const uint32_t node = ld_ro(M.ci + rs + slot);
                const uint4 nd = ld_node(M.node + node);
                s.ch_node[i] = node;
                s.ch_rs[i] = nd.y;
                s.ch_deg[i] = nd.z;
                s.so_idx[i] = i;
                loc += nd.z;
            }
            uint32_t tot;
            uint32_t off = block_scan1<B>(loc, tot, s.scanbuf[4]);
            for (uint32_t i = i0; i < i1; ++i) {
                s.so_eoff[i] = off;
                off += s.ch_deg[i];
            }
            if (t == 0) {
                s.so_eoff[cnt] = tot;
                s.Q = cnt;
                s.Qdeg = tot;
                s.npre = 0;
            }
            gsync<B>();
            place_and_claim(P0 + done, K0 + kdone, write_perm, reverse);
            gsync<B>();
            done += cnt;
            kdone += tot;
        }
    }
};

// ---------------------------------------------------------------------------
// One ordered BFS pass from `start` with pass key `base`.  Fills
// rec[0..placed) and, when write_perm, the output.  Returns false if the team
// must stop.  nlevels: number of levels; last_start: first position of the
// last level.  A level of wide_at nodes or more (0: none) hands the matrix to
// the level-synchronous engine.
// ---------------------------------------------------------------------------
template <int B, int EMAX, class TeamT>
__device__ bool bfs_pass(Smem<B, EMAX>& s, const MatrixView& M, TeamT& team, unsigned long long* agg,
                         uint32_t& step, const Options& opt, uint32_t start, uint32_t base, uint32_t wide_at,
                         bool sorted, bool write_perm, bool reverse, uint32_t& placed, uint32_t& nlevels,
                         uint32_t& last_start)
{
    Chunk<B, EMAX> ch{s, M, base};
    const uint32_t t = gtid<B>();
    const uint32_t G = team.size, R = team.rank;
    const uint32_t n = M.n;

    LevelState st;
    const uint4 sn = ld_node(M.node + start);
    const uint32_t rs0 = sn.y, deg0 = sn.z;
    st.a = 0;
    st.b = 1;
    st.Ka = 0;
    st.Kb = deg0;
    st.L = 0;
    st.last_start = 0;
    // CTA 0 places the start and claims its edges
    if (R == 0) {
        if (t == 0) {
            atomicMax(claim_ptr(M, start), base);
            __stcg(reinterpret_cast<uint4*>(M.rec), make_uint4(start, rs0, deg0, 0u));
            if (write_perm)
                M.perm[reverse ? n - 1 : 0] = start;
        }
        for (uint32_t k = t; k < deg0; k += B) {
            const uint32_t d = ld_ro(M.ci + rs0 + k);
            if (PB_CHECK(M.res, d < n, 110))
                atomicMax(claim_ptr(M, d), base - 1u - k);
        }
    }
    auto is_solo = [&](const LevelState& x) {
        return G == 1 || ((x.b - x.a) <= opt.solo_parents && (x.Kb - x.Ka) <= opt.solo_edges);
    };
    bool solo = is_solo(st);
    if (!solo) {
        if (!team.sync(2))
            return false;
    }
    // own: the next level's share [p_beg, p_end) is this CTA's own children;
    // carry: they are in shared memory, placed with edge base Kown
    bool own = false, carry = false;
    uint32_t p_beg = 0, p_end = 0, Kown = 0;
    while (true) {
        if (solo) {
            // ---- CTA 0 alone: chunk by chunk with running offsets ----------
            if (R == 0) {
                // carry: the frontier and its adjacency are still in shared
                // memory from the previous level (it fitted one chunk)
                carry = false;
                bool solo_fail = false;  // stop after handing the gate over
                while (true) {
                    uint32_t P = st.b, K = st.Kb;
                    bool next_carry = false;
                    if (carry) {
                        ch.form_from_children(st.Ka);
                        const Agg g = ch.collect(sorted, true);
                        ch.prefetch();
                        ch.place_and_claim(P, K, write_perm, reverse);
                        P += g.cnt;
                        K += g.esum;
                        next_carry = g.cnt > 0 && g.cnt <= (uint32_t)B && g.esum <= (uint32_t)EMAX &&
                                     s.npre == g.esum;
                        gsync<B>();
                    } else {
                        uint32_t p = st.a;
                        while (p < st.b) {
                            const uint32_t used = ch.form(p, st.b);
                            const bool single = p == st.a && used == st.b - st.a;
                            if (s.hub) {
                                const uint32_t r0 = s.peb[0] - st.Ka;
                                const Agg g = ch.hub_collect(r0, sorted);
                                ch.hub_place_and_claim(r0, g.cnt, P, K, write_perm, reverse);
                                P += g.cnt;
                                K += g.esum;
                            } else {
                                const Agg g = ch.collect(sorted);
                                if (single)
                                    ch.prefetch();
                                ch.place_and_claim(P, K, write_perm, reverse);
                                P += g.cnt;
                                K += g.esum;
                                next_carry = single && g.cnt > 0 && g.cnt <= (uint32_t)B &&
                                             g.esum <= (uint32_t)EMAX && s.npre == g.esum;
                            }
                            gsync<B>();
                            p += used;
                        }
                    }
                    carry = next_carry;
                    if (!team.block_ok()) {
                        solo_fail = true;
                        break;
                    }
                    const uint32_t tot = P - st.b;
                    if (tot == 0) {
                        st.a = st.b;  // an empty frontier marks the end of the pass
                        break;
                    }
                    st.last_start = st.b;
                    st.a = st.b;
                    st.b = P;
                    st.Ka = st.Kb;
                    st.Kb = K;
                    st.L += 1;
                    if (st.b > n) {
                        set_status(M.res, kErrCheck, 111);
                        solo_fail = true;
                        break;
                    }
                    if (G > 1)
                        team.beat();
                    if (!is_solo(st))
                        break;
                }
                if (G > 1) {
                    if (!team.gate_open(st, !solo_fail))
                        return false;
                } else if (solo_fail) {
                    return false;
                }
            } else {
                if (!team.gate_wait(st))
                    return false;
            }
            if (st.a == st.b)
                break;  // the pass ended during the solo run
            solo = false;
            carry = false;
            continue;
        }
        // ---- whole team ---------------------------------------------------
        // A CTA's children take consecutive positions, so as long as every
        // CTA's fit one chunk and cost no more than an equal share would,
        // each expands its own: they and their columns are still in shared
        // memory, which saves the level two of its six dependent round trips.
        // Else the level is split anew into equal runs of the queue.
        if (!own) {
            const uint32_t F = st.b - st.a;
            p_beg = st.a + (uint32_t)(((uint64_t)F * R) / G);
            p_end = st.a + (uint32_t)(((uint64_t)F * (R + 1)) / G);
        }
        // A1: collect and count.  A CTA whose parents take several chunks
        // stages each chunk's ranked children (M.stage, at the level-relative
        // edge offset of its first parent: the CTAs' regions are disjoint and
        // hold their children, which are at most their parents' edges), so
        // that placing them needs no second collect.
        uint32_t my_cnt = 0, my_esum = 0, nunits = 0;
        bool last_hub = false;
        bool staged = M.stage != nullptr;  // every unit staged (no hub among them)
        uint32_t stage_base = 0;
        uint32_t p = p_beg;
        if (carry && p < p_end) {
            ch.form_from_children(Kown);
            const Agg g = ch.collect(sorted, true);
            my_cnt = g.cnt;
            my_esum = g.esum;
            nunits = 1;
            p = p_end;
            gsync<B>();
        }
        while (p < p_end) {
            const uint32_t used = ch.form(p, p_end);
            if (nunits == 0)
                stage_base = s.peb[0] - st.Ka;
            Agg g;
            last_hub = s.hub != 0;
            if (last_hub) {
                g = ch.hub_collect(s.peb[0] - st.Ka, sorted);
                staged = false;
            } else {
                g = ch.collect(sorted);
                if (staged && !(nunits == 0 && used == p_end - p))
                    ch.stage_children(stage_base + my_cnt, my_esum);
            }
            my_cnt += g.cnt;
            my_esum += g.esum;
            ++nunits;
            p += used;
            gsync<B>();
        }
        // publish (level-tagged), then prefetch while the others finish
        ++step;
        team.ag_publish(my_cnt, my_esum, step, agg);
        const bool keep = nunits == 1 && !last_hub;
        if (keep)
            ch.prefetch();
        // all-gather of the per-CTA totals (a share costs by rounds of B edges:
        // own children while they take no more rounds than an equal share:
        // a 128^3 grid 5.60 ms with any share of one chunk, 5.37 so, 5.53
        // split anew every level)
        const uint32_t lim = min((uint32_t)EMAX, ((st.Kb - st.Ka) / G / (uint32_t)B + 1u) * (uint32_t)B);
        unsigned long long pre = 0, all = 0;
        bool over = false;
        if (!team.template ag_collect<B>(step, agg, lim, pre, all, over, s.gat64))
            return false;
        const uint32_t tot_cnt = (uint32_t)(all & 0xFFFFFFFFull);
        const uint32_t tot_esum = (uint32_t)(all >> 32);
        // (every CTA has the same totals and leaves)
        if (wide_at != 0 && tot_cnt >= wide_at) {
            if (R == 0 && t == 0)
                set_status(M.res, kNeedWide, 0);
            return false;
        }
        uint32_t P = st.b + (uint32_t)(pre & 0xFFFFFFFFull);
        uint32_t K = st.Kb + (uint32_t)(pre >> 32);
        const uint32_t p_old = p_beg, p_old_end = p_end;
        own = !over;
        carry = own && keep && s.npre == my_esum;
        Kown = K;
        p_beg = P;
        p_end = P + my_cnt;
        // A2: place (the only unit is still in shared memory, or all are staged)
        if (keep) {
            ch.place_and_claim(P, K, write_perm, reverse);
        } else if (nunits > 0 && staged) {
            ch.place_staged(stage_base, my_cnt, P, K, write_perm, reverse);
        } else if (nunits > 0) {
            p = p_old;
            while (p < p_old_end) {
                const uint32_t used = ch.form(p, p_old_end);
                if (s.hub) {
                    const uint32_t r0 = s.peb[0] - st.Ka;
                    const uint32_t q = __ldcg(ch.hk1() + r0);
                    const uint32_t qd = __ldcg(ch.hk1() + r0 + 1);
                    ch.hub_place_and_claim(r0, q, P, K, write_perm, reverse);
                    P += q;
                    K += qd;
                } else {
                    const Agg g = ch.collect(sorted);
                    ch.place_and_claim(P, K, write_perm, reverse);
                    P += g.cnt;
                    K += g.esum;
                }
                gsync<B>();
                p += used;
            }
        }
        if (!team.sync(5))
            return false;
        if (tot_cnt == 0)
            break;
        st.last_start = st.b;
        st.a = st.b;
        st.b += tot_cnt;
        st.Ka = st.Kb;
        st.Kb += tot_esum;
        st.L += 1;
        if (st.b > n) {
            set_status(M.res, kErrCheck, 112);
            return false;
        }
        solo = is_solo(st);
        own = own && !solo;
    }
    placed = st.b;
    nlevels = st.L + 1;
    last_start = st.last_start;
    return true;
}

// One breadth-first pass from `start`, unordered inside a level: what a
// start-search pass needs while its order does not matter (reorder_matrix).
// A node's first claim of the pass is the whole dedup.  Levels with a small
// frontier run on CTA 0 alone, as in bfs_pass, until one is too big; from
// then on the team works as follows.  A CTA keeps the children it claimed in
// shared memory and expands them itself in the next level, so a level is one
// round trip for the claims and one barrier, whose word also carries the
// level's totals and under which the next columns are loaded (the ordered
// pass: queue records, columns, node entries, all-gather, claims, barrier).
// When a CTA's share grows past a chunk it asks, in the same word, for a new
// split: all lists go to the queue behind an atomic counter and come back in
// equal runs.  Levels of more than 3/4 of a chunk a CTA go through the queue
// at once.
// Grid teams only; no row over EMAX.  first: the smallest key of this pass;
// base: its largest, the claim of every node.  The last level ends up at
// queue positions [last_start, placed).
template <int B, int EMAX>
__device__ bool level_pass(Smem<B, EMAX>& s, const MatrixView& M, Team& team, const Options& opt, uint32_t start,
                           uint32_t base, uint32_t first, uint32_t wide_at, uint32_t& slot, uint32_t& placed,
                           uint32_t& nlevels, uint32_t& last_start)
{
    Chunk<B, EMAX> ch{s, M, base};
    using List = typename Chunk<B, EMAX>::List;
    const uint32_t t = gtid<B>();
    const uint32_t G = team.size, R = team.rank, n = M.n;
    const uint4 sn = ld_node(M.node + start);
    LevelState st;
    st.a = 0;
    st.b = 1;
    st.Ka = 0;
    st.Kb = sn.z;  // Kb - Ka: entries of the frontier
    st.L = 0;
    st.last_start = 0;
    if (R == 0 && t == 0) {
        atomicMax(&M.node[start].claim, base);
        __stcg(reinterpret_cast<uint4*>(M.rec), make_uint4(start, sn.y, sn.z, 0u));
    }
    auto is_solo = [&](const LevelState& x) {
        return G == 1 || ((x.b - x.a) <= opt.solo_parents && (x.Kb - x.Ka) <= opt.solo_edges);
    };
    auto next_level = [&](uint32_t cnt, uint32_t esum) {
        st.last_start = st.b;
        st.a = st.b;
        st.b += cnt;
        st.Ka = st.Kb;
        st.Kb += esum;
        st.L += 1;
    };
    if (is_solo(st)) {
        bool ok = true;
        gsync<B>();
        if (R == 0) {
            uint32_t cur = 0, beat = 0;
            bool listed = false;  // the frontier is in list `cur`
            while (true) {
                const List P = ch.list(cur), out = ch.list(cur ^ 1u);
                uint32_t tail = st.b;  // queue positions taken
                Agg C{0, 0}, flushed{0, 0};
                auto flush = [&]() {
                    ch.place_list(out, tail, C.cnt);
                    tail += C.cnt;
                    flushed.esum += C.esum;
                    C = Agg{0, 0};
                    gsync<B>();
                };
                for (uint32_t p = st.a; p < st.b;) {
                    p += listed ? ch.form_list(P, p - st.a, st.b - st.a) : ch.form(p, st.b);
                    ch.collect_any(first, out, C, flush);
                }
                const uint32_t cnt = tail - st.b + C.cnt, esum = flushed.esum + C.esum;
                if (cnt == 0) {
                    if (listed) {
                        ch.place_list(P, st.a, st.b - st.a);
                        gsync<B>();
                    }
                    st.a = st.b;  // an empty frontier marks the end of the pass
                    break;
                }
                listed = tail == st.b;
                cur ^= 1u;
                next_level(cnt, esum);
                if (st.b > n) {
                    set_status(M.res, kErrCheck, 155);
                    ok = false;
                    break;
                }
                const bool stay = is_solo(st);
                if (!listed)
                    flush();
                else if (!stay)
                    ch.place_list(out, st.a, cnt);
                // the others' bounded wait, and an error posted elsewhere:
                // looked after every few levels
                if ((++beat & 7u) == 0) {
                    team.beat();
                    ok = team.block_ok();
                }
                if (!stay || !ok)
                    break;
            }
            gsync<B>();
            if (G > 1) {
                if (!team.gate_open(st, ok))
                    return false;
            } else if (!ok) {
                return false;
            }
        } else if (!team.gate_wait(st)) {
            return false;
        }
        if (st.a == st.b) {
            placed = st.b;
            nlevels = st.L + 1;
            last_start = st.last_start;
            return true;
        }
    } else if (!team.sync(2)) {
        return false;
    }
    // ---- the whole team
    constexpr int MAXEPT = Chunk<B, EMAX>::MAXEPT;
    uint32_t cur = 0, own = 0;
    bool listed = false;  // this CTA's share of the level is in list `cur` (own entries, one chunk)
    uint32_t col[MAXEPT];  // listed: the columns of its edges, on their way
    while (true) {
        const uint32_t F = st.b - st.a, E = st.Kb - st.Ka;
        const List P = ch.list(cur), out = ch.list(cur ^ 1u);
        Agg C{0, 0};
        bool split = false;  // some children are in the queue already
        auto flush = [&]() {
            if (C.cnt != 0) {
                if (t == 0)
                    s.bcast[0] = (uint32_t)atomicAdd(&team.gs->lvl[slot],
                                                     (unsigned long long)C.esum << 32 | C.cnt);
                gsync<B>();
                ch.place_list(out, st.b + s.bcast[0], C.cnt);
                gsync<B>();
            }
            C = Agg{0, 0};
            split = true;
        };
        // the children of this share go through the queue when the level
        // leaves no room for uneven shares, and a CTA asks for a new split
        // when its own next share would not fit one chunk (below that a share
        // costs the same whatever its size)
        const bool queue = E > G * (uint32_t)(EMAX / 4 * 3);
        auto too_big = [&](const Agg& g) { return g.cnt > (uint32_t)B || g.esum > (uint32_t)EMAX; };
        bool arrived = false;
        if (listed) {
            if (own != 0) {
                const bool alone = !queue;
                ch.claim_list(first, col, out, C, flush, [&](const Agg& g) {
                    if (alone)
                        team.level_arrive(g.cnt, g.esum, too_big(g));
                });
                arrived = alone;
            }
        } else {
            const uint32_t p_beg = st.a + (uint32_t)(((uint64_t)F * R) / G);
            const uint32_t p_end = st.a + (uint32_t)(((uint64_t)F * (R + 1)) / G);
            if (queue)
                ch.claim_wide(first, p_beg, p_end, out, C, st.b, &team.gs->lvl[slot]);
            else
                for (uint32_t p = p_beg; p < p_end;) {
                    p += ch.form(p, p_end);
                    ch.collect_any(first, out, C, flush);
                }
        }
        uint32_t cnt = 0, esum = 0;
        bool keep = false;
        if (!queue) {
            const bool ask = split || too_big(C);
            if (!arrived) {
                gsync<B>();
                team.level_arrive(C.cnt, C.esum, ask);
            }
            // the next level's columns while the others arrive
            if (!ask && C.cnt != 0) {
                ch.form_list(out, 0, C.cnt);
                ch.load_cols(col);
            }
            if (!team.level_wait(5, cnt, esum, keep))
                return false;
        }
        if (keep) {
            if (cnt == 0) {
                if (listed) {
                    // the last level to the queue, for the next start (the
                    // counter is next used behind another barrier)
                    if (own != 0) {
                        if (t == 0)
                            s.bcast[0] = (uint32_t)atomicAdd(&team.gs->lvl[slot], (unsigned long long)own);
                        gsync<B>();
                        ch.place_list(P, st.a + s.bcast[0], own);
                    }
                    if (!team.sync(9))
                        return false;
                    if (R == 0 && t == 0)
                        __stcg(&team.gs->lvl[slot], 0ull);
                }
                break;
            }
            listed = true;
            own = C.cnt;
            cur ^= 1u;
        } else {
            flush();
            if (!team.sync(13))
                return false;
            const unsigned long long all = __ldcg(&team.gs->lvl[slot]);
            cnt = (uint32_t)(all & 0xFFFFFFFFull);
            esum = (uint32_t)(all >> 32);
            // the counter of the level after next is free (everyone read it
            // before this barrier): cleared for it
            slot = slot == 2 ? 0 : slot + 1;
            if (R == 0 && t == 0)
                __stcg(&team.gs->lvl[slot == 2 ? 0 : slot + 1], 0ull);
            if (wide_at != 0 && cnt >= wide_at) {
                // a level this wide in the first pass: the level-synchronous
                // engine takes the matrix (every CTA has the same totals)
                if (R == 0 && t == 0)
                    set_status(M.res, kNeedWide, 0);
                return false;
            }
            if (cnt == 0)
                break;
            listed = false;
        }
        next_level(cnt, esum);
        if (st.b > n) {
            set_status(M.res, kErrCheck, 156);
            return false;
        }
    }
    placed = st.b;
    nlevels = st.L + 1;
    last_start = st.last_start;
    return true;
}

// Next start of the pseudo-peripheral search (simple_peripheral.cpp:110-127)
// from the ordered BFS just run: among the last min(outnodes, n-1) positions,
// those on the last level; the last of minimal valence.  Thread 0 computes.
__device__ __forceinline__ uint32_t next_peripheral_start(const MatrixView& M, uint32_t outnodes, uint32_t last_start)
{
    const uint32_t n = M.n;
    uint32_t lo = n - min(outnodes, n - 1);
    lo = max(lo, max(last_start, 1u));
    uint32_t best = 0, bestdeg = kUnvisited;
    for (uint32_t pos = lo; pos < n; ++pos) {
        const uint4 r = __ldcg(reinterpret_cast<const uint4*>(M.rec) + pos);
        if (r.z <= bestdeg) {
            bestdeg = r.z;
            best = r.x;
        }
    }
    return best;
}

// The node of minimal valence at positions [at, at + width), and how many have
// that valence (one warp).
__device__ __forceinline__ uint32_t unique_min_valence(const MatrixView& M, uint32_t at, uint32_t width, uint32_t& node)
{
    uint32_t d = kUnvisited, v = 0, same = 0;
    for (uint32_t i = threadIdx.x & 31u; i < width; i += 32) {
        const uint4 r = __ldcg(reinterpret_cast<const uint4*>(M.rec) + at + i);
        same = r.z < d ? 1u : same + (r.z == d ? 1u : 0u);
        if (r.z < d) {
            d = r.z;
            v = r.x;
        }
    }
    const uint32_t dm = __reduce_min_sync(kFull, d);
    node = __shfl_sync(kFull, v, __ffs(__ballot_sync(kFull, d == dm)) - 1);
    return __reduce_add_sync(kFull, d == dm ? same : 0u);
}

// Fills the node table (claim 0, row start, valence) of the matrix.
template <int B>
__device__ void init_nodes(const MatrixView& M, uint32_t R, uint32_t G)
{
    for (uint64_t v = (uint64_t)R * B + gtid<B>(); v < M.n; v += (uint64_t)G * B) {
        const uint32_t a = ld_ro(M.rp + v), e = ld_ro(M.rp + v + 1);
        __stcg(reinterpret_cast<uint4*>(M.node) + v, make_uint4(0u, a, e - a, 0u));
    }
}

// ---------------------------------------------------------------------------
// Full reorder of one matrix by one team: start search, final ordered pass,
// bandwidth.  Every CTA of the team runs this; CTA 0 thread 0 writes *res.
// ---------------------------------------------------------------------------
template <int B, int EMAX, class TeamT>
__device__ void reorder_matrix(Smem<B, EMAX>& s, const MatrixView& M, TeamT& team, unsigned long long* agg,
                               const Options& opt)
{
    const uint32_t t = gtid<B>();
    const uint32_t n = M.n;
    const uint32_t G = team.size, R = team.rank;
    uint32_t start = opt.start;
    uint32_t passes = 0, ecc = 0, placed = 0, nlevels = 0, last_start = 0;
    uint32_t step = 0, slot = 0;

    if (start != kUnvisited && start >= n) {
        if (R == 0 && t == 0)
            set_status(M.res, kErrArg, 2);
        return;
    }
    if (R == 0 && t == 0)
        M.res->t_begin = globaltimer();
    init_nodes<B>(M, R, G);
    if (!team.sync(1))
        return;
    // pass keys: pass p owns [p*kspan, p*kspan + nnz + 1]
    const uint32_t kspan = M.nnz + 2u;
    const uint32_t pmax = (uint32_t)(0xFFFFFFFFull / kspan) - 1u;
    uint32_t pass_id = 0;

    // pseudo-peripheral search (simple_peripheral.cpp:92-141), then the
    // degree-sorted pass that writes the permutation.
    //
    // A search pass has to deliver its level count and the next start, and
    // that start -- the last node of minimal valence among the last outnodes
    // discovered, on the last level -- does not depend on the order when the
    // last level has at most outnodes nodes and one of them alone has the
    // minimal valence.  So the search runs unordered (level_pass, about half
    // the time of an ordered level) and only repeats a pass in discovery
    // order where that fails: never on 5- and 7-point grids, which end in a
    // corner, about a third of the passes of random geometric graphs, every
    // pass on wider stencils (wide_stencil), which therefore begin in discovery
    // order.  A pass after a repeated one is ordered at once too, until one
    // would not have had to be (strips of 25-point stencils, 1,001 levels:
    // 24.2 ms with every pass tried unordered, 18.8 so).  From the third pass
    // on, which usually confirms the
    // eccentricity, the search pass is the sorted pass itself and its order
    // the result if it does.  (Matrices with rows over EMAX and cluster teams
    // search in discovery order.)
    enum : uint32_t { kLevels, kFifo, kSorted };
    const bool any_order = TeamT::kGrid && G <= 255u && __ldcg(&M.res->maxdeg) <= (uint32_t)EMAX;
    const bool full = opt.mode != kModeStartOnly;
    bool searching = start == kUnvisited && n > 1;
    bool repeat = false;  // this pass repeats the last one in discovery order
    uint32_t kind = kSorted, lastdist = 0;
    if (n == 1) {
        // one node: the start search runs one pass and records nothing
        passes = start == kUnvisited ? 1 : 0;
        start = 0;
    } else if (searching) {
        start = n / 2;
        passes = 1;
        kind = any_order && !wide_stencil(n, M.nnz, __ldcg(&M.res->maxdeg)) ? kLevels : kFifo;
    }
    while (searching || full) {
        if (pass_id + 1 > pmax) {
            for (uint64_t v = (uint64_t)R * B + t; v < n; v += (uint64_t)G * B)
                M.node[v].claim = 0u;
            pass_id = 0;
            if (!team.sync(7))
                return;
        }
        ++pass_id;
        const uint32_t base = pass_id * kspan + M.nnz + 1u;
        const uint32_t wide_at = passes <= 1 && G == gridDim.x ? opt.wide_at : 0u;
        // (one call site of each pass: they are large when inlined)
        if (kind == kLevels) {
            if constexpr (TeamT::kGrid) {
                if (!level_pass<B, EMAX>(s, M, team, opt, start, base, pass_id * kspan, wide_at, slot, placed,
                                         nlevels, last_start))
                    return;
            }
        } else {
            if (!bfs_pass<B, EMAX>(s, M, team, agg, step, opt, start, base, wide_at, kind == kSorted,
                                   kind == kSorted, kind == kSorted && opt.reverse != 0, placed, nlevels, last_start))
                return;
        }
        const uint32_t dist = nlevels - 1;
        const bool confirmed = dist == lastdist && !repeat;
        uint32_t next = 0;
        bool unique = false;
        if (!end_pass(team, [&]() {
                if (!searching || placed != n || confirmed)
                    return;
                // the next start
                const uint32_t width = n - last_start;
                if (t < 32) {
                    uint32_t v = 0, count = 0;
                    if (width <= min(opt.outnodes, n - 1))
                        count = unique_min_valence(M, last_start, width, v);
                    if (t == 0) {
                        s.bcast[0] = kind == kFifo ? next_peripheral_start(M, opt.outnodes, last_start) : v;
                        s.bcast[1] = count == 1u ? 1u : 0u;
                    }
                }
                gsync<B>();
                next = s.bcast[0];
                unique = s.bcast[1] != 0u;
                gsync<B>();
            }))
            return;
        if (!searching)
            break;
        if (placed != n) {
            if (R == 0 && t == 0)
                set_status(M.res, kErrDisconnected, 0);
            return;
        }
        if (confirmed) {
            ecc = dist;
            searching = false;
            if (kind == kSorted)
                break;  // confirmed by the sorted pass: the result
            kind = kSorted;  // the sorted pass from the same start comes next
            continue;
        }
        repeat = kind != kFifo && !unique;
        if (repeat) {
            kind = kFifo;
            continue;
        }
        start = next;
        lastdist = dist;
        if (passes > n) {  // eccentricities only grow; cannot happen on a valid run
            if (R == 0 && t == 0)
                set_status(M.res, kErrCheck, 3);
            return;
        }
        ++passes;
        kind = passes >= 3 && full ? kSorted : any_order && unique ? kLevels : kFifo;
    }
    if (opt.mode == kModeStartOnly) {
        if (R == 0 && t == 0) {
            M.res->start = start;
            M.res->passes = passes;
            M.res->ecc = ecc;
            M.res->placed = n;
        }
        return;
    }
    if (placed != n) {
        if (R == 0 && t == 0) {
            set_status(M.res, kErrDisconnected, 1);
            M.res->placed = placed;
        }
        return;
    }
    if (opt.want_bw) {
        // inverse permutation (CM positions) into node[].inv
        for (uint64_t pos = (uint64_t)R * B + t; pos < n; pos += (uint64_t)G * B) {
            const uint4 r = __ldcg(reinterpret_cast<const uint4*>(M.rec) + pos);
            M.node[r.x].inv = (uint32_t)pos;
        }
        if (!team.sync(6))
            return;
        unsigned long long bw = 0, bw0 = 0, plo = 0, phi = 0;
        for (uint64_t i = (uint64_t)R * B + t; i < n; i += (uint64_t)G * B) {
            const uint32_t a = ld_ro(M.rp + i), e = ld_ro(M.rp + i + 1);
            if (a == e)
                continue;
            const uint32_t me = __ldcg(&M.node[i].inv);
            uint32_t mnr = kUnvisited, mxr = 0;
            for (uint32_t k = a; k < e; ++k) {
                const uint32_t p = __ldcg(&M.node[ld_ro(M.ci + k)].inv);
                mnr = min(mnr, p);
                mxr = max(mxr, p);
            }
            // computeBandwidth (main.cpp:143-184): max(row - min, max - row), >= 0
            const unsigned long long b1 = me >= mnr ? (unsigned long long)(me - mnr) : 0ull;
            const unsigned long long b2 = mxr >= me ? (unsigned long long)(mxr - me) : 0ull;
            bw = max(bw, max(b1, b2));
            // profile of the CM order (row - min col) and of its reverse (max col - row)
            plo += b1;
            phi += b2;
            // initial bandwidth: first / last stored column (main.cpp:114-129)
            const uint32_t c0 = ld_ro(M.ci + a), c1 = ld_ro(M.ci + e - 1);
            const unsigned long long i0 = i >= c0 ? i - c0 : 0, i1 = c1 >= i ? c1 - i : 0;
            bw0 = max(bw0, max(i0, i1));
        }
        bw = block_reduce_max<B, unsigned long long>(bw, s.tmp64);
        bw0 = block_reduce_max<B, unsigned long long>(bw0, s.tmp64);
        block_reduce_sum2<B>(plo, phi, s.tmp64);
        if (t == 0) {
            atomicMax(&M.res->bandwidth, bw);
            atomicMax(&M.res->initial_bw, bw0);
            atomicAdd(&M.res->profile_lo, plo);
            atomicAdd(&M.res->profile_hi, phi);
        }
    }
    if (R == 0 && t == 0) {
        M.res->start = start;
        M.res->passes = passes;
        M.res->ecc = ecc;
        M.res->levels = nlevels;
        M.res->placed = placed;
        M.res->t_end = globaltimer();
    }
}

// ---------------------------------------------------------------------------
// CSR check of one matrix by one thread group (the batch kernels; the
// single-matrix path runs k_validate over the whole GPU instead): rows
// ordered and inside [0, nnz], every column below n, and the largest valence
// (decides whether hub scratch is needed) into res->maxdeg.  Coalesced.
template <int B>
__device__ void validate_group(const MatrixView& M, uint32_t* red)
{
    const uint32_t t = gtid<B>();
    uint32_t mx = 0;
    bool bad = false;
    for (uint32_t i = t; i < M.n; i += B) {
        const uint32_t a = ld_ro(M.rp + i), b = ld_ro(M.rp + i + 1);
        if (b < a || b > M.nnz)
            bad = true;
        else
            mx = max(mx, b - a);
    }
    if (t == 0 && (ld_ro(M.rp) != 0 || ld_ro(M.rp + M.n) != M.nnz))
        bad = true;
#pragma unroll 4
    for (uint32_t k = t; k < M.nnz; k += B)
        if (ld_ro(M.ci + k) >= M.n)
            bad = true;
    if (bad)
        set_status(M.res, kErrArg, 200);
    mx = block_reduce_max<B, uint32_t>(mx, red);
    if (t == 0)
        atomicMax(&M.res->maxdeg, mx);
    gsync<B>();
}

// validate_group without the column pass: row pointers and the largest
// valence (the solo batch kernel tests the columns while it builds the edge
// records, solo_build_edges).
template <int B>
__device__ void validate_rows(const MatrixView& M, uint32_t* red)
{
    const uint32_t t = gtid<B>();
    uint32_t mx = 0;
    bool bad = false;
    for (uint32_t i = t; i < M.n; i += B) {
        const uint32_t a = ld_ro(M.rp + i), b = ld_ro(M.rp + i + 1);
        if (b < a || b > M.nnz)
            bad = true;
        else
            mx = max(mx, b - a);
    }
    if (t == 0 && (ld_ro(M.rp) != 0 || ld_ro(M.rp + M.n) != M.nnz))
        bad = true;
    if (bad)
        set_status(M.res, kErrArg, 200);
    mx = block_reduce_max<B, uint32_t>(mx, red);
    if (t == 0)
        atomicMax(&M.res->maxdeg, mx);
    gsync<B>();
}

// Bounded wait of a thread group for a matrix's CSR to arrive (the word
// `ready` is written by a host-to-device copy after the CSR's copies).  A
// wait that runs out posts PBRCM_ERR_TIMEOUT for the matrix.  The word is
// read with acquire semantics; the CSR's lines are read only afterwards, and
// no other matrix shares them (every CSR starts on a 128-byte boundary).
template <int B>
__device__ void wait_ready(const uint32_t* ready, unsigned long long wait_ns, DevResult* res, int* flag)
{
    if (gtid<B>() == 0) {
        int ok = 1;
        unsigned long long t0 = 0;
        uint32_t spins = 0;
        while (ld_acquire(ready) == 0u) {
            if ((++spins & 63u) == 0) {
                const unsigned long long now = globaltimer();
                if (t0 == 0) {
                    t0 = now;
                } else if (now - t0 > wait_ns) {
                    set_status(res, kErrTimeout, 210);
                    ok = 0;
                    break;
                }
            }
            __nanosleep(spins > 4096 ? 1024 : 128);
        }
        *flag = ok;
    }
    gsync<B>();
}

// ---------------------------------------------------------------------------
// Early exits shared by the reorder kernels.  Returns true if the matrix must
// not be processed.  Every CTA reads the same values, so all agree.
template <int EMAX>
__device__ __forceinline__ bool skip_matrix(const MatrixView& M, bool first_thread)
{
    if (read_status(M.res) != 0)
        return true;
    if (__ldcg(&M.res->maxdeg) > (uint32_t)EMAX && M.hub == nullptr) {
        if (first_thread)
            set_status(M.res, kNeedHub, 0);
        return true;
    }
    return false;
}

}  // namespace pbrcm
