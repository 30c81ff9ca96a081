// Searches of low-degree graphs (lattices, road networks: no list of more than
// LOW_DEGREE edges), depth labels: one kernel for every strategy.
//
// Such a search is a chain of hundreds or thousands of small levels, and its
// time is the latency of a level: the dependent round trips of its body and
// the barrier that ends it.  Both are kept as short as the hardware allows:
//   * The frontier holds the vertices discovered by the level before, each
//     with its row range (start, and the list length in the top bits of the
//     id), so a level's chain is entry -> column entries -> visited-mask claims
//     with the claimed vertices' row offsets behind them -> append.  A thread
//     takes one vertex and its whole list at once.  (An edge frontier holds
//     every edge and claims a level later; a plain vertex frontier reads the
//     row range as one more round trip.)
//   * Levels of a few thousand vertices run on ONE thread-block cluster with
//     the frontier in distributed shared memory.  Each CTA deals its
//     discoveries out to the cluster's CTAs in turn, into the region of the
//     receiver's queue that belongs to the sender, so no reservation leaves
//     the CTA, and every receiver gets an even share.  There is no barrier at
//     the level's end: the entries and counts travel as st.async, and a CTA
//     goes on when its mbarrier has the arrivals and bytes of every sender: no
//     release waits for the level's label stores and no acquire drops the L1
//     lines the next level reads (the wait is 250 of a level's 2400 cycles).
//   * Larger levels run on the whole grid, frontier in global memory.  A CTA
//     takes a contiguous share of it and writes what it discovers to a segment
//     of its own, publishing the count; after the grid barrier every CTA scans
//     the counts.  No reservation is in the chain, and because shares and
//     segments keep their order, an SM stays in its part of the graph (its
//     address translations and cache lines) from level to level.
// The kernel changes between the two as the frontier grows and shrinks.
// Contract-expand, a search: 1024^2 lattice 7.43 -> 2.2 ms (1.5 us a level),
// 256^3 lattice 4.4 -> 3.96 ms (4.6 us a level of 3,000 vertices, 8 us of 55,000:
// its column, row-offset and label sectors come from DRAM), 100^3 1.13 -> 0.81 ms.
//
// The strategies differ only in what they report (search depth, total_queued,
// the level log); see Account.  The reference's level loops are cited there.

#include <cuda_runtime.h>

#include <algorithm>

#include "bfs_kernels.cuh"

namespace b40c_b200 {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int THREADS = 512;
constexpr int WARPS = THREADS / 32;
constexpr int LEN_SHIFT = 27;  // list length above, vertex id below (nodes < 2^27)
static_assert(LOW_DEGREE <= 16, "a list has a group of at most 16 lanes; its length takes 5 bits");
constexpr unsigned ID_MASK = (1u << LEN_SHIFT) - 1u;
// Vertices a CTA may discover in one level on the cluster: its regions in the
// receivers' queues hold DEAL / TEAM entries each.
constexpr int DEAL = 2048;
// Levels on the cluster between two grid barriers, so that the waiting CTAs'
// time limit counts about a millisecond of them.
constexpr int CLUSTER_LEVELS = 1024;

template <int TEAM>
struct Smem {
    union {
        int2 region[2][TEAM][DEAL / TEAM];  // cluster: frontier entries dealt by each CTA, by level parity
        int2 stage[2 * DEAL];               // grid: this CTA's discoveries, until it reserves room for them
    };
    uint2 count[2][TEAM];        // what each CTA discovered: vertices, their edges
    unsigned long long full[2];  // mbarriers: region[b] and count[b] have landed
    unsigned found[2], edges[2];  // this CTA's discoveries of the level
    unsigned base;               // compact grid level: this CTA's room in the queue
    unsigned prefix[THREADS + 1];  // grid level: frontier entries of the segments before each
    unsigned warp_n[WARPS], warp_e[WARPS];
    unsigned first;              // the segment this CTA's share starts in
    int it;                      // after the cluster's levels: the level
    unsigned flag;               // after a grid barrier: the error word
};

__device__ __forceinline__ bool leader() { return blockIdx.x == 0 && threadIdx.x == 0; }

__device__ __forceinline__ void put_record(const BfsParams &p, int idx, unsigned frontier, bool instant) {
    if (p.levels && idx < p.level_cap) {
        LevelRecord r;
        r.t_start = globaltimer_ns();
        r.frontier = frontier;
        r.chunks = r.wchunks = r.bottom_up = 0u;
        if (instant) r.t_work_end = r.t_start;
        p.levels[idx] = r;
    }
}

// What the strategies report for a search that runs as vertex levels: step it
// expands the nf vertices of depth it (mf edges) and discovers depth it + 1.
//   * expand-contract: level it's frontier is the nf vertices; iteration it at
//     the end (enactor_expand_contract.cuh:258-373).
//   * contract-expand, hybrid: level it + 1's frontier is the mf edges, level
//     0's the source; a level that finds nothing new counts
//     (enactor_contract_expand.cuh:259-407).
//   * two-phase: as contract-expand, each level's vertices logged as well; a
//     contract that finds nothing ends the search uncounted
//     (enactor_two_phase.cuh:416-596).
struct Account {
    int strategy;
    int last = -1;  // log record whose work the current step is
    unsigned long long queued = 0;

    __device__ __forceinline__ void step(const BfsParams &p, int it, unsigned nf, unsigned mf) {
        if (strategy == STRATEGY_EXPAND_CONTRACT) {
            queued += nf;
            last = it;
            put_record(p, it, nf, false);
        } else {
            const bool two = strategy == STRATEGY_TWO_PHASE;
            if (it == 0) {
                queued += 1;
                put_record(p, 0, 1u, true);
            }
            if (two) put_record(p, 2 * it + 1, nf, true);
            last = -1;
            if (mf) {
                queued += mf;
                last = two ? 2 * it + 2 : it + 1;
                put_record(p, last, mf, false);
            }
        }
    }
    __device__ __forceinline__ void work_end(const BfsParams &p) const {
        if (p.levels && last >= 0 && last < p.level_cap) p.levels[last].t_work_end = globaltimer_ns();
    }
    // it: the first depth without vertices; mf: the edges of the depth before.
    __device__ __forceinline__ void finish(const BfsParams &p, int it, unsigned mf) const {
        const bool extra = (strategy == STRATEGY_CONTRACT_EXPAND || strategy == STRATEGY_HYBRID) && mf != 0u;
        p.ctr->total_queued = queued;
        p.ctr->iteration = it + (extra ? 1 : 0);
        put_record(p, strategy == STRATEGY_TWO_PHASE ? 2 * it + 2 : p.ctr->iteration, 0u, false);
        atomicOr(&p.ctr->sticky, ld_relaxed_gpu(&p.ctr->error));
    }
};

// ---- data between the CTAs of a cluster -------------------------------------------
__device__ __forceinline__ unsigned map_rank(const void *p, unsigned rank) {  // shared::cluster address
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// An 8-byte store into another CTA's shared memory that counts its bytes on
// that CTA's mbarrier.
__device__ __forceinline__ void send8(unsigned to, unsigned bar, int2 v) {
    const unsigned long long x = (unsigned)v.x | ((unsigned long long)(unsigned)v.y << 32);
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to), "l"(x),
                 "r"(bar)
                 : "memory");
}
// This CTA's arrival at another CTA's mbarrier, after `bytes` sent to it.
// Relaxed: what the receiver reads is ordered by the bytes' own completion.
__device__ __forceinline__ void arrive_remote(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Waits, within wait_ns, for the phase of the given parity.
__device__ __forceinline__ bool wait_full(const BfsParams &p, unsigned long long *bar, unsigned parity) {
    unsigned ok = 0;
    unsigned long long t0 = 0;
    for (;;) {
        asm volatile(
            "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, "
            "q;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        else if (t - t0 > p.wait_ns) return false;
    }
}

// One edge per lane and element u: lane j of a vertex's group takes entry j of
// its list (bit u of have: there is one; at[u]: its column position).  Claims
// the neighbours for depth `label`; bit u of the result: this lane got it, its
// frontier entry in e[u].  The U column loads go out together, then the U
// claims.  eager: the row offsets of every neighbour are loaded behind the
// claims, one round trip less; else only the claimed ones', a sixth of the
// requests on a 3D lattice.
template <int U, bool EAGER>
__device__ __forceinline__ unsigned claim(const BfsParams &p, unsigned have, const int (&at)[U], int label,
                                          int2 (&e)[U]) {
    int x[U], r0[U], r1[U];
    unsigned old[U], ok = 0, got = 0;
#pragma unroll
    for (int u = 0; u < U; u++) x[u] = (have >> u) & 1u ? __ldg(p.col + at[u]) : -1;
#pragma unroll
    for (int u = 0; u < U; u++)
        if ((unsigned)x[u] < (unsigned)p.nodes) ok |= 1u << u;
    unsigned seen[U];
#pragma unroll
    for (int u = 0; u < U; u++)
        seen[u] = !EAGER && ((ok >> u) & 1u) ? __ldca(p.mask + ((unsigned)x[u] >> 5)) : ~0u;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const unsigned bit = 1u << ((unsigned)x[u] & 31u);
        old[u] = bit;
        r0[u] = r1[u] = 0;
        if (EAGER ? (ok >> u) & 1u : !(seen[u] & bit)) {
            old[u] = atomicOr(p.mask + ((unsigned)x[u] >> 5), bit);
            if (EAGER) {
                r0[u] = __ldg(p.row_offsets + x[u]);
                r1[u] = __ldg(p.row_offsets + x[u] + 1);
            }
        }
    }
    if (have != ok) atomicOr(&p.ctr->error, ERR_BAD_VERTEX);
#pragma unroll
    for (int u = 0; u < U; u++)
        if (!(old[u] & (1u << ((unsigned)x[u] & 31u)))) got |= 1u << u;
    if (!EAGER) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            if ((got >> u) & 1u) {
                r0[u] = __ldg(p.row_offsets + x[u]);
                r1[u] = __ldg(p.row_offsets + x[u] + 1);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        if ((got >> u) & 1u) p.labels[x[u]] = label;
        e[u] = make_int2(int((unsigned)x[u] | (unsigned(r1[u] - r0[u]) << LEN_SHIFT)), r0[u]);
    }
    return got;
}

// Places for the warp's claimed entries among the CTA's discoveries of the
// level (sm.found / sm.edges [b]); called by all lanes together.
template <int TEAM, int U>
__device__ __forceinline__ void place(Smem<TEAM> &sm, int b, unsigned got, const int2 (&e)[U], unsigned (&at)[U]) {
    const unsigned lt = lanemask_lt();
    unsigned total = 0, edges = 0, base = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const unsigned m = __ballot_sync(FULL, (got >> u) & 1u);
        at[u] = total + __popc(m & lt);
        total += __popc(m);
        edges += (got >> u) & 1u ? (unsigned)e[u].x >> LEN_SHIFT : 0u;
    }
    if (total == 0u) return;  // warp-uniform
    if (lane_id() == 0) base = atomicAdd(&sm.found[b], total);
    edges = __reduce_add_sync(FULL, edges);
    if (lane_id() == 0) atomicAdd(&sm.edges[b], edges);
    base = __shfl_sync(FULL, base, 0);
#pragma unroll
    for (int u = 0; u < U; u++) at[u] += base;
}

// The grid barrier of bfs_device.cuh with the level cluster 0 left off at
// (Counters::cur_it) read behind it.  Polls back off further: a CTA may wait
// for a thousand levels of cluster 0.
template <int TEAM>
__device__ __forceinline__ bool grid_sync(const BfsParams &p, Smem<TEAM> &sm) {
    Counters *c = p.ctr;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long arrived = atom_add_acqrel_gpu_u64(&c->bar_total, 1ull);
        const unsigned long long target = (arrived / gridDim.x + 1ull) * gridDim.x;
        if (arrived + 1ull != target) {
            const unsigned long long t0 = globaltimer_ns();
            for (unsigned polls = 0; ld_acquire_gpu_u64(&c->bar_total) < target; polls++) {
                if (ld_relaxed_gpu(&c->error) != 0u) break;
                const unsigned long long waited = globaltimer_ns() - t0;
                if (waited > p.wait_ns) {
                    atomicOr(&c->error, ERR_BARRIER_TIMEOUT);
                    break;
                }
                if (waited > 20000ull) __nanosleep(500);
            }
        }
        sm.it = __ldcg(&c->cur_it);
        sm.flag = ld_relaxed_gpu(&c->error);
    }
    __syncthreads();
    return sm.flag == 0u;
}

// What every CTA knows of the level: its frontier's size and edges, and where
// the entries are: at their index (compact), or in the segments the CTAs of
// the level before wrote, segment c from share(before, c) * max_degree.
struct Level {
    int it;
    unsigned nf, mf, before;
    bool compact;
};

// Start of CTA c's share of n entries.
__device__ __forceinline__ unsigned share(unsigned n, unsigned c) {
    return unsigned((unsigned long long)n * c / gridDim.x);
}

// Reads the counts the CTAs published for level v.it: the frontier's totals,
// and for segments the prefix sums and the segment this CTA's share starts in.
template <int TEAM>
__device__ __forceinline__ void read_level(const LowDegreeParams &a, Smem<TEAM> &sm, Level &v) {
    const unsigned t = threadIdx.x, lane = lane_id(), warp = t >> 5;
    const uint2 n = t < gridDim.x ? __ldcg(a.counts + (v.it & 1) * THREADS + t) : make_uint2(0u, 0u);
    const unsigned incl = unsigned(warp_inclusive_scan(int(n.x))), e = __reduce_add_sync(FULL, n.y);
    if (lane == 31u) {
        sm.warp_n[warp] = incl;
        sm.warp_e[warp] = e;
    }
    __syncthreads();
    const unsigned wn = lane < WARPS ? sm.warp_n[lane] : 0u, we = lane < WARPS ? sm.warp_e[lane] : 0u;
    v.nf = __reduce_add_sync(FULL, wn);
    v.mf = __reduce_add_sync(FULL, we);
    const unsigned upto = __reduce_add_sync(FULL, lane < warp ? wn : 0u) + incl;
    sm.prefix[t + 1u] = upto;
    if (t == 0) sm.prefix[0] = 0u;
    const unsigned lo = share(v.nf, blockIdx.x);
    if (n.x && upto - n.x <= lo && lo < upto) sm.first = t;
    __syncthreads();
}

// Rounds [r0, r1) of a CTA's share [lo, hi) of a grid level, U in flight together.
template <int TEAM, int G, int U, bool EAGER>
__device__ __forceinline__ void grid_rounds(const BfsParams &p, const LowDegreeParams &a, Smem<TEAM> &sm,
                                            const Level &v, unsigned lo, unsigned hi, unsigned r0, unsigned r1) {
    constexpr unsigned VPR = THREADS / G;  // vertices per round of the CTA
    const int *q_in = p.queue[v.it & 1], *s_in = a.starts[v.it & 1];
    const unsigned j = threadIdx.x % G;
    for (unsigned r = r0; r < r1; r += U) {
        int col[U];
        unsigned have = 0, at[U], pos[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned i = lo + (r + u) * VPR + threadIdx.x / G;
            pos[u] = i < hi ? i : ~0u;
            if (!v.compact && i < hi) {
                unsigned seg = sm.first;
                while (i >= sm.prefix[seg + 1u]) seg++;
                pos[u] = share(v.before, seg) * unsigned(a.max_degree) + (i - sm.prefix[seg]);
            }
        }
        unsigned w[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            w[u] = pos[u] != ~0u ? (unsigned)ld_cg(q_in + pos[u]) : 0u;
            col[u] = pos[u] < a.starts_cap ? ld_cg(s_in + pos[u]) : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (pos[u] >= a.starts_cap && pos[u] != ~0u) col[u] = __ldg(p.row_offsets + (w[u] & ID_MASK));
            if (j < w[u] >> LEN_SHIFT) have |= 1u << u;
            col[u] += int(j);
        }
        int2 e[U];
        const unsigned got = claim<U, EAGER>(p, have, col, v.it + 1, e);
        place(sm, 0, got, e, at);
#pragma unroll
        for (int u = 0; u < U; u++)
            if ((got >> u) & 1u) sm.stage[at[u]] = e[u];
    }
}

// One level on the whole grid.  A CTA stages its discoveries in shared memory
// and writes them to its segment; when the segments (max_degree entries for
// each entry of the shares) would not fit the queue, or one batch the stage,
// to compact room reserved by an atomicAdd per batch.  Returns whether the
// next frontier is compact.
template <int TEAM, int G>
__device__ __forceinline__ bool grid_level(const BfsParams &p, const LowDegreeParams &a, Smem<TEAM> &sm,
                                           const Level &v) {
    constexpr unsigned VPR = THREADS / G;             // vertices per round of the CTA
    constexpr unsigned BATCH = 2 * DEAL / THREADS;    // rounds that fit the stage
    static_assert(BATCH % 4 == 0, "a batch is whole groups of the rounds in flight together");
    int *q_out = p.queue[(v.it + 1) & 1], *s_out = a.starts[(v.it + 1) & 1];
    const unsigned lo = share(v.nf, blockIdx.x), hi = share(v.nf, blockIdx.x + 1u);
    const unsigned rounds = (hi - lo + VPR - 1u) / VPR;
    const bool compact = ((long long)v.nf + gridDim.x) * a.max_degree > p.qcap ||
                         v.nf / gridDim.x + 1u > BATCH * VPR;  // every CTA alike
    unsigned wrote = 0, edges = 0;
    for (unsigned r0 = 0; r0 == 0 || r0 < rounds; r0 += BATCH) {  // CTA-uniform
        if (rounds == 1u) grid_rounds<TEAM, G, 1, true>(p, a, sm, v, lo, hi, 0u, 1u);
        else grid_rounds<TEAM, G, 4, false>(p, a, sm, v, lo, hi, r0, min(rounds, r0 + BATCH));
        __syncthreads();
        const unsigned total = sm.found[0];
        edges += sm.edges[0];
        unsigned base = lo * unsigned(a.max_degree);
        if (compact) {
            if (threadIdx.x == 0 && total) sm.base = atomicAdd(&p.ctr->qlen[(v.it + 1) & 3], total);
            __syncthreads();
            base = sm.base;
        }
        for (unsigned k = threadIdx.x; k < total; k += THREADS) {
            const unsigned pos = base + k;
            if ((long long)pos < p.qcap) {
                q_out[pos] = sm.stage[k].x;
                if (pos < a.starts_cap) s_out[pos] = sm.stage[k].y;
            } else {
                atomicOr(&p.ctr->error, ERR_OVERFLOW);
            }
        }
        wrote += total;
        __syncthreads();
        if (threadIdx.x == 0) sm.found[0] = sm.edges[0] = 0u;
        if (r0 + BATCH < rounds) __syncthreads();
    }
    if (threadIdx.x == 0) a.counts[((v.it + 1) & 1) * THREADS + blockIdx.x] = make_uint2(wrote, edges);
    return compact;
}

// Whether a frontier of nf vertices goes to the cluster: at most PASSES passes
// of its lanes (a pass takes about 1.1 us, the smallest grid level 4.6), and a
// CTA's share (even, but for up to one entry per sender) can then discover at
// most DEAL vertices.
constexpr unsigned PASSES = 3;
template <int TEAM, int G>
__device__ __forceinline__ bool on_cluster(unsigned nf) {
    static_assert((PASSES * THREADS / G + TEAM) * G <= DEAL, "the regions hold what a level discovers");
    return nf <= PASSES * TEAM * (THREADS / G);
}

// The queue a strategy's frontier would be in overflows (csr_problem.cuh:600-641
// sizes it): edges for the edge-frontier strategies, vertices otherwise.
__device__ __forceinline__ bool overflows(const BfsParams &p, const LowDegreeParams &a, unsigned nf, unsigned mf) {
    const long long n = a.strategy == STRATEGY_EXPAND_CONTRACT ? (long long)nf : (long long)mf;
    return n > p.qcap || (long long)nf > p.qcap;
}

// Levels on cluster 0, from the frontier v until it is too large, empty, or
// CLUSTER_LEVELS levels ran.  Leaves the frontier in global memory, its counts
// published and the level in Counters::cur_it.  Every CTA leaves on the same counts.  phase: the parity each
// mbarrier completes next.
template <int TEAM, int G>
__device__ __forceinline__ void cluster_levels(const BfsParams &p, const LowDegreeParams &a, Smem<TEAM> &sm,
                                               Account &acct, unsigned &phase, const Level &v, unsigned &mf_before) {
    int it = v.it;
    unsigned nf = v.nf, mf = v.mf;
    const unsigned r = blockIdx.x, lane = lane_id(), here = smem_u32(&sm);
    // Groups of G lanes take the regions' entries in turn, row by row: the
    // regions hold about the same number of entries, so the first warps'
    // groups fill up and the other warps have nothing to issue.
    constexpr unsigned STEP = THREADS / G / TEAM;
    const unsigned group = threadIdx.x / G, j = threadIdx.x % G;
    const unsigned s = group % TEAM, row = group / TEAM;
    Counters *c = p.ctr;
    // Deal the frontier out as if one CTA had: entry i to CTA i % TEAM, there
    // to region (i / TEAM) % TEAM.
    unsigned mine = 0;  // entries in this group's region
    {
        const int *q_in = p.queue[it & 1], *s_in = a.starts[it & 1];
        const unsigned o = s * TEAM + r;  // and on in steps of TEAM * TEAM
        mine = nf > o ? (nf - o + TEAM * TEAM - 1u) / (TEAM * TEAM) : 0u;
        for (unsigned k = row + STEP * j; k < mine; k += STEP * G) {
            const unsigned i = k * TEAM * TEAM + o;
            unsigned pos = i;
            if (!v.compact) {
                unsigned lo = 0, hi = gridDim.x;  // the last segment whose prefix is at most i
                while (hi - lo > 1u) {
                    const unsigned mid = (lo + hi) >> 1;
                    if (sm.prefix[mid] <= i) lo = mid;
                    else hi = mid;
                }
                pos = share(v.before, lo) * unsigned(a.max_degree) + (i - sm.prefix[lo]);
            }
            const unsigned w = (unsigned)ld_cg(q_in + pos);
            sm.region[0][s][k] =
                make_int2(int(w), pos < a.starts_cap ? ld_cg(s_in + pos) : __ldg(p.row_offsets + (w & ID_MASK)));
        }
        if (threadIdx.x < 2) sm.found[threadIdx.x] = sm.edges[threadIdx.x] = 0u;
        cluster_sync_all();
    }
    unsigned senders = 0;  // lanes below TEAM: the entries each CTA dealt in the last level
    bool ok = true;       // no wait ran out
    int b = 0;
    for (int steps = 0;; steps++, b ^= 1) {
        if (leader()) acct.step(p, it, nf, mf);
        if (threadIdx.x == 0) sm.found[b ^ 1] = sm.edges[b ^ 1] = 0u;
        for (unsigned k = row; __any_sync(FULL, k < mine); k += STEP) {
            const int2 q = k < mine ? sm.region[b][s][k] : make_int2(0, 0);
            const int col[1] = {q.y + int(j)};
            int2 e[1];
            unsigned at[1];
            const unsigned got = claim<1, true>(p, j < (unsigned)q.x >> LEN_SHIFT ? 1u : 0u, col, it + 1, e);
            place(sm, b, got, e, at);
            if (got) {  // at: below DEAL (on_cluster)
                const unsigned to = map_rank(&sm, at[0] % TEAM);
                send8(to + (smem_u32(&sm.region[b ^ 1][r][at[0] / TEAM]) - here),
                      to + (smem_u32(&sm.full[b ^ 1]) - here), e[0]);
            }
        }
        if (__syncthreads_or(!ok)) {  // a wait ran out in this CTA; the others' will, too
            ok = false;
            break;
        }
        if (threadIdx.x < TEAM) {
            const unsigned k = sm.found[b], to = threadIdx.x, there = map_rank(&sm, to);
            const unsigned bar = there + (smem_u32(&sm.full[b ^ 1]) - here);
            send8(there + (smem_u32(&sm.count[b ^ 1][r]) - here), bar, make_int2(int(k), int(sm.edges[b])));
            arrive_remote(bar, 8u * (1u + (k > to ? (k - to + TEAM - 1u) / TEAM : 0u)));
        }
        if (leader()) acct.work_end(p);
        ok = wait_full(p, &sm.full[b ^ 1], (phase >> (b ^ 1)) & 1u);
        if (!ok) {  // this level and its regions are not read; the error ends the search at the next barrier
            atomicOr(&c->error, ERR_BARRIER_TIMEOUT);
            mine = 0;
            continue;
        }
        phase ^= 1u << (b ^ 1);
        const unsigned from = sm.count[b ^ 1][s].x;
        const uint2 n2 = lane < TEAM ? sm.count[b ^ 1][lane] : make_uint2(0u, 0u);
        mf_before = mf;
        nf = __reduce_add_sync(FULL, n2.x);
        mf = __reduce_add_sync(FULL, n2.y);
        mine = from > r ? (from - r + TEAM - 1u) / TEAM : 0u;
        senders = n2.x;
        it++;
        if (nf == 0u || steps + 1 >= CLUSTER_LEVELS || !on_cluster<TEAM, G>(nf) || overflows(p, a, nf, mf)) break;
    }
    if (!ok) return;
    if (overflows(p, a, nf, mf)) {
        if (leader()) atomicOr(&c->error, ERR_OVERFLOW);
    } else {
        int *q = p.queue[it & 1], *st = a.starts[it & 1];
        const unsigned upto = unsigned(warp_inclusive_scan(int(senders))) - senders;
        const unsigned before = __shfl_sync(FULL, upto, s);  // entries of the senders before region s's
        for (unsigned k = row + STEP * j; k < mine; k += STEP * G) {
            const int2 e = sm.region[b ^ 1][s][k];
            const unsigned pos = before + k * TEAM + r;  // the sender's k * TEAM + r-th entry
            q[pos] = e.x;
            if (pos < a.starts_cap) st[pos] = e.y;
        }
    }
    if (threadIdx.x < 2) sm.found[threadIdx.x] = sm.edges[threadIdx.x] = 0u;
    // The frontier is compact: all of it counts as CTA 0's segment.
    if (r == 0) {
        a.counts[(it & 1) * THREADS + threadIdx.x] = threadIdx.x == 0 ? make_uint2(nf, mf) : make_uint2(0u, 0u);
        if (threadIdx.x < 4) c->qlen[threadIdx.x] = 0u;
        if (threadIdx.x == 0) c->cur_it = it;
    }
}

template <int TEAM, int G>
__global__ void __launch_bounds__(THREADS, 2) low_degree_kernel(BfsParams p, LowDegreeParams a) {
    extern __shared__ __align__(128) unsigned char dyn_smem[];
    Smem<TEAM> &sm = *reinterpret_cast<Smem<TEAM> *>(dyn_smem);
    Counters *c = p.ctr;
    Account acct{a.strategy};
    unsigned long long busy = 0, t0 = 0;
    if (threadIdx.x < 2) sm.found[threadIdx.x] = sm.edges[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        mbar_init(&sm.full[0], TEAM);
        mbar_init(&sm.full[1], TEAM);
        mbar_init_fence();
    }
    unsigned phase = 0;
    cluster_sync_all();  // the cluster's CTAs run, and their barriers are ready, before any writes into another's memory
    Level v{0, 0u, 0u, 0u, true};
    unsigned mf_before = 0;
    for (;;) {
        read_level(a, sm, v);
        if (v.nf == 0u) break;
        if (p.cta_busy && threadIdx.x == 0) t0 = globaltimer_ns();
        if (level_limit_hit(v.it, p.nodes)) {  // every CTA alike
            if (leader()) atomicOr(&c->error, ERR_LEVEL_LIMIT);
            break;
        }
        const bool small = on_cluster<TEAM, G>(v.nf);
        if (!small) {
            if (leader()) {
                acct.step(p, v.it, v.nf, v.mf);
                c->qlen[(v.it + 2) & 3] = 0u;
                if (overflows(p, a, v.nf, v.mf)) atomicOr(&c->error, ERR_OVERFLOW);
            }
            const bool compact = grid_level<TEAM, G>(p, a, sm, v);
            if (leader()) acct.work_end(p);
            mf_before = v.mf;
            v.before = v.nf;
            v.compact = compact;
        } else if (blockIdx.x < TEAM) {
            cluster_levels<TEAM, G>(p, a, sm, acct, phase, v, mf_before);
        }
        if (p.cta_busy) {
            __syncthreads();
            if (threadIdx.x == 0 && (!small || blockIdx.x < TEAM)) busy += globaltimer_ns() - t0;
        }
        if (!grid_sync(p, sm)) break;
        if (small) {
            v.it = sm.it;
            v.compact = true;
        } else {
            v.it++;
        }
    }
    if (p.cta_busy && threadIdx.x == 0) p.cta_busy[blockIdx.x] = busy;
    if (leader()) acct.finish(p, v.it, mf_before);
    cluster_sync_all();  // no CTA leaves while another may still write into it
}

// Counters to zero; the source labelled, marked and queued with its row range.
__global__ void low_degree_init_kernel(BfsParams p, LowDegreeParams a) {
    Counters *c = p.ctr;
    unsigned *w = reinterpret_cast<unsigned *>(c);
    constexpr int WORDS = int(offsetof(Counters, sticky) / 4);  // everything but the sticky error
    for (int i = threadIdx.x; i < WORDS; i += blockDim.x) w[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < THREADS; i += blockDim.x) a.counts[i] = make_uint2(0u, 0u);
    __syncthreads();
    if (threadIdx.x != 0) return;
    const int st = p.row_offsets[p.src];
    const unsigned len = unsigned(p.row_offsets[p.src + 1] - st);
    p.labels[p.src] = 0;
    p.mask[unsigned(p.src) >> 5] |= 1u << (unsigned(p.src) & 31u);
    p.queue[0][0] = int(unsigned(p.src) | (len << LEN_SHIFT));
    a.starts[0][0] = st;
    a.counts[0] = make_uint2(1u, len);
}

typedef void (*LowDegreeFn)(BfsParams, LowDegreeParams);

template <int TEAM>
LowDegreeFn pick(int max_degree) {
    return max_degree <= 4 ? low_degree_kernel<TEAM, 4> : max_degree <= 8 ? low_degree_kernel<TEAM, 8>
                                                                          : low_degree_kernel<TEAM, 16>;
}

cudaLaunchConfig_t config(int grid, cudaStream_t stream, cudaLaunchAttribute (&attr)[2]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = sizeof(Smem<LF_TEAM>);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = LF_TEAM;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

}  // namespace

cudaError_t low_degree_grid_limit(int max_degree, int *grid) {
    *grid = 0;
    const void *fn = (const void *)pick<LF_TEAM>(max_degree);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(Smem<LF_TEAM>)));
    if (!e && LF_TEAM > 8) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e) return e;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = config(LF_TEAM, nullptr, attr);
    cfg.numAttrs = 1;
    int clusters = 0;
    if ((e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg))) return e;
    *grid = std::min(clusters, THREADS / LF_TEAM) * LF_TEAM;  // a thread reads each CTA's counts
    return cudaSuccess;
}

cudaError_t launch_low_degree(const BfsParams &p, const LowDegreeParams &a, int grid, cudaStream_t stream) {
    low_degree_init_kernel<<<1, 64, 0, stream>>>(p, a);
    cudaError_t e = cudaGetLastError();
    if (e) return e;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = config(grid, stream, attr);
    return cudaLaunchKernelEx(&cfg, pick<LF_TEAM>(a.max_degree), p, a);
}

}  // namespace b40c_b200
