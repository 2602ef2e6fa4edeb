// Neighbour sampling and the Fused-Map id mapping for sm_100a.
//
// One persistent, cooperatively launched kernel walks every hop of every mini-batch it is given.  Its
// CTAs are split into teams; a team owns one mini-batch at a time and one slice of the hashtable that is
// small enough to stay in the 126 MB L2, and synchronises with a team-local barrier, so that several
// mini-batches are in flight and one team's barrier latency is covered by the others' memory traffic.
//
// Per hop, for the current node list (the seeds of the hop), in the fused kernel:
//   B  sample    block-CSR offsets by a scan over the edge counts of the hop's node tiles, which were added up when the
//                nodes joined the list; each seed is served by a group of 8/16/32 lanes that choose
//                the picks (Philox4x32-10; Floyd's algorithm for a k-subset, run by the group in registers), read the
//                picked sources and insert them into the open-addressing table (64-bit slots {key, value}, atomicCAS
//                to claim, atomicMin of the edge number to find the first occurrence).  A thread that claims a slot or
//                lowers its edge number marks its edge "possibly first" and moves one unit of the per-CTA count of
//                first occurrences from the displaced edge's CTA to its own, so no counting pass is needed
//   D  rank      scan over the possibly-first edges that still hold their slot -> local id, publish it in the slot,
//                append the node (and for the next hop its adjacency offset, its degree and min(degree, next fanout)
//                in its tile's edge count) to the list
//   E  relabel   replace the slot position kept in the remaining edge entries by the local id
// Two barriers per hop: after B and after D.  E needs none behind it: it reads slots that hold their final id, and the
// next hop's inserts touch only empty and pending ones.
// With FGL_MAP_ARRIVAL_ORDER the claiming thread takes the next id from a warp-aggregated counter in phase B and
// phase D is skipped.  The drop-in kernels (fgl_sample: a counting pass A over the seeds, then B without a table;
// fgl_map: explicit edges) keep a counting pass (C) between B and D.
//
// Replaces sample_node_cuda (sample.cu:102-203), transfer_edge_id_cuda (id_map.cu:386-493) and the
// hashtable of id_map.cu:26-255 / cuda_hashtable.cuh.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace fgl {

#ifndef FGL_SM_THREADS
#define FGL_SM_THREADS 512
#endif
constexpr int kThreads = FGL_SM_THREADS;
constexpr int kMinCtas = 1024 / FGL_SM_THREADS;
constexpr int kWarps = kThreads / 32;
constexpr unsigned long long kEmpty = ~0ULL;
constexpr uint32_t kPending = 0x80000000u;

enum { MODE_FUSED = 0, MODE_SAMPLE = 1, MODE_MAP = 2 };

struct KParams {
    // graph
    const void* indptr;
    const int32_t* indices;
    int64_t n_nodes;
    // batch geometry
    int32_t n_batches, n_hops;
    int32_t fanout[FGL_MAX_HOPS];
    int32_t flags;
    int32_t n_teams, team_size;
    uint64_t rng_seed, rng_ctr;
    const int32_t* seeds;
    int64_t seed_stride;
    const int32_t* seed_counts;  // device; if NULL every batch has n_seeds_host seeds
    int32_t n_seeds_host;
    int32_t* nodes;
    int64_t nodes_stride;
    int32_t* counts;
    int32_t* blk_indptr[FGL_MAX_HOPS];
    int64_t blk_indptr_stride[FGL_MAX_HOPS];
    int32_t* blk_src[FGL_MAX_HOPS];
    int64_t blk_src_stride[FGL_MAX_HOPS];
    int32_t* out_dst;  // MODE_SAMPLE: global seed id per edge (may be NULL)
    int32_t* blk_dst[FGL_MAX_HOPS];  // MODE_FUSED, one mini-batch: local destination id per edge (may be NULL)
    int32_t tile_shift[FGL_MAX_HOPS];  // MODE_FUSED: a hop's node tile has 2^shift nodes
    // MODE_MAP: explicit edges
    int32_t* map_src;
    int32_t* map_dst;
    int64_t map_edges;
    // workspace
    unsigned long long* table;
    int64_t table_slots;  // drop-in map: slots, a power of two
    int32_t table_shift;  // 32 - log2(buckets)
    int32_t table_log2_first, table_log2_max;  // fused: smallest and largest table of a team (see hop_table)
    unsigned long long* barriers;  // one per team, 16 words apart
    int32_t* team_sums;            // drop-in kernels: per-CTA counts
    int32_t* tile_sums;            // [n_teams][3][kMaxTiles]: edge counts of the node tiles (hops rotate through three)
    int32_t* team_cnt;             // [n_teams][3][team_size]: per-CTA counts of first occurrences (likewise)
    long long* node_start;         // [n_teams][deg_stride]: adjacency offset of every node that can still be a seed
    int32_t* node_deg;             // [n_teams][deg_stride]: and its degree
    int64_t deg_stride;
    int32_t* status;               // [0] first error, [1] abort flag
    int32_t* counts_host;          // pinned host copies (may be NULL)
    int32_t* status_host;
    int32_t seq;                   // closes a counts row on the host
};

// ----------------------------------------------------------------------------------------------
// hashtable: 64-bit slots, key in the high word; low word = local id (bit 31 clear) or, while the
// key's id is not assigned yet, kPending | (smallest edge number that carries the key).
// Four slots make a bucket, one 32-byte sector: a key goes to the first free slot of its bucket (then of the next
// ones), and a probe reads a bucket at once, so that a second round trip to the L2 is left to the one key in twenty
// whose bucket is full and not to every neighbour of an occupied slot.
// ----------------------------------------------------------------------------------------------
constexpr int kBucket = 4;

struct Table {
    unsigned long long* slots;
    uint32_t mask;  // buckets - 1
    int shift;      // 32 - log2(buckets)
};

__device__ __forceinline__ uint32_t hash_bucket(const Table& t, uint32_t key) { return (key * 0x9E3779B1u) >> t.shift; }

// Read in the L2, where the claims and the ids appear (an old value is as good: a claim or a minimum returns the new one).
__device__ __forceinline__ unsigned long long ld_slot(const unsigned long long* p) { return __ldcg(p); }

__device__ __forceinline__ void ld_bucket(const Table& t, uint32_t bucket, unsigned long long (&s)[kBucket]) {
    const unsigned long long* p = t.slots + (size_t)bucket * kBucket;
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(s[0]), "=l"(s[1]) : "l"(p));
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(s[2]), "=l"(s[3]) : "l"(p + 2));
}

// The same under a predicate, and a predicated claim: without a branch the loads and claims of several keys stay together.
__device__ __forceinline__ void ld_bucket_if(bool on, const Table& t, uint32_t bucket, unsigned long long (&s)[kBucket]) {
    const unsigned long long* p = t.slots + (size_t)bucket * kBucket;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
        "mov.u64 %0, -1;\n\tmov.u64 %1, -1;\n\tmov.u64 %2, -1;\n\tmov.u64 %3, -1;\n\t"
        "@q ld.global.cg.v2.u64 {%0, %1}, [%4];\n\t@q ld.global.cg.v2.u64 {%2, %3}, [%4 + 16];\n\t}"
        : "=&l"(s[0]), "=&l"(s[1]), "=&l"(s[2]), "=&l"(s[3])
        : "l"(p), "r"((int)on));
}

__device__ __forceinline__ unsigned long long claim_if(bool on, unsigned long long* slot, unsigned long long mine,
                                                       unsigned long long otherwise) {
    unsigned long long old;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %4, 0;\n\tmov.u64 %0, %3;\n\t"
        "@q atom.global.cas.b64 %0, [%1], -1, %2;\n\t}"
        : "=&l"(old)
        : "l"(slot), "l"(mine), "l"(otherwise), "r"((int)on)
        : "memory");
    return old;
}

// First slot of a bucket that holds the key or is free (kBucket: neither), and what it holds.
__device__ __forceinline__ int match_bucket(const unsigned long long (&s)[kBucket], uint32_t key, unsigned long long& cur) {
    int at = kBucket;
    cur = kEmpty;
#pragma unroll
    for (int i = kBucket - 1; i >= 0; --i) {
        if (s[i] == kEmpty || (uint32_t)(s[i] >> 32) == key) {
            at = i;
            cur = s[i];
        }
    }
    return at;
}

// A picked neighbour id is read once and never again: a hub's list has thousands of entries and a pick touches one
// 32-byte sector of it.  The load tells the L2 to evict that line first and keeps it out of L1, so the picks do not
// push the teams' tables and the next phase's entries out of the L2 (measured: 7 % off the launch; marking the table
// accesses evict-last on top of it bought nothing and slowed the aggregation kernel that shares the L2).
__device__ __forceinline__ int ld_adjacency(const int32_t* p) {
    int v;
    uint64_t policy;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(policy));
    return v;
}

// A probe sequence gives up after kProbeLimit buckets (or the whole table, if smaller): at the load factors the
// tables are sized for a key is a bucket or two away from its own, so only a table that is too small for its
// mini-batch gets there.  The failure is recorded and the launch is told to stop at its next team barrier, so an
// undersized table costs milliseconds, not a scan of the table per key.
constexpr uint32_t kProbeLimit = 1u << 11;

__device__ __forceinline__ uint32_t probe_limit(const Table& t) { return t.mask < kProbeLimit ? t.mask : kProbeLimit; }

__device__ __forceinline__ void probe_failed(int32_t* status) {
    set_status(status, FGL_ERR_PROBE);
    atomicExch(status + 1, 1);
}

// Slot of a key: the one that holds it (cur = its content), or a free one that this call claimed with `mine` (cur =
// kEmpty), or -1 when the probes ran out.
__device__ __forceinline__ int table_find_or_claim(const Table& t, uint32_t key, unsigned long long mine, unsigned long long& cur,
                                                   int32_t* status) {
    uint32_t bucket = hash_bucket(t, key);
    for (uint32_t probe = 0; probe <= probe_limit(t);) {
        unsigned long long s[kBucket];
        ld_bucket(t, bucket, s);
        const int i = match_bucket(s, key, cur);
        if (i < kBucket) {
            const int pos = (int)(bucket * kBucket) + i;
            if (cur == kEmpty) {
                cur = atomicCAS(t.slots + pos, kEmpty, mine);
                if (cur != kEmpty && (uint32_t)(cur >> 32) != key) continue;  // another key took the slot: look again
            }
            return pos;
        }
        bucket = (bucket + 1) & t.mask;
        ++probe;
    }
    probe_failed(status);
    return -1;
}

// Seed i gets local id i; of two equal seeds the later position wins, as a sequential run of
// id_map.cu:259-287 leaves it.
__device__ __forceinline__ void table_insert_seed(const Table& t, uint32_t key, uint32_t local, int32_t* status) {
    const unsigned long long mine = ((unsigned long long)key << 32) | local;
    unsigned long long cur;
    const int pos = table_find_or_claim(t, key, mine, cur, status);
    if (pos >= 0 && cur != kEmpty) atomicMax(t.slots + pos, mine);
}

// Lowers the edge number kept in a pending slot to `edge` if that is smaller.  Returns the edge number that lost
// its place as the key's first occurrence, or -1 if nothing changed.
__device__ __forceinline__ int table_lower_edge(const Table& t, uint32_t pos, uint32_t key, uint32_t edge) {
    const unsigned long long mine = ((unsigned long long)key << 32) | (kPending | edge);
    const unsigned long long old = atomicMin(t.slots + pos, mine);
    const uint32_t old_lo = (uint32_t)old;
    return ((old_lo & kPending) && old_lo > (kPending | edge)) ? (int)(old_lo & ~kPending) : -1;
}

// Inserts edge number `edge` of source `key`.  Returns the local id (>= 0) if the key already has one, else ~pos of its
// slot (< 0).  created is set for the thread that claimed the slot; displaced is the edge that this one displaced as the
// key's first occurrence (-1: none; never in arrival order).  created or displaced >= 0 means "edge may be the key's
// first occurrence".
template <bool ARRIVAL>
__device__ __forceinline__ int table_insert(const Table& t, uint32_t key, uint32_t edge, int32_t* status, bool& created,
                                            int& displaced) {
    displaced = -1;
    unsigned long long cur;
    const int pos = table_find_or_claim(t, key, ((unsigned long long)key << 32) | (ARRIVAL ? kPending : (kPending | edge)), cur, status);
    created = pos >= 0 && cur == kEmpty;
    if (pos < 0) return 0;
    const uint32_t lo = (uint32_t)cur;
    if (!created && !(lo & kPending)) return (int)lo;
    if (!ARRIVAL && !created && lo > (kPending | edge)) displaced = table_lower_edge(t, (uint32_t)pos, key, edge);
    return ~pos;
}

// Value of a key that must be present (a seed); missing keys report FGL_ERR_BOUNDS and map to 0.
__device__ __forceinline__ int table_lookup(const Table& t, uint32_t key, int32_t* status) {
    uint32_t bucket = hash_bucket(t, key);
    for (uint32_t probe = 0; probe <= probe_limit(t); ++probe) {
        unsigned long long s[kBucket], cur;
        ld_bucket(t, bucket, s);
        const int i = match_bucket(s, key, cur);
        if (i < kBucket && cur == kEmpty) break;
        if (i < kBucket) return (int)((uint32_t)cur & ~kPending);
        bucket = (bucket + 1) & t.mask;
    }
    set_status(status, FGL_ERR_BOUNDS);
    return 0;
}

// ----------------------------------------------------------------------------------------------
// per-hop state
// ----------------------------------------------------------------------------------------------
struct Hop {
    int32_t* nodes;        // this mini-batch's unique list
    int64_t nodes_cap;
    int32_t* counts;       // this mini-batch's counts row
    int32_t* blk_indptr;   // may be NULL (MODE_SAMPLE without CSR output)
    int32_t* blk_src;      // edge array: global ids (MODE_SAMPLE) or local ids / pending entries
    int32_t* out_dst;      // destination of every edge: global seed id (MODE_SAMPLE), local id (fused); may be NULL
    long long* node_start; // fused: adjacency offset and degree of the nodes that can still become seeds
    int32_t* node_deg;
    int64_t deg_cap;
    int32_t* sums;         // fused: edge counts of this hop's node tiles ...
    int32_t* next_sums;    // ... and of the next hop's, which this hop's new nodes are added to
    int tile_shift, next_shift, next_fanout;
    int hop, fanout, n_seeds, n_first;  // n_first: the mini-batch's own seeds, which may hold a node twice
    bool last_hop;
    uint64_t ctr;
};

constexpr int kMaxTiles = 8 * kThreads;  // node tiles per hop; a thread scans eight of their counts
constexpr int kMinTileShift = 3;
constexpr int kMaxTeam = 512;    // CTAs per team (a cooperative grid of 512-thread CTAs has at most a few hundred)

struct Smem {
    int scan[40];
    int v[kThreads];
    long long start[kThreads];
    int deg[kThreads];
    int off[kThreads];
    int prefix[kMaxTiles + 1];  // fused: first edge of every node tile (offsets, and the owner of an edge number)
    int first_tile[kMaxTeam + 1];  // fused: first node tile of every CTA of the team ...
    int first_edge[kMaxTeam + 1];  // ... and its first edge
    int moved[kMaxTeam];        // fused: first occurrences that this CTA's edges took from every CTA of the team
    float owner_scale;          // fused: CTAs per edge
};

// Fused kernel, first-occurrence order: an edge entry is a local id (>= 0) or, while the id is pending,
// ~(slot | kTentative if the edge may be the first occurrence of its key).  Slots are below 2^29.
constexpr int kTentative = 1 << 29;
constexpr int kSlotMask = kTentative - 1;

__device__ __forceinline__ void chunk_of(int n, int rank, int size, int& lo, int& hi) {
    const int per = (n + size - 1) / size;
    lo = min(n, rank * per);
    hi = min(n, lo + per);
}

template <typename PtrT>
__device__ __forceinline__ void load_adj(const KParams& p, int v, long long& start, int& deg) {
    const PtrT* ptr = (const PtrT*)p.indptr;
    if (v < 0 || (int64_t)v >= p.n_nodes) {
        set_status(p.status, FGL_ERR_BOUNDS);
        start = 0;
        deg = 0;
        return;
    }
    const long long a = (long long)ptr[v], b = (long long)ptr[v + 1];
    start = a;
    const long long d = b - a;
    deg = d < 0 ? 0 : (d > 0x7fffffffLL ? 0x7fffffff : (int)d);
}

// The CTAs of a team share a hop's node tiles by work, not by number: the nodes at the front of the list are the
// mini-batch's own seeds and their picks, the ones behind them were reached through an edge and have more edges
// themselves (with equal numbers of nodes the last CTA took 1.6 times as long as the first).  A tile's position is the
// edges and nodes before it; CTA r owns the tiles at positions from r / size of the total on.
__device__ __forceinline__ int first_tile_of(const Smem& sm, int n_tiles, int shift, int rank, int size) {
    const long long work = sm.prefix[n_tiles] + ((long long)n_tiles << shift);
    int lo = 0, hi = n_tiles;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((sm.prefix[mid] + ((long long)mid << shift)) * size >= rank * work) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// The CTA of the team whose edge range holds edge number e: the ranges are of nearly equal size, so a guess is at most a
// step or two away.
__device__ __forceinline__ int edge_owner(const Smem& sm, int size, int e) {
    int r = min(size - 1, (int)((float)e * sm.owner_scale));
    while (e < sm.first_edge[r]) --r;
    while (e >= sm.first_edge[r + 1]) ++r;
    return r;
}

// A node that joins the list with local id `local`: what the next hop needs of it.  Returns its edges there.
__device__ __forceinline__ int note_node(const Hop& h, int local, long long start, int deg) {
    if ((int64_t)local >= h.deg_cap) return 0;
    __stcg(h.node_start + local, start);
    __stcg(h.node_deg + local, deg);
    return min(deg, h.next_fanout);
}

// Second half of an insert in arrival-order mode: the claiming thread takes the next local id and publishes it.
template <typename PtrT>
__device__ __forceinline__ int arrival_assign(const KParams& p, const Hop& h, const Table& tab, int32_t* team_cnt, int g, int r) {
    cg::coalesced_group grp = cg::coalesced_threads();  // one atomicAdd per group of claiming lanes
    int base = 0;
    if (grp.thread_rank() == 0) base = h.n_seeds + atomicAdd(team_cnt, (int)grp.size());
    base = grp.shfl(base, 0);
    const int local = base + (int)grp.thread_rank();
    const uint32_t pos = (uint32_t)~r;
    if ((int64_t)local < h.nodes_cap) {
        h.nodes[local] = g;
        if (!h.last_hop) {
            long long start;
            int deg;
            load_adj<PtrT>(p, g, start, deg);
            const int k = note_node(h, local, start, deg);
            if (k > 0) atomicAdd(h.next_sums + (local >> h.next_shift), k);
        }
        atomicExch(tab.slots + pos, ((unsigned long long)(uint32_t)g << 32) | (uint32_t)local);
        return local;
    }
    set_status(p.status, FGL_ERR_CAPACITY);
    atomicExch(tab.slots + pos, ((unsigned long long)(uint32_t)g << 32));
    return 0;
}

// One sampled edge of the wide-fanout path: picked source `g` of destination `v`, edge number e within the hop.
// first_cnt counts the edges of this thread that may be first occurrences (fused, first-occurrence order).
template <typename PtrT, int MODE, bool ARRIVAL>
__device__ __forceinline__ void emit_edge(const KParams& p, const Hop& h, const Table& tab, Smem& sm,
                                          int32_t* team_cnt, int v, int g, int e, int& first_cnt) {
    if (h.out_dst) h.out_dst[e] = v;
    if (MODE == MODE_SAMPLE) {
        h.blk_src[e] = g;
        return;
    }
    if (g < 0 || (int64_t)g >= p.n_nodes) {
        set_status(p.status, FGL_ERR_BOUNDS);
        h.blk_src[e] = 0;
        return;
    }
    bool created;
    int displaced;
    int r = table_insert<ARRIVAL>(tab, (uint32_t)g, (uint32_t)e, p.status, created, displaced);
    if (ARRIVAL) {
        if (created) r = arrival_assign<PtrT>(p, h, tab, team_cnt, g, r);
    } else if (r < 0 && (created || displaced >= 0)) {
        r = ~((~r) | kTentative);
        ++first_cnt;
        if (displaced >= 0) atomicSub(&sm.moved[edge_owner(sm, p.team_size, displaced)], 1);
    }
    h.blk_src[e] = r;
}

// Fanouts up to 32: a group of G lanes per seed, one lane per pick; a group works on kSeedsPerIter seeds at a time.
// Picks: a Philox block holds the words of four consecutive pick slots, so lane 4b + q of a group computes block b of the
// group's q-th seed and a 4 x 4 transposition inside the quads hands every lane its words.  A k-subset is Floyd's
// algorithm (slot i draws t in [0, deg-k+i] and takes deg-k+i instead if an earlier slot already holds t) for all slots
// at once: slot i is replaced if an earlier slot drew the same t -- whoever holds it by then -- or if t is the
// replacement deg-k+j of an earlier slot j that was replaced itself; the second rule is iterated on ballots until nothing
// changes, nearly always once.  (Walking the slots one after the other and drawing a block per lane were half of the
// phase's instructions.)
// The dependent loads of the group's seeds -- picked sources, buckets, claims -- are issued seed by seed before the
// first is used, so that kSeedsPerIter round trips are in flight per lane; a key whose bucket is full goes round again
// together with the others' retries.  (Requesting the next round's sources before this round's inserts, CTAs of 256 or 384
// threads with more registers, and three or four seeds per round were all measured: none is faster.)
// Element (i, j) of the 4 x 4 words of a quad of lanes (lane i holds row i) goes to (j, i).
__device__ __forceinline__ void quad_transpose(uint4& w) {
    const bool odd = threadIdx.x & 1, high = threadIdx.x & 2;
    uint32_t t = __shfl_xor_sync(0xffffffffu, odd ? w.x : w.y, 1);
    if (odd) w.x = t; else w.y = t;
    t = __shfl_xor_sync(0xffffffffu, odd ? w.z : w.w, 1);
    if (odd) w.z = t; else w.w = t;
    t = __shfl_xor_sync(0xffffffffu, high ? w.x : w.z, 2);
    if (high) w.x = t; else w.z = t;
    t = __shfl_xor_sync(0xffffffffu, high ? w.y : w.w, 2);
    if (high) w.y = t; else w.w = t;
}

#ifndef FGL_SM_KS
#define FGL_SM_KS 2
#endif
constexpr int kSeedsPerIter = FGL_SM_KS;
constexpr int kGroupPathMaxFanout = 32;

template <typename PtrT, int MODE, bool ARRIVAL, int G>
__device__ __forceinline__ void sample_tile_groups(const KParams& p, const Hop& h, const Table& tab, Smem& sm,
                                                   int32_t* team_cnt, int tile0, int tile_n, int& first_cnt) {
    const bool replace = (p.flags & FGL_SAMPLE_REPLACE) != 0;
    const int fanout = h.fanout;
    constexpr int kGroups = kThreads / G;
    constexpr int KS = kSeedsPerIter;
    const int gid = threadIdx.x / G, gl = threadIdx.x % G;
    const int gbase = (threadIdx.x & 31) & ~(G - 1);  // first lane of the group within its warp
    // Stage 1 of a round of seeds: the picks, and the requests for the picked sources.
    auto picks = [&](int it, int (&g)[KS]) {
        int deg[KS];
        long long start[KS];
        uint32_t pk[KS];
        bool any_hub = false;
#pragma unroll
        for (int q = 0; q < KS; ++q) {
            const int j = (it * KS + q) * kGroups + gid;
            g[q] = 0;
            deg[q] = 0;
            start[q] = 0;
            if (j < tile_n) {
                deg[q] = sm.deg[j];
                start[q] = sm.start[j];
            }
            pk[q] = (uint32_t)gl;
            any_hub |= deg[q] > fanout;
        }
        // the picks of the rows that have more edges than the fanout
        if (__any_sync(0xffffffffu, any_hub)) {  // warp-uniform
            uint4 w = make_uint4(0, 0, 0, 0);
            const int wq = gl & 3;
            if (wq < KS) w = philox_block(p.rng_seed, h.ctr, (uint32_t)(tile0 + (it * KS + wq) * kGroups + gid), (uint32_t)(gl >> 2));
            quad_transpose(w);
            const uint32_t draw[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < KS; ++q) {
                const bool pick = deg[q] > fanout && gl < fanout;
                if (replace) {
                    if (pick) pk[q] = __umulhi(draw[q], (uint32_t)deg[q]);
                } else {
                    const int floor_q = deg[q] - fanout;
                    const uint32_t jj = (uint32_t)(floor_q + gl);
                    const uint32_t tt = __umulhi(draw[q], jj + 1u);
                    const unsigned same = __match_any_sync(0xffffffffu, pick ? tt : (0x80000000u | (unsigned)gl));
                    const unsigned earlier = (1u << gl) - 1u;
                    unsigned replaced = __ballot_sync(0xffffffffu, pick && ((same >> gbase) & earlier)) >> gbase;
                    const int ref = (int)tt - floor_q;  // the slot whose replacement t is
                    const bool may = pick && ref >= 0 && ref < gl;
                    for (;;) {
                        const unsigned more = __ballot_sync(0xffffffffu, may && !((replaced >> gl) & 1u) && ((replaced >> ref) & 1u));
                        if (!more) break;
                        replaced |= more >> gbase;
                    }
                    if (pick) pk[q] = ((replaced >> gl) & 1u) ? jj : tt;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < KS; ++q)
            if (gl < min(deg[q], fanout)) g[q] = ld_adjacency(p.indices + start[q] + (long long)pk[q]);
    };
    const int rounds = (tile_n + kGroups * KS - 1) / (kGroups * KS);
    int g[KS];
    for (int it = 0; it < rounds; ++it) {
        picks(it, g);
        int v[KS], off[KS];
        bool has[KS];
#pragma unroll
        for (int q = 0; q < KS; ++q) {
            const int j = (it * KS + q) * kGroups + gid;
            v[q] = 0;
            off[q] = 0;
            has[q] = false;
            if (j < tile_n) {
                has[q] = gl < min(sm.deg[j], fanout);
                v[q] = sm.v[j];
                off[q] = sm.off[j];
            }
        }
        if (h.out_dst) {
#pragma unroll
            for (int q = 0; q < KS; ++q)
                if (has[q]) h.out_dst[off[q] + gl] = v[q];
        }
        if (MODE == MODE_SAMPLE) {
#pragma unroll
            for (int q = 0; q < KS; ++q)
                if (has[q]) h.blk_src[off[q] + gl] = g[q];
        } else {
        // stage 2: find or claim the slots.  open: sources that are still looking for theirs
        uint32_t bucket[KS];
        int r[KS];
        unsigned open = 0;
#pragma unroll
        for (int q = 0; q < KS; ++q) {
            if (has[q] && (g[q] < 0 || (int64_t)g[q] >= p.n_nodes)) {
                set_status(p.status, FGL_ERR_BOUNDS);
                h.blk_src[off[q] + gl] = 0;
                has[q] = false;
            }
            bucket[q] = hash_bucket(tab, (uint32_t)g[q]);
            r[q] = 0;
            if (has[q]) open |= 1u << q;
        }
        unsigned created = 0, lower = 0;
#pragma unroll 1
        for (uint32_t probe = 0; open != 0; ++probe) {
            if (probe > probe_limit(tab) + 64u) {  // the odd round more: a claim that lost its slot looks again
                probe_failed(p.status);
                break;
            }
            unsigned long long cur[KS];
            int at[KS];
            {
                unsigned long long s[KS][kBucket];
#pragma unroll
                for (int q = 0; q < KS; ++q) ld_bucket_if(open >> q & 1u, tab, bucket[q], s[q]);
#pragma unroll
                for (int q = 0; q < KS; ++q) at[q] = match_bucket(s[q], (uint32_t)g[q], cur[q]);
            }
            unsigned claimed = 0;
#pragma unroll
            for (int q = 0; q < KS; ++q) {
                const bool claim = (open >> q & 1u) && at[q] < kBucket && cur[q] == kEmpty;
                const uint32_t e = (uint32_t)(off[q] + gl);
                cur[q] = claim_if(claim, tab.slots + bucket[q] * kBucket + at[q],
                                  ((unsigned long long)(uint32_t)g[q] << 32) | (ARRIVAL ? kPending : (kPending | e)), cur[q]);
                if (claim) claimed |= 1u << q;
            }
#pragma unroll
            for (int q = 0; q < KS; ++q) {
                const bool full = at[q] == kBucket;
                const bool mine = (claimed >> q & 1u) && cur[q] == kEmpty;
                const bool hit = (open >> q & 1u) && !full && (mine || (uint32_t)(cur[q] >> 32) == (uint32_t)g[q]);
                const uint32_t lo = (uint32_t)cur[q];
                const bool pending = mine || (lo & kPending);
                if (hit) r[q] = pending ? ~((int)(bucket[q] * kBucket) + at[q]) : (int)lo;
                if (hit && mine) {
                    created |= 1u << q;
                    if (!ARRIVAL && !h.last_hop)  // the ranking phase reads this node's offsets
                        asm volatile("prefetch.global.L2 [%0];" ::"l"((const PtrT*)p.indptr + g[q]));
                }
                if (!ARRIVAL && hit && pending && !mine && lo > (kPending | (uint32_t)(off[q] + gl))) lower |= 1u << q;
                if (hit) open &= ~(1u << q);
                if (full) bucket[q] = (bucket[q] + 1) & tab.mask;
            }
        }
        // stage 3: settle every edge
        int displaced[KS];
        if (!ARRIVAL) {
#pragma unroll
            for (int q = 0; q < KS; ++q)
                displaced[q] = (lower >> q & 1u) ? table_lower_edge(tab, (uint32_t)~r[q], (uint32_t)g[q], (uint32_t)(off[q] + gl)) : -1;
        }
#pragma unroll
        for (int q = 0; q < KS; ++q) {
            if (!has[q]) continue;
            if (ARRIVAL) {
                if (created >> q & 1u) r[q] = arrival_assign<PtrT>(p, h, tab, team_cnt, g[q], r[q]);
            } else if ((created >> q & 1u) || displaced[q] >= 0) {
                r[q] = ~((~r[q]) | kTentative);
                ++first_cnt;
                if (displaced[q] >= 0) atomicSub(&sm.moved[edge_owner(sm, p.team_size, displaced[q])], 1);
            }
            h.blk_src[off[q] + gl] = r[q];
        }
        }  // MODE != MODE_SAMPLE
    }
}

// Any fanout up to FGL_MAX_FANOUT: one warp per seed, picks in shared memory.
template <typename PtrT, int MODE, bool ARRIVAL>
__device__ __forceinline__ void sample_tile_wide(const KParams& p, const Hop& h, const Table& tab, Smem& sm,
                                                 int32_t* team_cnt, uint32_t* picks_all, int tile0, int tile_n, int& first_cnt) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool replace = (p.flags & FGL_SAMPLE_REPLACE) != 0;
    const int fanout = h.fanout;
    uint32_t* picks = picks_all + (size_t)warp * fanout;
    for (int j = warp; j < tile_n; j += kWarps) {
        const int v = sm.v[j], deg = sm.deg[j], off = sm.off[j];
        const long long start = sm.start[j];
        if (deg <= fanout) {
            for (int i = lane; i < deg; i += 32)
                emit_edge<PtrT, MODE, ARRIVAL>(p, h, tab, sm, team_cnt, v, p.indices[start + i], off + i, first_cnt);
        } else if (replace) {
            for (int i = lane; i < fanout; i += 32) {
                const uint32_t r = philox_draw(p.rng_seed, h.ctr, (uint32_t)(tile0 + j), (uint32_t)i);
                emit_edge<PtrT, MODE, ARRIVAL>(p, h, tab, sm, team_cnt, v,
                                               ld_adjacency(p.indices + start + (long long)__umulhi(r, (uint32_t)deg)), off + i, first_cnt);
            }
        } else {
            uint32_t r = 0;
            for (int i = 0; i < fanout; ++i) {
                if ((i & 31) == 0) {
                    r = (i + lane < fanout) ? philox_draw(p.rng_seed, h.ctr, (uint32_t)(tile0 + j), (uint32_t)(i + lane)) : 0u;
                }
                const uint32_t ri = __shfl_sync(0xffffffffu, r, i & 31);
                const uint32_t jj = (uint32_t)(deg - fanout + i);
                const uint32_t t = __umulhi(ri, jj + 1u);
                bool hit = false;
                for (int q = lane; q < i; q += 32) hit |= (picks[q] == t);
                const bool any = __any_sync(0xffffffffu, hit);
                if (lane == 0) picks[i] = any ? jj : t;
                __syncwarp();
            }
            for (int i = lane; i < fanout; i += 32)
                emit_edge<PtrT, MODE, ARRIVAL>(p, h, tab, sm, team_cnt, v, ld_adjacency(p.indices + start + (long long)picks[i]), off + i,
                                               first_cnt);
        }
        __syncwarp();
    }
}

// Phase A of the drop-in sampler: per-CTA sum of min(deg, fanout) over the CTA's slice of the seeds.
template <typename PtrT>
__device__ __forceinline__ void phase_count_seeds(const KParams& p, const Hop& h, const Team& t, Smem& sm,
                                                  int32_t* team_sums) {
    int s0, s1;
    chunk_of(h.n_seeds, t.rank, t.size, s0, s1);
    int acc = 0;
    for (int s = s0 + (int)threadIdx.x; s < s1; s += 4 * kThreads) {
        int v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = (s + q * kThreads < s1) ? __ldcg(h.nodes + s + q * kThreads) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (s + q * kThreads < s1) {
                long long start;
                int deg;
                load_adj<PtrT>(p, v[q], start, deg);
                acc += min(deg, h.fanout);
            }
        }
    }
    const int total = block_sum(acc, sm.scan);
    if (threadIdx.x == 0) __stcg(team_sums + t.rank, total);
}

// The nodes that are in the list already are destinations of the next hop too: their edges, by tile (of eight nodes or
// more: eight lanes, or all of a warp, meet in one addition).
__device__ __forceinline__ void phase_count_old(const Hop& h, const Team& t) {
    for (int s0 = t.rank * kThreads; s0 < h.n_seeds; s0 += t.size * kThreads) {
        const int s = s0 + (int)threadIdx.x;
        int k = s < h.n_seeds ? min(__ldcg(h.node_deg + s), h.next_fanout) : 0;
        const int lanes = h.next_shift >= 5 ? 32 : 1 << kMinTileShift;
        for (int o = 1; o < lanes; o <<= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
        if ((s & (lanes - 1)) == 0 && k > 0) atomicAdd(h.next_sums + (s >> h.next_shift), k);
    }
}

// Sum of the team's partials before `rank` and over the whole team.
__device__ __forceinline__ void team_prefix(const int32_t* team_sums, const Team& t, Smem& sm, int& before, int& total) {
    // every warp for itself: a few loads more, but no barriers of the CTA
    int a = 0, b = 0;
    for (int q = threadIdx.x & 31; q < t.size; q += 32) {
        const int x = __ldcg(team_sums + q);
        b += x;
        if (q < t.rank) a += x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    before = a;
    total = b;
}

// The fused kernel's table of 2^log2 slots: it lies at slot 2^log2 of the team's region, so the tables of a mini-batch do
// not overlap.  A mini-batch starts with a small one and moves to a larger one when a hop could fill it -- once the hop's
// edge count is known, not for the worst case: the random accesses of all teams have to stay in the L2, where a slot
// costs the 128-byte line that it lies in.  (With worst-case tables, 16 MB for each of eight teams at the benchmark's
// sizes, the inserts of the last hop took longer than the adjacency reads.)
__device__ __forceinline__ Table hop_table(const KParams& p, int team_id, int log2) {
    Table tab;
    tab.slots = p.table + ((size_t)team_id << (p.table_log2_max + 1)) + ((size_t)1 << log2);
    tab.mask = (1u << (log2 - 2)) - 1u;
    tab.shift = 34 - log2;
    return tab;
}

// Room for every node in the list and a new one for every edge, at a load of at most 0.8 (in practice a third of it).
__device__ __forceinline__ int table_log2_for(const KParams& p, int log2, long long keys) {
    while (log2 < p.table_log2_max && (4LL << log2) < 5 * keys) ++log2;
    return log2;
}

// Phase B: offsets, picks, source reads, table inserts.  Returns the CTA's first edge and edge count; false: aborted.
template <typename PtrT, int MODE, bool ARRIVAL>
__device__ __forceinline__ bool phase_sample(const KParams& p, const Hop& h, Table& tab, int& log2, unsigned& used, int team_id,
                                             Team& t, Smem& sm, uint32_t* picks, const int32_t* team_sums, int32_t* team_cnt,
                                             int& e0, int& e1) {
    int before, total, s0, s1;
    if (MODE == MODE_FUSED) {
        // first edge of every node tile of the hop; the CTAs own runs of tiles
        constexpr int kPer = kMaxTiles / kThreads;
        const int n_tiles = (h.n_seeds + (1 << h.tile_shift) - 1) >> h.tile_shift;
        const int q0 = (int)threadIdx.x * kPer;
        int c[kPer], mine = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            c[q] = q0 + q < n_tiles ? __ldcg(h.sums + q0 + q) : 0;
            mine += c[q];
        }
        int excl = block_excl_scan(mine, sm.scan, total);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (q0 + q < n_tiles) sm.prefix[q0 + q] = excl;
            excl += c[q];
        }
        if (threadIdx.x == 0) {
            sm.prefix[n_tiles] = total;
            sm.owner_scale = (float)t.size / (float)max(total, 1);
        }
        __syncthreads();
        for (int i = threadIdx.x; i <= t.size; i += kThreads) {
            const int tile = i == t.size ? n_tiles : first_tile_of(sm, n_tiles, h.tile_shift, i, t.size);
            sm.first_tile[i] = tile;
            sm.first_edge[i] = sm.prefix[tile];
            if (i < t.size) sm.moved[i] = 0;
        }
        __syncthreads();
        before = sm.first_edge[t.rank];
        s0 = min(h.n_seeds, sm.first_tile[t.rank] << h.tile_shift);
        s1 = min(h.n_seeds, sm.first_tile[t.rank + 1] << h.tile_shift);
    } else {
        team_prefix(team_sums, t, sm, before, total);
        chunk_of(h.n_seeds, t.rank, t.size, s0, s1);
    }
    if (MODE == MODE_FUSED) {
        const int want = table_log2_for(p, log2, (long long)h.n_seeds + total);
        if (want > log2) {  // the same for every CTA of the team
            log2 = want;
            used |= 1u << log2;
            tab = hop_table(p, team_id, log2);
            for (int s = t.rank * kThreads + (int)threadIdx.x; s < h.n_seeds; s += t.size * kThreads) {
                const int v = __ldcg(h.nodes + s);
                if (v >= 0 && (int64_t)v < p.n_nodes) table_insert_seed(tab, (uint32_t)v, (uint32_t)s, p.status);
            }
            if (!team_barrier(t)) return false;
        }
    }
    if (t.rank == 0 && threadIdx.x == 0) {
        h.counts[8 + h.hop] = total;
        if (h.blk_indptr) h.blk_indptr[h.n_seeds] = total;
    }
    int running = before;
    int first_cnt = 0;
    e0 = before;
    for (int tile0 = s0; tile0 < s1; tile0 += kThreads) {
        const int s = tile0 + (int)threadIdx.x;
        int k = 0;
        if (s < s1) {
            const int v = __ldcg(h.nodes + s);
            long long start;
            int deg;
            if (MODE == MODE_FUSED) {
                start = __ldcg(h.node_start + s);
                deg = __ldcg(h.node_deg + s);
            } else {
                load_adj<PtrT>(p, v, start, deg);
            }
            k = min(deg, h.fanout);
            // what goes into out_dst: the seed itself, or its local id (of two equal seeds, the later one's)
            sm.v[threadIdx.x] = (MODE == MODE_FUSED && h.out_dst) ? (s < h.n_first && k > 0 ? table_lookup(tab, (uint32_t)v, p.status) : s) : v;
            sm.start[threadIdx.x] = start;
            sm.deg[threadIdx.x] = deg;
        }
        int tile_total;
        const int excl = block_excl_scan(k, sm.scan, tile_total);
        if (s < s1) {
            sm.off[threadIdx.x] = running + excl;
            if (h.blk_indptr) h.blk_indptr[s] = running + excl;
        }
        __syncthreads();
        const int tile_n = min(kThreads, s1 - tile0);
        if (h.fanout <= 8)
            sample_tile_groups<PtrT, MODE, ARRIVAL, 8>(p, h, tab, sm, team_cnt, tile0, tile_n, first_cnt);
        else if (h.fanout <= 16)
            sample_tile_groups<PtrT, MODE, ARRIVAL, 16>(p, h, tab, sm, team_cnt, tile0, tile_n, first_cnt);
        else if (h.fanout <= kGroupPathMaxFanout)
            sample_tile_groups<PtrT, MODE, ARRIVAL, 32>(p, h, tab, sm, team_cnt, tile0, tile_n, first_cnt);
        else
            sample_tile_wide<PtrT, MODE, ARRIVAL>(p, h, tab, sm, team_cnt, picks, tile0, tile_n, first_cnt);
        running += tile_total;
        __syncthreads();
    }
    e1 = running;
    if (MODE == MODE_FUSED && !ARRIVAL) {
        // The counts of first occurrences that moved between CTAs meet here, in one addition per pair of CTAs: added edge
        // by edge, the few dozen counters of a team are a handful of L2 lines that tens of thousands of atomics wait for.
        const int mine = block_sum(first_cnt, sm.scan);
        if (threadIdx.x == 0) sm.moved[t.rank] += mine;
        __syncthreads();
        for (int i = threadIdx.x; i < t.size; i += kThreads)
            if (sm.moved[i] != 0) atomicAdd(team_cnt + i, sm.moved[i]);
    }
    return true;
}

// ---- fused kernel, first-occurrence order ------------------------------------------------------------------------------
// Phase D: the possibly-first edges that still hold their slot are the first occurrences.  Local ids in edge order;
// the node, its adjacency offset and degree (unless this is the last hop) join the list; the edge entry becomes the id.
// kPer (4 or 8) consecutive edges per thread: 128-bit loads of entries, then up to kPer slot loads in flight, then as many of
// the new nodes' offsets.
template <typename PtrT, int kPer>
__device__ __forceinline__ int phase_rank_tracked(const KParams& p, const Hop& h, const Table& tab, int32_t* edges, int e0, int e1,
                                                  int n_before, const Team& t, Smem& sm, const int32_t* team_cnt) {
    int before, total;
    team_prefix(team_cnt, t, sm, before, total);
    int running = n_before + before;
    for (int tile0 = e0 & ~3; tile0 < e1; tile0 += kPer * kThreads) {
        const int eb = tile0 + kPer * (int)threadIdx.x;
        int m[kPer];
#pragma unroll
        for (int part = 0; part < kPer / 4; ++part) {
            const int at = eb + 4 * part;
            int4 x = make_int4(0, 0, 0, 0);
            if (at + 3 >= e0 && at + 3 < e1) {
                x = __ldcg(reinterpret_cast<const int4*>(edges + at));  // the row is 16-byte aligned
            } else if (at < e1 && at + 3 >= e0) {  // the range's last entries: never read beyond e1
                x.x = __ldcg(edges + at);
                if (at + 1 < e1) x.y = __ldcg(edges + at + 1);
                if (at + 2 < e1) x.z = __ldcg(edges + at + 2);
            }
            m[4 * part + 0] = x.x;
            m[4 * part + 1] = x.y;
            m[4 * part + 2] = x.z;
            m[4 * part + 3] = x.w;
        }
        unsigned long long cur[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const bool mine = eb + q >= e0 && eb + q < e1 && m[q] < 0 && ((~m[q]) & kTentative);
            if (!mine) m[q] = 0;
            cur[q] = mine ? ld_slot(tab.slots + ((~m[q]) & kSlotMask)) : 0ULL;
        }
        int firsts = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (!(m[q] < 0 && (uint32_t)cur[q] == (kPending | (uint32_t)(eb + q)))) m[q] = 0;  // keep first occurrences
            firsts += m[q] < 0 ? 1 : 0;
        }
        // the new nodes' adjacency offsets and degrees, all on their way before the first is stored
        long long start[kPer];
        int deg[kPer];
        if (!h.last_hop) {
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                start[q] = 0;
                deg[q] = 0;
                if (m[q] < 0) load_adj<PtrT>(p, (int)(cur[q] >> 32), start[q], deg[q]);
            }
        }
        int tile_total;
        int local = running + block_excl_scan(firsts, sm.scan, tile_total);
        int node_tile = -1, node_sum = 0;  // this thread's new nodes have consecutive ids: mostly one tile
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (m[q] < 0) {
                const uint32_t pos = (uint32_t)((~m[q]) & kSlotMask);
                const uint32_t key = (uint32_t)(cur[q] >> 32);
                if ((int64_t)local < h.nodes_cap) {
                    h.nodes[local] = (int)key;
                    tab.slots[pos] = ((unsigned long long)key << 32) | (uint32_t)local;
                    edges[eb + q] = local;
                    if (!h.last_hop) {
                        const int k = note_node(h, local, start[q], deg[q]);
                        if ((local >> h.next_shift) != node_tile) {
                            if (node_sum > 0) atomicAdd(h.next_sums + node_tile, node_sum);
                            node_tile = local >> h.next_shift;
                            node_sum = 0;
                        }
                        node_sum += k;
                    }
                } else {
                    set_status(p.status, FGL_ERR_CAPACITY);
                    tab.slots[pos] = ((unsigned long long)key << 32);
                    edges[eb + q] = 0;
                }
                ++local;
            }
        }
        if (!h.last_hop) {
            // A warp's nodes are consecutive too: one addition where they lie in one tile.  (Tiles of 512 nodes, which large
            // mini-batches have, took 512 additions at one address.)
            const unsigned act = __ballot_sync(0xffffffffu, node_sum > 0);
            if (act != 0) {
                const int leader = __ffs(act) - 1;
                const int lead_tile = __shfl_sync(0xffffffffu, node_tile, leader);
                if (__all_sync(0xffffffffu, node_sum == 0 || node_tile == lead_tile)) {
                    const int sum = __reduce_add_sync(0xffffffffu, node_sum);
                    if ((int)(threadIdx.x & 31) == leader) atomicAdd(h.next_sums + lead_tile, sum);
                } else if (node_sum > 0) {
                    atomicAdd(h.next_sums + node_tile, node_sum);
                }
            }
        }
        running += tile_total;
    }
    return n_before + total;
}

// Phase E: the entries that are still pending take the local id their slot now holds.
__device__ __forceinline__ void phase_relabel_tracked(const Table& tab, int32_t* edges, int e0, int e1) {
    constexpr int kPer = 8;
    for (int tile0 = e0 & ~3; tile0 < e1; tile0 += kPer * kThreads) {
        const int eb = tile0 + kPer * (int)threadIdx.x;
        int m[kPer];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int at = eb + 4 * half;
            int4 x = make_int4(0, 0, 0, 0);
            if (at + 3 >= e0 && at + 3 < e1) {
                x = __ldcg(reinterpret_cast<const int4*>(edges + at));
            } else if (at < e1 && at + 3 >= e0) {  // the range's last entries: never read beyond e1
                x.x = __ldcg(edges + at);
                if (at + 1 < e1) x.y = __ldcg(edges + at + 1);
                if (at + 2 < e1) x.z = __ldcg(edges + at + 2);
            }
            m[4 * half + 0] = x.x;
            m[4 * half + 1] = x.y;
            m[4 * half + 2] = x.z;
            m[4 * half + 3] = x.w;
        }
        unsigned long long cur[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const bool mine = eb + q >= e0 && eb + q < e1 && m[q] < 0;
            if (!mine) m[q] = 0;
            cur[q] = mine ? ld_slot(tab.slots + ((~m[q]) & kSlotMask)) : 0ULL;
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q)
            if (m[q] < 0) edges[eb + q] = (int)((uint32_t)cur[q] & ~kPending);
    }
}

// ---- drop-in id map (fgl_map): counting pass, rank, relabel over entries that are local ids or ~slot --------------------
// Phase C: number of first occurrences among the CTA's edges.
__device__ __forceinline__ void phase_count_first(const Table& tab, const int32_t* edges, int e0, int e1, const Team& t,
                                                  Smem& sm, int32_t* team_sums) {
    int acc = 0;
    for (int e = e0 + (int)threadIdx.x; e < e1; e += 4 * kThreads) {
        int m[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = (e + q * kThreads < e1) ? __ldcg(edges + e + q * kThreads) : 0;
        unsigned long long cur[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) cur[q] = (m[q] < 0) ? ld_slot(tab.slots + (uint32_t)~m[q]) : 0ULL;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            acc += (m[q] < 0 && (uint32_t)cur[q] == (kPending | (uint32_t)(e + q * kThreads))) ? 1 : 0;
    }
    const int total = block_sum(acc, sm.scan);
    if (threadIdx.x == 0) __stcg(team_sums + t.rank, total);
}

// Phase D: local ids in first-occurrence order; returns the new node count.
__device__ __forceinline__ int phase_rank(const KParams& p, const Table& tab, const int32_t* edges, int e0, int e1,
                                          int32_t* nodes, int64_t nodes_cap, int n_before, const Team& t, Smem& sm,
                                          const int32_t* team_sums) {
    int before, total;
    team_prefix(team_sums, t, sm, before, total);
    int running = n_before + before;
    // every thread ranks four consecutive edges: their entries and slots are loaded together
    for (int tile0 = e0; tile0 < e1; tile0 += 4 * kThreads) {
        const int eb = tile0 + 4 * (int)threadIdx.x;
        int m[4];
        unsigned long long cur[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = (eb + q < e1) ? __ldcg(edges + eb + q) : 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) cur[q] = (m[q] < 0) ? ld_slot(tab.slots + (uint32_t)~m[q]) : 0ULL;
        int mine = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!(m[q] < 0 && (uint32_t)cur[q] == (kPending | (uint32_t)(eb + q)))) m[q] = 0;  // keep first occurrences
            mine += m[q] < 0 ? 1 : 0;
        }
        int tile_total;
        int local = running + block_excl_scan(mine, sm.scan, tile_total);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (m[q] < 0) {
                const uint32_t pos = (uint32_t)~m[q];
                const uint32_t key = (uint32_t)(cur[q] >> 32);
                if ((int64_t)local < nodes_cap) {
                    nodes[local] = (int)key;
                    tab.slots[pos] = ((unsigned long long)key << 32) | (uint32_t)local;
                } else {
                    set_status(p.status, FGL_ERR_CAPACITY);
                    tab.slots[pos] = ((unsigned long long)key << 32);
                }
                ++local;
            }
        }
        running += tile_total;
    }
    return n_before + total;
}

// Phase E: slot positions -> local ids.
__device__ __forceinline__ void phase_relabel(const Table& tab, int32_t* edges, int e0, int e1) {
    for (int e = e0 + (int)threadIdx.x; e < e1; e += 4 * kThreads) {
        int m[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = (e + q * kThreads < e1) ? __ldcg(edges + e + q * kThreads) : 0;
        unsigned long long cur[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) cur[q] = (m[q] < 0) ? ld_slot(tab.slots + (uint32_t)~m[q]) : 0ULL;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (m[q] < 0) edges[e + q * kThreads] = (int)((uint32_t)cur[q] & ~kPending);
    }
}

// ----------------------------------------------------------------------------------------------
// kernels
// ----------------------------------------------------------------------------------------------
// The launch reports an error to the host itself (see fgl_fused_extra); true where the caller returns.
__device__ __forceinline__ bool given_up(const KParams& p, bool ok) {
    if (!ok && p.status_host && threadIdx.x == 0) *(volatile int32_t*)p.status_host = *(volatile int32_t*)p.status;
    return !ok;
}

// The mini-batch's numbers are settled (behind the barrier after its last ranking): the team's first warp, which wrote them,
// copies them to the host.  What is left -- relabelling the last hop, emptying the tables -- goes on while the host prepares
// what comes next.
__device__ __forceinline__ void tell_host(const KParams& p, const Hop& h, int b, int rank) {
    if (p.counts_host == nullptr || rank != 0 || threadIdx.x >= 32) return;
    __syncwarp();
    volatile int32_t* row = p.counts_host + (size_t)b * FGL_COUNTS_STRIDE;
    if (threadIdx.x < FGL_COUNTS_STRIDE - 1) row[threadIdx.x] = *(volatile int32_t*)(h.counts + threadIdx.x);
    if (threadIdx.x == 31) {
        const int32_t code = *(volatile int32_t*)p.status;
        if (code != FGL_OK) *(volatile int32_t*)p.status_host = code;
    }
    __threadfence_system();
    __syncwarp();
    if (threadIdx.x == 0) row[FGL_COUNTS_STRIDE - 1] = p.seq;
}

template <typename PtrT, int MODE, bool ARRIVAL>
__global__ void __launch_bounds__(kThreads, kMinCtas) sample_map_kernel(const __grid_constant__ KParams p) {
    __shared__ Smem sm;
    extern __shared__ uint32_t picks[];
    const int team_id = blockIdx.x / p.team_size;
    if (team_id >= p.n_teams) return;
    if (given_up(p, *(volatile int32_t*)(p.status + 1) == 0)) return;  // an earlier launch gave up: wait for fgl_ws_check
    Team t;
    t.rank = blockIdx.x % p.team_size;
    t.size = p.team_size;
    t.epoch = 0;
    t.bar = p.barriers + (size_t)team_id * 16;
    t.status = p.status;
    int32_t* tile_sums = MODE == MODE_FUSED ? p.tile_sums + (size_t)team_id * 3 * kMaxTiles : nullptr;
    int32_t* team_cnt = MODE == MODE_FUSED ? p.team_cnt + (size_t)team_id * 3 * p.team_size : nullptr;
    // The tile sums and the first-occurrence counts of a hop live in one of three buffers, used in turn over all hops of
    // all mini-batches: while a hop's phase B reads (and its new nodes add to the next one), the third is zeroed.
    int turn = 0;

    for (int b = team_id; b < p.n_batches; b += p.n_teams) {
        Hop h;
        h.nodes = p.nodes + (size_t)b * p.nodes_stride;
        h.nodes_cap = p.nodes_stride;
        h.counts = p.counts + (size_t)b * FGL_COUNTS_STRIDE;
        h.out_dst = p.out_dst;
        h.node_start = nullptr;
        h.node_deg = nullptr;
        h.sums = h.next_sums = nullptr;
        h.deg_cap = 0;
        int n0 = p.seed_counts ? __ldg(p.seed_counts + b) : p.n_seeds_host;
        n0 = max(0, min(n0, (int)min((int64_t)0x7fffffff, p.seed_stride)));
        const int32_t* seeds = p.seeds + (size_t)b * p.seed_stride;
        h.n_first = n0;

        int log2 = p.table_log2_first;
        unsigned used = 1u << log2;
        Table tab{};
        if (MODE == MODE_FUSED) {
            tab = hop_table(p, team_id, log2);
            // The team's tables are empty here: the host cleared them once and every mini-batch empties them again at its
            // end.  Insert the seeds with local id = position; cache their adjacency offsets and degrees.
            h.node_start = p.node_start + (size_t)team_id * p.deg_stride;
            h.node_deg = p.node_deg + (size_t)team_id * p.deg_stride;
            h.deg_cap = p.deg_stride;
            if (t.rank == 0 && threadIdx.x < FGL_COUNTS_STRIDE) h.counts[threadIdx.x] = threadIdx.x == 0 ? n0 : 0;
            int32_t* sums = tile_sums + turn * kMaxTiles;
            for (int s = t.rank * kThreads + (int)threadIdx.x; s < n0; s += t.size * kThreads) {
                const int v = seeds[s];
                h.nodes[s] = v;
                long long start = 0;
                int deg = 0;
                if (v < 0 || (int64_t)v >= p.n_nodes) {
                    set_status(p.status, FGL_ERR_BOUNDS);
                } else {
                    table_insert_seed(tab, (uint32_t)v, (uint32_t)s, p.status);
                    load_adj<PtrT>(p, v, start, deg);
                }
                __stcg(h.node_start + s, start);
                __stcg(h.node_deg + s, deg);
                if (deg > 0) atomicAdd(sums + (s >> p.tile_shift[0]), min(deg, p.fanout[0]));
            }
            if (given_up(p, team_barrier(t))) return;
        } else {
            h.nodes = const_cast<int32_t*>(seeds);  // MODE_SAMPLE reads the seeds in place
        }

        int n_cur = n0;
        for (int hop = 0; hop < p.n_hops; ++hop) {
            h.hop = hop;
            h.last_hop = hop + 1 == p.n_hops;
            h.fanout = p.fanout[hop];
            h.n_seeds = n_cur;
            h.ctr = p.rng_ctr + (uint64_t)b * 8u + (uint64_t)hop;
            h.blk_indptr = p.blk_indptr[hop] ? p.blk_indptr[hop] + (size_t)b * p.blk_indptr_stride[hop] : nullptr;
            h.blk_src = p.blk_src[hop] + (size_t)b * p.blk_src_stride[hop];

            int32_t* cnt = nullptr;
            if (MODE == MODE_FUSED) {
                const int next = turn == 2 ? 0 : turn + 1, spare = next == 2 ? 0 : next + 1;
                h.out_dst = p.blk_dst[hop];
                h.sums = tile_sums + turn * kMaxTiles;
                h.next_sums = tile_sums + next * kMaxTiles;
                h.tile_shift = p.tile_shift[hop];
                h.next_shift = h.last_hop ? 0 : p.tile_shift[hop + 1];
                h.next_fanout = h.last_hop ? 0 : p.fanout[hop + 1];
                cnt = team_cnt + turn * p.team_size;
                int32_t* zero = tile_sums + spare * kMaxTiles;
                for (int i = t.rank * kThreads + (int)threadIdx.x; i < kMaxTiles; i += t.size * kThreads) __stcg(zero + i, 0);
                if (threadIdx.x == 0) __stcg(team_cnt + spare * p.team_size + t.rank, 0);
                turn = next;
            } else {
                phase_count_seeds<PtrT>(p, h, t, sm, p.team_sums);
                if (given_up(p, team_barrier(t))) return;
            }

            if (MODE == MODE_FUSED && !h.last_hop) phase_count_old(h, t);
            int e0, e1;
            if (given_up(p, phase_sample<PtrT, MODE, ARRIVAL>(p, h, tab, log2, used, team_id, t, sm, picks, p.team_sums, cnt, e0, e1))) return;
            if (MODE == MODE_SAMPLE) break;
            if (given_up(p, team_barrier(t))) return;

            if (!ARRIVAL) {
                n_cur = h.last_hop ? phase_rank_tracked<PtrT, 8>(p, h, tab, h.blk_src, e0, e1, n_cur, t, sm, cnt)
                                   : phase_rank_tracked<PtrT, 4>(p, h, tab, h.blk_src, e0, e1, n_cur, t, sm, cnt);
                n_cur = (int)min((int64_t)n_cur, h.nodes_cap);
                if (t.rank == 0 && threadIdx.x == 0) h.counts[hop + 1] = n_cur;
                if (given_up(p, team_barrier(t))) return;
                if (h.last_hop) tell_host(p, h, b, t.rank);
                phase_relabel_tracked(tab, h.blk_src, e0, e1);
            } else {
                n_cur = (int)min((int64_t)n_cur + __ldcg(cnt), h.nodes_cap);
                if (t.rank == 0 && threadIdx.x == 0) h.counts[hop + 1] = n_cur;
                if (h.last_hop) tell_host(p, h, b, t.rank);
                phase_relabel(tab, h.blk_src, e0, e1);
            }
        }
        if (MODE == MODE_SAMPLE) break;
        // Once every CTA has finished reading the tables, empty them for the next mini-batch: a coalesced sweep of the
        // team's (L2-resident) slots, a 16-byte store per two.
        if (given_up(p, team_barrier(t))) return;
        for (unsigned m = used; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            uint4* base = reinterpret_cast<uint4*>(hop_table(p, team_id, k).slots);
            const uint4 ones = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
            for (int i = t.rank * kThreads + (int)threadIdx.x; i < (1 << (k - 1)); i += t.size * kThreads) base[i] = ones;
        }
        if (b + p.n_teams < p.n_batches) {
            if (given_up(p, team_barrier(t))) return;
        }
    }
}

// Explicit-edge mapping (the drop-in transfer_edge_id).  The table was cleared by the host.
template <bool ARRIVAL>
__global__ void __launch_bounds__(kThreads, kMinCtas) map_kernel(const __grid_constant__ KParams p) {
    __shared__ Smem sm;
    Team t;
    t.rank = blockIdx.x;
    t.size = gridDim.x;
    t.epoch = 0;
    t.bar = p.barriers;
    t.status = p.status;
    int32_t* team_sums = p.team_sums;
    Table tab;
    tab.slots = p.table;
    tab.mask = (uint32_t)(p.table_slots / kBucket - 1);
    tab.shift = p.table_shift;
    const int n_seeds = p.n_seeds_host;
    const int n_edges = (int)p.map_edges;
    int32_t* unique = p.nodes;
    const int64_t nodes_cap = p.nodes_stride;

    int s0, s1;
    chunk_of(n_seeds, t.rank, t.size, s0, s1);
    for (int s = s0 + (int)threadIdx.x; s < s1; s += kThreads) {
        const int v = p.seeds[s];
        unique[s] = v;  // id_map.cu:285
        if (v < 0)
            set_status(p.status, FGL_ERR_BOUNDS);
        else
            table_insert_seed(tab, (uint32_t)v, (uint32_t)s, p.status);
    }
    if (t.rank == 0 && threadIdx.x == 0) p.counts[1] = n_seeds;
    if (!team_barrier(t)) return;

    int e0, e1;
    chunk_of(n_edges, t.rank, t.size, e0, e1);
    for (int e = e0 + (int)threadIdx.x; e < e1; e += kThreads) {
        const int g = p.map_src[e];
        if (g < 0) {
            set_status(p.status, FGL_ERR_BOUNDS);
            p.map_src[e] = 0;
        } else {
            // same table as the fused kernel; n_nodes is not known here
            bool created;
            int displaced;
            int r = table_insert<ARRIVAL>(tab, (uint32_t)g, (uint32_t)e, p.status, created, displaced);
            if (ARRIVAL && created) {
                cg::coalesced_group grp = cg::coalesced_threads();
                int base = 0;
                if (grp.thread_rank() == 0) base = atomicAdd(p.counts + 1, (int)grp.size());
                base = grp.shfl(base, 0);
                const int local = base + (int)grp.thread_rank();
                const uint32_t pos = (uint32_t)~r;
                if ((int64_t)local < nodes_cap) {
                    unique[local] = g;
                    atomicExch(tab.slots + pos, ((unsigned long long)(uint32_t)g << 32) | (uint32_t)local);
                    r = local;
                } else {
                    set_status(p.status, FGL_ERR_CAPACITY);
                    atomicExch(tab.slots + pos, ((unsigned long long)(uint32_t)g << 32));
                    r = 0;
                }
            }
            p.map_src[e] = r;
        }
        if (p.map_dst) {  // id_map.cu:378-381; the seeds all have their ids since the barrier
            const int d = p.map_dst[e];
            p.map_dst[e] = d < 0 ? 0 : table_lookup(tab, (uint32_t)d, p.status);
            if (d < 0) set_status(p.status, FGL_ERR_BOUNDS);
        }
    }
    if (!team_barrier(t)) return;
    if (!ARRIVAL) {
        phase_count_first(tab, p.map_src, e0, e1, t, sm, team_sums);
        if (!team_barrier(t)) return;
        const int n_total = phase_rank(p, tab, p.map_src, e0, e1, unique, nodes_cap, n_seeds, t, sm, team_sums);
        if (t.rank == 0 && threadIdx.x == 0) p.counts[1] = (int)min((int64_t)n_total, nodes_cap);
        if (!team_barrier(t)) return;
    }
    phase_relabel(tab, p.map_src, e0, e1);
}

// ----------------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------------
constexpr int64_t kMaxTableBytes = 1LL << 30;

constexpr int64_t kSmallTable = 1 << 16;
constexpr int64_t kResidentTables = 48LL << 20;   // bytes

static int64_t pow2_at_least(int64_t n) {
    int64_t p = 1024;
    while (p < n) p <<= 1;
    return p;
}

static int log2_of(int64_t pow2) {
    int l = 0;
    while ((1LL << l) < pow2) ++l;
    return l;
}

template <auto kernel>
static int max_coresident(Workspace* ws, size_t dyn_smem, int* out) {
    if (dyn_smem > 48 * 1024)
        FGL_CUDA_OK(ws, cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem));
    // the answer does not change, and asking costs more than a launch (one static per kernel; the dynamic shared memory
    // is zero except for wide fanouts)
    static std::atomic<int> cached{0};
    int per_sm = dyn_smem == 0 ? cached.load(std::memory_order_relaxed) : 0;
    if (per_sm == 0) {
        FGL_CUDA_OK(ws, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, dyn_smem));
        if (dyn_smem == 0) cached.store(per_sm, std::memory_order_relaxed);
    }
    if (per_sm < 1) {
        ws->last_error = "kernel does not fit on an SM";
        return FGL_ERR_CUDA;
    }
    *out = per_sm * ws->sm_count;
    return FGL_OK;
}

template <typename K>
static int launch_coop(Workspace* ws, K kernel, int grid, size_t dyn_smem, KParams* kp, cudaStream_t st) {
    if (dyn_smem > 48 * 1024)
        FGL_CUDA_OK(ws, cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem));
    void* args[] = {(void*)kp};
    timing_begin(ws, st);
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(kThreads), args, dyn_smem, st);
    timing_end(ws, st);
    FGL_CUDA_OK(ws, e);
    return FGL_OK;
}

// scratch layout of the drop-in kernels: [barrier: 16 u64][team_sums: grid i32][counts: 16 i32]
// of the fused kernel: [barriers: n_teams * 16 u64][tile_sums: n_teams * 3 * kMaxTiles i32][team_cnt: 3 * grid i32]
//                      [node_start: n_teams * deg_stride i64][node_deg: n_teams * deg_stride i32]
// Only the part before node_start is zeroed per call.
static int64_t sums_bytes(int64_t words) { return ((words * 4 + 127) / 128) * 128; }

static int64_t scratch_head(int grid) { return 128 + sums_bytes(grid) + 128; }

static void place_scratch(Workspace* ws, KParams& kp, int grid, int32_t** call_counts) {
    char* base = ws->scratch;
    kp.barriers = (unsigned long long*)base;
    kp.team_sums = (int32_t*)(base + 128);
    *call_counts = (int32_t*)(base + scratch_head(grid) - 128);
    kp.status = ws->status;
}

static int64_t fused_head(int n_teams, int grid) {
    return (int64_t)n_teams * 128 + (int64_t)n_teams * 3 * kMaxTiles * 4 + sums_bytes(3 * (int64_t)grid);
}

static int64_t fused_need(int n_teams, int grid, int64_t deg_stride) {
    return fused_head(n_teams, grid) + (int64_t)n_teams * deg_stride * 12;
}

static void place_fused(Workspace* ws, KParams& kp, int n_teams, int grid, int64_t deg_stride) {
    char* base = ws->scratch;
    kp.barriers = (unsigned long long*)base;
    base += (size_t)n_teams * 128;
    kp.tile_sums = (int32_t*)base;
    base += (size_t)n_teams * 3 * kMaxTiles * 4;
    kp.team_cnt = (int32_t*)base;
    base = ws->scratch + fused_head(n_teams, grid);
    kp.node_start = (long long*)base;
    base += (size_t)n_teams * deg_stride * 8;
    kp.node_deg = (int32_t*)base;
    kp.deg_stride = deg_stride;
    kp.status = ws->status;
}

template <int MODE>
static int launch_sample_map(Workspace* ws, KParams& kp, bool is64, bool arrival, int grid, size_t dyn, cudaStream_t st) {
#define FGL_LAUNCH(PT, AR) launch_coop(ws, sample_map_kernel<PT, MODE, AR>, grid, dyn, &kp, st)
    if (is64) return arrival ? FGL_LAUNCH(int64_t, true) : FGL_LAUNCH(int64_t, false);
    return arrival ? FGL_LAUNCH(int32_t, true) : FGL_LAUNCH(int32_t, false);
#undef FGL_LAUNCH
}

template <int MODE>
static int occupancy_sample_map(Workspace* ws, bool is64, bool arrival, size_t dyn, int* out) {
#define FGL_OCC(PT, AR) max_coresident<sample_map_kernel<PT, MODE, AR>>(ws, dyn, out)
    if (is64) return arrival ? FGL_OCC(int64_t, true) : FGL_OCC(int64_t, false);
    return arrival ? FGL_OCC(int32_t, true) : FGL_OCC(int32_t, false);
#undef FGL_OCC
}

// dynamic shared memory: a row of picks per warp for fanouts beyond 32 (narrower fanouts keep their picks in registers)
static size_t picks_smem(int max_fanout) {
    return max_fanout > kGroupPathMaxFanout ? (size_t)kWarps * max_fanout * sizeof(uint32_t) : 0;
}

}  // namespace fgl

using namespace fgl;

extern "C" {

int fgl_fused_capacity(int64_t n_nodes, int32_t max_seeds, int32_t n_hops, const int32_t* fanout, int64_t* cap_nodes) {
    if (n_nodes <= 0 || max_seeds < 0 || n_hops < 1 || n_hops > FGL_MAX_HOPS || !fanout || !cap_nodes) return FGL_ERR_INVALID;
    cap_nodes[0] = max_seeds;
    for (int h = 0; h < n_hops; ++h) {
        if (fanout[h] < 1 || fanout[h] > FGL_MAX_FANOUT) return FGL_ERR_INVALID;
        const int64_t grown = cap_nodes[h] * (1 + (int64_t)fanout[h]);
        cap_nodes[h + 1] = std::max<int64_t>(cap_nodes[h], std::min<int64_t>(n_nodes, grown));
        if (cap_nodes[h] * (int64_t)fanout[h] > 0x7fffffffLL) return FGL_ERR_INVALID;
    }
    return FGL_OK;
}

int fgl_sample(fgl_ws* ws, const void* indptr, int indptr_is_64, const int32_t* indices, int64_t n_nodes,
               const int32_t* seeds, int32_t n_seeds, int32_t fanout, int32_t flags, uint64_t rng_seed,
               uint64_t rng_ctr, int32_t* out_indptr, int32_t* out_src, int32_t* out_dst, int64_t* n_edges_host,
               void* stream) {
    if (!ws || !indptr || !indices || n_nodes <= 0 || n_seeds < 0 || fanout < 1 || fanout > FGL_MAX_FANOUT ||
        (n_seeds > 0 && (!seeds || !out_src)) || (int64_t)n_seeds * fanout > 0x7fffffffLL)
        return FGL_ERR_INVALID;
    std::lock_guard<std::mutex> lock(ws->mu);
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    const size_t dyn = picks_smem(fanout);
    int max_grid = 0;
    int rc = occupancy_sample_map<MODE_SAMPLE>(ws, indptr_is_64 != 0, false, dyn, &max_grid);
    if (rc != FGL_OK) return rc;
    const int lanes = fanout <= 8 ? 8 : (fanout <= 16 ? 16 : 32);
    const int64_t seeds_per_cta = kThreads / lanes;
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(max_grid, (n_seeds + seeds_per_cta - 1) / seeds_per_cta));
    rc = ws_ensure(ws, 0, scratch_head(grid));
    if (rc != FGL_OK) return rc;
    KParams kp;
    std::memset(&kp, 0, sizeof(kp));
    int32_t* call_counts = nullptr;
    place_scratch(ws, kp, grid, &call_counts);
    kp.indptr = indptr;
    kp.indices = indices;
    kp.n_nodes = n_nodes;
    kp.n_batches = 1;
    kp.n_hops = 1;
    kp.fanout[0] = fanout;
    kp.flags = flags;
    kp.n_teams = 1;
    kp.team_size = grid;
    kp.rng_seed = rng_seed;
    kp.rng_ctr = rng_ctr;
    kp.seeds = seeds;
    kp.seed_stride = n_seeds;
    kp.seed_counts = nullptr;
    kp.n_seeds_host = n_seeds;
    kp.nodes = nullptr;
    kp.nodes_stride = n_seeds;
    kp.counts = call_counts;
    kp.blk_indptr[0] = out_indptr;
    kp.blk_src[0] = out_src;
    kp.out_dst = out_dst;
    kp.table = nullptr;
    kp.table_slots = 1024;
    kp.table_shift = 24;
    FGL_CUDA_OK(ws, cudaMemsetAsync(ws->scratch, 0, (size_t)scratch_head(grid), st));
    rc = launch_sample_map<MODE_SAMPLE>(ws, kp, indptr_is_64 != 0, false, grid, dyn, st);
    if (rc != FGL_OK) return rc;
    if (n_edges_host) {
        FGL_CUDA_OK(ws, cudaMemcpyAsync(ws->host_pinned, call_counts + 8, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        FGL_CUDA_OK(ws, cudaMemcpyAsync(ws->host_pinned + 1, ws->status, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        FGL_CUDA_OK(ws, cudaStreamSynchronize(st));
        *n_edges_host = ws->host_pinned[0];
        const int code = ws->host_pinned[1];
        if (code != FGL_OK) {
            FGL_CUDA_OK(ws, cudaMemsetAsync(ws->status, 0, 2 * sizeof(int32_t), st));
            ws->last_error = std::string("fgl_sample: ") + fgl_status_str(code);
            return code;
        }
    }
    return FGL_OK;
}

int fgl_map(fgl_ws* ws, int32_t* src, int32_t* dst, const int32_t* seeds, int32_t n_seeds, int64_t n_edges,
            int32_t* unique, int64_t unique_cap, int32_t flags, int64_t* n_unique_host, void* stream) {
    if (!ws || n_seeds < 0 || n_edges < 0 || n_edges > 0x7fffffffLL || (n_seeds > 0 && !seeds) || (n_edges > 0 && !src) ||
        !unique || unique_cap < n_seeds)
        return FGL_ERR_INVALID;
    std::lock_guard<std::mutex> lock(ws->mu);
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    const bool arrival = (flags & FGL_MAP_ARRIVAL_ORDER) != 0;
    int max_grid = 0;
    int rc = arrival ? max_coresident<map_kernel<true>>(ws, 0, &max_grid) : max_coresident<map_kernel<false>>(ws, 0, &max_grid);
    if (rc != FGL_OK) return rc;
    const int64_t work = std::max<int64_t>(n_edges, n_seeds);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(max_grid, (work + 2 * kThreads - 1) / (2 * kThreads)));
    // at most n_seeds + min(n_edges, unique_cap - n_seeds) distinct keys; load factor <= 2/3
    const int64_t max_keys = (int64_t)n_seeds + n_edges;
    const int64_t slots = pow2_at_least(max_keys + max_keys / 2 + 1);
    if (slots > (1LL << 31)) return FGL_ERR_CAPACITY;
    rc = ws_ensure(ws, slots, scratch_head(grid));
    if (rc != FGL_OK) return rc;
    KParams kp;
    std::memset(&kp, 0, sizeof(kp));
    int32_t* call_counts = nullptr;
    place_scratch(ws, kp, grid, &call_counts);
    kp.n_nodes = 0x7fffffff;
    kp.flags = flags;
    kp.n_teams = 1;
    kp.team_size = grid;
    kp.seeds = seeds;
    kp.n_seeds_host = n_seeds;
    kp.nodes = unique;
    kp.nodes_stride = unique_cap;
    kp.counts = call_counts;
    kp.map_src = src;
    kp.map_dst = dst;
    kp.map_edges = n_edges;
    kp.table = ws->table;
    kp.table_slots = slots;
    kp.table_shift = 32 - log2_of(slots / kBucket);
    FGL_CUDA_OK(ws, cudaMemsetAsync(ws->scratch, 0, (size_t)scratch_head(grid), st));
    FGL_CUDA_OK(ws, cudaMemsetAsync(ws->table, 0xFF, sizeof(unsigned long long) * (size_t)slots, st));
    ws->table_dirty = true;  // this call leaves its keys in the table
    rc = arrival ? launch_coop(ws, map_kernel<true>, grid, 0, &kp, st) : launch_coop(ws, map_kernel<false>, grid, 0, &kp, st);
    if (rc != FGL_OK) return rc;
    if (n_unique_host) {
        FGL_CUDA_OK(ws, cudaMemcpyAsync(ws->host_pinned, call_counts + 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        FGL_CUDA_OK(ws, cudaMemcpyAsync(ws->host_pinned + 1, ws->status, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        FGL_CUDA_OK(ws, cudaStreamSynchronize(st));
        *n_unique_host = ws->host_pinned[0];
        const int code = ws->host_pinned[1];
        if (code != FGL_OK) {
            FGL_CUDA_OK(ws, cudaMemsetAsync(ws->status, 0, 2 * sizeof(int32_t), st));
            ws->last_error = std::string("fgl_map: ") + fgl_status_str(code);
            return code;
        }
    }
    return FGL_OK;
}

int fgl_sample_map_fused(fgl_ws* ws, const fgl_fused_args* a, void* stream) {
    if (!a || !a->seed_counts) return FGL_ERR_INVALID;
    return fgl_sample_map_fused_extra(ws, a, nullptr, stream);
}

int fgl_sample_map_fused_extra(fgl_ws* ws, const fgl_fused_args* a, const fgl_fused_extra* extra, void* stream) {
    if (!ws || !a || !a->indptr || !a->indices || a->n_nodes <= 0 || a->n_batches < 0 || a->n_hops < 1 ||
        a->n_hops > FGL_MAX_HOPS || !a->seeds || !a->nodes || !a->counts || a->seed_stride < 0)
        return FGL_ERR_INVALID;
    if (a->n_batches == 0) return FGL_OK;
    int64_t cap[FGL_MAX_HOPS + 1];
    if (a->seed_stride > 0x7fffffffLL) return FGL_ERR_INVALID;
    int rc = fgl_fused_capacity(a->n_nodes, (int32_t)a->seed_stride, a->n_hops, a->fanout, cap);
    if (rc != FGL_OK) return rc;
    int max_fanout = 0;
    for (int h = 0; h < a->n_hops; ++h) {
        max_fanout = std::max(max_fanout, (int)a->fanout[h]);
        if (!a->block_indptr[h] || !a->block_src[h] || a->block_indptr_stride[h] < cap[h] + 1 ||
            a->block_src_stride[h] < cap[h] * a->fanout[h])
            return FGL_ERR_INVALID;
    }
    if (a->nodes_stride < cap[a->n_hops]) return FGL_ERR_INVALID;
    for (int h = 0; extra && h < a->n_hops; ++h)
        if (extra->block_dst[h] && a->n_batches != 1) return FGL_ERR_INVALID;
    for (int h = 0; h < a->n_hops; ++h)   // the relabelling passes read and write the edge entries four at a time
        if (((uintptr_t)a->block_src[h] & 15) != 0 || a->block_src_stride[h] % 4 != 0) return FGL_ERR_INVALID;
    const int64_t deg_stride = (cap[a->n_hops - 1] + 31) / 32 * 32;   // nodes that can still become seeds
    std::lock_guard<std::mutex> lock(ws->mu);
    DeviceGuard guard(ws->device);
    cudaStream_t st = (cudaStream_t)stream;
    const bool arrival = (a->flags & FGL_MAP_ARRIVAL_ORDER) != 0;
    const bool is64 = a->indptr_is_64 != 0;
    const size_t dyn = picks_smem(max_fanout);
    int max_grid = 0;
    rc = occupancy_sample_map<MODE_FUSED>(ws, is64, arrival, dyn, &max_grid);
    if (rc != FGL_OK) return rc;
    // The largest table of a team: sized for the worst case, or by the caller's hint (if it fills up the launch reports
    // FGL_ERR_PROBE and the caller retries without a hint).  All tables of a team together take twice that.
    int64_t slots = pow2_at_least(cap[a->n_hops] + cap[a->n_hops] / 2 + 1);
    if (a->table_slots_hint > 0) slots = std::min(slots, pow2_at_least(a->table_slots_hint));
    if (slots > (1LL << 29)) return FGL_ERR_CAPACITY;   // pending edge entries keep a slot number in 29 bits
    // A team per mini-batch of the window, up to 16: the small hops and the barriers of one mini-batch are covered by
    // the others' traffic.  Beyond four teams the tables together stay below kMaxTableBytes.
    int n_teams = a->n_teams;
    if (n_teams <= 0) n_teams = (int)std::max<int64_t>(4, std::min<int64_t>(16, kMaxTableBytes / (slots * 16)));
    n_teams = std::max(1, std::min(std::min(n_teams, (int)a->n_batches), max_grid));
    // CTAs per team: two edges per thread at the widest hop's worst case is all a small mini-batch can use
    int64_t widest = cap[0];
    for (int h = 0; h < a->n_hops; ++h) widest = std::max(widest, cap[h] * a->fanout[h]);
    const int team_size = (int)std::max<int64_t>(1, std::min<int64_t>(max_grid / n_teams, (widest + 2 * kThreads - 1) / (2 * kThreads)));
    if (team_size > kMaxTeam) return FGL_ERR_INVALID;
    const int grid = team_size * n_teams;
    rc = ws_ensure(ws, 2 * slots * n_teams, fused_need(n_teams, grid, deg_stride));
    if (rc != FGL_OK) return rc;
    if (ws->table_dirty) {
        FGL_CUDA_OK(ws, cudaMemsetAsync(ws->table, 0xFF, sizeof(unsigned long long) * (size_t)ws->table_slots, st));
        ws->table_dirty = false;
    }
    KParams kp;
    std::memset(&kp, 0, sizeof(kp));
    place_fused(ws, kp, n_teams, grid, deg_stride);
    kp.indptr = a->indptr;
    kp.indices = a->indices;
    kp.n_nodes = a->n_nodes;
    kp.n_batches = a->n_batches;
    kp.n_hops = a->n_hops;
    for (int h = 0; h < a->n_hops; ++h) {
        kp.fanout[h] = a->fanout[h];
        kp.tile_shift[h] = kMinTileShift;
        while ((cap[h] >> kp.tile_shift[h]) >= kMaxTiles) ++kp.tile_shift[h];
        kp.blk_indptr[h] = a->block_indptr[h];
        kp.blk_indptr_stride[h] = a->block_indptr_stride[h];
        kp.blk_src[h] = a->block_src[h];
        kp.blk_src_stride[h] = a->block_src_stride[h];
    }
    kp.flags = a->flags;
    kp.n_teams = n_teams;
    kp.team_size = team_size;
    kp.rng_seed = a->rng_seed;
    kp.rng_ctr = a->rng_ctr;
    kp.seeds = a->seeds;
    kp.seed_stride = a->seed_stride;
    kp.seed_counts = a->seed_counts;
    kp.n_seeds_host = (int32_t)a->seed_stride;  // without counts every mini-batch is full
    kp.nodes = a->nodes;
    kp.nodes_stride = a->nodes_stride;
    kp.counts = a->counts;
    if (extra) {
        kp.counts_host = extra->counts_host;
        kp.status_host = extra->status_host;
        kp.seq = extra->seq;
        for (int h = 0; h < a->n_hops; ++h) kp.blk_dst[h] = extra->block_dst[h];
    }
    kp.table = ws->table;
    // The first table covers the first hop's worst case, and every small mini-batch as a whole.  Tables that all fit the
    // L2 together are as large as they get from the start: moving to a larger one re-inserts the nodes.
    kp.table_log2_max = log2_of(slots);
    kp.table_log2_first = slots * n_teams * 8 <= kResidentTables
                              ? kp.table_log2_max
                              : log2_of(std::min(slots, std::max(kSmallTable, pow2_at_least(cap[1] + cap[1] / 4))));
    FGL_CUDA_OK(ws, cudaMemsetAsync(ws->scratch, 0, (size_t)fused_head(n_teams, grid), st));
    return launch_sample_map<MODE_FUSED>(ws, kp, is64, arrival, grid, dyn, st);
}

}  // extern "C"
