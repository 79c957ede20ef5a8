// Launch interfaces of the engine's kernels (internal to libgowalker.so).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "gw_step.cuh"

namespace gw {

constexpr int kWalkThreads = 256;   // threads per CTA of the walk kernels
constexpr uint64_t kL2Bytes = 126ull << 20;
// Whether a CSR's ids take more of the L2 than walks leave them (two thirds).
inline bool past_l2(uint64_t nedges) { return 6 * nedges > kL2Bytes; }

// Work / statistics counters of one run (device, zeroed per run).
enum Counter : int {
    kCtrCursor = 0,   // next walker index to hand out
    kCtrSteps = 1,
    kCtrTrials = 2,
    kCtrDone = 3,
    kCtrHashSum = 4,  // wrapping sum of finished walkers' path hashes
    kCtrCoopSmall = 5,     // hard steps decided from candidate positions (prev degree < 32)
    kCtrCoopSmallAtt = 6,  // attempts those steps took
    kCtrCoopLarge = 7,     // hard steps evaluated with candidate loads and searches
    kCtrCoopLargeAtt = 8,  // attempts those steps took
    kCtrZcSectors = 9,     // out-of-core zero-copy tail: 32-byte sectors read from mapped host memory
    kCtrModelSectors = 10, // out-of-core, blocks resident: the sectors those steps would read from mapped memory
    kCtrRunnable = 11,     // out-of-core: walkers handed to the step kernels (sum over launches)
    kCtrCount = 12
};
// Behind the counters of an in-core run and the error word: the sum of a
// borrowed graph's contents (CsrCheck::sum) and that check's own error word.
constexpr int kCtrGraphSum = kCtrCount + 1, kCtrWords = kCtrCount + 3;

// Per-warp statistics a walk kernel keeps in shared memory and adds to the
// Counter slots when it ends.
enum WarpStat : int {
    kWsSteps = 0,
    kWsTrials,
    kWsDone,
    kWsHash,
    kWsCoopSmall,
    kWsCoopSmallAtt,
    kWsCoopLarge,
    kWsCoopLargeAtt,
    kWsCount
};

// Error word bits set by kernels instead of trapping.
enum ErrBit : uint32_t {
    kErrVertexRange = 1u,   // a neighbour id >= nverts
    kErrSource = 2u,        // a walker source >= nverts
    kErrBlock = 4u,         // a vertex outside every block, or a block scheduled absent
    kErrTrials = 8u,        // a step exceeded kMaxAttempts rejection trials
    kErrWeight = 16u,       // an edge weight that is not a positive finite number
};

// Rejection trials allowed for one step before the walker is stopped with
// kErrTrials.  Only degenerate parameters get near it (e.g. alpha = 1 on a
// directed graph whose N(cur) and N(prev) are disjoint): the worst R-MAT case
// of the SOPR rule, a step from a degree-1 vertex into a hub of degree d,
// needs 1 + alpha*d/(1-alpha) trials on average (~1.3e6 for d = 5e6), so a
// cap of 2^26 is never reached by a valid walk.
constexpr uint32_t kMaxAttempts = 1u << 26;

struct WalkerInit {
    uint32_t mode;       // GW_INIT_*
    uint32_t algo;       // GW_NODE2VEC / GW_SOPR / GW_SOSR
    uint32_t wps;        // walkers per vertex
    uint32_t numwalks;   // total walkers (single-source / random)
    uint32_t nverts;
    uint32_t key0, key1; // walk seed (random init)
};

struct IncoreArgs {
    StepConsts c;
    WalkerInit init;
    const uint64_t *beg;       // nverts+1 global offsets
    const uint32_t *csr;       // nedges neighbour ids
    uint64_t nedges;
    int search;                // Search: what of the index below the walk reads
    Levels levels;             // kLevels
    // kTable
    const uint4 *verts;        // {first edge (low word), degree, first bucket, mod_magic(degree)} per vertex
    const uint32_t *heads_hi;  // high words of the first edges; null when all are 0
    const uint32_t *table;     // membership tables (table_has)
    uint32_t nverts;
    uint32_t nwalkers;         // walkers of this launch: ids wid_base + i, i < nwalkers
    uint32_t wid_base;
    uint32_t out_base;         // first walker id of the population: outputs are indexed by wid - out_base
    uint32_t chunk;            // walkers a warp claims per atomic (incore_plan)
    uint32_t slots;            // walkers of a warp at a time (incore_plan)
    uint32_t claims_end;       // nwalkers; 0: a claim for every warp, by the warps' places and not by atomics
    uint32_t *paths;           // rows indexed by walker id, or null
    uint32_t stride;           // maxhops + 1
    uint32_t *lens;            // vertices per path
    uint64_t *hashes;          // FNV-1a per path
    unsigned long long *ctr;   // Counter slots
    uint32_t *err;             // ErrBit word
    const uint2 *alias;        // weighted Node2vec: {prob bits, alias column} per edge; null when unweighted
};

// Source vertex of walker `wid` (engine/walk.hpp:32-49 per-vertex ids
// v*wps+i; 82-95 and 355-384 single source 1, or 1 and 3 for SOSR).
__device__ __forceinline__ uint32_t walker_source(const WalkerInit &in, uint32_t wid)
{
    if (in.mode == 0u) return wid / in.wps;
    if (in.mode == 1u) {
        if (in.algo == 2u) return wid < in.numwalks / 2 ? 1u : 3u;
        return 1u;
    }
    const U4 r = philox4x32_10(wid, 0xFFFFFFFFu, 0u, kTagInit, in.key0, in.key1);
    return r.x % in.nverts;
}

// What a step reads of a vertex v < nverts.
struct Vertex {
    uint64_t head;   // first edge
    uint32_t deg;
    uint32_t bucket; // first bucket of its membership table
    uint32_t magic;  // mod_magic(deg)
};
// INDEX: from the vertex index, else from the offsets.  CHECK: offsets that are
// no valid list's (a borrowed CSR, written since it was checked) give a dead end.
template <bool INDEX, bool CHECK = false>
__device__ __forceinline__ Vertex load_vertex(const IncoreArgs &a, uint32_t v)
{
    if constexpr (INDEX) {
        const uint4 e = __ldg(a.verts + v);
        return Vertex{a.heads_hi ? ((uint64_t)__ldg(a.heads_hi + v) << 32) | e.x : e.x, e.y, e.z, e.w};
    }
    const uint64_t head = __ldg(a.beg + v), end = __ldg(a.beg + v + 1);
    uint32_t deg = (uint32_t)(end - head);
    if (CHECK && (head > end || end > a.nedges)) deg = 0;
    return Vertex{head, deg, 0u, deg ? mod_magic(deg) : 0u};
}

// Lanes of a warp in groups of `size`, one walker a group: every lane of a
// group holds the walker's whole state and evaluates one of its next `size`
// attempts, and the first one in order that decides the step counts.  A walk is
// a chain of trials, so where lanes are to spare -- few walkers, or the end of a
// run -- groups shorten it by the attempts that reject.
struct Group {
    uint32_t shift = 0;  // size = 2^shift
    __device__ uint32_t size() const { return 1u << shift; }
    __device__ uint32_t sub(uint32_t lane) const { return lane & (size() - 1u); }
    __device__ uint32_t base(uint32_t lane) const { return lane & ~(size() - 1u); }
    // this lane's group's bits of a ballot, from bit 0
    __device__ unsigned mine(unsigned ballot, uint32_t lane) const
    {
        return (ballot >> base(lane)) & (0xFFFFFFFFu >> (32u - size()));
    }
};
constexpr uint32_t kMaxGroupShift = 3;  // 8 attempts: 1 step in 12 of a 0.27 acceptance needs more

// Groups for a warp whose `act` (ballot) lanes hold the last walkers it will
// get: grown while all walkers fit.  Returns the lane whose state this lane
// takes over (itself when nothing changes), and whether it then holds a walker.
__device__ __forceinline__ uint32_t regroup(Group &g, unsigned act, uint32_t lane, bool &holds)
{
    const unsigned bases[] = {0xFFFFFFFFu, 0x55555555u, 0x11111111u, 0x01010101u};
    const unsigned b = act & bases[g.shift];  // a bit per walker
    const uint32_t n = (uint32_t)__popc(b);
    while (g.shift < kMaxGroupShift && (n << (g.shift + 1)) <= 32u) ++g.shift;
    const uint32_t slot = lane >> g.shift;
    holds = slot < n;
    return holds ? __fns(b, 0, (int)slot + 1) : lane;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}

// How an in-core run is launched.
struct IncorePlan {
    int grid;               // CTAs
    uint32_t slots, chunk, one_wave;  // IncoreArgs
    uint32_t ctas_per_sm;   // the kernel's register cap: CTAs of an SM it is built for
};
// `grid` CTAs as asked for, or (0) as many as are resident at once.
IncorePlan incore_plan(uint64_t nwalkers, uint64_t nedges, bool sopr, bool paths, bool coop, bool weighted,
                       int search, bool sure, int grid, int num_sms);
// a.alias set: weighted Node2vec.
cudaError_t launch_walk_incore(const IncoreArgs &a, bool sopr, bool coop, int grid, cudaStream_t s);

// One launch per hop (gw_walk_hop.cu): walker state between launches.
struct HopState {
    uint32_t *prev, *cur, *hop;
    uint64_t *hash;
};
// Launch `round` (0 .. maxhops-1) of the one-launch-per-hop walk: round 0
// starts every walker; each advances every live walker by one step.
cudaError_t launch_walk_hop(const IncoreArgs &a, const HopState &st, bool sopr, uint32_t round, int num_sms,
                            cudaStream_t s);

// Whether a run needs the warp-cooperative path for hard steps: always for
// SOPR/SOSR (acceptance ~ deg(prev)/deg(cur) next to hubs); for Node2vec
// only when max/min of {1/p, 1/q, 1} exceeds 8 (otherwise a step accepts
// within 1/ratio >= 1/8 per trial and never gets hard).
inline bool needs_coop(uint32_t algo, const StepConsts &c)
{
    return algo != 0u || c.n2v_maxv > 8.0f * c.n2v_minv;
}
// Whether every Node2vec trial accepts: 1/p, 1/q and 1 are one value, which no
// rand value exceeds.
inline bool sure_steps(bool sopr, const StepConsts &c) { return !sopr && c.n2v_maxv == c.n2v_minv; }
// One pass over a resident CSR before any walk reads it: error bits for
// offsets that are not monotone within [0, nedges] and ids >= nverts, and, in
// the same pass, the vertex index (verts null: none) with a place for every
// vertex's table; *nbuckets counts the buckets.
struct CsrCheck {
    const uint64_t *beg;
    const uint32_t *csr;
    uint32_t nverts;
    uint64_t nedges;
    uint32_t *err;
    uint4 *verts;
    uint32_t *heads_hi;            // null: offsets below 2^32
    unsigned long long *nbuckets;
    unsigned long long *sum;       // null, or a 64-bit sum over the contents is added here
};
cudaError_t launch_validate_csr(const CsrCheck &a, int num_sms, cudaStream_t s);
// Walkers an in-core kernel holds at a time: the lanes of `walk_ctas` CTAs an SM.
uint64_t walk_lanes(int num_sms);
// Whether a run reads sample levels when it has no tables: Node2vec past the L2
// (one walker a vertex, without and with paths: 16 M edges 1.72 and 1.87 ms, by
// quarters 1.52 and 1.83; 23 M 1.33 and 1.44 / 1.34 and 1.64; 31 M 2.21 and 2.47
// / 2.09 to 2.42 and 3.14), with walkers for a quarter of the lanes (fewer wait
// for the chain of loads, which is longer: 64 M edges, 10,000 walkers 0.45 ms,
// 0.39 by quarters, 100,000 0.67 / 0.82; SOPR searches little: 128 M edges 28.2
// ms, 27.3 by quarters).
bool wants_levels(uint64_t nwalkers, uint64_t nedges, bool sopr, bool sure, int num_sms);
// dst[j] = src[32 * j] for j < n.
cudaError_t launch_sample_level(const uint32_t *src, uint64_t n, uint32_t *dst, int num_sms, cudaStream_t s);
// Fills the membership tables of a validated CSR; every slot is kEmptySlot before.
cudaError_t launch_build_table(const uint64_t *beg, const uint4 *verts, uint32_t nverts, const uint32_t *csr,
                               uint64_t nedges, uint32_t *table, int num_sms, cudaStream_t s);

}  // namespace gw
