// Step kernels of the walk engine (replace GOWalker gpu/gpuwalk.hpp:87-319).
//
// In-core kernel: one persistent grid sized to fill the SMs.  Each lane owns
// one walker at a time and takes it to the end; a warp claims walker ids in
// claims of a few with one atomic and hands them to its idle lanes, so lanes
// whose walks end early (SOPR termination, dead ends) pick up new walkers
// instead of idling -- the work-stealing loop that replaces the reference's
// grid-stride loop (gpu/gpuwalk.hpp:200) and its one-walker-per-thread
// imbalance.  The loop body is one rejection-sampling trial, so lanes of a
// warp stay converged at trial granularity whatever their walk lengths.
//
// Walkers of the in-core kernel are generated from their id on the fly
// (engine/walk.hpp:32-49 for per-vertex init), so no walker record is read
// or written; per walker the kernel writes its path row (optional), length
// and 64-bit path hash.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include "gw_kernels.cuh"
#include "../../include/gowalker.h"

namespace gw {

// Words of a lane's walker parked in shared memory while its warp serves hard
// steps.
enum ParkWord : int {
    kPkWid = 0, kPkPrev, kPkCur, kPkHop, kPkAttempt, kPkDeg, kPkPdeg, kPkHeadLo, kPkHeadHi, kPkPheadLo,
    kPkPheadHi, kPkBucket, kPkPbucket, kPkMagic, kPkHashLo, kPkHashHi, kPkThr0, kPkThr1, kPkThr2, kPkTrials, kPkCount
};

// CTAs of an SM the kernel is built for: 5 leave 48 registers a thread, 4 leave
// 64.  Measured, 5 against 4: n2v_large-like 3.17 / 3.31 ms, SOPR over 128 M
// edges 29.6 / 30.8, weighted 0.67 / 0.70, L2-resident Node2vec 1.75 / 1.72;
// Node2vec with hard steps (p 0.25, q 4) spills at 48: 3.81 / 3.25.  (6 and 8
// spill everywhere and lose 5-100 %.)
__host__ __device__ constexpr int walk_ctas(bool sopr, bool coop) { return coop && !sopr ? 4 : 5; }

// W: weighted Node2vec -- the trial's candidate is alias column r.x % deg,
// kept when float(r.w >> 8) * 2^-24 < its probability, else its alias (the
// alias tables of gw_weighted.cu); everything else is the unweighted step.
//
// One round of the loop is one trial of every active lane: the draw, the
// candidate, then the new vertex's record and (where the verdict needs it) the
// search of N(prev), in flight together.  A warp spends the time of its
// longest lane in each part, so the parts that differ between lanes are kept
// short: one draw for accepted, rejected and new walkers alike, a membership
// table (csr_contains), one load for a vertex's record.  GROUPS: with fewer
// walkers than lanes several lanes share one (Group); runs that fill the lanes
// are bound by instructions, and groups at their end alone lose (n2v_corpus-like
// runs 1.70 / 1.88 ms without / with).
//
// SURE: every trial accepts (p = q = 1, first-order walks): no verdict, no
// search, nothing of the previous vertex, and no groups, which only save
// attempts that reject (3,878 walkers of length 80: 0.15 ms, 0.20 with groups;
// 200,000 of length 40: 0.20 ms, 0.25 with the verdict).  8 CTAs an SM are 8 %
// slower on a million walkers.
template <bool SOPR, bool PATHS, bool COOP, bool W, int SEARCH, bool GROUPS, bool SURE>
__global__ void __launch_bounds__(kWalkThreads, walk_ctas(SOPR, COOP))
    k_walk_incore(const __grid_constant__ IncoreArgs a)
{
    __shared__ uint32_t s_iv[COOP ? kWalkThreads / 32 : 1][kCoopScratchWords];  // scratch of warp_first_accept
    __shared__ unsigned long long s_ws[kWalkThreads / 32][kWsCount];  // per-warp statistics
    __shared__ unsigned long long s_hash[kWalkThreads], s_steps[kWalkThreads];  // per lane, of finished walkers
    __shared__ uint32_t s_done[kWalkThreads];
    __shared__ uint32_t s_park[COOP ? kWalkThreads / 32 : 1][kPkCount][32];  // lane state during hard steps
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if (lane < kWsCount) s_ws[warp][lane] = 0;
    s_hash[threadIdx.x] = s_steps[threadIdx.x] = 0;
    s_done[threadIdx.x] = 0;
    __syncwarp();
    constexpr bool INDEX = SEARCH == kTable;
    constexpr int kHard = INDEX ? kTable : kQuarter;  // a hard step's list stays in the L1
    const auto ix = [&]() {
        if constexpr (SEARCH == kLevels) return CsrIndex<kLevels>{a.csr, &a.levels};
        else return CsrIndex<SEARCH>{a.csr, a.table};
    }();
    const uint32_t *__restrict__ csr = a.csr;
    const uint32_t maxhops = a.c.maxhops;
    const uint32_t chunk = a.chunk;
    Group grp;
    if constexpr (GROUPS)
        while (grp.shift < kMaxGroupShift && (a.slots << (grp.shift + 1)) <= 32u) ++grp.shift;

    uint32_t q_next = 0, q_end = 0;  // warp-uniform claimed range
    constexpr bool kOneWave = GROUPS || SURE;  // (the others, which fill the lanes, lose 9 % by these lines)
    if (kOneWave && a.claims_end == 0) {
        const unsigned long long base = ((unsigned long long)warp * gridDim.x + blockIdx.x) * chunk;
        q_next = (uint32_t)min(base, (unsigned long long)a.nwalkers);
        q_end = (uint32_t)min(base + chunk, (unsigned long long)a.nwalkers);
    }
    bool exhausted = false;          // warp-uniform
    bool active = false;

    // Lane state.  Statistics live in shared memory and the path row is
    // recomputed from wid, so the registers hold only what the next trial
    // reads.  `attempt` is the attempt the next trial evaluates.
    uint32_t wid = 0, prev = 0, cur = 0, hop = 0, attempt = 0;
    uint32_t deg = 0, pdeg = 0, bucket = 0, pbucket = 0, magic = 0;
    uint64_t head = 0, phead = 0, h = 0;
    StepThr t{0.f, 0.f, 0.f};
    uint32_t n_trials = 0;  // trials not yet added to s_ws

    // A walker's steps are its hops: every accepted trial moves it one hop.
    // Lane 0 of a group writes what its walker writes.
    auto leads = [&]() { return grp.sub(lane) == 0; };
    auto finish = [&]() {
        active = false;
        if (!leads()) return;
        a.hashes[wid - a.out_base] = h;
        a.lens[wid - a.out_base] = hop + 1;
        s_steps[threadIdx.x] += hop;
        s_hash[threadIdx.x] += h;
        s_done[threadIdx.x] += 1;
    };

    for (;;) {
        // Hand walkers to idle groups.
        for (;;) {
            const unsigned need = __ballot_sync(0xFFFFFFFFu, !active && (!(GROUPS || SURE) || (lane >> grp.shift) < a.slots));
            if (need == 0 || exhausted) break;
            if (q_next >= q_end) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&a.ctr[kCtrCursor], (unsigned long long)chunk);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                if (base >= (kOneWave ? a.claims_end : a.nwalkers)) {
                    exhausted = true;
                    break;
                }
                q_next = (uint32_t)base;
                q_end = (uint32_t)min(base + chunk, (unsigned long long)a.nwalkers);
            }
            const uint32_t avail = q_end - q_next;
            const uint32_t rank = __popc(need & ((1u << grp.base(lane)) - 1u)) >> grp.shift;
            if (((need >> lane) & 1u) && rank < avail) {
                wid = a.wid_base + q_next + rank;
                const uint32_t src = walker_source(a.init, wid);
                prev = cur = src;
                hop = 0;
                attempt = 0;
                h = hash_init(src);
                if (PATHS && leads()) a.paths[(uint64_t)(wid - a.out_base) * a.stride] = src;
                Vertex vx{0, 0, 0, 0};
                if (src >= a.nverts) atomicOr(a.err, kErrSource);
                else if (maxhops != 0) vx = load_vertex<INDEX, SEARCH == kLevels>(a, src);
                deg = vx.deg;
                if (deg == 0) {
                    finish();  // bad source, no steps asked for, or a dead end (engine/engine.hpp:196-199)
                } else {
                    phead = head = vx.head;
                    pbucket = bucket = vx.bucket;
                    pdeg = deg;
                    magic = vx.magic;
                    t = step_thresholds<SOPR>(a.c, deg, pdeg);
                    active = true;
                }
            }
            q_next += min((uint32_t)__popc(need) >> grp.shift, avail);
        }
        const unsigned act = __ballot_sync(0xFFFFFFFFu, active);
        if (act == 0) break;
        if (GROUPS && exhausted && grp.shift < kMaxGroupShift && 2 * __popc(act) <= 32) {
            // the last walkers spread over the lanes that have none left
            const int from = (int)regroup(grp, act, lane, active);
            wid = __shfl_sync(0xFFFFFFFFu, wid, from);
            prev = __shfl_sync(0xFFFFFFFFu, prev, from);
            cur = __shfl_sync(0xFFFFFFFFu, cur, from);
            hop = __shfl_sync(0xFFFFFFFFu, hop, from);
            attempt = __shfl_sync(0xFFFFFFFFu, attempt, from);
            deg = __shfl_sync(0xFFFFFFFFu, deg, from);
            pdeg = __shfl_sync(0xFFFFFFFFu, pdeg, from);
            bucket = __shfl_sync(0xFFFFFFFFu, bucket, from);
            pbucket = __shfl_sync(0xFFFFFFFFu, pbucket, from);
            magic = __shfl_sync(0xFFFFFFFFu, magic, from);
            head = shfl64(head, from);
            phead = shfl64(phead, from);
            h = shfl64(h, from);
            t = shfl_thr<SOPR>(t, from);
        }

        // Walkers whose step keeps rejecting (a low-degree prev next to a hub
        // under SOPR) are served one at a time by the whole warp, which finds
        // their accepting attempt; the lane then takes it below.  Meanwhile
        // every lane's walker is parked in shared memory: the registers go to
        // the attempt loop, and lane L's fields reach all lanes as broadcast
        // loads.
        if (COOP) {
            const unsigned hm = __ballot_sync(0xFFFFFFFFu, active && attempt >= kHardAttempts && leads());
            if (hm) {
                uint32_t(*pk)[32] = s_park[COOP ? warp : 0];
                pk[kPkWid][lane] = wid;
                pk[kPkPrev][lane] = prev;
                pk[kPkCur][lane] = cur;
                pk[kPkHop][lane] = hop;
                pk[kPkAttempt][lane] = attempt;
                pk[kPkDeg][lane] = deg;
                pk[kPkPdeg][lane] = pdeg;
                pk[kPkHeadLo][lane] = (uint32_t)head;
                pk[kPkHeadHi][lane] = (uint32_t)(head >> 32);
                pk[kPkPheadLo][lane] = (uint32_t)phead;
                pk[kPkPheadHi][lane] = (uint32_t)(phead >> 32);
                pk[kPkBucket][lane] = bucket;
                pk[kPkPbucket][lane] = pbucket;
                pk[kPkMagic][lane] = magic;
                pk[kPkHashLo][lane] = (uint32_t)h;
                pk[kPkHashHi][lane] = (uint32_t)(h >> 32);
                pk[kPkThr0][lane] = __float_as_uint(t.inv_deg);
                pk[kPkThr1][lane] = __float_as_uint(t.sum);
                pk[kPkThr2][lane] = __float_as_uint(t.t_prev);
                pk[kPkTrials][lane] = n_trials;
                __syncwarp();
                for (unsigned m = hm; m; m &= m - 1) {
                    const int L = __ffs(m) - 1;
                    const uint32_t p0 = pk[kPkAttempt][L];
                    const uint32_t Lprev = pk[kPkPrev][L], Lcur = pk[kPkCur][L], Lpdeg = pk[kPkPdeg][L];
                    const uint64_t hd = ((uint64_t)pk[kPkHeadHi][L] << 32) | pk[kPkHeadLo][L];
                    const uint64_t ph = ((uint64_t)pk[kPkPheadHi][L] << 32) | pk[kPkPheadLo][L];
                    const StepThr tl{__uint_as_float(pk[kPkThr0][L]), __uint_as_float(pk[kPkThr1][L]),
                                     __uint_as_float(pk[kPkThr2][L])};
                    const uint32_t astar = warp_first_accept<SOPR>(
                        a.c, tl, pk[kPkWid][L], pk[kPkHop][L], p0, kMaxAttempts, csr + hd, pk[kPkDeg][L],
                        pk[kPkMagic][L], Lprev, Lcur, CsrIndex<kHard>{csr + ph, a.table}, pk[kPkPbucket][L], Lpdeg,
                        s_iv[COOP ? warp : 0]);
                    __syncwarp();  // every lane has read lane L's fields
                    if (lane == 0) {
                        pk[kPkAttempt][L] = astar;
                        const bool by_pos = by_position<SOPR>(tl, Lpdeg, Lprev, Lcur);
                        s_ws[warp][by_pos ? kWsCoopSmall : kWsCoopLarge] += 1ull;
                        s_ws[warp][by_pos ? kWsCoopSmallAtt : kWsCoopLargeAtt] += (unsigned long long)(astar - p0 + 1);
                    }
                }
                __syncwarp();
                wid = pk[kPkWid][lane];
                prev = pk[kPkPrev][lane];
                cur = pk[kPkCur][lane];
                hop = pk[kPkHop][lane];
                attempt = pk[kPkAttempt][grp.base(lane)];
                deg = pk[kPkDeg][lane];
                pdeg = pk[kPkPdeg][lane];
                head = ((uint64_t)pk[kPkHeadHi][lane] << 32) | pk[kPkHeadLo][lane];
                phead = ((uint64_t)pk[kPkPheadHi][lane] << 32) | pk[kPkPheadLo][lane];
                bucket = pk[kPkBucket][lane];
                pbucket = pk[kPkPbucket][lane];
                magic = pk[kPkMagic][lane];
                h = ((uint64_t)pk[kPkHashHi][lane] << 32) | pk[kPkHashLo][lane];
                t.inv_deg = __uint_as_float(pk[kPkThr0][lane]);
                t.sum = __uint_as_float(pk[kPkThr1][lane]);
                t.t_prev = __uint_as_float(pk[kPkThr2][lane]);
                n_trials = pk[kPkTrials][lane];
                if (active && attempt >= kMaxAttempts) {
                    atomicOr(a.err, kErrTrials);
                    finish();
                }
                __syncwarp();
            }
        }

        // One rejection-sampling trial a lane.
        if (!GROUPS && !active) continue;
        const bool last = hop + 1 >= maxhops;
        bool end = false;    // the step's termination draw ends the walk
        int verdict = 0;
        uint32_t x = 0;
        Vertex vx{0, 0, 0, 0};
        if (active) {
            const uint32_t att = attempt + grp.sub(lane);
            const U4 r = draw(a.c, wid, hop, att);
            end = att == 0 && hop != 0 && terminates(a.c, r.z);
            if (!GROUPS && end) {
                finish();
                continue;
            }
            const uint32_t pos = SURE && !INDEX ? r.x % deg : mod_by(r.x, deg, magic);
            const float rv = rand_val(r.y, thr_max<SOPR>(a.c, t));
            uint32_t col = pos;
            if constexpr (W) {
                const uint2 e = __ldg(a.alias + head + pos);
                // (a column past the list: a borrowed graph was written since its tables were built)
                if (!(__uint2float_rn(r.w >> 8) * 0x1p-24f < __uint_as_float(e.x))) col = e.y < deg ? e.y : pos;
            }
            x = __ldg(csr + head + col);
            if (SURE) verdict = 1;
            else if (!GROUPS || (!end && att < kMaxAttempts)) verdict = accept_without_prev<SOPR>(a.c, t, rv, x, prev, cur);
            // the record of a vertex that is, or may be, the next one
            if (verdict != 0 && !last && x < a.nverts) vx = load_vertex<INDEX, SEARCH == kLevels>(a, x);
            if (!SURE && verdict < 0)
                verdict = csr_contains(ix, pbucket, phead, pdeg, x) ? rv < thr_found<SOPR>(a.c, t)
                                                                    : rv < thr_notfound<SOPR>(a.c, t);
        }
        uint32_t first = 0;  // the accepting attempt, from `attempt`
        if (GROUPS && grp.shift) {
            const unsigned acc = grp.mine(__ballot_sync(0xFFFFFFFFu, verdict != 0), lane);
            end = grp.mine(__ballot_sync(0xFFFFFFFFu, end), lane) != 0;
            first = acc ? (uint32_t)__ffs(acc) - 1 : 0u;
            verdict = acc != 0;
            const int from = (int)(grp.base(lane) + first);
            x = __shfl_sync(0xFFFFFFFFu, x, from);
            vx.head = shfl64(vx.head, from);
            vx.deg = __shfl_sync(0xFFFFFFFFu, vx.deg, from);
            vx.bucket = __shfl_sync(0xFFFFFFFFu, vx.bucket, from);
            vx.magic = __shfl_sync(0xFFFFFFFFu, vx.magic, from);
        }
        if (GROUPS && !active) continue;
        if (GROUPS && end) {
            finish();
        } else if (verdict) {
            if (leads()) {
                n_trials += attempt + first + 1;  // a step's trials are counted when it is taken
                if (PATHS) a.paths[(uint64_t)(wid - a.out_base) * a.stride + hop + 1] = x;
                if (n_trials & 0x80000000u) {  // a step adds < 2^27: no wrap
                    atomicAdd(&s_ws[warp][kWsTrials], (unsigned long long)n_trials);
                    n_trials = 0;
                }
            }
            hop++;
            h = hash_step(h, x);
            attempt = 0;
            prev = cur;
            phead = head;
            pdeg = deg;
            pbucket = bucket;
            cur = x;
            head = vx.head;
            deg = vx.deg;
            bucket = vx.bucket;
            magic = vx.magic;
            if (!last && x >= a.nverts) atomicOr(a.err, kErrVertexRange);
            if (deg == 0) finish();  // the last hop, a bad id, or a dead end
            else t = step_thresholds<SOPR>(a.c, deg, pdeg);
        } else {
            attempt += grp.size();
            if (attempt >= kMaxAttempts) {
                atomicOr(a.err, kErrTrials);
                finish();
            }
        }
    }

    __syncwarp();
    const unsigned long long trials = warp_sum((unsigned long long)n_trials);
    const unsigned long long steps = warp_sum(s_steps[threadIdx.x]);
    const unsigned long long hashes = warp_sum(s_hash[threadIdx.x]);
    const unsigned long long done = warp_sum((unsigned long long)s_done[threadIdx.x]);
    if (lane == 0) {
        atomicAdd(&a.ctr[kCtrSteps], steps);
        atomicAdd(&a.ctr[kCtrTrials], trials + s_ws[warp][kWsTrials]);
        atomicAdd(&a.ctr[kCtrDone], done);
        atomicAdd(&a.ctr[kCtrHashSum], hashes);
        if (COOP) {
            atomicAdd(&a.ctr[kCtrCoopSmall], s_ws[warp][kWsCoopSmall]);
            atomicAdd(&a.ctr[kCtrCoopSmallAtt], s_ws[warp][kWsCoopSmallAtt]);
            atomicAdd(&a.ctr[kCtrCoopLarge], s_ws[warp][kWsCoopLarge]);
            atomicAdd(&a.ctr[kCtrCoopLargeAtt], s_ws[warp][kWsCoopLargeAtt]);
        }
    }
}

// Memory-safety check of a resident CSR before any walk reads it: offsets
// non-decreasing and within [0, nedges], every neighbour id < nverts; the
// vertex index is written from the same reads of the offsets.  (Adjacency
// order is a precondition -- the reference's `sorted` option -- and affects
// results, not safety.)  Bound by reading the CSR once: eight ids (one sector)
// per thread and load.  A warp takes its vertices' buckets with one atomic.
//
// a.sum: a sum over every offset and id, each mixed with its place, by which a
// later run sees that a borrowed CSR has been written.  One id's change always
// changes it (each mix is a bijection of the word), several do but for one time
// in 2^64.  Two ids a multiplication, so the pass stays bound by its reads.
constexpr uint64_t kSumA = 0x9E3779B97F4A7C15ull, kSumB = 0xD1342543DE82EF95ull, kSumC = 0xBF58476D1CE4E5B9ull;
__device__ __forceinline__ uint64_t sum_mix(uint64_t h, uint64_t w)
{
    h = (h ^ w) * kSumC;
    return h ^ (h >> 32);
}
__global__ void __launch_bounds__(256) k_validate_csr(const __grid_constant__ CsrCheck a)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    bool bad = false;
    uint64_t sum = 0;
    for (uint64_t v0 = t0 - lane; v0 < a.nverts; v0 += stride) {
        const uint64_t v = v0 + lane;
        uint64_t b = 0, e = 0;
        if (v < a.nverts) {
            b = a.beg[v];
            e = a.beg[v + 1];
            bad |= (b > e) | (e > a.nedges);
            if (a.sum) sum += sum_mix(v * kSumA, b * kSumB + e) * kSumB;
        }
        if (a.verts) {
            const uint32_t d = (uint32_t)(e - b);
            const uint32_t n = table_buckets(d);
            uint32_t x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            unsigned long long base = 0;
            if (lane == 31 && x) base = atomicAdd(a.nbuckets, (unsigned long long)x);
            base = __shfl_sync(0xFFFFFFFFu, base, 31);
            if (v < a.nverts) {
                a.verts[v] = make_uint4((uint32_t)b, d, (uint32_t)base + x - n, d ? mod_magic(d) : 0u);
                if (a.heads_hi) a.heads_hi[v] = (uint32_t)(b >> 32);
            }
        }
    }
    uint64_t done = 0;
    if (((uintptr_t)a.csr & 31u) == 0) {
        const uint64_t sectors = a.nedges / 8;
        for (uint64_t j = t0; j < sectors; j += stride) {
            uint32_t v[8];
            load_sector(a.csr + 8 * j, v);
#pragma unroll
            for (int i = 0; i < 8; ++i) bad |= v[i] >= a.nverts;
            if (a.sum) {
                uint64_t h = ~j * kSumA;
#pragma unroll
                for (int i = 0; i < 8; i += 2) h = sum_mix(h, ((uint64_t)v[i + 1] << 32) | v[i]);
                sum += h * kSumB;
            }
        }
        done = 8 * sectors;
    }
    for (uint64_t i = done + t0; i < a.nedges; i += stride) {
        const uint32_t x = __ldg(a.csr + i);
        bad |= x >= a.nverts;
        if (a.sum) sum += sum_mix(~i * kSumA, x) * kSumB;
    }
    if (a.sum) {
        sum = warp_sum((unsigned long long)sum);
        if (lane == 0) atomicAdd(a.sum, (unsigned long long)sum);
    }
    if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicOr(a.err, kErrVertexRange);
}

cudaError_t launch_validate_csr(const CsrCheck &a, int num_sms, cudaStream_t s)
{
    const uint64_t need = (std::max<uint64_t>(a.nverts, a.nedges / 8) + 255) / 256;  // one round of every thread
    k_validate_csr<<<(int)std::min<uint64_t>(need + 1, 8ull * num_sms), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// The membership tables: a thread takes `per` consecutive edges, finds the first
// one's vertex by halving the offsets and goes on from there, so hubs and
// isolated vertices cost alike.  An id claims the first free slot of its home
// bucket, from its own first slot round (table_slot), and of the buckets after
// it; an id met twice takes the same way and keeps one slot.  Bound by the
// claims, atomics into the L2, one after another in a thread: from each bucket's
// first slot on they were twice as many (31 M edges 1.43 ms, 1.05 so).  A small
// graph's edges are spread over all threads (30,000 edges: 106 us at 32 a
// thread, 14 us so), a large one's taken 16 at a time (63 M, claims from the
// first slot: 4.8 / 4.1 / 3.2 / 3.1 / 3.4 ms at 2 / 4 / 8 / 16 / 32; fewer repeat
// the search, more lengthen the last wave).
constexpr uint64_t kTableEdges = 16;
__global__ void __launch_bounds__(256) k_build_table(const uint64_t *__restrict__ beg, const uint4 *__restrict__ verts,
                                                     uint32_t nverts, const uint32_t *__restrict__ csr,
                                                     uint64_t nedges, uint32_t per, uint32_t *table)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * per;
    for (uint64_t e0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * per; e0 < nedges; e0 += stride) {
        uint32_t v = 0, hi = nverts;  // beg[v] <= e0 < beg[hi]
        while (hi - v > 1) {
            const uint32_t m = v + ((hi - v) >> 1);
            if (__ldg(beg + m) <= e0) v = m;
            else hi = m;
        }
        uint64_t end = __ldg(beg + v + 1);
        uint32_t buckets = 0, first = 0;
        const uint64_t e1 = min(e0 + per, nedges);
        for (uint64_t e = e0; e < e1; ++e) {
            while (e >= end) {
                ++v;
                end = __ldg(beg + v + 1);
                buckets = 0;
            }
            if (buckets == 0) {
                const uint4 r = __ldg(verts + v);
                buckets = table_buckets(r.y);
                first = r.z;
            }
            const uint32_t x = __ldg(csr + e);
            uint32_t b = table_home(x, buckets);
            for (bool placed = false; !placed;) {  // the slots outnumber the ids
                uint32_t *slot = table + ((uint64_t)first + b) * 8u;
                uint32_t k = table_slot(x);
                for (uint32_t i = 0; i < 8 && !placed; ++i) {
                    const uint32_t was = atomicCAS(slot + (i < 7 ? k : 7u), kEmptySlot, x);
                    placed = was == kEmptySlot || was == x;
                    k = k == 6 ? 0u : k + 1;
                }
                b = b + 1 == buckets ? 0u : b + 1;
            }
        }
    }
}

cudaError_t launch_build_table(const uint64_t *beg, const uint4 *verts, uint32_t nverts, const uint32_t *csr,
                               uint64_t nedges, uint32_t *table, int num_sms, cudaStream_t s)
{
    if (nedges == 0) return cudaSuccess;
    const uint64_t threads = 2048ull * num_sms;  // all resident
    const uint32_t per = (uint32_t)std::min(kTableEdges, (nedges + threads - 1) / threads);
    const uint64_t need = (nedges + 256ull * per - 1) / (256ull * per);
    k_build_table<<<(int)std::min<uint64_t>(need, 8ull * num_sms), 256, 0, s>>>(beg, verts, nverts, csr, nedges, per,
                                                                              table);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_sample_level(const uint32_t *__restrict__ src, uint64_t n,
                                                      uint32_t *__restrict__ dst)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) dst[j] = __ldg(src + 32 * j);
}

cudaError_t launch_sample_level(const uint32_t *src, uint64_t n, uint32_t *dst, int num_sms, cudaStream_t s)
{
    k_sample_level<<<(int)std::min<uint64_t>((n + 255) / 256, 8ull * num_sms), 256, 0, s>>>(src, n, dst);
    return cudaGetLastError();
}

bool wants_levels(uint64_t nwalkers, uint64_t nedges, bool sopr, bool sure, int num_sms)
{
    return !sopr && !sure && past_l2(nedges) && 4 * nwalkers > walk_lanes(num_sms);
}

uint64_t walk_lanes(int num_sms) { return (uint64_t)walk_ctas(false, false) * kWalkThreads * num_sms; }

template <bool SOPR, bool PATHS, bool COOP, bool W, int SEARCH, bool SURE>
static int resident_grid(int num_sms)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk_incore<SOPR, PATHS, COOP, W, SEARCH, false, SURE>,
                                                  kWalkThreads, 0);
    return (per_sm < 1 ? 1 : per_sm) * num_sms;
}

// f called with the kernel's template arguments as compile-time constants.
template <class F>
static auto walk_kernel(bool sopr, bool paths, bool coop, bool weighted, int search, bool sure, F &&f)
{
    using yes = std::true_type;
    using no = std::false_type;
    using quarter = std::integral_constant<int, kQuarter>;
    using levels = std::integral_constant<int, kLevels>;
    using table = std::integral_constant<int, kTable>;
    const auto by_search = [&](auto s, auto p, auto c, auto w, auto u) {
        if (search == kTable) return f(s, p, c, w, table{}, u);
        if constexpr (!s() && !u())
            if (search == kLevels) return f(s, p, c, w, levels{}, u);
        return f(s, p, c, w, quarter{}, u);
    };
    const auto by_paths = [&](auto s, auto c, auto w, auto u) {
        return paths ? by_search(s, yes{}, c, w, u) : by_search(s, no{}, c, w, u);
    };
    if (weighted) return sure ? by_paths(no{}, no{}, yes{}, yes{}) : by_paths(no{}, no{}, yes{}, no{});
    if (sopr) return by_paths(yes{}, yes{}, no{}, no{});  // SOPR steps get hard
    if (sure) return by_paths(no{}, no{}, no{}, yes{});
    return coop ? by_paths(no{}, yes{}, no{}, no{}) : by_paths(no{}, no{}, no{}, no{});
}

// Slots and claims by the number of walkers, which is what decides them first:
// - few walkers are spread over the warps, down to one each, as long as a
//   scheduler then has about four warps: a round costs a warp the instructions
//   of all its lanes' branches, so fewer walkers are faster until the schedulers
//   are busy (1,024 walkers of length 30, one lane a walker: 0.093 ms at one a
//   warp, 0.154 at 32; 65,536: 0.23 ms at 32, 0.32 at 16); walks of sure steps
//   go four a warp at least (3,878 walkers 0.107 ms at two, 0.080 at four);
// - a claim fills a warp when the run is one wave, so that no more warps than
//   needed share the walkers; later waves claim eight at a time, which evens
//   out the end of the run (600,000 walkers: 1.75 ms at 8, 1.82 at 32, 1.98 at
//   64; weighted 200,000: 0.67 / 0.77 / 0.76; hard Node2vec steps 3.25 / 4.44
//   / 4.62; SOPR on 16.8 M walkers: no difference); walks of sure steps end
//   together, so a claim fills the warp again; walks of a CSR past the L2
//   without tables wait for memory, and sixteen lanes a warp wait less than
//   thirty-two, so theirs are claims of eight in one wave too (100,000 walkers
//   on 64 M edges 0.66 ms, 0.82 at 32, through levels 0.67 / 0.90);
// - one wave's claims go to the first warp of every CTA, then to the second: taken
//   as warps come, they fell to the CTAs that started first, on some devices
//   several to an SM and none on others (180,000 walks of length 200 on one of
//   them 2.70 ms, 1.47 so; 100,000 sure ones 0.084, 0.057; elsewhere the same);
// - no more CTAs than walkers need where each gets an SM to itself: the others
//   find none, but take 12 us to come and go (3,878 sure walks 0.080 -> 0.062
//   ms, 1,024 of Node2vec 0.062 -> 0.049).
IncorePlan incore_plan(uint64_t nwalkers, uint64_t nedges, bool sopr, bool paths, bool coop, bool weighted,
                       int search, bool sure, int grid, int num_sms)
{
    IncorePlan p{};
    p.ctas_per_sm = (uint32_t)walk_ctas(sopr, coop);
    p.grid = grid > 0 ? grid
                      : walk_kernel(sopr, paths, coop, weighted, search, sure,
                                    [&](auto s, auto pa, auto c, auto w, auto i, auto u) {
                                        return resident_grid<s(), pa(), c(), w(), i(), u()>(num_sms);
                                    });
    const uint64_t warps = (uint64_t)p.grid * (kWalkThreads / 32), busy = std::min<uint64_t>(warps, 16ull * num_sms);
    p.slots = sure ? 4 : 1;
    while (p.slots < 32 && p.slots * busy < nwalkers) p.slots *= 2;
    const bool waits = !sure && search != kTable && past_l2(nedges);
    p.chunk = nwalkers <= 32 * warps ? (waits ? std::min(p.slots, 8u) : p.slots) : sure ? 32 : 8;
    const uint64_t need = (nwalkers + p.slots * (kWalkThreads / 32) - 1) / (p.slots * (kWalkThreads / 32));
    if (grid <= 0 && need <= (uint64_t)num_sms) p.grid = (int)need;
    p.one_wave = p.chunk == p.slots && need <= (uint64_t)p.grid;
    return p;
}

cudaError_t launch_walk_incore(const IncoreArgs &a, bool sopr, bool coop, int grid, cudaStream_t s)
{
    walk_kernel(sopr, a.paths != nullptr, coop, a.alias != nullptr, a.search, sure_steps(sopr, a.c),
                [&](auto so, auto pa, auto c, auto w, auto i, auto u) {
                    // (levels are read by runs that fill the lanes)
                    if (!u() && i() != kLevels && (a.slots < 32 || a.claims_end == 0))
                        k_walk_incore<so(), pa(), c(), w(), i(), !u() && i() != kLevels, u()><<<grid, kWalkThreads, 0, s>>>(a);
                    else
                        k_walk_incore<so(), pa(), c(), w(), i(), false, u()><<<grid, kWalkThreads, 0, s>>>(a);
                    return 0;
                });
    return cudaGetLastError();
}

}  // namespace gw
