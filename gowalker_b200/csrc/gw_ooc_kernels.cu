// Out-of-core kernels (replace GOWalker gpu/gpuwalk.hpp:87-372 and the host
// block choice of engine/schedule.hpp:70-138).
//
//  k_init_walkers  walker records from ids (engine/walk.hpp:32-95)
//  k_count         walkers per (prev block, cur block) bucket before the first
//                  step, warp-aggregated atomics (one atomic per distinct bucket
//                  per warp instead of one per walker, gpu/gpuwalk.hpp:179)
//  k_plan          exclusive scan of the bucket counts in one CTA (coalesced warp segments;
//                  the reference scans them on one thread, gpu/gpuwalk.hpp:321-338), with
//                  everything else the next decision and the scatter read
//  k_scatter       walkers into bucket order, finished walkers dropped
//                  (gpu/gpuwalk.hpp:340-360 + the spill of engine/walk.hpp:484-525)
//  k_runnable      ranges of the buckets whose two blocks are resident, and their
//                  counts cleared
//  k_schedule      GOwalker_scheduler_t::max_choose_blocks on the device
//  k_walk_ooc      the step kernel over runnable walkers; a walker stops when
//                  its next vertex lies in a block that is not resident, and
//                  counts itself in its new bucket
#include <cuda_runtime.h>
#include <cstdint>
#include "gw_ooc_kernels.cuh"

namespace gw {


__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t block_of(const uint32_t *vs, uint32_t nb, uint32_t v)
{
    // largest b with vs[b] <= v (vs[nb] = nverts > v)
    uint32_t lo = 0, hi = nb;  // invariant vs[lo] <= v < vs[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (vs[mid] <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t bucket_of(const WalkerRec &r, uint32_t nb)
{
    if (r.prev_blk == kFinished) return kNoBucket;
    return ((r.cur_blk & kNeedPrev) ? nb * nb : 0u) + r.prev_blk * nb + (r.cur_blk & ~kNeedPrev);
}

__global__ void k_init_walkers(WalkerInit in, const uint32_t *__restrict__ vstart, uint32_t nb, uint32_t wid0,
                               uint64_t n, WalkerRec *__restrict__ out, uint32_t *__restrict__ order,
                               uint32_t *__restrict__ keys, uint32_t *__restrict__ paths, uint32_t stride)
{
    __shared__ uint32_t s_vs[kMaxBlocks + 1];
    for (uint32_t i = threadIdx.x; i <= nb; i += blockDim.x) s_vs[i] = vstart[i];
    __syncthreads();
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const uint32_t wid = wid0 + (uint32_t)i;
        const uint32_t src = walker_source(in, wid);
        const uint32_t b = block_of(s_vs, nb, src);
        const uint64_t h = hash_init(src);
        WalkerRec r;
        r.wid = wid;
        r.prev = src;
        r.cur = src;
        r.hop = 0;
        r.prev_blk = b;
        r.cur_blk = b;
        r.hash_lo = (uint32_t)h;
        r.hash_hi = (uint32_t)(h >> 32);
        out[i] = r;
        order[i] = (uint32_t)i;
        keys[i] = bucket_of(r, nb);
        if (paths) paths[i * stride] = src;
    }
}

__global__ void k_count(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ n_ptr, uint32_t *__restrict__ counts)
{
    const uint64_t n = *n_ptr;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; base < n; base += step) {
        const uint64_t i = base + lane;
        const uint32_t b = (i < n) ? keys[i] : kNoBucket;
        const unsigned grp = __match_any_sync(0xFFFFFFFFu, b);
        if (b != kNoBucket && lane == (uint32_t)(__ffs(grp) - 1)) atomicAdd(&counts[b], (uint32_t)__popc(grp));
    }
}

// Half the threads an SM holds, so that the runnable pass and the block choice
// (1,024 threads each) find room beside it instead of behind it: they start 3 us
// after the plan, not 8.  Four rounds of 32 walkers in flight a warp make up for
// it (10 us for a million walkers either way).
__global__ void __launch_bounds__(256) k_scatter(const uint32_t *__restrict__ keys_in,
                                                 const uint32_t *__restrict__ order_in,
                                                 const uint32_t *__restrict__ n_ptr, uint32_t *__restrict__ cursor,
                                                 uint32_t *__restrict__ keys_out, uint32_t *__restrict__ order_out,
                                                 OocClock *clock)
{
    constexpr uint32_t R = 4;
    const uint64_t n = *n_ptr;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * R;
    for (uint64_t base = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull) * R; base < n; base += step) {
        uint32_t r[R], b[R], pos[R];
        unsigned grp[R];
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint64_t i = base + 32 * k + lane;
            b[k] = i < n ? keys_in[i] : kNoBucket;
            r[k] = i < n ? order_in[i] : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            grp[k] = __match_any_sync(0xFFFFFFFFu, b[k]);
            pos[k] = 0;
            if (b[k] != kNoBucket && (grp[k] & lt) == 0) pos[k] = atomicAdd(&cursor[b[k]], (uint32_t)__popc(grp[k]));
        }
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint32_t at = __shfl_sync(0xFFFFFFFFu, pos[k], __ffs(grp[k]) - 1) + (uint32_t)__popc(grp[k] & lt);
            if (b[k] != kNoBucket) {
                keys_out[at] = b[k];
                order_out[at] = r[k];
            }
        }
    }
    if (threadIdx.x == 0) atomicMax(&clock->scatter_end, global_ns());
}

// One-CTA scans over at most 2^21 entries (nblocks <= 1024).
constexpr int kScanThreads = 1024;


// Warp w of the CTA owns entries [w * seg, (w + 1) * seg) and walks them 32
// at a time, so every load and store of a round is one coalesced line; the
// warps' totals are scanned once through shared memory.
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, uint32_t lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    return x;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
    return x;
}

// Exclusive scan of the warps' totals: warp w gets the sum of warps < w.
__device__ __forceinline__ uint32_t cta_warp_base(uint32_t wtotal, uint32_t *total)
{
    __shared__ uint32_t s_t[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) s_t[warp] = wtotal;
    __syncthreads();
    if (warp == 0) {
        const uint32_t v = lane < (blockDim.x >> 5) ? s_t[lane] : 0u;
        const uint32_t inc = warp_incl_scan(v, lane);
        s_t[lane] = inc - v;
        if (lane == 31 && total) *total = inc;
    }
    __syncthreads();
    const uint32_t b = s_t[warp];
    __syncthreads();
    return b;
}

// Between the step and the scatter, all that needs one CTA: bucket offsets
// (and the scatter's cursors, which start there), the new number of sorted
// positions, per-pair totals (when `pairs` is given), and the counters and error
// word into mapped host memory.  Five launches and two copies of 2-5 us each
// before; the next decision may start as soon as this is done, beside the
// scatter.
__global__ void __launch_bounds__(kScanThreads) k_plan(const uint32_t *__restrict__ counts, uint32_t nn,
                                                       uint32_t *__restrict__ offsets, uint32_t *__restrict__ cursor,
                                                       uint32_t *__restrict__ pairs, uint32_t *__restrict__ n_out,
                                                       const unsigned long long *__restrict__ ctr,
                                                       const uint32_t *__restrict__ err, unsigned long long *snap,
                                                       OocClock *clock)
{
    __shared__ uint32_t s_total;
    if (threadIdx.x == 0) {
        const unsigned long long now = global_ns();
        if (clock->walk_start) clock->walk_ns += clock->walk_end - clock->walk_start;
        if (clock->plan_start) clock->bucket_ns += clock->scatter_end - clock->plan_start;
        clock->walk_start = 0;
        clock->plan_start = pairs ? now : clock->pairs_start;
    }
    const uint32_t n = 2 * nn;
    if (threadIdx.x <= kCtrCount) {
        snap[threadIdx.x] = threadIdx.x < kCtrCount ? ctr[threadIdx.x] : *err;
        __threadfence_system();
    }
    if (pairs)
        for (uint32_t k = threadIdx.x; k < nn; k += blockDim.x) pairs[k] = counts[k] + counts[nn + k];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t seg = ((n + nw - 1) / nw + 31u) & ~31u;
    const uint32_t lo = min(warp * seg, n), hi = min(lo + seg, n);
    uint32_t part = 0;
#pragma unroll 4
    for (uint32_t i = lo + lane; i < hi; i += 32) part += counts[i];
    uint32_t base = cta_warp_base(warp_sum(part), &s_total);  // (every thread is past its pairs)
#pragma unroll 4
    for (uint32_t i0 = lo; i0 < hi; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t v = i < hi ? counts[i] : 0u;
        const uint32_t inc = warp_incl_scan(v, lane);
        if (i < hi) {
            offsets[i] = cursor[i] = base + inc - v;
        }
        base += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        offsets[n] = s_total;
        *n_out = s_total;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_runnable(const uint32_t *__restrict__ offsets,
                                                           const __grid_constant__ TablePatch patch, uint32_t nb,
                                                           uint32_t lazy, uint32_t *__restrict__ counts,
                                                           const uint32_t **__restrict__ blk_csr,
                                                           unsigned long long *cursor, uint32_t *__restrict__ run_pre,
                                                           uint32_t *__restrict__ run_off, uint32_t *__restrict__ nrun)
{
    __shared__ uint8_t s_res[kMaxBlocks];
    __shared__ uint32_t s_cnt, s_sum;
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) {
        bool resident = blk_csr[i] != nullptr;
        for (uint32_t k = 0; k < patch.n; ++k)
            if (patch.block[k] == i) {
                blk_csr[i] = patch.csr[k];
                blk_csr[nb + i] = patch.alias[k];
                resident = patch.csr[k] != nullptr;
            }
        s_res[i] = resident;
    }
    if (threadIdx.x == 0) *cursor = 0;
    __syncthreads();
    const uint32_t nn = nb * nb, n = 2 * nn;
    // unflagged walkers need their current block (and, unless lazy, the
    // previous one); flagged walkers need both
    auto runnable = [&](uint32_t b) {
        const uint32_t pc = b < nn ? b : b - nn;
        const bool cur_ok = s_res[pc % nb] != 0, prev_ok = s_res[pc / nb] != 0;
        return cur_ok && (prev_ok || (lazy && b < nn));
    };
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t seg = ((n + nw - 1) / nw + 31u) & ~31u;
    const uint32_t lo = min(warp * seg, n), hi = min(lo + seg, n);
    uint32_t pc = 0, ps = 0;
#pragma unroll 4
    for (uint32_t b = lo + lane; b < hi; b += 32) {
        const uint32_t c = offsets[b + 1] - offsets[b];
        if (c && runnable(b)) {
            pc++;
            ps += c;
        }
    }
    uint32_t kb = cta_warp_base(warp_sum(pc), &s_cnt);
    uint32_t sb = cta_warp_base(warp_sum(ps), &s_sum);
#pragma unroll 4
    for (uint32_t b0 = lo; b0 < hi; b0 += 32) {
        const uint32_t b = b0 + lane;
        const uint32_t c = b < hi ? offsets[b + 1] - offsets[b] : 0u;
        const bool f = c && runnable(b);
        const unsigned fm = __ballot_sync(0xFFFFFFFFu, f);
        const uint32_t v = f ? c : 0u;
        const uint32_t inc = warp_incl_scan(v, lane);
        if (f) {
            const uint32_t k = kb + (uint32_t)__popc(fm & lt);
            run_off[k] = offsets[b];
            run_pre[k] = sb + inc - v;
            counts[b] = 0;  // the step takes all of them, and counts each where it stops
        }
        kb += (uint32_t)__popc(fm);
        sb += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *nrun = s_cnt;
        run_pre[s_cnt] = s_sum;
    }
}

// Block choice, GOwalker_scheduler_t::max_choose_blocks (engine/schedule.hpp:70-138):
//  cache not full: for every uncached block i, score = sum over cached c of
//    walkers(i,c) + walkers(c,i), plus walkers(i,i); the best block is added.
//  cache full: for every uncached i, s_j = walkers(i,c_j) + walkers(c_j,i);
//    score = sum_j s_j - min_j s_j and i replaces the cached block with the
//    smallest s_j (first such j).
//  A block is taken only if its score is > 0 and > zero_threshold; ties go to
//  the lowest block id (the reference's std::sort leaves their order open).
// Rescue choice, for runs without the zero-copy tail (where the reference
// would switch to it): the fullest bucket with an absent block; load its first
// absent block, evicting the cached block with the fewest incident walkers
// outside that bucket -- after at most two rescues the bucket runs, so every
// run ends.  `pred` (optional, the learned policy): each block's forecast of
// log1p(incident walkers over the next iterations); with a full cache the
// chosen block then replaces the cached block with the lowest forecast
// instead of the one with the smallest link (pred_weight is unused).
// One CTA on the path from a plan to the next block's copy.  Up to
// kSchedShared blocks the counts come into shared memory in one round trip, and
// the choices are reduced by shuffles, not by an atomic for every bucket: 7.5 us
// at 24 blocks, 12 before.
constexpr uint32_t kSchedShared = 64;  // 16 KB of counts
__device__ __forceinline__ unsigned long long warp_max(unsigned long long x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xFFFFFFFFu, x, o));
    return x;
}
__device__ __forceinline__ unsigned long long warp_min(unsigned long long x) { return ~warp_max(~x); }

struct CachedList {
    uint16_t block[kMaxBlocks];  // an argument: no read of mapped host memory on the decision's path
};
// 32 registers: with 64 it waits for an SM of its own.
__global__ void __launch_bounds__(1024, 2) k_schedule(const uint32_t *__restrict__ all_counts,
                                                   const uint32_t *__restrict__ live, uint32_t nb,
                                                   const __grid_constant__ CachedList cached, uint32_t ncached,
                                                   uint32_t nslots, uint32_t zero_threshold,
                                                   const float *__restrict__ pred, float pred_weight,
                                                   Decision *__restrict__ out)
{
    __shared__ uint8_t s_cached[kMaxBlocks];
    __shared__ uint32_t s_list[kMaxBlocks];
    __shared__ uint32_t s_pos[kMaxBlocks];
    __shared__ unsigned long long s_inc[kMaxBlocks];
    __shared__ unsigned long long s_wbest[32], s_wbucket[32];
    __shared__ uint32_t s_counts[kSchedShared * (kSchedShared + 1)];
    const uint32_t nbk = nb * nb;
    const uint32_t *counts = all_counts;
    uint32_t ld = nb;
    if (nb <= kSchedShared) {
        ld = nb | 1u;  // odd: a column's entries lie in different banks
#pragma unroll 4
        for (uint32_t b = threadIdx.x; b < nbk; b += blockDim.x) s_counts[b / nb * ld + b % nb] = all_counts[b];
        counts = s_counts;
    }
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) s_cached[i] = 0;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < ncached; j += blockDim.x) {
        s_list[j] = cached.block[j];
        s_cached[cached.block[j]] = 1;
    }
    __syncthreads();
    const bool full = ncached >= nslots;
    // one warp per block i: lanes split the row / column and the cached list
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long best = 0;  // of the warp's blocks: (score << 11) | (2047 - block)
    for (uint32_t i = warp; i < nb; i += nw) {
        unsigned long long incident = 0;  // walkers in buckets touching i (row + column, diagonal once)
        for (uint32_t c = lane; c < nb; c += 32)
            incident += (unsigned long long)counts[i * ld + c] + (c != i ? counts[c * ld + i] : 0u);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) incident += __shfl_xor_sync(0xFFFFFFFFu, incident, o);
        if (lane == 0) s_inc[i] = incident;
        if (s_cached[i]) continue;  // warp-uniform
        unsigned long long score = 0;
        uint32_t pos = 0;
        if (!full) {
            for (uint32_t j = lane; j < ncached; j += 32) {
                const uint32_t c = s_list[j];
                score += (unsigned long long)counts[i * ld + c] + counts[c * ld + i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) score += __shfl_xor_sync(0xFFFFFFFFu, score, o);
            score += counts[i * ld + i];
        } else {
            // all minus the smallest link; the first position on ties
            unsigned long long all = 0, key = ~0ull;  // (value << 32) | position
            for (uint32_t j = lane; j < ncached; j += 32) {
                const uint32_t c = s_list[j];
                const unsigned long long v = (unsigned long long)counts[i * ld + c] + counts[c * ld + i];
                all += v;
                const unsigned long long kv = (v << 32) | j;
                key = kv < key ? kv : key;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                all += __shfl_xor_sync(0xFFFFFFFFu, all, o);
                const unsigned long long ko = __shfl_xor_sync(0xFFFFFFFFu, key, o);
                key = ko < key ? ko : key;
            }
            score = all - (key >> 32);
            pos = (uint32_t)key;
        }
        if (lane == 0) s_pos[i] = pos;
        best = max(best, (score << 11) | (2047u - i));
    }
    // fullest bucket with an absent block: (count << 21) | (0x1FFFFF - bucket)
    unsigned long long bucket = 0;
    for (uint32_t b = threadIdx.x; b < nbk; b += blockDim.x) {
        const uint32_t c = counts[b / nb * ld + b % nb];
        if (c && !(s_cached[b / nb] && s_cached[b % nb]))
            bucket = max(bucket, ((unsigned long long)c << 21) | (0x1FFFFFu - b));
    }
    bucket = warp_max(bucket);
    if (lane == 0) {
        s_wbest[warp] = best;
        s_wbucket[warp] = bucket;
    }
    __syncthreads();
    if (warp != 0) return;
    best = warp_max(s_wbest[lane]);  // 32 warps
    bucket = warp_max(s_wbucket[lane]);
    // the cached block with the fewest incident walkers outside the bucket; the first on ties
    unsigned long long fewest = ~0ull;
    const uint32_t bp = (0x1FFFFFu - (uint32_t)(bucket & 0x1FFFFFu)) / nb;
    const uint32_t bc = (0x1FFFFFu - (uint32_t)(bucket & 0x1FFFFFu)) % nb;
    if (full && bucket)
        for (uint32_t j = lane; j < ncached; j += 32) {
            const uint32_t blk = s_list[j];
            if (blk != bp && blk != bc) fewest = min(fewest, (s_inc[blk] << 11) | j);
        }
    fewest = warp_min(fewest);
    if (lane == 0) {
        Decision d{};
        const uint64_t score = best >> 11;
        const int32_t bi = (int32_t)(2047u - (uint32_t)(best & 2047u));
        d.score = score;
        d.live = *live;
        if (score > 0 && score > zero_threshold) {
            d.action = full ? 2 : 1;
            d.block = bi;
            d.position = full ? (int32_t)s_pos[bi] : (int32_t)ncached;
            if (full && pred) {
                // learned eviction: the cached block with the lowest forecast
                // of incident walkers over the next iterations (first on ties)
                float mn = 3.0e38f;
                for (uint32_t j = 0; j < ncached; ++j)
                    if (pred[s_list[j]] < mn) {
                        mn = pred[s_list[j]];
                        d.position = (int32_t)j;
                    }
            }
        } else {
            d.action = 0;
            d.block = -1;
            d.position = -1;
        }
        d.rescue_block = -1;
        d.rescue_position = -1;
        if (bucket) {
            d.rescue_block = (int32_t)(s_cached[bc] ? bp : bc);  // the current block first: lazy walkers need only it
            if (fewest != ~0ull) d.rescue_position = (int32_t)(fewest & 2047u);
        }
        *out = d;
        __threadfence_system();  // `out` may be mapped host memory
    }
}

// W: weighted Node2vec -- the candidate is alias column r.x % deg, kept when
// float(r.w >> 8) * 2^-24 < its probability, else its alias (the block's
// alias tables sit behind its neighbour list), as in the in-core kernel.
// ZC: the zero-copy tail -- the blocks marked in a.mapped are read through
// mapped host memory; every read of one is counted as a 32-byte sector in
// kCtrZcSectors (an upper bound of the host-link bytes: each probe of a
// binary search counts as its own sector).  Without ZC the same count is
// taken as if every block were mapped (kCtrModelSectors): what these steps
// would cost in the zero-copy tail, the learned policy's switch estimate.
//
// An iteration ends with its longest walk, a few dozen trials one after
// another, so what bounds it is the chain of dependent loads in a trial: the
// block table lives in shared memory, the next vertex's offsets load while
// N(prev) is searched, resident lists are searched by quarters (list_has;
// mapped ones by halving, which reads fewer sectors), few walkers are spread
// over many warps, so that one lane's search does not hold up the others, and
// lanes to spare share a walker's attempts (Group), from the start when the
// walkers are few and at the end of every iteration.
template <bool SOPR, bool PATHS, bool COOP, bool W = false, bool ZC = false>
__global__ void __launch_bounds__(kWalkThreads) k_walk_ooc(const __grid_constant__ OocStepArgs a)
{
    __shared__ uint32_t s_vs[kMaxBlocks + 1];
    __shared__ const uint32_t *s_csr[kMaxBlocks];  // block neighbours; null = absent
    __shared__ uint64_t s_es[kMaxBlocks];          // first edge of each block
    __shared__ uint8_t s_mapped[ZC ? kMaxBlocks : 1];
    __shared__ uint32_t s_iv[COOP ? kWalkThreads / 32 : 1][kCoopScratchWords];
    __shared__ unsigned long long s_ws[kWalkThreads / 32][kWsCount];  // per-warp statistics
    const uint32_t nrun = *a.nrun;
    const uint32_t total = a.run_pre[nrun];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.clock->walk_start = global_ns();
        atomicAdd(&a.ctr[kCtrRunnable], (unsigned long long)total);
    }
    // slots and claims by the number of walkers, as incore_plan chooses them
    const uint32_t warps = gridDim.x * (kWalkThreads / 32);
    uint32_t slots = 1;
    while (slots < 32 && (uint64_t)slots * a.busy_warps < total) slots *= 2;
    const uint32_t chunk = total <= 32ull * warps ? slots : 8u;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if ((uint64_t)blockIdx.x * (kWalkThreads / 32) * chunk >= total && blockIdx.x != 0 && chunk == slots)
        return;  // one wave: the CTAs before this one take every walker
    Group grp;
    while (grp.shift < kMaxGroupShift && (slots << (grp.shift + 1)) <= 32u) ++grp.shift;
    for (uint32_t i = threadIdx.x; i <= a.nb; i += blockDim.x) {
        s_vs[i] = a.vstart[i];
        if (i < a.nb) {
            s_csr[i] = a.blk_csr[i];
            s_es[i] = a.estart[i];
            if constexpr (ZC) s_mapped[i] = a.mapped[i];
        }
    }
    if (lane < kWsCount) s_ws[warp][lane] = 0;
    __syncthreads();
    constexpr int kSearch = ZC ? kHalve : kQuarter;
    uint32_t zc_sectors = 0;
    // sectors of a plain binary search over n ids plus the final read: at most
    // bit_length(n) + 1
    auto search_sectors = [](uint32_t n) { return 33u - (uint32_t)__clz(n); };

    const uint32_t maxhops = a.c.maxhops;

    uint32_t q_next = 0, q_end = 0;
    uint32_t bkt = 0, bkt_start = 0, bkt_end = 0;  // bucket of the claim's first walker; lane j: end of bucket bkt + j
    bool exhausted = false;
    bool active = false;

    uint32_t wid = 0, prev = 0, cur = 0, hop = 0, hop0 = 0, attempt = 0, pb = 0, cb = 0, deg = 0, pdeg = 0, idx = 0;
    uint64_t h = 0;
    const uint32_t *cadj = nullptr, *padj = nullptr;  // N(cur), N(prev); padj null: prev's block is absent
    const uint2 *calias = nullptr;                    // W: the current vertex's alias table
    StepThr t{0.f, 0.f, 0.f};
    uint32_t n_trials = 0;  // trials not yet added to s_ws

    // Lane 0 of a group writes what its walker writes.
    auto leads = [&]() { return grp.sub(lane) == 0; };
    // Statistics of the walker leaving this lane (finished or parked): its
    // steps in this launch are the hops it made since it was loaded.
    auto flush = [&]() { atomicAdd(&s_ws[warp][kWsSteps], (unsigned long long)(hop - hop0)); };
    auto finish = [&]() {
        active = false;
        if (!leads()) return;
        a.hashes[wid - a.out_base] = h;
        a.lens[wid - a.out_base] = hop + 1;
        a.keys[idx] = kNoBucket;
        atomicAdd(&s_ws[warp][kWsHash], (unsigned long long)h);
        atomicAdd(&s_ws[warp][kWsDone], 1ull);
        flush();
    };
    auto park = [&](uint32_t cur_blk) {
        active = false;
        if (!leads()) return;
        WalkerRec rec;
        rec.wid = wid;
        rec.prev = prev;
        rec.cur = cur;
        rec.hop = hop;
        rec.prev_blk = pb;
        rec.cur_blk = cur_blk;
        rec.hash_lo = (uint32_t)h;
        rec.hash_hi = (uint32_t)(h >> 32);
        a.recs[__ldg(a.order + idx)] = rec;
        const uint32_t b = bucket_of(rec, a.nb);
        a.keys[idx] = b;
        atomicAdd(a.counts + b, 1u);
        flush();
    };
    // Enter a step at vertex cur (block cb, edges [b0, b1)), prev adjacency
    // already set.  The termination draw is the step's first.
    auto enter = [&](uint64_t b0, uint64_t b1) {
        attempt = 0;
        deg = (uint32_t)(b1 - b0);
        cadj = s_csr[cb] + (b0 - s_es[cb]);
        if constexpr (W) calias = a.blk_alias[cb] + (b0 - s_es[cb]);
        if (deg == 0) finish();
        else t = step_thresholds<SOPR>(a.c, deg, pdeg);
    };

    for (;;) {
        for (;;) {
            const unsigned need = __ballot_sync(0xFFFFFFFFu, !active && (lane >> grp.shift) < slots);
            if (need == 0 || exhausted) break;
            if (q_next >= q_end) {
                uint32_t base = 0;
                if (lane == 0) base = (uint32_t)min(atomicAdd(&a.ctr[kCtrCursor], (unsigned long long)chunk), 0xFFFFFFFFull);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                if (base >= total) {
                    exhausted = true;
                    break;
                }
                q_next = base;
                q_end = min(base + chunk, total);
                // its bucket: the last one that starts at or before it, 32
                // probes a round.  Buckets are not empty, so the claim's
                // walkers lie in this one and the 31 after it.
                uint32_t lo = 0, hi = nrun;  // run_pre[lo] <= base < run_pre[hi]
                while (hi - lo > 1) {
                    const uint32_t step = (hi - lo + 32) / 33, q = lo + step * (lane + 1);
                    const uint32_t c =
                        (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, q < hi && __ldg(a.run_pre + q) <= base));
                    hi = min(hi, lo + step * (c + 1));
                    lo += step * c;
                }
                bkt = lo;
                bkt_start = __ldg(a.run_pre + lo);
                bkt_end = __ldg(a.run_pre + min(lo + 1 + lane, nrun));
            }
            const uint32_t avail = q_end - q_next;
            const uint32_t rank = __popc(need & ((1u << grp.base(lane)) - 1u)) >> grp.shift;
            const uint32_t g = q_next + min(rank, avail - 1);
            uint32_t k = 0;  // buckets of the window that end at or before g
#pragma unroll
            for (uint32_t o = 16; o > 0; o >>= 1)
                if (__shfl_sync(0xFFFFFFFFu, bkt_end, (int)(k + o - 1)) <= g) k += o;
            const uint32_t k_end = __shfl_sync(0xFFFFFFFFu, bkt_end, (int)(k ? k - 1 : 0));
            if (((need >> lane) & 1u) && rank < avail) {
                idx = __ldg(a.run_off + bkt + k) + (g - (k ? k_end : bkt_start));
                const WalkerRec rec = a.recs[__ldg(a.order + idx)];
                wid = rec.wid;
                prev = rec.prev;
                cur = rec.cur;
                hop = rec.hop;
                hop0 = hop;
                pb = rec.prev_blk;
                cb = rec.cur_blk & ~kNeedPrev;
                h = ((uint64_t)rec.hash_hi << 32) | rec.hash_lo;
                // lazy mode: the previous block may be absent; its offsets are
                // resident, so deg(prev) is known either way
                const uint32_t *pcsr = s_csr[pb];
                if (hop >= maxhops) {
                    finish();
                } else if (pcsr == nullptr && !a.lazy) {
                    atomicOr(a.err, kErrBlock);  // scheduled without its previous block
                    finish();
                } else {
                    const uint64_t p0 = __ldg(a.beg + prev), p1 = __ldg(a.beg + prev + 1);
                    const uint64_t c0 = __ldg(a.beg + cur), c1 = __ldg(a.beg + cur + 1);
                    pdeg = (uint32_t)(p1 - p0);
                    padj = pcsr ? pcsr + (p0 - s_es[pb]) : nullptr;
                    active = true;
                    enter(c0, c1);
                }
            }
            q_next += min((uint32_t)__popc(need) >> grp.shift, avail);
        }
        const unsigned act = __ballot_sync(0xFFFFFFFFu, active);
        if (act == 0) break;
        if (exhausted && grp.shift < kMaxGroupShift && 2 * __popc(act) <= 32) {
            // the last walkers spread over the lanes that have none left
            const int from = (int)regroup(grp, act, lane, active);
            wid = __shfl_sync(0xFFFFFFFFu, wid, from);
            prev = __shfl_sync(0xFFFFFFFFu, prev, from);
            cur = __shfl_sync(0xFFFFFFFFu, cur, from);
            hop = __shfl_sync(0xFFFFFFFFu, hop, from);
            hop0 = __shfl_sync(0xFFFFFFFFu, hop0, from);
            attempt = __shfl_sync(0xFFFFFFFFu, attempt, from);
            pb = __shfl_sync(0xFFFFFFFFu, pb, from);
            cb = __shfl_sync(0xFFFFFFFFu, cb, from);
            deg = __shfl_sync(0xFFFFFFFFu, deg, from);
            pdeg = __shfl_sync(0xFFFFFFFFu, pdeg, from);
            idx = __shfl_sync(0xFFFFFFFFu, idx, from);
            h = shfl64(h, from);
            cadj = shfl_ptr(cadj, from);
            padj = shfl_ptr(padj, from);
            if constexpr (W) calias = shfl_ptr(calias, from);
            t = shfl_thr<SOPR>(t, from);
        }

        // hard steps: the whole warp evaluates 32 attempts per round
        for (unsigned hm = COOP ? __ballot_sync(0xFFFFFFFFu, active && leads() && attempt >= kHardAttempts) : 0u;
             hm; hm &= hm - 1) {
            const int L = __ffs(hm) - 1;
            const uint32_t p0 = __shfl_sync(0xFFFFFFFFu, attempt, L);
            const uint32_t Ldeg = __shfl_sync(0xFFFFFFFFu, deg, L);
            const CsrIndex<kSearch> pix{shfl_ptr(padj, L), nullptr};
            const uint32_t astar = warp_first_accept<SOPR>(
                a.c, shfl_thr<SOPR>(t, L), __shfl_sync(0xFFFFFFFFu, wid, L), __shfl_sync(0xFFFFFFFFu, hop, L), p0,
                kMaxAttempts, shfl_ptr(cadj, L), Ldeg, mod_magic(Ldeg), __shfl_sync(0xFFFFFFFFu, prev, L),
                __shfl_sync(0xFFFFFFFFu, cur, L), pix, 0u, __shfl_sync(0xFFFFFFFFu, pdeg, L), s_iv[COOP ? warp : 0]);
            if (grp.base(lane) == (uint32_t)L) {
                if (leads()) {
                    if constexpr (ZC)  // every attempt: a candidate and, at most, a search of N(prev)
                        zc_sectors +=
                            (astar - p0) * ((s_mapped[cb] ? 1u : 0u) + (s_mapped[pb] ? search_sectors(pdeg) : 0u));
                    else
                        zc_sectors += (astar - p0) * (1u + search_sectors(pdeg));
                }
                attempt = astar;
                if (astar >= kMaxAttempts) {
                    atomicOr(a.err, kErrTrials);
                    finish();
                }
            }
        }

        // One rejection-sampling trial a lane.
        const bool last = hop + 1 >= maxhops;
        bool end = false;  // the step's termination draw ends the walk
        int verdict = 0;
        uint32_t x = 0, sectors = 0;
        uint64_t n0 = 0, n1 = 0;  // offsets of a vertex that is, or may be, the next one
        float rv = 0.0f;
        if (active) {
            const uint32_t att = attempt + grp.sub(lane);
            const U4 r = draw(a.c, wid, hop, att);
            end = att == 0 && hop > 0 && terminates(a.c, r.z);
            const uint32_t pos = r.x % deg;
            rv = rand_val(r.y, thr_max<SOPR>(a.c, t));
            uint32_t col = pos;
            if constexpr (W) {
                const uint2 e = __ldg(calias + pos);
                if (!(__uint2float_rn(r.w >> 8) * 0x1p-24f < __uint_as_float(e.x))) col = e.y;
            }
            x = __ldg(cadj + col);
            if (!end && att < kMaxAttempts) {
                verdict = accept_without_prev<SOPR>(a.c, t, rv, x, prev, cur);
                if (!ZC || s_mapped[cb]) sectors += 1u;
            }
            if (verdict != 0 && !last && x < a.nverts) {
                n0 = __ldg(a.beg + x);
                n1 = __ldg(a.beg + x + 1);
            }
        }
        // N(prev) is searched only when the verdict depends on it, then only if
        // its block is resident (or mapped), and only if no attempt before this
        // one decides the step without: the whole warp waits for a search.  Each
        // search and each candidate counts its sectors.
        bool search = verdict < 0 && padj != nullptr;
        if (grp.shift) {
            const unsigned sure = grp.mine(__ballot_sync(0xFFFFFFFFu, end || (verdict != 0 && !search)), lane);
            if (sure & ((1u << grp.sub(lane)) - 1u)) search = false;
        }
        if (search) {
            if (!ZC || s_mapped[pb]) sectors += search_sectors(pdeg);
            const bool found = csr_contains(CsrIndex<kSearch>{padj, nullptr}, 0u, 0ull, pdeg, x);
            verdict = (found ? rv < thr_found<SOPR>(a.c, t) : rv < thr_notfound<SOPR>(a.c, t)) ? 1 : 0;
        }
        uint32_t first = 0;  // the deciding attempt, from `attempt`
        if (grp.shift) {
            const unsigned dec = grp.mine(__ballot_sync(0xFFFFFFFFu, verdict != 0), lane);
            end = grp.mine(__ballot_sync(0xFFFFFFFFu, end), lane) != 0;
            first = dec ? (uint32_t)__ffs(dec) - 1 : 0u;
            if (dec && grp.sub(lane) > first) sectors = 0;  // one lane alone would not have come this far
            const int from = (int)(grp.base(lane) + first);
            verdict = __shfl_sync(0xFFFFFFFFu, verdict, from);
            if (!dec) verdict = 0;
            x = __shfl_sync(0xFFFFFFFFu, x, from);
            n0 = shfl64(n0, from);
            n1 = shfl64(n1, from);
        }
        if (!active) continue;
        zc_sectors += end ? 0u : sectors;
        if (end) {
            finish();
        } else if (verdict < 0) {
            // Needs N(prev), whose block is absent: park the walker flagged in
            // bucket (prev block, cur block).  The step restarts at attempt 0
            // once both blocks are resident (the draws are counter-based), so
            // its attempts so far are not counted.
            park(cb | kNeedPrev);
        } else if (verdict > 0) {
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
            prev = cur;
            pb = cb;
            pdeg = deg;
            padj = cadj;
            cur = x;
            if (last) {
                finish();
            } else if (x >= a.nverts) {
                atomicOr(a.err, kErrVertexRange);
                finish();
            } else {
                if (x < s_vs[cb] || x >= s_vs[cb + 1]) cb = block_of(s_vs, a.nb, x);
                if (s_csr[cb] == nullptr) park(cb);  // next block absent: bucket (pb, cb)
                else enter(n0, n1);
            }
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
    if (lane == 0) {
        atomicAdd(&a.ctr[kCtrSteps], s_ws[warp][kWsSteps]);
        atomicAdd(&a.ctr[kCtrTrials], trials + s_ws[warp][kWsTrials]);
        atomicAdd(&a.ctr[kCtrDone], s_ws[warp][kWsDone]);
        atomicAdd(&a.ctr[kCtrHashSum], s_ws[warp][kWsHash]);
        atomicMax(&a.clock->walk_end, global_ns());
    }
    {
        const unsigned long long zs = warp_sum((unsigned long long)zc_sectors);
        if (lane == 0 && zs) atomicAdd(&a.ctr[ZC ? kCtrZcSectors : kCtrModelSectors], zs);
    }
}

// ------------------------------------------------------------------ learned policy

// Per-block features of the demand predictor (all log1p-scaled counts):
//  0 waiting at i (cur block i)   1 leaving i (prev block i)   2 diagonal (i,i)
//  3 walkers between i and resident blocks   4 walkers that run if i is resident
//  5 resident   6 edge share   7 vertex share   8 arrival EMA   9 arrivals
// 10 live fraction  11 iteration/256  12 waiting share  13 incident
// 14 leaving, off-diagonal  15 waiting, off-diagonal
__global__ void __launch_bounds__(1024) k_features(const FeatureArgs f)
{
    __shared__ uint8_t s_res[kMaxBlocks];
    const uint32_t nb = f.nb;
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) s_res[i] = f.blk_csr[i] != nullptr;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) {
        uint64_t col = 0, row = 0, cross = 0, ready = 0;
        for (uint32_t p = 0; p < nb; ++p) {
            const uint32_t cpi = f.counts[p * nb + i], cip = f.counts[i * nb + p];
            col += cpi;
            row += cip;
            if (s_res[p]) cross += (uint64_t)cpi + cip;
            if (s_res[p] || p == i) ready += cpi;
        }
        const uint32_t diag = f.counts[i * nb + i];
        const float colf = (float)col;
        const float arr = fmaxf(colf - f.prev_col[i], 0.f);
        const float ema = 0.7f * f.ema_arr[i] + 0.3f * arr;
        f.prev_col[i] = colf;
        f.ema_arr[i] = ema;
        float *x = f.x + (uint64_t)i * 16;
        x[0] = log1pf(colf);
        x[1] = log1pf((float)row);
        x[2] = log1pf((float)diag);
        x[3] = log1pf((float)cross);
        x[4] = log1pf((float)ready);
        x[5] = s_res[i] ? 1.f : 0.f;
        x[6] = f.emass[i];
        x[7] = f.vfrac[i];
        x[8] = log1pf(ema);
        x[9] = log1pf(arr);
        x[10] = f.live_frac;
        x[11] = 0.f;  // (the iteration count: left out, it only grows past what training saw)
        x[12] = colf * f.inv_live * (float)nb;
        x[13] = log1pf((float)(row + col - diag));
        x[14] = log1pf((float)(row - diag));
        x[15] = log1pf((float)(col - diag));
        f.col[i] = (float)(row + col - diag);  // incident walkers: the forecast's quantity
    }
}

// Training set from the trace ring (ring slots of kMlpIn features and of
// incident walkers per block -- walkers whose current or previous block it
// is; iteration t lives in slot t % ring): samples t0 .. t0+T-1 gathered in
// order, with targets y = log1p(mean incident walkers over the next k
// iterations) - x[13] (x[13] = log1p of the incident walkers then), so the
// network learns the change of that log demand and an untrained one
// forecasts no change.
__global__ void k_gather_train(const float *ring_x, const float *ring_col, uint32_t t0, uint32_t ring, uint32_t T,
                               uint32_t k, uint32_t nb, float *train_x, float *y)
{
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= T * nb) return;
    const uint32_t j = idx / nb, i = idx % nb;
    const uint32_t t = t0 + j;
    const float *xs = ring_x + ((uint64_t)(t % ring) * nb + i) * 16;
    float *xd = train_x + (uint64_t)idx * 16;
    for (int f = 0; f < 16; ++f) xd[f] = xs[f];
    float s = 0.f;
    for (uint32_t d = 1; d <= k; ++d) s += ring_col[(uint64_t)((t + d) % ring) * nb + i];
    y[idx] = log1pf(s / (float)k) - xs[13];
}

// level[i] = res[i] + x[i][13]: the forecast change back to log incident walkers.
__global__ void k_add_level(const float *res, const float *x, float *level, uint32_t nb)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nb) level[i] = res[i] + x[(uint64_t)i * 16 + 13];
}


cudaError_t launch_features(const FeatureArgs &f, cudaStream_t s)
{
    k_features<<<1, 1024, 0, s>>>(f);
    return cudaGetLastError();
}

cudaError_t launch_gather_train(const float *ring_x, const float *ring_col, uint32_t t0, uint32_t ring, uint32_t T,
                                uint32_t k, uint32_t nb, float *train_x, float *y, cudaStream_t s)
{
    const uint32_t n = T * nb;
    k_gather_train<<<(n + 255) / 256, 256, 0, s>>>(ring_x, ring_col, t0, ring, T, k, nb, train_x, y);
    return cudaGetLastError();
}

cudaError_t launch_add_level(const float *res, const float *x, float *level, uint32_t nb, cudaStream_t s)
{
    k_add_level<<<(nb + 255) / 256, 256, 0, s>>>(res, x, level, nb);
    return cudaGetLastError();
}


// ------------------------------------------------------------------ launchers

cudaError_t launch_init_walkers(const WalkerInit &in, const uint32_t *vstart, uint32_t nb, uint32_t wid0, uint64_t n,
                                WalkerRec *recs, uint32_t *order, uint32_t *keys, uint32_t *paths, uint32_t stride,
                                int num_sms, cudaStream_t s)
{
    k_init_walkers<<<num_sms * 8, 256, 0, s>>>(in, vstart, nb, wid0, n, recs, order, keys, paths, stride);
    return cudaGetLastError();
}

cudaError_t launch_count(const uint32_t *keys, const uint32_t *n, uint32_t *counts, int num_sms, cudaStream_t s)
{
    k_count<<<num_sms * 8, 256, 0, s>>>(keys, n, counts);
    return cudaGetLastError();
}

__global__ void k_combine(const uint32_t *__restrict__ counts, uint32_t nn, uint32_t *__restrict__ combined,
                          OocClock *clock)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) clock->pairs_start = global_ns();
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x)
        combined[k] = counts[k] + counts[nn + k];
}

cudaError_t launch_plan(const uint32_t *counts, uint32_t nb, uint32_t *offsets, uint32_t *cursor, uint32_t *pairs,
                        uint32_t *n_out, const unsigned long long *ctr, const uint32_t *err, unsigned long long *snap,
                        OocClock *clock, int num_sms, cudaStream_t s)
{
    // many blocks' pair totals are too much for one CTA (8 words a thread at 64
    // blocks, 128 at 256)
    const bool apart = nb > 64;
    if (apart) {
        k_combine<<<num_sms, 256, 0, s>>>(counts, nb * nb, pairs, clock);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_plan<<<1, kScanThreads, 0, s>>>(counts, nb * nb, offsets, cursor, apart ? nullptr : pairs, n_out, ctr, err, snap,
                                    clock);
    return cudaGetLastError();
}

cudaError_t launch_scatter(const uint32_t *keys_in, const uint32_t *order_in, const uint32_t *n, uint32_t *cursor,
                           uint32_t *keys_out, uint32_t *order_out, OocClock *clock, int num_sms, cudaStream_t s)
{
    k_scatter<<<num_sms * 4, 256, 0, s>>>(keys_in, order_in, n, cursor, keys_out, order_out, clock);
    return cudaGetLastError();
}

cudaError_t launch_runnable(const uint32_t *offsets, const TablePatch &patch, uint32_t nb, uint32_t lazy,
                            uint32_t *counts, const uint32_t **blk_csr, unsigned long long *cursor, uint32_t *run_pre,
                            uint32_t *run_off, uint32_t *nrun, cudaStream_t s)
{
    k_runnable<<<1, kScanThreads, 0, s>>>(offsets, patch, nb, lazy, counts, blk_csr, cursor, run_pre, run_off, nrun);
    return cudaGetLastError();
}

cudaError_t launch_schedule(const uint32_t *counts, const uint32_t *live, uint32_t nb, const uint32_t *h_cached,
                            uint32_t ncached, uint32_t nslots, uint32_t zero_threshold, const float *pred,
                            float pred_weight, Decision *out, cudaStream_t s)
{
    CachedList cached;
    for (uint32_t j = 0; j < kMaxBlocks; ++j) cached.block[j] = j < ncached ? (uint16_t)h_cached[j] : 0u;
    k_schedule<<<1, 1024, 0, s>>>(counts, live, nb, cached, ncached, nslots, zero_threshold, pred, pred_weight, out);
    return cudaGetLastError();
}

template <bool SOPR, bool PATHS, bool COOP, bool W = false>
static int ooc_grid_for(int num_sms)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk_ooc<SOPR, PATHS, COOP, W>, kWalkThreads, 0);
    return (per_sm < 1 ? 1 : per_sm) * num_sms;
}

template <bool SOPR, bool PATHS, bool COOP, bool W = false>
static void ooc_launch_one(const OocStepArgs &a, int grid, cudaStream_t s)
{
    if (a.mapped) k_walk_ooc<SOPR, PATHS, COOP, W, true><<<grid, kWalkThreads, 0, s>>>(a);
    else k_walk_ooc<SOPR, PATHS, COOP, W><<<grid, kWalkThreads, 0, s>>>(a);
}

int ooc_grid(bool sopr, bool paths, bool coop, int num_sms, bool weighted)
{
    if (weighted) return paths ? ooc_grid_for<false, true, false, true>(num_sms) : ooc_grid_for<false, false, false, true>(num_sms);
    const int v = (sopr ? 4 : 0) | (paths ? 2 : 0) | (coop ? 1 : 0);
    switch (v) {
    case 0: return ooc_grid_for<false, false, false>(num_sms);
    case 1: return ooc_grid_for<false, false, true>(num_sms);
    case 2: return ooc_grid_for<false, true, false>(num_sms);
    case 3: return ooc_grid_for<false, true, true>(num_sms);
    case 4: return ooc_grid_for<true, false, false>(num_sms);
    case 5: return ooc_grid_for<true, false, true>(num_sms);
    case 6: return ooc_grid_for<true, true, false>(num_sms);
    default: return ooc_grid_for<true, true, true>(num_sms);
    }
}

cudaError_t launch_walk_ooc(const OocStepArgs &a, bool sopr, bool coop, bool weighted, int grid, cudaStream_t s)
{
    if (weighted) {
        if (sopr || coop || !a.blk_alias) return cudaErrorInvalidValue;  // weighted walks are Node2vec walks
        if (a.paths) ooc_launch_one<false, true, false, true>(a, grid, s);
        else ooc_launch_one<false, false, false, true>(a, grid, s);
        return cudaGetLastError();
    }
    const int v = (sopr ? 4 : 0) | (a.paths ? 2 : 0) | (coop ? 1 : 0);
    switch (v) {
    case 0: ooc_launch_one<false, false, false>(a, grid, s); break;
    case 1: ooc_launch_one<false, false, true>(a, grid, s); break;
    case 2: ooc_launch_one<false, true, false>(a, grid, s); break;
    case 3: ooc_launch_one<false, true, true>(a, grid, s); break;
    case 4: ooc_launch_one<true, false, false>(a, grid, s); break;
    case 5: ooc_launch_one<true, false, true>(a, grid, s); break;
    case 6: ooc_launch_one<true, true, false>(a, grid, s); break;
    default: ooc_launch_one<true, true, true>(a, grid, s); break;
    }
    return cudaGetLastError();
}

}  // namespace gw
