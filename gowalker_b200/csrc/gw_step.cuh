// The second-order walk step, shared by every walk kernel.
//
// Semantics follow the reference CPU step (GOWalker engine/engine.hpp:158-404)
// with every draw taken from Philox4x32-10 keyed by the walk seed and
// countered by (walker id, hop, attempt, 0):
//   lane x -> rand_pos = x % deg                                (util/util.hpp:294)
//   lane y -> rand_val = float(y >> 8) * 2^-24 * max_val        (one fp32 multiply)
//   lane z -> SOPR/SOSR termination draw at hop >= 1 (attempt 0)
// Acceptance keeps the reference's precision mix:
//   Node2vec: fp32 thresholds 1/p, 1, 1/q, min and max of the three
//             (engine/engine.hpp:169-172, 209-258)
//   SOPR/SOSR: inv_deg = (float)((1-alpha)/deg) in fp64, inv_prev_deg =
//             alpha/(float)prev_deg in fp32 (323-326); the x==prev compare is
//             fp64 (341), the others fp32 (334, 368, 373).
// Every rounding step is an explicit _rn intrinsic so no contraction or
// fast-math flag can change a bit.  The fp64 compare is carried out in fp32
// without changing a verdict: for a float rv and a double T,
// (double)rv < T  <=>  rv < RU(T), RU(T) the smallest float >= T (if T is a
// float, RU(T) = T; otherwise every float below RU(T) is below T).
#pragma once
#include <cstdint>
#include "gw_philox.cuh"

namespace gw {

// Per-run constants, computed on the host.
struct StepConsts {
    uint32_t maxhops;
    uint32_t key0, key1;
    float n2v_maxv, n2v_minv;  // max / min of {1/p, 1/q, 1}
    float inv_p, inv_q;        // 1.0f/p, 1.0f/q
    float alpha;               // SOPR/SOSR
    float term_prob;           // 0 = no termination draw
    double one_m_alpha;        // 1.0 - (double)alpha
    uint32_t rk0[10], rk1[10]; // Philox key schedule: round r uses key + r * Weyl constant
};

// Per-step thresholds.  Node2vec's are run constants and live in
// StepConsts; SOPR/SOSR's depend on deg and prev_deg and take three floats.
struct StepThr {
    float inv_deg;  // (float)((1-alpha)/deg), divided in fp64
    float sum;      // inv_deg + alpha/(float)prev_deg
    float t_prev;   // RU((1-alpha)/deg): x == prev accepts iff rv < t_prev
};

template <bool SOPR>
__device__ __forceinline__ StepThr step_thresholds(const StepConsts &c, uint64_t deg, uint64_t pdeg)
{
    StepThr t{0.f, 0.f, 0.f};
    if constexpr (SOPR) {
        const double tp = __ddiv_rn(c.one_m_alpha, (double)deg);
        t.inv_deg = __double2float_rn(tp);
        const float inv_prev = __fdiv_rn(c.alpha, __ull2float_rn((unsigned long long)pdeg));
        t.sum = __fadd_rn(t.inv_deg, inv_prev);
        t.t_prev = __double2float_ru(tp);
    }
    return t;
}

// The five thresholds of a trial (engine/engine.hpp:209-258, 334-375).
template <bool SOPR>
__device__ __forceinline__ float thr_max(const StepConsts &c, const StepThr &t)
{
    if constexpr (SOPR) return (t.inv_deg < t.sum) ? t.sum : t.inv_deg;  // std::max(inv_deg, sum)
    else return c.n2v_maxv;
}
template <bool SOPR>
__device__ __forceinline__ float thr_min(const StepConsts &c, const StepThr &t)
{
    if constexpr (SOPR) return (t.sum < t.inv_deg) ? t.sum : t.inv_deg;  // std::min(inv_deg, sum)
    else return c.n2v_minv;
}
template <bool SOPR>
__device__ __forceinline__ float thr_prev(const StepConsts &c, const StepThr &t)
{
    if constexpr (SOPR) return t.t_prev;
    else return c.inv_p;
}
template <bool SOPR>
__device__ __forceinline__ float thr_found(const StepConsts &c, const StepThr &t)
{
    if constexpr (SOPR) return t.sum;
    else return 1.0f;
}
template <bool SOPR>
__device__ __forceinline__ float thr_notfound(const StepConsts &c, const StepThr &t)
{
    if constexpr (SOPR) return t.inv_deg;
    else return c.inv_q;
}

// The walk draw.  The key schedule comes precomputed in the kernel's
// parameters, so each round is two wide multiplies and two three-way xors
// with a constant operand.
__device__ __forceinline__ U4 draw(const StepConsts &c, uint32_t wid, uint32_t hop, uint32_t attempt)
{
    return philox4x32_10_sched(wid, hop, attempt, kTagWalk, c.rk0, c.rk1);
}

__device__ __forceinline__ float rand_val(uint32_t y, float maxv)
{
    return __fmul_rn(__uint2float_rn(y >> 8) * 0x1p-24f, maxv);
}

__device__ __forceinline__ bool terminates(const StepConsts &c, uint32_t z)
{
    return c.term_prob > 0.0f && __uint2float_rn(z >> 8) * 0x1p-24f < c.term_prob;
}

// Neighbour array of the graph (or of one block), with the membership table of
// its vertices (table_has), and how a neighbour is searched.
enum Search : int {
    kHalve,    // mapped host memory: fewest sectors
    kQuarter,  // device memory: fewest dependent loads without an index
    kLevels,   // device memory past the L2: fewest lines without a table
    kTable
};
template <int SEARCH>
struct CsrIndex {
    const uint32_t *csr;
    const uint32_t *table;  // kTable: buckets of eight ids, on 32-byte boundaries
};
// Sample levels of a whole CSR: level L holds csr[j * 32^L] for every j, about
// 3 % of the CSR in all.
constexpr int kIdxLevels = 6;
struct Levels {
    const uint32_t *lvl[kIdxLevels];
    uint32_t n;
};
template <>
struct CsrIndex<kLevels> {
    const uint32_t *csr;  // the whole CSR: levels are by global position
    const Levels *levels;
};

// Membership table of one vertex's neighbours: table_buckets(d) buckets of
// eight slots, an id in its home bucket (table_home) or, that one being full,
// in the next that was not, the eighth slot filled last, empty ones kEmptySlot.
// The slots number more than d, so a search ends at a bucket with room.
constexpr uint32_t kEmptySlot = 0xFFFFFFFFu;  // no id: ids are below a 32-bit vertex count
__host__ __device__ __forceinline__ uint32_t table_buckets(uint32_t d)
{
    return d ? (d >> 2) + (d >> 4) + 1u : 0u;  // 3.2 ids a bucket: fewer than 1 in 100 buckets overflow
}
__device__ __forceinline__ uint32_t table_hash(uint32_t id)
{
    // two rounds: the product alone sends some arithmetic progressions to one bucket
    const uint32_t h = id * 0x9E3779B1u;
    return (h ^ (h >> 15)) * 0x85EBCA77u;
}
__device__ __forceinline__ uint32_t table_home(uint32_t id, uint32_t buckets) { return __umulhi(table_hash(id), buckets); }
// The slot an id tries first, of the first seven (it goes round them, then to
// the eighth): a hash of its own decides, so most find it empty.
__device__ __forceinline__ uint32_t table_slot(uint32_t id) { return __umulhi(table_hash(id) * 0xC2B2AE3Du, 7u); }

// One aligned 32-byte sector: eight consecutive words in one load.
__device__ __forceinline__ void load_sector(const uint32_t *p, uint32_t (&v)[8])
{
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// Whether x is among the d ids whose table starts at bucket `first`.
__device__ __forceinline__ bool table_has(const uint32_t *table, uint32_t first, uint32_t d, uint32_t x)
{
    const uint32_t n = table_buckets(d);
    uint32_t b = n ? table_home(x, n) : 0u;
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t v[8];
        load_sector(table + ((uint64_t)first + b) * 8u, v);
        bool found = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) found |= v[k] == x;
        if (found) return true;
        if (v[7] == kEmptySlot) return false;
        b = b + 1 == n ? 0u : b + 1;
    }
    return false;
}

// First position p in [lo, hi) with csr[p] >= y, or hi (csr[lo, hi) sorted,
// hi - lo < 2^32).
__device__ __forceinline__ uint64_t csr_lower_bound(const uint32_t *csr, uint64_t lo, uint64_t hi, uint32_t y)
{
    const uint32_t *__restrict__ p = csr + lo;
    uint32_t a = 0, b = (uint32_t)(hi - lo);
    while (a < b) {
        const uint32_t m = (a + b) >> 1;
        if (__ldg(p + m) < y) a = m + 1;
        else b = m;
    }
    return lo + a;
}

// How many of the sorted p[0, n) are below y, by quarters (see list_has).
__device__ __forceinline__ uint32_t list_below(const uint32_t *__restrict__ p, uint32_t n, uint32_t y)
{
    uint32_t lo = 0, len = n;  // the answer lies in [lo, lo + len]
    while (len > 3) {
        const uint32_t q = len >> 2;
        const uint32_t v1 = __ldg(p + lo + q), v2 = __ldg(p + lo + 2 * q), v3 = __ldg(p + lo + 3 * q);
        if (v3 < y) {
            lo += 3 * q + 1;
            len -= 3 * q + 1;
        } else {
            len = v1 < y ? q - 1 : q;
            lo += v2 < y ? 2 * q + 1 : v1 < y ? q + 1 : 0u;
        }
    }
    uint32_t c = lo;
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
        if (i < len && __ldg(p + lo + i) < y) c = lo + i + 1;
    return c;
}

// Membership of x in the sorted p[0, n), quartering: three independent probes
// a round, so half the dependent loads of halving for half as many again in
// all -- what counts where no table is at hand and few walkers hide a load.
__device__ __forceinline__ bool list_has(const uint32_t *__restrict__ p, uint32_t n, uint32_t x)
{
    uint32_t lo = 0, len = n;  // x can only be in [lo, lo + len)
    while (len > 4) {
        const uint32_t q = len >> 2;
        const uint32_t v1 = __ldg(p + lo + q), v2 = __ldg(p + lo + 2 * q), v3 = __ldg(p + lo + 3 * q);
        len = v3 <= x ? len - 3 * q : q;
        lo += v3 <= x ? 3 * q : v2 <= x ? 2 * q : v1 <= x ? q : 0u;
    }
    bool found = false;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
        if (i < len) found |= __ldg(p + lo + i) == x;
    return found;
}

// Membership of x in the sorted csr[lo, lo + n) through the sample levels: down
// from the highest with more than two entries inside (level L qualifies when
// the range is longer than 2 * 32^L), each a binary search that narrows the
// range 32-fold, the last one in the CSR itself; 64 ids and fewer go there at
// once.  All but that one stay in the L2.
__device__ __forceinline__ bool levels_have(const CsrIndex<kLevels> &ix, uint64_t lo, uint32_t n, uint32_t x)
{
    const Levels &lv = *ix.levels;
    const uint64_t end = lo + n;
    uint64_t hi = end;
    if (n > 64) {
        int L = min((int)lv.n, (30 - __clz((int)n)) / 5);  // (floor(log2 n) - 1) / 5
        for (; L >= 1; --L) {
            const uint32_t sh = 5u * (uint32_t)L;
            if (hi - lo <= (2ull << sh)) continue;
            const uint32_t *__restrict__ g = lv.lvl[L - 1];
            const uint64_t j0 = (lo + (1ull << sh) - 1) >> sh, j1 = (hi - 1) >> sh;
            uint32_t a = 0, b = (uint32_t)(j1 - j0) + 1;  // first j in [j0, j1] with csr[j << sh] >= x
            while (a < b) {
                const uint32_t m = (a + b) >> 1;
                if (__ldg(g + j0 + m) < x) a = m + 1;
                else b = m;
            }
            if (a > 0) lo = ((j0 + a - 1) << sh) + 1;
            if (j0 + a <= j1) hi = (j0 + a) << sh;
        }
    }
    const uint64_t p = csr_lower_bound(ix.csr, lo, hi, x);
    return p < end && __ldg(ix.csr + p) == x;
}

// Membership of x in the sorted csr[lo, lo + n), whose table starts at bucket
// `first`.
//
// What bounds it: every probe of a search is a dependent load of a line of its
// own and a warp waits for the longest chain of its lanes.  Halving takes 12
// probes (a hundred instructions) for the thousands of neighbours of the
// vertices walks visit most; a bucket is one load and eight compares.  Sample
// levels of 32, eight-way levels and eight-way trees were all measured too:
// fewer lines than halving, but no fewer instructions.  Fewer lines count where
// the L2 does not keep the CSR and no table is there (Node2vec on 64 M edges:
// 4.23 ms by levels of 32, 4.92 by quarters, 5.38 by halving, 3.25 by tables;
// on 16 M 1.72 / 1.52 / - / 1.03).
template <int SEARCH>
__device__ __forceinline__ bool csr_contains(const CsrIndex<SEARCH> &ix, uint32_t first, uint64_t lo, uint32_t n,
                                             uint32_t x)
{
    if constexpr (SEARCH == kTable) {
        return table_has(ix.table, first, n, x);
    } else if constexpr (SEARCH == kLevels) {
        return levels_have(ix, lo, n, x);
    } else if constexpr (SEARCH == kQuarter) {
        return list_has(ix.csr + lo, n, x);
    } else {
        const uint64_t p = csr_lower_bound(ix.csr, lo, lo + n, x);
        return p < lo + n && __ldg(ix.csr + p) == x;
    }
}

// Verdict on candidate x drawn with rand value rv (engine/engine.hpp:209-258,
// 334-375) without N(prev): 1 accept, 0 reject, -1 when it depends on x in
// N(prev) (the found and not-found thresholds disagree at rv).
template <bool SOPR>
__device__ __forceinline__ int accept_without_prev(const StepConsts &c, const StepThr &t, float rv, uint32_t x,
                                                   uint32_t prev, uint32_t cur)
{
    if (rv <= thr_min<SOPR>(c, t)) return 1;
    if (x == prev) return rv < thr_prev<SOPR>(c, t) ? 1 : 0;
    const bool af = rv < thr_found<SOPR>(c, t);
    // x is drawn from N(cur); when prev == cur the search must succeed.
    if (prev == cur) return af ? 1 : 0;
    const bool an = rv < thr_notfound<SOPR>(c, t);
    return af == an ? (af ? 1 : 0) : -1;
}

// The verdict with N(prev) = pix.csr[phead, phead + pdeg) at hand.  N(prev)
// is searched only when the verdict depends on it: for Node2vec a trial whose
// rand value lies on the same side of both thresholds (1 and 1/q) needs no
// search, so p = 0.5, q = 2 searches on a quarter of the trials and p = 2,
// q = 0.5 on a half, where every rand value above the smallest threshold
// (three quarters of them) used to search.  The step kernels are bound by the
// distinct lines their loads touch (one L1 tag access per cycle), most of
// them probes of this search.
template <bool SOPR, int SEARCH>
__device__ __forceinline__ bool accept_candidate(const StepConsts &c, const StepThr &t, float rv, uint32_t x,
                                                 uint32_t prev, uint32_t cur, const CsrIndex<SEARCH> &pix, uint32_t pbucket,
                                                 uint64_t phead, uint32_t pdeg)
{
    const int v = accept_without_prev<SOPR>(c, t, rv, x, prev, cur);
    if (v >= 0) return v != 0;
    return csr_contains(pix, pbucket, phead, pdeg, x) ? (rv < thr_found<SOPR>(c, t)) : (rv < thr_notfound<SOPR>(c, t));
}

// A walker whose step has rejected this many attempts is served by the whole
// warp (warp_first_accept).
constexpr uint32_t kHardAttempts = 4;

__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src)
{
    const uint32_t lo = __shfl_sync(0xFFFFFFFFu, (uint32_t)v, src);
    const uint32_t hi = __shfl_sync(0xFFFFFFFFu, (uint32_t)(v >> 32), src);
    return ((uint64_t)hi << 32) | lo;
}

template <typename T>
__device__ __forceinline__ T *shfl_ptr(T *p, int src)
{
    return reinterpret_cast<T *>(shfl64(reinterpret_cast<uint64_t>(p), src));
}

template <bool SOPR>
__device__ __forceinline__ StepThr shfl_thr(const StepThr &t, int src)
{
    StepThr o{0.f, 0.f, 0.f};
    if constexpr (SOPR) {
        o.inv_deg = __shfl_sync(0xFFFFFFFFu, t.inv_deg, src);
        o.sum = __shfl_sync(0xFFFFFFFFu, t.sum, src);
        o.t_prev = __shfl_sync(0xFFFFFFFFu, t.t_prev, src);
    }
    return o;
}

// Per-warp shared scratch of a cooperative step, in 32-bit words: run starts
// (32), run ends (32), and a filter of 2^kFilterBits buckets, one bit each.
constexpr uint32_t kFilterBits = 12;
constexpr int kCoopScratchWords = 64 + (1 << kFilterBits) / 32;

// Smallest k in [0, 2^24] for which `pred(k)` fails, where pred holds on a
// prefix of [0, 2^24).  rand_val(k << 8, maxv) is non-decreasing in k (an
// exact scaling followed by one rounded multiply by a positive constant), so
// every "rv <= T" / "rv < T" test of a step is such a prefix, and comparing
// k = y >> 8 with its bound gives the same verdict bit for bit.
template <class Pred>
__device__ __forceinline__ uint32_t rand_prefix(Pred pred)
{
    uint32_t lo = 0, hi = 1u << 24;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (pred(mid)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Integer bounds of a step's four rand-value tests, found by the whole warp:
// lanes 8w..8w+7 compute bound w (0: rv <= min, 1: rv < prev, 2: rv < found,
// 3: rv < notfound) and lane 8w returns it.  Each group tests the eight k
// around the estimate bound / maxv * 2^24, within three of the true bound when
// maxv and the bound are normal floats (the quotient is rounded once, and one
// rounding of k * 2^-24 * maxv moves it by at most half an ulp: each at most
// one step of k); a group whose window does not bracket the bound falls back
// to rand_prefix.
template <bool SOPR>
__device__ __forceinline__ uint32_t rand_bounds(const StepConsts &c, const StepThr &t)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t which = lane >> 3;
    const float maxv = thr_max<SOPR>(c, t);
    const float bound = which == 0 ? thr_min<SOPR>(c, t) : which == 1 ? thr_prev<SOPR>(c, t)
                      : which == 2 ? thr_found<SOPR>(c, t) : thr_notfound<SOPR>(c, t);
    auto pred = [&](uint32_t k) {
        const float rv = rand_val(k << 8, maxv);
        return which == 0 ? (rv <= bound) : (rv < bound);
    };
    const float est = __fmul_rn(__fdiv_rn(bound, maxv), 0x1p24f);
    const bool est_ok = est >= 0.0f && est <= 0x1p24f;  // false for NaN
    const int32_t base = (est_ok ? (int32_t)est : 0) - 4;
    const int32_t kc = base + (int32_t)(lane & 7u);
    const bool q = kc < 0 ? true : (kc >= (1 << 24) ? false : pred((uint32_t)kc));
    const unsigned g = (__ballot_sync(0xFFFFFFFFu, q) >> (lane & 24u)) & 0xFFu;
    // a bracket: true at the first candidate, false at the last, ones then zeros
    if (est_ok && (g & 1u) && !(g & 0x80u) && g == (1u << __popc(g)) - 1u) return (uint32_t)(base + __popc(g));
    return rand_prefix(pred);
}

// Whether a hard step is decided from candidate positions
// (warp_first_accept_runs) or by evaluating candidates 32 at a time.
// Positions need prev's neighbours to fit a lane each.  Setting them up (a
// search of N(cur) per neighbour, the filter) costs about as much as seven
// rounds of 32 candidates, and an attempt then half of one; a SOPR trial
// accepts with at least inv_deg / sum, so steps expected to take fewer than
// 192 attempts are evaluated.
template <bool SOPR>
__device__ __forceinline__ bool by_position(const StepThr &t, uint32_t pdeg, uint32_t prev, uint32_t cur)
{
    return pdeg < 32 && prev != cur && !(SOPR && t.sum <= 192.0f * t.inv_deg);
}

// Hard steps whose prev has fewer than 32 neighbours are decided without
// touching the candidate: a trial's verdict depends on x = N(cur)[pos] only
// through "x == prev" and "x in N(prev)", i.e. through whether pos falls in
// the run of prev, or of some y in N(prev), inside the sorted N(cur).  Those
// runs are located once per step (one search per lane).
//
// Trials then run on integers only.  The rand-value tests become bounds on
// k = y >> 8 (rand_bounds).  pos = x mod deg is not formed on the common path:
// with Lemire's fraction f = M*x mod 2^64 (M = ceil(2^64/deg)), pos =
// floor(f*deg / 2^64) and f lies in [M*pos, M*pos + 2^32), so its top kFilterBits
// bits name a bucket of positions.  A per-warp bitmap marks every bucket a run
// can reach; a trial whose bucket is unmarked is in no run and its verdict is
// k < max(k_min, k_notfound).  A round in which some trial passes that or is
// marked is looked at again exactly (pos, run lookup in `iv`).
//
// What bounds it: the Philox multiplies (17 wide products a draw, four cycles
// each per warp: 70 of the cycles of 32 attempts), then the set-up's loads.
template <bool SOPR>
__device__ __forceinline__ uint32_t warp_first_accept_runs(const StepConsts &c, const StepThr &t, uint32_t wid,
                                                           uint32_t hop, uint32_t p0, uint32_t limit,
                                                           const uint32_t *cadj, uint32_t deg, uint32_t magic,
                                                           uint32_t prev, const uint32_t *padj, uint32_t pdeg,
                                                           uint32_t *iv)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t *bm = iv + 64;
    constexpr uint32_t kFilterWords = (1u << kFilterBits) / 32;
    for (uint32_t w = lane; w < kFilterWords; w += 32) bm[w] = 0;
    // lane k < pdeg: run of N(prev)[k]; lane pdeg: run of prev
    uint32_t lo = 0, hi = 0;
    if (lane <= pdeg) {
        const uint32_t y = (lane < pdeg) ? __ldg(padj + lane) : prev;
        lo = list_below(cadj, deg, y);
        hi = lo;
        while (hi < deg && __ldg(cadj + hi) == y) hi++;
    }
    if (lane < pdeg) {
        iv[lane] = lo;
        iv[32 + lane] = hi;
    }
    const uint64_t M = fastmod_magic_by(deg, magic, __frcp_rn(__uint2float_rn(deg)));
    __syncwarp();
    if (hi > lo) {
        const uint32_t b0 = fraction_first(lo, M) >> (32 - kFilterBits), b1 = fraction_last(hi, M) >> (32 - kFilterBits);
        for (uint32_t w = b0 >> 5; w <= (b1 >> 5); ++w) {
            const uint32_t from = (w == (b0 >> 5)) ? (b0 & 31u) : 0u;
            const uint32_t to = (w == (b1 >> 5)) ? (b1 & 31u) : 31u;
            const uint32_t mask = (0xFFFFFFFFu >> (31u - to)) & (0xFFFFFFFFu << from);
            atomicOr(bm + w, mask);
        }
    }
    // integer bounds of the four rand-value tests
    const uint32_t kq = rand_bounds<SOPR>(c, t);
    const uint32_t k_min = __shfl_sync(0xFFFFFFFFu, kq, 0), k_prev = __shfl_sync(0xFFFFFFFFu, kq, 8);
    const uint32_t k_found = __shfl_sync(0xFFFFFFFFu, kq, 16), k_nf = __shfl_sync(0xFFFFFFFFu, kq, 24);
    const uint32_t k_fast = max(k_min, k_nf);
    const uint32_t plo = __shfl_sync(0xFFFFFFFFu, lo, (int)pdeg), phi = __shfl_sync(0xFFFFFFFFu, hi, (int)pdeg);
    __syncwarp();

    // exact verdict of a trial whose bucket is marked
    auto exact = [&](uint32_t x, uint32_t k) -> bool {
        if (k < k_min) return true;
        const uint32_t pos = fastmod(x, M, deg);
        if (pos >= plo && pos < phi) return k < k_prev;
        // last run whose start is <= pos (runs are in N(prev) order, so sorted)
        int r = -1;
        uint32_t a = 0, b = pdeg;
        while (a < b) {
            const uint32_t m = (a + b) >> 1;
            if (iv[m] <= pos) {
                r = (int)m;
                a = m + 1;
            } else {
                b = m;
            }
        }
        const bool found = r >= 0 && pos < iv[32 + r];
        return found ? (k < k_found) : (k < k_nf);
    };
    auto marked = [&](uint32_t x) -> bool {
        const uint32_t b = fraction_top(x, M);
        return (__funnelshift_r(bm[b >> (37 - kFilterBits)], 0u, b >> (32 - kFilterBits)) & 1u) != 0;
    };
    // 64 attempts per round, two independent Philox chains per lane
    for (uint32_t base = p0; base < limit; base += 64) {
        const U4 r0 = draw(c, wid, hop, base + lane), r1 = draw(c, wid, hop, base + 32 + lane);
        const uint32_t k0 = r0.y >> 8, k1 = r1.y >> 8;
        const bool in0 = marked(r0.x), in1 = marked(r1.x);
        if (!__any_sync(0xFFFFFFFFu, in0 || in1 || k0 < k_fast || k1 < k_fast)) continue;
        const bool acc0 = base + lane < limit && (in0 ? exact(r0.x, k0) : k0 < k_fast);
        const bool acc1 = base + 32 + lane < limit && (in1 ? exact(r1.x, k1) : k1 < k_fast);
        const unsigned m0 = __ballot_sync(0xFFFFFFFFu, acc0);
        const unsigned m1 = __ballot_sync(0xFFFFFFFFu, acc1);
        if (m0 | m1) return base + (m0 ? 0u : 32u) + (uint32_t)__ffs(m0 ? m0 : m1) - 1;
    }
    return limit;
}

// All 32 lanes, with identical (broadcast) arguments, evaluate attempts
// p0+lane, p0+32+lane, ... of one walker's step and return the first accepting
// attempt in attempt order -- the one a single thread evaluating them one by
// one would take.  Returns `limit` if none of the attempts below `limit`
// accepts.  N(cur) is cadj[0, deg), magic its mod_magic; N(prev) is
// pix.csr[0, pdeg), its table at bucket pbucket.
template <bool SOPR, int SEARCH>
__device__ __forceinline__ uint32_t warp_first_accept(const StepConsts &c, const StepThr &t, uint32_t wid,
                                                      uint32_t hop, uint32_t p0, uint32_t limit,
                                                      const uint32_t *cadj, uint32_t deg, uint32_t magic,
                                                      uint32_t prev, uint32_t cur, const CsrIndex<SEARCH> &pix,
                                                      uint32_t pbucket, uint32_t pdeg, uint32_t *iv)
{
    uint32_t first = limit;
    if (by_position<SOPR>(t, pdeg, prev, cur)) {
        first = warp_first_accept_runs<SOPR>(c, t, wid, hop, p0, limit, cadj, deg, magic, prev, pix.csr, pdeg, iv);
    } else {
        const uint32_t lane = threadIdx.x & 31u;
        const float maxv = thr_max<SOPR>(c, t);
        for (uint32_t base = p0; base < limit; base += 32) {
            const uint32_t att = base + lane;
            bool acc = false;
            if (att < limit) {
                const U4 r = draw(c, wid, hop, att);
                const float rv = rand_val(r.y, maxv);
                const uint32_t x = __ldg(cadj + mod_by(r.x, deg, magic));
                acc = accept_candidate<SOPR>(c, t, rv, x, prev, cur, pix, pbucket, 0ull, pdeg);
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, acc);
            if (m) {
                first = base + (uint32_t)__ffs(m) - 1;
                break;
            }
        }
    }
    __syncwarp();
    return first;
}

}  // namespace gw
