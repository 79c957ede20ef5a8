// Weighted Node2vec walks, in-core (the reference has no counterpart: it loads
// edge weights, engine/cache.hpp:71, gpu/memory.hpp:134-137, and never samples
// with them).
//
// Semantics: from cur (with prev), candidate x is drawn in proportion to the
// weight of cur -> x, then accepted by the unweighted rule (1/p if x == prev,
// 1 if x is a neighbour of prev, 1/q otherwise, with the reference's
// thresholds and precision, engine/engine.hpp:209-258): P(x) is proportional
// to w(cur, x) times the Node2vec bias, the usual weighted Node2vec.
// The candidate comes from Walker's alias table of cur's out-edges: column
// i = lane x % deg of the trial's draw (the unweighted rand_pos), coin =
// float(lane w >> 8) * 2^-24; the trial takes column i when coin < prob[i],
// its alias otherwise.  Lanes y (rand value) and z (termination) keep their
// meaning, so a graph whose weights are all equal walks exactly as unweighted.
// The walk itself is the in-core kernel (gw_walk.cu) with its W flag; this
// file builds the alias tables.
//
// Alias tables (Vose's method, per vertex: one thread each, a CTA for each
// vertex above 256 neighbours, below): the weights are
// summed in double in index order, scaled to p_i = w_i * deg / sum, split
// into a queue of p < 1 and a queue of p >= 1 in index order; repeatedly the
// next small s takes the front large l as its alias (prob[s] = (float)p_s)
// and p_l = (p_l + p_s) - 1, l moving to the back of the small queue when it
// drops below 1; leftovers get probability 1.  Every operation is an IEEE
// double rounded to nearest, so the oracle's C restatement builds the same
// table bit for bit.
#include <cuda_runtime.h>
#include <cstdint>
#include "gw_kernels.cuh"
#include "gw_weighted.cuh"

namespace gw {

constexpr uint64_t kHubDeg = 256;  // vertices above this degree get a CTA each

// Vose's loop for one vertex whose probabilities p[0, d) are scaled; the
// queues hold indices in the order they are pushed.  p and the queues may be
// shared or global memory.
__device__ void vose_loop(uint64_t d, double *p, uint32_t *small, uint32_t *large, AliasEntry *out)
{
    uint64_t ns = 0, nl = 0, hs = 0, hl = 0;
    for (uint64_t i = 0; i < d; ++i) {
        if (p[i] < 1.0) small[ns++] = (uint32_t)i;
        else large[nl++] = (uint32_t)i;
    }
    while (hs < ns && hl < nl) {
        const uint32_t sidx = small[hs++], lidx = large[hl];
        out[sidx] = AliasEntry{__double2float_rn(p[sidx]), lidx};
        p[lidx] = __dsub_rn(__dadd_rn(p[lidx], p[sidx]), 1.0);
        if (p[lidx] < 1.0) {
            ++hl;
            small[ns++] = lidx;
        }
    }
    while (hl < nl) {
        const uint32_t lidx = large[hl++];
        out[lidx] = AliasEntry{1.f, lidx};
    }
    while (hs < ns) {
        const uint32_t sidx = small[hs++];
        out[sidx] = AliasEntry{1.f, sidx};
    }
}

// Vertices of degree at most kHubDeg: one thread each.
__global__ void k_build_alias(const uint64_t *__restrict__ beg, const float *__restrict__ w, uint32_t nverts,
                              double *__restrict__ pd, uint32_t *__restrict__ qs, uint32_t *__restrict__ ql,
                              AliasEntry *__restrict__ out, uint32_t *err)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nverts; v += stride) {
        const uint64_t h = beg[v], d = beg[v + 1] - h;
        if (d == 0 || d > kHubDeg) continue;
        double sum = 0.0;
        bool bad = false;
        for (uint64_t i = 0; i < d; ++i) {
            const float wi = w[h + i];
            bad |= !(wi > 0.f && wi < __int_as_float(0x7F800000));
            sum = __dadd_rn(sum, (double)wi);
        }
        if (bad) {
            atomicOr(err, kErrWeight);
            for (uint64_t i = 0; i < d; ++i) out[h + i] = AliasEntry{1.f, (uint32_t)i};
            continue;
        }
        for (uint64_t i = 0; i < d; ++i) pd[h + i] = __ddiv_rn(__dmul_rn((double)w[h + i], (double)d), sum);
        vose_loop(d, pd + h, qs + h, ql + h, out + h);
    }
}

// The vertices of degree in (lo, hi], appended to the list work[2 + i]
// (work[0] counts it) that the CTAs of k_build_alias_hubs take one vertex at
// a time from (work[1]): R-MAT hubs sit at ids with many zero bits, so a
// fixed stride would give a few CTAs most of the work.  Listing the largest
// first lets their serial loops start first.
__global__ void k_list_hubs(const uint64_t *__restrict__ beg, uint32_t nverts, uint64_t lo, uint64_t hi,
                            uint32_t *__restrict__ work)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < nverts; b += stride) {
        const uint64_t v = b + threadIdx.x;
        const bool hub = v < nverts && beg[v + 1] - beg[v] > lo && beg[v + 1] - beg[v] <= hi;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, hub);
        uint32_t base = 0;
        if (lane == 0 && m) base = atomicAdd(work, (uint32_t)__popc(m));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (hub) work[2 + base + __popc(m & ((1u << lane) - 1u))] = (uint32_t)v;
    }
}

// Vertices of degree above kHubDeg: one CTA each, taken from the list.
//
// Vose's loop is one chain of double operations (each step's residual is the
// next one's input), and so is the weight sum; they are what bounds the build:
// the largest hub's length times a step.  One thread runs each chain out of
// shared memory -- two dependent additions and a compare a step -- and the
// whole CTA does everything else around it, kWin entries at a time: gathers the
// probabilities the next steps will read and writes the entries the last ones
// decided.
//
// Both queues are read in order.  The large queue is the initial larges (index
// order), each one's probability untouched until it is the current large, whose
// residual r stays in a register.  Every consumed large has dropped below 1 and
// joined the small queue, so the small queue is the initial smalls (index
// order) followed by the larges in order, with their residuals: entry j >= ns0
// is large j - ns0, and ql[0, hl) need not be written again.
//
// Measured (R-MAT, 200,003 vertices, 16 edges drawn for each): 5.5 ms with a
// warp in lockstep that fetched the queues by shuffles, 1.7 ms so.
constexpr uint32_t kWin = 1024;
__global__ void __launch_bounds__(128)
    k_build_alias_hubs(const uint64_t *__restrict__ beg, const float *__restrict__ w, uint32_t *__restrict__ work,
                       double *__restrict__ pd, uint32_t *__restrict__ qs, uint32_t *__restrict__ ql,
                       AliasEntry *__restrict__ out, uint32_t *err)
{
    __shared__ uint32_t s_next;
    __shared__ double s_sum;
    __shared__ uint32_t s_cnt[2][4];  // per warp: smalls, larges of the current 128 indices
    __shared__ uint32_t s_tot[2];     // smalls, larges so far
    __shared__ __align__(16) double s_sp[kWin], s_lp[kWin], s_lr[kWin];  // small queue; larges: initial, residual once dropped
    __shared__ uint32_t s_si[kWin], s_li[kWin];            // their indices
    __shared__ uint16_t s_ord[kWin];                       // the large each small was joined with
    __shared__ uint32_t s_adv[2];                          // entries of the windows consumed
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t nhubs = work[0];
    for (;;) {
        __syncthreads();  // the previous vertex is done with the shared memory
        if (threadIdx.x == 0) {
            s_next = atomicAdd(work + 1, 1u);
            s_tot[0] = s_tot[1] = 0;
        }
        __syncthreads();
        if (s_next >= nhubs) break;
        const uint64_t v = work[2 + s_next];
        const uint64_t h = beg[v], d = beg[v + 1] - h;
        // the weight sum: one in-order chain of double additions over weights
        // that the other warps bring in, a window ahead
        float *buf = reinterpret_cast<float *>(s_sp);  // two windows of kWin floats
        bool bad = false;
        auto fetch = [&](uint64_t at, float *to, uint32_t t0, uint32_t nt) {
            for (uint32_t i = t0; i < kWin && at + i < d; i += nt) {
                const float x = w[h + at + i];
                bad |= !(x > 0.f && x < __int_as_float(0x7F800000));
                to[i] = x;
            }
        };
        fetch(0, buf, threadIdx.x, blockDim.x);
        __syncthreads();
        double sum = 0.0;
        for (uint64_t at = 0, k = 0; at < d; at += kWin, ++k) {
            const float *cur = buf + (k & 1) * kWin;
            if (warp != 0) {
                fetch(at + kWin, buf + ((k + 1) & 1) * kWin, threadIdx.x - 32, blockDim.x - 32);
            } else if (lane == 0) {
                const uint32_t n = (uint32_t)min((uint64_t)kWin, d - at);
                uint32_t i = 0;
                for (; i + 8 <= n; i += 8) {
                    const float4 a = *reinterpret_cast<const float4 *>(cur + i);
                    const float4 b = *reinterpret_cast<const float4 *>(cur + i + 4);
                    sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sum, (double)a.x), (double)a.y), (double)a.z), (double)a.w);
                    sum = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(sum, (double)b.x), (double)b.y), (double)b.z), (double)b.w);
                }
                for (; i < n; ++i) sum = __dadd_rn(sum, (double)cur[i]);
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) s_sum = sum;
        bad = __syncthreads_or(bad);
        if (bad) {
            if (threadIdx.x == 0) atomicOr(err, kErrWeight);
            for (uint64_t i = threadIdx.x; i < d; i += blockDim.x) out[h + i] = AliasEntry{1.f, (uint32_t)i};
            continue;
        }
        // scale, and split the indices into the two queues in index order
        sum = s_sum;
        for (uint64_t b = 0; b < d; b += blockDim.x) {
            const uint64_t i = b + threadIdx.x;
            double p = 0.0;
            if (i < d) {
                p = __ddiv_rn(__dmul_rn((double)w[h + i], (double)d), sum);
                pd[h + i] = p;
            }
            const bool sm = i < d && p < 1.0, lg = i < d && !(p < 1.0);
            const unsigned bs = __ballot_sync(0xFFFFFFFFu, sm), bl = __ballot_sync(0xFFFFFFFFu, lg);
            if (lane == 0) {
                s_cnt[0][warp] = __popc(bs);
                s_cnt[1][warp] = __popc(bl);
            }
            __syncthreads();
            uint32_t os = s_tot[0], ol = s_tot[1];
            for (uint32_t k = 0; k < warp; ++k) {
                os += s_cnt[0][k];
                ol += s_cnt[1][k];
            }
            const unsigned lt = (1u << lane) - 1u;
            if (sm) qs[h + os + __popc(bs & lt)] = (uint32_t)i;
            if (lg) ql[h + ol + __popc(bl & lt)] = (uint32_t)i;
            __syncthreads();
            if (threadIdx.x == 0)
                for (uint32_t k = 0; k < blockDim.x / 32; ++k) {
                    s_tot[0] += s_cnt[0][k];
                    s_tot[1] += s_cnt[1][k];
                }
            __syncthreads();
        }
        const uint32_t ns0 = s_tot[0], nl = s_tot[1];
        // Vose's loop: hs smalls and hl larges are consumed so far
        uint32_t hs = 0, hl = 0;
        double r = 0.0;  // thread 0: residual of large hl
        bool have_r = false;
        while (hs < ns0 + hl && hl < nl) {
            const uint32_t ns = min(kWin, ns0 + hl - hs), ng = min(kWin, nl - hl);
            for (uint32_t i = threadIdx.x; i < ns; i += blockDim.x) {
                const uint32_t j = hs + i, idx = j < ns0 ? qs[h + j] : ql[h + j - ns0];
                s_si[i] = idx;
                s_sp[i] = pd[h + idx];
            }
            for (uint32_t i = threadIdx.x; i < ng; i += blockDim.x) {
                const uint32_t idx = ql[h + hl + i];
                s_li[i] = idx;
                s_lp[i] = pd[h + idx];
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t k = 0, l = 0, n = ns;
                if (!have_r) r = s_lp[0];
                have_r = true;
                double ps = s_sp[0];
                for (;;) {
                    const double next = s_sp[min(k + 1, kWin - 1)];  // read ahead of the chain
                    const double t = __dsub_rn(__dadd_rn(r, ps), 1.0);
                    s_ord[k] = (uint16_t)l;
                    ++k;
                    ps = next;
                    r = t;
                    if (t < 1.0) {
                        // the large drops: small number ns0 + hl + l
                        s_lr[l] = t;
                        const uint32_t at = ns0 + hl + l - hs;
                        if (at < kWin) {
                            s_sp[at] = t;
                            s_si[at] = s_li[l];
                            n = at + 1;
                            if (at == k) ps = t;
                        }
                        if (++l == ng) {
                            have_r = false;
                            break;
                        }
                        r = s_lp[l];
                    }
                    if (k == n) break;
                }
                s_adv[0] = k;
                s_adv[1] = l;
            }
            __syncthreads();
            const uint32_t k = s_adv[0], l = s_adv[1];
            for (uint32_t i = threadIdx.x; i < k; i += blockDim.x)
                out[h + s_si[i]] = AliasEntry{__double2float_rn(s_sp[i]), s_li[s_ord[i]]};
            for (uint32_t i = threadIdx.x; i < l; i += blockDim.x) pd[h + s_li[i]] = s_lr[i];
            hs += k;
            hl += l;
            __syncthreads();  // the windows are read, the residuals written
        }
        // what is left keeps its own column: the larges from the current one
        // on, and the smalls not consumed
        for (uint32_t k = hl + threadIdx.x; k < nl; k += blockDim.x) {
            const uint32_t i = ql[h + k];
            out[h + i] = AliasEntry{1.f, i};
        }
        for (uint32_t k = hs + threadIdx.x; k < ns0 + hl; k += blockDim.x) {
            const uint32_t i = k < ns0 ? qs[h + k] : ql[h + (k - ns0)];
            out[h + i] = AliasEntry{1.f, i};
        }
    }
}

cudaError_t launch_build_alias(const uint64_t *beg, const float *w, uint32_t nverts, double *pd, uint32_t *qs,
                               uint32_t *ql, uint32_t *work, AliasEntry *out, uint32_t *err, int num_sms, cudaStream_t s)
{
    k_build_alias<<<num_sms * 8, 128, 0, s>>>(beg, w, nverts, pd, qs, ql, out, err);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(work, 0, 2 * sizeof(uint32_t), s)) != cudaSuccess) return e;
    k_list_hubs<<<num_sms * 4, 256, 0, s>>>(beg, nverts, 16 * kHubDeg, ~0ull, work);
    k_list_hubs<<<num_sms * 4, 256, 0, s>>>(beg, nverts, kHubDeg, 16 * kHubDeg, work);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_build_alias_hubs<<<num_sms * 4, 128, 0, s>>>(beg, w, work, pd, qs, ql, out, err);
    return cudaGetLastError();
}


}  // namespace gw
