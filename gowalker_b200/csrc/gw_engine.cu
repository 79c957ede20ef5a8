// C ABI of the walk engine: handle, graph residency, walker population, runs.
//
// Replaces the device-side plumbing of GOWalker's graph_engine
// (engine/engine.hpp:54-102, 406-638), gpu/memory.hpp and the walker
// creation of engine/walk.hpp:272-389.  Every failure returns a status and
// records a message; nothing exits the process.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>
#include <sys/mman.h>
#include "gw_engine.cuh"
#include "gw_memory.cuh"

using namespace gw;

// ------------------------------------------------------------------ helpers

int gw_handle::fail(int status, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    err = buf;
    return status;
}

int gw_handle::cuda(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return GW_OK;
    cudaGetLastError();
    const int st = (e == cudaErrorMemoryAllocation) ? GW_ERR_NOMEM : GW_ERR_CUDA;
    return fail(st, "%s: %s", what, cudaGetErrorString(e));
}

int gw_handle::dev_alloc(void **p, uint64_t bytes, const char *what)
{
    return cuda(device_malloc_any(p, bytes, this), what);
}

// Every engine, so that one's index can give way to another's allocation.  The
// lists and gw_handle::in_call are guarded by the mutex; an index is dropped
// under it, or by a call of its own engine, which others see by in_call.
namespace {
struct Engines {
    std::mutex mu;
    std::vector<gw_handle *> all;
};
Engines &engines()
{
    static Engines *e = new Engines;  // outlives every static
    return *e;
}
struct InCall {
    explicit InCall(gw_handle *h) : h(h) { set(true); }
    ~InCall() { set(false); }
    void set(bool v)
    {
        std::lock_guard<std::mutex> l(engines().mu);
        h->in_call = v;
    }
    gw_handle *h;
};
}  // namespace

cudaError_t gw::device_malloc_any(void **p, size_t bytes, gw_handle *self)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> l(engines().mu);
    for (gw_handle *h : engines().all) {
        if (h->cfg.device != dev || (h->in_call && h != self) || !h->d_index) continue;
        cudaGetLastError();
        cudaStreamSynchronize(h->s_compute);
        h->drop_index();
        h->index_refused = true;
        if ((e = cudaMalloc(p, bytes)) != cudaErrorMemoryAllocation) break;
    }
    return e;
}

void gw::consts_from_config(const gw_config &c, StepConsts &k)
{
    k.maxhops = c.maxhops;
    k.key0 = (uint32_t)c.seed;
    k.key1 = (uint32_t)(c.seed >> 32);
    // engine/engine.hpp:169-172, in fp32 exactly as the reference writes them
    const float inv_p = 1.0f / c.p;
    const float inv_q = 1.0f / c.q;
    const float mx_q1 = (inv_q < 1.0f) ? 1.0f : inv_q;
    const float mn_q1 = (1.0f < inv_q) ? 1.0f : inv_q;
    k.n2v_maxv = (inv_p < mx_q1) ? mx_q1 : inv_p;
    k.n2v_minv = (mn_q1 < inv_p) ? mn_q1 : inv_p;
    k.inv_p = inv_p;
    k.inv_q = inv_q;
    k.alpha = c.alpha;
    k.term_prob = c.term_prob;
    k.one_m_alpha = 1.0 - (double)c.alpha;
    philox_schedule(k.key0, k.key1, k.rk0, k.rk1);
}

static bool config_ok(const gw_config &c, std::string &why)
{
    if (c.algorithm > GW_SOSR) { why = "algorithm must be 0 (node2vec), 1 (SOPR) or 2 (SOSR)"; return false; }
    if (!(c.p > 0.0f) || !(c.q > 0.0f)) { why = "p and q must be positive"; return false; }
    if (!(c.alpha >= 0.0f) || !(c.alpha <= 1.0f)) { why = "alpha must lie in [0, 1]"; return false; }
    if (!(c.term_prob >= 0.0f) || !(c.term_prob < 1.0f)) { why = "term_prob must lie in [0, 1)"; return false; }
    if (c.init_mode > GW_INIT_RANDOM) { why = "unknown init_mode"; return false; }
    if (c.record_paths > GW_PATHS_FULL) { why = "unknown record_paths"; return false; }
    if (c.launch_mode > GW_LAUNCH_PER_HOP) { why = "unknown launch_mode"; return false; }
    if (c.learned_mode & ~(GW_LEARNED_EVICT | GW_LEARNED_ZERO_SWITCH)) { why = "unknown learned_mode bits"; return false; }
    if (c.threadperblock != 0 && (c.threadperblock % 32 != 0 || c.threadperblock > 1024)) {
        why = "threadperblock must be a multiple of 32 up to 1024";
        return false;
    }
    return true;
}

// ------------------------------------------------------------------ ABI: basics

extern "C" int gw_version(void) { return GW_ABI_VERSION; }

extern "C" const char *gw_status_string(int s)
{
    switch (s) {
    case GW_OK: return "ok";
    case GW_ERR_ARG: return "invalid argument";
    case GW_ERR_CUDA: return "CUDA runtime error";
    case GW_ERR_NOMEM: return "out of memory";
    case GW_ERR_STATE: return "call out of order";
    case GW_ERR_TIMEOUT: return "device wait timed out";
    case GW_ERR_DEVICE: return "kernel reported an error";
    case GW_ERR_GRAPH: return "graph failed validation";
    default: return "unknown status";
    }
}

extern "C" int gw_config_default(gw_config *c)
{
    if (!c) return GW_ERR_ARG;
    memset(c, 0, sizeof(*c));
    c->cache_size = 4ull << 30;    // "memory" 4 GB (api/constants.hpp MEMORY_CACHE)
    c->blocksize = 1024ull << 20;  // "blocksize" 1024 MB
    c->algorithm = GW_NODE2VEC;
    c->p = 0.5f;
    c->q = 2.0f;
    c->alpha = 0.2f;
    c->maxhops = 30;
    c->walkpersource = 1;
    c->numwalks = 0;
    c->init_mode = GW_INIT_PER_VERTEX;
    c->term_prob = 0.0f;
    c->seed = 42;
    c->record_paths = GW_PATHS_NONE;
    c->device = 0;
    return GW_OK;
}

extern "C" int gw_create(const gw_config *cfg, gw_handle **out)
{
    if (!cfg || !out) return GW_ERR_ARG;
    *out = nullptr;
    std::string why;
    if (!config_ok(*cfg, why)) return GW_ERR_ARG;
    gw_handle *h = new (std::nothrow) gw_handle();
    if (!h) return GW_ERR_NOMEM;
    h->cfg = *cfg;
    int st = h->init_device();
    if (st != GW_OK) {
        delete h;
        return st;
    }
    *out = h;
    return GW_OK;
}

extern "C" int gw_destroy(gw_handle *h)
{
    if (!h) return GW_ERR_ARG;
    h->release();
    delete h;
    return GW_OK;
}

extern "C" int gw_last_error(gw_handle *h, char *buf, size_t n)
{
    if (!h || !buf || n == 0) return GW_ERR_ARG;
    snprintf(buf, n, "%s", h->err.c_str());
    return GW_OK;
}

extern "C" int gw_set_config(gw_handle *h, const gw_config *cfg)
{
    if (!h || !cfg) return GW_ERR_ARG;
    std::string why;
    if (!config_ok(*cfg, why)) return h->fail(GW_ERR_ARG, "%s", why.c_str());
    if (cfg->device != h->cfg.device) return h->fail(GW_ERR_ARG, "device cannot change on a live handle");
    const bool paths_grow = cfg->record_paths == GW_PATHS_FULL &&
                            (h->cfg.record_paths != GW_PATHS_FULL || cfg->maxhops != h->cfg.maxhops);
    h->cfg = *cfg;
    if (paths_grow) h->walkers_ready = false;
    return GW_OK;
}

extern "C" int gw_stream(gw_handle *h, void **stream)
{
    if (!h || !stream) return GW_ERR_ARG;
    *stream = (void *)h->s_compute;
    return GW_OK;
}

// ------------------------------------------------------------------ handle internals

int gw_handle::init_device()
{
    int ndev = 0;
    int st = cuda(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
    if (st) return st;
    if (cfg.device < 0 || cfg.device >= ndev) return fail(GW_ERR_ARG, "device %d of %d", cfg.device, ndev);
    if ((st = cuda(cudaSetDevice(cfg.device), "cudaSetDevice"))) return st;
    // the attribute alone: all of a device's properties take 2.4 ms to collect
    if ((st = cuda(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, cfg.device), "SM count"))) return st;
    if ((st = cuda(cudaStreamCreateWithFlags(&s_compute, cudaStreamNonBlocking), "stream"))) return st;
    if ((st = cuda(cudaStreamCreateWithFlags(&s_copy, cudaStreamNonBlocking), "stream"))) return st;
    if ((st = cuda(cudaEventCreate(&ev_start), "event"))) return st;
    if ((st = cuda(cudaEventCreate(&ev_kernel0), "event"))) return st;
    if ((st = cuda(cudaEventCreate(&ev_kernel1), "event"))) return st;
    if ((st = cuda(cudaEventCreate(&ev_stop), "event"))) return st;
    if ((st = dev_alloc(d_ctr, sizeof(unsigned long long) * kCtrWords, "counters"))) return st;
    d_err = reinterpret_cast<uint32_t *>(d_ctr + kCtrCount);
    if ((st = cuda(cudaMallocHost(&h_ctr, sizeof(unsigned long long) * kCtrWords), "pinned counters")))
        return st;
    memset(h_ctr, 0, sizeof(unsigned long long) * kCtrWords);
    std::lock_guard<std::mutex> l(engines().mu);
    engines().all.push_back(this);
    return GW_OK;
}

void gw_handle::release()
{
    {
        std::lock_guard<std::mutex> l(engines().mu);
        auto &all = engines().all;
        all.erase(std::remove(all.begin(), all.end(), this), all.end());
    }
    cudaSetDevice(cfg.device);
    if (s_compute) cudaStreamSynchronize(s_compute);
    if (s_copy) cudaStreamSynchronize(s_copy);
    free_own_graph();
    cudaFree(own_w);
    cudaFree(d_alias);
    own_w = nullptr;
    d_alias = nullptr;
    alias_ready = false;
    cudaFree(d_paths);
    cudaFree(d_hashes);
    cudaFree(d_ctr);
    drop_index();
    if (h_ctr) cudaFreeHost(h_ctr);
    ooc_release();
    if (ev_start) cudaEventDestroy(ev_start);
    if (ev_kernel0) cudaEventDestroy(ev_kernel0);
    if (ev_kernel1) cudaEventDestroy(ev_kernel1);
    if (ev_stop) cudaEventDestroy(ev_stop);
    if (s_compute) cudaStreamDestroy(s_compute);
    if (s_copy) cudaStreamDestroy(s_copy);
    d_paths = nullptr;
    d_lens = nullptr;
    d_hashes = nullptr;
}

void gw_handle::free_own_graph()
{
    cudaFree(own_beg);
    cudaFree(own_csr_apart);
    own_beg = nullptr;
    own_csr = own_csr_apart = nullptr;
}

uint64_t gw_handle::graph_bytes() const
{
    return ((uint64_t)nverts + 1) * sizeof(uint64_t) + nedges * sizeof(uint32_t) +
           (weighted ? nedges * (sizeof(float) + sizeof(gw::AliasEntry)) : 0);
}

bool gw_handle::host_graph_complete() const
{
    if (nblocks == 0 || host_beg.size() != nblocks) return false;
    for (uint32_t b = 0; b < nblocks; ++b)
        if (!host_beg[b] || (!host_csr[b] && eblocks[b + 1] > eblocks[b])) return false;
    return true;
}

// Copy every host block into one contiguous device CSR.  Blocks are
// consecutive vertex ranges and their offsets are absolute, so block b's
// nverts offsets land at vblocks[b] and its neighbours at eblocks[b].
int gw_handle::upload_whole_graph(cudaStream_t s, uint64_t *h2d)
{
    int st;
    if (!own_beg) {
        const uint64_t beg_bytes = (((uint64_t)nverts + 1) * sizeof(uint64_t) + 255) & ~255ull;
        const uint64_t csr_bytes = (nedges ? nedges : 1) * sizeof(uint32_t);
        const bool apart = beg_bytes < kShareBytes && csr_bytes < kShareBytes;
        if ((st = dev_alloc(own_beg, beg_bytes + (apart ? 0 : csr_bytes), "graph"))) return st;
        own_csr = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(own_beg) + beg_bytes);
        if (apart) {
            if ((st = dev_alloc(own_csr_apart, csr_bytes, "graph"))) {
                free_own_graph();
                return st;
            }
            own_csr = own_csr_apart;
        }
    }
    uint64_t bytes = 0;
    for (uint32_t b = 0; b < nblocks; ++b) {
        const uint64_t nv = (uint64_t)vblocks[b + 1] - vblocks[b];
        const uint64_t ne = eblocks[b + 1] - eblocks[b];
        const uint64_t nvc = (b + 1 == nblocks) ? nv + 1 : nv;
        if (nvc) {
            if ((st = cuda(cudaMemcpyAsync(own_beg + vblocks[b], host_beg[b], nvc * sizeof(uint64_t),
                                           cudaMemcpyHostToDevice, s), "block offsets H2D")))
                return st;
            bytes += nvc * sizeof(uint64_t);
        }
        if (ne) {
            if ((st = cuda(cudaMemcpyAsync(own_csr + eblocks[b], host_csr[b], ne * sizeof(uint32_t),
                                           cudaMemcpyHostToDevice, s), "block neighbours H2D")))
                return st;
            bytes += ne * sizeof(uint32_t);
        }
    }
    if (weighted && !device_graph) {
        if (!own_w && (st = dev_alloc(own_w, (nedges ? nedges : 1) * sizeof(float), "edge weights")))
            return st;
        for (uint32_t b = 0; b < nblocks; ++b) {
            const uint64_t ne = eblocks[b + 1] - eblocks[b];
            if (!ne) continue;
            if ((st = cuda(cudaMemcpyAsync(own_w + eblocks[b], host_w[b], ne * sizeof(float), cudaMemcpyHostToDevice,
                                           s), "block weights H2D")))
                return st;
            bytes += ne * sizeof(float);
        }
        dev_w = own_w;
        alias_ready = false;
    }
    dev_beg = own_beg;
    dev_csr = own_csr;
    resident = true;
    validated = false;
    if (h2d) *h2d += bytes;
    return GW_OK;
}

int gw_handle::ensure_outputs()
{
    const uint64_t n = nwalkers;
    const uint32_t stride = cfg.maxhops + 1;
    int st;
    if (n > cap_walkers) {
        cudaFree(d_hashes);
        d_hashes = nullptr;
        d_lens = nullptr;
        cap_walkers = 0;
        if ((st = dev_alloc(d_hashes, n * (sizeof(uint64_t) + sizeof(uint32_t)), "path hashes and lengths")))
            return st;
        d_lens = reinterpret_cast<uint32_t *>(d_hashes + n);
        cap_walkers = n;
        cap_path_walkers = 0;
    }
    if (cfg.record_paths == GW_PATHS_FULL) {
        const uint64_t need = n * (uint64_t)stride;
        if (need > cap_path_words) {
            cudaFree(d_paths);
            d_paths = nullptr;
            cap_path_words = 0;
            cap_path_walkers = 0;
            if ((st = dev_alloc(d_paths, need * sizeof(uint32_t), "paths"))) return st;
            cap_path_words = need;
        }
        path_stride = stride;
        cap_path_walkers = n;
    }
    return GW_OK;
}

// ------------------------------------------------------------------ ABI: graph

extern "C" int gw_set_graph_meta(gw_handle *h, uint32_t nverts, uint64_t nedges, uint32_t nblocks,
                                 const uint32_t *vblocks, const uint64_t *eblocks)
{
    if (!h) return GW_ERR_ARG;
    if (!vblocks || !eblocks || nblocks == 0) return h->fail(GW_ERR_ARG, "block table missing");
    if (vblocks[0] != 0 || vblocks[nblocks] != nverts)
        return h->fail(GW_ERR_GRAPH, "vertex blocks must start at 0 and end at nverts");
    if (eblocks[0] != 0 || eblocks[nblocks] != nedges)
        return h->fail(GW_ERR_GRAPH, "edge blocks must start at 0 and end at nedges");
    for (uint32_t b = 0; b < nblocks; ++b) {
        if (vblocks[b + 1] < vblocks[b] || eblocks[b + 1] < eblocks[b])
            return h->fail(GW_ERR_GRAPH, "block table is not monotone at block %u", b);
    }
    cudaSetDevice(h->cfg.device);
    cudaStreamSynchronize(h->s_compute);
    h->nverts = nverts;
    h->nedges = nedges;
    h->nblocks = nblocks;
    h->vblocks.assign(vblocks, vblocks + nblocks + 1);
    h->eblocks.assign(eblocks, eblocks + nblocks + 1);
    h->host_beg.assign(nblocks, nullptr);
    h->host_csr.assign(nblocks, nullptr);
    h->host_w.assign(nblocks, nullptr);
    h->weighted = false;
    h->dev_w = nullptr;
    cudaFree(h->own_w);
    h->own_w = nullptr;
    cudaFree(h->d_alias);  // sized for the edges of the graph before
    h->d_alias = nullptr;
    h->alias_ready = false;
    h->dev_beg = nullptr;
    h->dev_csr = nullptr;
    h->resident = false;
    h->validated = false;
    h->free_own_graph();
    h->ooc_release();
    h->walkers_ready = false;
    std::lock_guard<std::mutex> l(engines().mu);
    h->index_search = kQuarter;
    // its memory serves a graph of like size (337 MB take 1.7 ms to free and take again)
    if (h->index_cap >= gw_handle::kSmallIndex && h->index_cap > 2 * h->index_layout(kTable).bytes) h->drop_index();
    return GW_OK;
}

extern "C" int gw_host_block(gw_handle *h, uint32_t blk, const uint64_t *beg, const uint32_t *csr)
{
    if (!h) return GW_ERR_ARG;
    if (blk >= h->nblocks) return h->fail(GW_ERR_ARG, "block %u out of range (%u blocks)", blk, h->nblocks);
    if (!beg) return h->fail(GW_ERR_ARG, "block %u offsets missing", blk);
    const uint64_t nv = (uint64_t)h->vblocks[blk + 1] - h->vblocks[blk];
    if (beg[0] != h->eblocks[blk] || beg[nv] != h->eblocks[blk + 1])
        return h->fail(GW_ERR_GRAPH, "block %u offsets disagree with the edge block table", blk);
    h->host_beg[blk] = beg;
    h->host_csr[blk] = csr;
    h->resident = false;
    h->ooc_invalidate(true);
    return GW_OK;
}

extern "C" int gw_device_graph(gw_handle *h, const uint64_t *d_beg, const uint32_t *d_csr)
{
    if (!h) return GW_ERR_ARG;
    if (h->nblocks == 0) return h->fail(GW_ERR_STATE, "set the graph meta first");
    if (!d_beg || (!d_csr && h->nedges)) return h->fail(GW_ERR_ARG, "device graph pointers missing");
    cudaSetDevice(h->cfg.device);
    h->free_own_graph();
    h->dev_beg = d_beg;
    h->dev_csr = d_csr;
    h->resident = true;
    h->device_graph = true;
    h->validated = false;
    h->alias_ready = false;
    return GW_OK;
}

extern "C" int gw_host_weights(gw_handle *h, uint32_t blk, const float *w)
{
    if (!h) return GW_ERR_ARG;
    if (blk >= h->nblocks) return h->fail(GW_ERR_ARG, "block %u out of range (%u blocks)", blk, h->nblocks);
    if (h->device_graph) return h->fail(GW_ERR_STATE, "the graph is on the device: use gw_device_weights");
    if (!w && h->eblocks[blk + 1] > h->eblocks[blk]) return h->fail(GW_ERR_ARG, "block %u weights missing", blk);
    h->host_w[blk] = w;
    bool all = true;
    for (uint32_t b = 0; b < h->nblocks; ++b) all &= h->host_w[b] != nullptr || h->eblocks[b + 1] == h->eblocks[b];
    h->weighted = all;
    h->resident = false;  // the next in-core run uploads the weights with the graph
    h->alias_ready = false;
    h->ooc_release();  // the out-of-core slots and alias tables follow the weights
    return GW_OK;
}

extern "C" int gw_device_weights(gw_handle *h, const float *d_w)
{
    if (!h) return GW_ERR_ARG;
    if (!h->device_graph) return h->fail(GW_ERR_STATE, "gw_device_weights needs a device graph (gw_device_graph)");
    if (!d_w && h->nedges) {
        h->weighted = false;
        h->dev_w = nullptr;
        return GW_OK;
    }
    cudaSetDevice(h->cfg.device);
    cudaFree(h->own_w);
    h->own_w = nullptr;
    h->dev_w = d_w;
    h->weighted = true;
    h->alias_ready = false;
    return GW_OK;
}

extern "C" int gw_cache_reset(gw_handle *h)
{
    if (!h) return GW_ERR_ARG;
    if (h->device_graph) return GW_OK;
    h->resident = false;
    h->ooc_invalidate(false);
    return GW_OK;
}

// ------------------------------------------------------------------ ABI: walkers

extern "C" int gw_init_walkers(gw_handle *h, uint32_t algo, uint32_t wps, uint64_t seed)
{
    return gw_init_walker_range(h, algo, wps, seed, 0, ~0ull);
}

extern "C" int gw_init_walker_range(gw_handle *h, uint32_t algo, uint32_t wps, uint64_t seed, uint64_t first,
                                    uint64_t count)
{
    if (!h) return GW_ERR_ARG;
    if (h->nblocks == 0) return h->fail(GW_ERR_STATE, "set the graph meta first");
    if (algo > GW_SOSR) return h->fail(GW_ERR_ARG, "unknown algorithm %u", algo);
    h->cfg.algorithm = algo;
    h->cfg.seed = seed;
    uint64_t n = 0;
    switch (h->cfg.init_mode) {
    case GW_INIT_PER_VERTEX:
        if (wps == 0) return h->fail(GW_ERR_ARG, "walkpersource must be positive");
        h->cfg.walkpersource = wps;
        n = (uint64_t)h->nverts * wps;
        break;
    case GW_INIT_SINGLE_SOURCE:
        if (h->nverts <= (algo == GW_SOSR ? 3u : 1u))
            return h->fail(GW_ERR_ARG, "single-source walks start at vertex 1 (and 3): graph too small");
        n = h->cfg.numwalks ? h->cfg.numwalks : (uint64_t)h->nverts * (wps ? wps : 1);
        break;
    default:
        n = h->cfg.numwalks ? h->cfg.numwalks : (uint64_t)h->nverts * (wps ? wps : 1);
        break;
    }
    if (n > 0xFFFFFFFFull) return h->fail(GW_ERR_ARG, "walker ids are 32-bit (wid_t); %llu walkers", (unsigned long long)n);
    if (n == 0) return h->fail(GW_ERR_ARG, "no walkers");
    if (first < n && count == ~0ull) count = n - first;  // to the end of the population
    if (first >= n || count == 0 || count > n - first)
        return h->fail(GW_ERR_ARG, "walker range [%llu, +%llu) outside the %llu walkers", (unsigned long long)first,
                       (unsigned long long)count, (unsigned long long)n);
    cudaSetDevice(h->cfg.device);
    h->walkers_ready = false;  // until the new population has its outputs
    h->nwalkers = count;
    h->wid_first = (uint32_t)first;
    h->numwalks_eff = (uint32_t)n;
    int st = h->ensure_outputs();
    if (st) {
        h->nwalkers = 0;  // what is left of the outputs is no population's
        return st;
    }
    h->walkers_ready = true;
    h->ooc_walkers_stale = true;
    return GW_OK;
}

extern "C" int gw_num_walkers(gw_handle *h, uint64_t *n)
{
    if (!h || !n) return GW_ERR_ARG;
    *n = h->walkers_ready ? h->nwalkers : 0;
    return GW_OK;
}

// ------------------------------------------------------------------ ABI: run

// The index of a resident CSR for walks that search by `search`.
// kTable: per vertex 16 bytes (first edge, degree, first bucket, the degree's
// reciprocal), which a step loads at once in place of two offsets and a
// division, and the membership tables (10 bytes per edge and up to 32 per
// vertex).  kLevels: the sample levels (0.13 bytes per edge).
gw_handle::IndexLayout gw_handle::index_layout(int search) const
{
    IndexLayout l{};
    if (search == kTable) {
        // buckets: 5/16 of an edge's and one more per vertex at most (table_buckets)
        l.buckets = nedges / 4 + nedges / 16 + nverts + 1;
        l.heads_hi = ((uint64_t)nverts * sizeof(uint4) + 255) & ~255ull;
        l.table = l.heads_hi + (nedges >= (1ull << 32) ? ((uint64_t)nverts * sizeof(uint32_t) + 255) & ~255ull : 0);
        l.bytes = l.table + l.buckets * 32;
    } else if (search == kLevels) {
        for (uint64_t m = nedges; l.nlevels < (uint32_t)kIdxLevels && m > 64; ++l.nlevels) {
            m = (m + 31) / 32;
            l.level[l.nlevels] = m;
            l.bytes += m * sizeof(uint32_t);
        }
    }
    return l;
}

// Memory for that index.  An index is worth having, not needed: a large one
// takes at most a quarter of what is free, and none is no error; after a refusal
// another attempt is made only where it has room.
bool gw_handle::reserve_index(int search)
{
    const IndexLayout l = index_layout(search);
    if (l.buckets >= (1ull << 32)) return false;  // bucket numbers are 32-bit
    if (l.bytes <= index_cap) return true;
    size_t free_bytes = 0, all_bytes = 0;
    if (l.bytes >= kSmallIndex || index_refused) {
        if (cudaMemGetInfo(&free_bytes, &all_bytes) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (l.bytes > (l.bytes >= kSmallIndex ? free_bytes / 4 : free_bytes)) {
            index_refused = true;
            return false;
        }
    }
    drop_index();
    index_refused = cudaMalloc(&d_index, l.bytes) != cudaSuccess;
    if (index_refused) {
        cudaGetLastError();
        d_index = nullptr;
        return false;
    }
    index_cap = l.bytes;
    return true;
}

void gw_handle::drop_index()
{
    cudaFree(d_index);
    d_index = nullptr;
    index_cap = 0;
    index_search = kQuarter;
}

// The search a run is worth an index for.  Tables cost a pass of atomics over
// the edges (7.6 M edges 0.24 ms, 64 M 2.8 ms) and save part of each step, so
// they are built when the steps of the runs on this graph so far and of this one
// come to so many an edge:
// - 1 where graph and tables fit the L2 (a first run of 27 steps an edge on 1.8 M
//   edges 1.66 ms, 2.81 without; of 2.8 on 7.6 M 1.44 / 1.77; of 0.14 0.43 / 0.22),
// - 6 past it (a first run of 2.6 on 64 M edges 6.0 / 4.5 ms, on 31 M 2.77 / 2.20,
//   of 5.2 on 16 M with paths 2.34 / 1.89; the run after it 3.3 / 4.3, 1.53 / 2.20
//   and 1.45 / 1.89), 1 for SOPR and SOSR, whose steps take more trials (128 M
//   edges, 0.8: 30.4 / 27.5 ms, then 24.3 / 27.2).
// Steps that always accept search nothing.
int gw_handle::wanted_search(bool sopr, bool sure) const
{
    if (cfg.launch_mode == GW_LAUNCH_PER_HOP || sure) return kQuarter;
    const double steps = index_steps + run_steps();
    if (steps >= (double)nedges * (sopr || 14 * nedges <= kL2Bytes ? 1.0 : 6.0)) return kTable;
    return wants_levels(nwalkers, nedges, sopr, sure, num_sms) ? kLevels : kQuarter;
}

// Steps of a run at most: every walker to its last hop, or to its mean by the
// termination draws.  Fewer walkers than lanes take as long as many.
double gw_handle::run_steps() const
{
    double hops = cfg.maxhops;
    if (cfg.term_prob > 0.f) hops = std::min(hops, 1.0 / (double)cfg.term_prob);
    return (double)std::max(nwalkers, walk_lanes(num_sms)) * hops;
}

// Checks the resident CSR, and builds its index for walks that search by
// `search`, where it has memory.
int gw_handle::validate_graph(cudaStream_t s, int search)
{
    int st;
    index_search = kQuarter;
    // the memory of a small index is taken with the first check, so that the
    // run that builds it, maybe a short one, does not wait for an allocation
    // (first: a reservation that fails leaves nothing of the one before)
    if (search != kTable && !index_refused && index_layout(kTable).bytes < kSmallIndex) reserve_index(kTable);
    if (!reserve_index(search)) search = kQuarter;
    const IndexLayout l = index_layout(search);
    const bool index = search == kTable;
    CsrCheck check{};
    check.beg = dev_beg;
    check.csr = dev_csr;
    check.nverts = nverts;
    check.nedges = nedges;
    check.err = d_err;
    check.sum = device_graph ? d_ctr + kCtrGraphSum : nullptr;
    if (index) {
        d_verts = reinterpret_cast<uint4 *>(d_index);
        d_heads_hi = l.table > l.heads_hi ? reinterpret_cast<uint32_t *>(d_index + l.heads_hi) : nullptr;
        d_table = reinterpret_cast<uint32_t *>(d_index + l.table);
        check.verts = d_verts;
        check.heads_hi = d_heads_hi;
        check.nbuckets = d_ctr;
    }
    uint64_t ends[2] = {1, 0};
    const size_t ctr_bytes = sizeof(unsigned long long) * kCtrWords;
    if ((st = cuda(cudaMemsetAsync(d_ctr, 0, ctr_bytes, s), "memset")) ||
        (st = cuda(launch_validate_csr(check, num_sms, s), "validate")) ||
        (st = cuda(cudaMemcpyAsync(h_ctr, d_ctr, ctr_bytes, cudaMemcpyDeviceToHost, s), "buckets D2H")) ||
        (st = cuda(cudaMemcpyAsync(&ends[0], dev_beg, sizeof(uint64_t), cudaMemcpyDeviceToHost, s), "beg[0]")) ||
        (st = cuda(cudaMemcpyAsync(&ends[1], dev_beg + nverts, sizeof(uint64_t), cudaMemcpyDeviceToHost, s), "beg[V]")) ||
        (st = cuda(cudaStreamSynchronize(s), "validate")))
        return st;
    if ((uint32_t)h_ctr[kCtrCount] != 0) {
        h_ctr[kCtrCount] = 0;
        return fail(GW_ERR_GRAPH, "graph failed validation: offsets not monotone or a neighbour id >= %u", nverts);
    }
    if (ends[0] != 0 || ends[1] != nedges)
        return fail(GW_ERR_GRAPH, "graph offsets must run from 0 to nedges (%llu..%llu)", (unsigned long long)ends[0],
                    (unsigned long long)ends[1]);
    if (index) {
        if ((st = cuda(cudaMemsetAsync(d_table, 0xFF, h_ctr[0] * 32, s), "memset")) ||
            (st = cuda(launch_build_table(dev_beg, d_verts, nverts, dev_csr, nedges, d_table, num_sms, s),
                       "membership tables")))
            return st;
    }
    const uint32_t *src = dev_csr;
    uint32_t *dst = reinterpret_cast<uint32_t *>(d_index);
    for (uint32_t i = 0; i < l.nlevels; ++i) {
        if ((st = cuda(launch_sample_level(src, l.level[i], dst, num_sms, s), "sample level"))) return st;
        levels.lvl[i] = src = dst;
        dst += l.level[i];
    }
    levels.n = l.nlevels;
    index_search = search;
    index_sum = h_ctr[kCtrGraphSum];
    validated = true;
    return GW_OK;
}

// Alias tables of every vertex from the resident weights: 8 bytes per edge
// kept, 16 bytes per edge of scratch for the construction.
int gw_handle::build_alias(cudaStream_t s)
{
    int st;
    if (!d_alias && (st = dev_alloc(d_alias, (nedges ? nedges : 1) * sizeof(AliasEntry), "alias tables")))
        return st;
    double *pd = nullptr;
    uint32_t *q = nullptr;
    if ((st = dev_alloc(pd, (nedges ? nedges : 1) * sizeof(double), "alias scratch"))) return st;
    if ((st = dev_alloc(q, (2 * (nedges ? nedges : 1) + nverts + 2) * sizeof(uint32_t), "alias scratch"))) {
        cudaFree(pd);
        return st;
    }
    st = cuda(cudaMemsetAsync(d_err, 0, sizeof(uint32_t), s), "memset");
    if (!st) st = cuda(launch_build_alias(dev_beg, dev_w, nverts, pd, q, q + nedges,
                                                      q + 2 * (nedges ? nedges : 1), d_alias, d_err, num_sms, s),
                       "alias build");
    if (!st) st = cuda(cudaMemcpyAsync(h_ctr + kCtrCount, d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, s), "D2H");
    if (!st) st = cuda(cudaStreamSynchronize(s), "alias build");
    cudaFree(pd);
    cudaFree(q);
    if (st) return st;
    if ((uint32_t)h_ctr[kCtrCount] != 0) {
        h_ctr[kCtrCount] = 0;
        return fail(GW_ERR_GRAPH, "edge weights must be positive finite numbers");
    }
    alias_ready = true;
    return GW_OK;
}

int gw_handle::run_incore(gw_stats *stats)
{
    int st;
    cudaStream_t s = s_compute;
    uint64_t h2d = 0;
    if ((st = cuda(cudaEventRecord(ev_start, s), "event"))) return st;
    if (!resident) {
        if ((st = upload_whole_graph(s, &h2d))) return st;
    }
    StepConsts consts;
    consts_from_config(cfg, consts);
    const bool sopr = cfg.algorithm != GW_NODE2VEC;
    const bool sure = sure_steps(sopr, consts);
    if (!validated) index_steps = 0;
    const int wanted = wanted_search(sopr, sure);
    const bool unchecked = !validated || (wanted > index_search && reserve_index(wanted));
    if (unchecked && (st = validate_graph(s, wanted))) return st;
    if (weighted) {
        if (cfg.algorithm != GW_NODE2VEC)
            return fail(GW_ERR_ARG, "weighted walks are Node2vec walks (algorithm %u given)", cfg.algorithm);
        if (!alias_ready && (st = build_alias(s))) return st;
    }
    IncoreArgs a{};
    a.c = consts;
    a.init.mode = cfg.init_mode;
    a.init.algo = cfg.algorithm;
    a.init.wps = cfg.walkpersource;
    a.init.numwalks = numwalks_eff;
    a.init.nverts = nverts;
    a.init.key0 = (uint32_t)cfg.seed;
    a.init.key1 = (uint32_t)(cfg.seed >> 32);
    a.beg = dev_beg;
    a.csr = dev_csr;
    a.nedges = nedges;
    // A borrowed CSR is summed before its index is read, so a run of few steps
    // leaves the index alone and reads the CSR as it is
    const bool indexed = !device_graph || unchecked || (!sure && 8.0 * run_steps() >= (double)nedges);
    a.search = indexed ? index_search : kQuarter;
    if (a.search == kLevels && !wants_levels(nwalkers, nedges, sopr, sure, num_sms)) a.search = kQuarter;
    a.levels = levels;
    a.verts = d_verts;
    a.heads_hi = d_heads_hi;
    a.table = d_table;
    a.nverts = nverts;
    a.nwalkers = (uint32_t)nwalkers;
    a.wid_base = wid_first;
    a.out_base = wid_first;
    a.paths = (cfg.record_paths == GW_PATHS_FULL) ? d_paths : nullptr;
    a.stride = cfg.maxhops + 1;
    a.lens = d_lens;
    a.hashes = d_hashes;
    a.ctr = d_ctr;
    a.err = d_err;
    const bool coop = !weighted && needs_coop(cfg.algorithm, a.c);
    a.alias = weighted ? reinterpret_cast<const uint2 *>(d_alias) : nullptr;
    if (cfg.launch_mode == GW_LAUNCH_PER_HOP) {
        // ---- the plain form: one launch per hop, walker state in memory
        if (weighted) return fail(GW_ERR_ARG, "one launch per hop runs unweighted walks only");
        HopState hs{};
        const uint64_t n = nwalkers;
        int rc = GW_OK;
        if ((rc = dev_alloc(hs.prev, n * 4, "hop state")) || (rc = dev_alloc(hs.cur, n * 4, "hop state")) ||
            (rc = dev_alloc(hs.hop, n * 4, "hop state")) || (rc = dev_alloc(hs.hash, n * 8, "hop state"))) {
            cudaFree(hs.prev);
            cudaFree(hs.cur);
            cudaFree(hs.hop);
            cudaFree(hs.hash);
            return rc;
        }
        const uint32_t rounds = cfg.maxhops ? cfg.maxhops : 1;
        if (!(rc = cuda(cudaMemsetAsync(d_ctr, 0, sizeof(unsigned long long) * kCtrWords, s), "memset")) &&
            !(rc = cuda(cudaEventRecord(ev_kernel0, s), "event"))) {
            for (uint32_t k = 0; k < rounds && !rc; ++k) rc = cuda(launch_walk_hop(a, hs, sopr, k, num_sms, s), "hop launch");
        }
        if (!rc && !(rc = cuda(cudaEventRecord(ev_kernel1, s), "event")) &&
            !(rc = cuda(cudaMemcpyAsync(h_ctr, d_ctr, sizeof(unsigned long long) * kCtrWords,
                                        cudaMemcpyDeviceToHost, s),
                        "counters D2H")) &&
            !(rc = cuda(cudaEventRecord(ev_stop, s), "event")))
            rc = cuda(cudaStreamSynchronize(s), "walk");
        cudaStreamSynchronize(s);
        cudaFree(hs.prev);
        cudaFree(hs.cur);
        cudaFree(hs.hop);
        cudaFree(hs.hash);
        if (rc) return rc;
        last_hash_sum = h_ctr[kCtrHashSum];
        last_steps = h_ctr[kCtrSteps];
        if (stats) {
            memset(stats, 0, sizeof(*stats));
            stats->steps = h_ctr[kCtrSteps];
            stats->trials = h_ctr[kCtrTrials];
            stats->walkers = h_ctr[kCtrDone];
            stats->h2d_bytes = h2d;
            stats->d2h_bytes = sizeof(unsigned long long) * kCtrCount + sizeof(uint32_t);
            stats->block_loads = h2d ? nblocks : 0;
            stats->iterations = rounds;
            stats->launches = rounds;
            stats->kernel_variant = 0xFFFFFFFFu;
            cudaEventElapsedTime(&stats->kernel_ms, ev_kernel0, ev_kernel1);
            cudaEventElapsedTime(&stats->total_ms, ev_start, ev_stop);
        }
        const uint32_t errw = (uint32_t)h_ctr[kCtrCount];
        if (errw) return fail(GW_ERR_DEVICE, "walk kernel error word 0x%x", errw);
        if (h_ctr[kCtrDone] != nwalkers)
            return fail(GW_ERR_DEVICE, "per-hop walk finished %llu of %llu walkers", (unsigned long long)h_ctr[kCtrDone],
                        (unsigned long long)nwalkers);
        return GW_OK;
    }
    const IncorePlan plan = incore_plan(nwalkers, nedges, sopr, a.paths != nullptr, coop, weighted, a.search, sure,
                                        (int)cfg.blockpergrid, num_sms);
    a.slots = plan.slots;
    a.chunk = plan.chunk;
    a.claims_end = plan.one_wave ? 0u : a.nwalkers;
    const size_t ctr_bytes = sizeof(unsigned long long) * (kCtrCount + 1);  // with the error word
    // A borrowed CSR may have been written since its index was built: its
    // contents are summed beside the walk, which is done again if they are not
    // the same.  (Records, tables and levels of another graph of these sizes
    // lead no read out of range.)  A walk that fills the device leaves the sum no
    // room until its end, so there the sum goes first.  64 M edges: 65 us of a
    // walk of 3.2 ms, and of one of 0.15 ms that leaves room.
    const bool summed = device_graph && a.search != kQuarter && !unchecked;
    const bool sum_first = nwalkers >= walk_lanes(num_sms);
    auto sum_graph = [&]() {
        CsrCheck check{};
        check.beg = dev_beg;
        check.csr = dev_csr;
        check.nverts = nverts;
        check.nedges = nedges;
        check.sum = d_ctr + kCtrGraphSum;
        check.err = reinterpret_cast<uint32_t *>(check.sum + 1);
        int e;
        // behind what the caller put on the compute stream before this run
        if ((e = cuda(cudaStreamWaitEvent(s_copy, ev_start, 0), "graph sum")) ||
            (e = cuda(cudaMemsetAsync(check.sum, 0, 2 * sizeof(unsigned long long), s_copy), "memset")) ||
            (e = cuda(launch_validate_csr(check, num_sms, s_copy), "graph sum")))
            return e;
        return cuda(cudaMemcpyAsync(h_ctr + kCtrGraphSum, check.sum, sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, s_copy),
                    "graph sum");
    };
    if (summed && sum_first && (st = sum_graph())) return st;
    if ((st = cuda(cudaMemsetAsync(d_ctr, 0, ctr_bytes, s), "memset")) ||
        (st = cuda(cudaEventRecord(ev_kernel0, s), "event")) ||
        (st = cuda(launch_walk_incore(a, sopr, coop, plan.grid, s), "walk kernel launch")) ||
        (st = cuda(cudaEventRecord(ev_kernel1, s), "event")) ||
        (summed && !sum_first && (st = sum_graph())) ||
        (st = cuda(cudaMemcpyAsync(h_ctr, d_ctr, ctr_bytes, cudaMemcpyDeviceToHost, s), "counters D2H")) ||
        (st = cuda(cudaEventRecord(ev_stop, s), "event")) || (st = cuda(cudaStreamSynchronize(s), "walk")) ||
        (summed && (st = cuda(cudaStreamSynchronize(s_copy), "graph sum"))))
        return st;
    if (summed && h_ctr[kCtrGraphSum] != index_sum) {  // written: checked and indexed anew, then walked
        h_ctr[kCtrCount] = 0;
        validated = false;
        alias_ready = false;
        return run_incore(stats);
    }
    last_hash_sum = h_ctr[kCtrHashSum];
    last_steps = h_ctr[kCtrSteps];
    index_steps += run_steps();
    const uint32_t errw = (uint32_t)h_ctr[kCtrCount];
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->steps = h_ctr[kCtrSteps];
        stats->trials = h_ctr[kCtrTrials];
        stats->walkers = h_ctr[kCtrDone];
        stats->h2d_bytes = h2d;
        stats->d2h_bytes = sizeof(unsigned long long) * kCtrCount + sizeof(uint32_t);
        stats->block_loads = h2d ? nblocks : 0;
        stats->iterations = 1;
        stats->launches = 1;
        stats->kernel_variant = plan.ctas_per_sm;
        stats->walker_chunk = a.chunk;
        stats->coop_small_steps = h_ctr[kCtrCoopSmall];
        stats->coop_small_attempts = h_ctr[kCtrCoopSmallAtt];
        stats->coop_large_steps = h_ctr[kCtrCoopLarge];
        stats->coop_large_attempts = h_ctr[kCtrCoopLargeAtt];
        cudaEventElapsedTime(&stats->kernel_ms, ev_kernel0, ev_kernel1);
        cudaEventElapsedTime(&stats->total_ms, ev_start, ev_stop);
    }
    if (errw) return fail(GW_ERR_DEVICE, "walk kernel error word 0x%x (graph ids out of range)", errw);
    if (h_ctr[kCtrDone] != nwalkers)
        return fail(GW_ERR_DEVICE, "walk kernel finished %llu of %llu walkers", (unsigned long long)h_ctr[kCtrDone],
                    (unsigned long long)nwalkers);
    return GW_OK;
}

extern "C" int gw_run(gw_handle *h, uint32_t policy, gw_stats *stats)
{
    if (!h) return GW_ERR_ARG;
    if (policy > GW_POLICY_SA) return h->fail(GW_ERR_ARG, "unknown policy %u", policy);
    if (h->nblocks == 0) return h->fail(GW_ERR_STATE, "no graph");
    if (!h->walkers_ready) return h->fail(GW_ERR_STATE, "call gw_init_walkers first");
    cudaSetDevice(h->cfg.device);
    InCall in_call(h);
    int st = h->ensure_outputs();
    if (st) return st;
    const bool incore = h->device_graph || h->graph_bytes() <= h->cfg.cache_size;
    if (incore) {
        if (!h->resident && !h->host_graph_complete())
            return h->fail(GW_ERR_STATE, "graph blocks missing: call gw_host_block for every block");
        return h->run_incore(stats);
    }
    if (!h->host_graph_complete())
        return h->fail(GW_ERR_STATE, "graph blocks missing: call gw_host_block for every block");
    return h->run_ooc(policy, stats);
}

// ------------------------------------------------------------------ ABI: results

namespace {
// Zero every path-row entry past its walk's length (the kernels write a row
// only up to the length; the rest holds whatever the buffer held before).
__global__ void k_zero_tails(uint32_t *rows, const uint32_t *lens, uint64_t n, uint32_t stride)
{
    const uint64_t total = n * stride;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i / stride;
        if (i - row * stride >= __ldg(lens + row)) rows[i] = 0u;
    }
}
}  // namespace

// Pages of a large pageable destination, brought in by several threads before
// the copy: a device-to-host copy that meets fresh pages takes each fault on
// its one thread (64 MB: 31 ms, 3.2 ms into resident pages).  A destination
// that is pinned, or whose pages are there already, is left alone.
static void touch_pages(void *dst, uint64_t bytes)
{
    constexpr uint64_t kPage = 4096, kLeast = 4ull << 20;
    cudaPointerAttributes at{};
    if (!dst || bytes < kLeast) return;
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (at.type != cudaMemoryTypeUnregistered) return;
    char *const p = (char *)dst;
    uint64_t there = 0;
    for (uint64_t k = 0; k < 16; ++k) {
        unsigned char in = 0;
        char *q = (char *)((uintptr_t)(p + (bytes - 1) / 16 * k) & ~(uintptr_t)(kPage - 1));
        there += mincore(q, kPage, &in) == 0 && (in & 1u);
    }
    if (there == 16) return;
    const unsigned n = std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
    const uint64_t part = (bytes / n + kPage - 1) / kPage * kPage;
    auto touch = [=](uint64_t lo) {
        for (uint64_t o = lo; o < std::min(lo + part, bytes); o += kPage) ((volatile char *)p)[o] = 0;
    };
    std::vector<std::thread> pool;
    try {
        pool.reserve(n);
        for (unsigned k = 1; k < n; ++k) pool.emplace_back(touch, k * part);
    } catch (...) {  // fewer threads: the copy brings in the rest
    }
    touch(0);
    for (auto &t : pool) t.join();
}

extern "C" int gw_path_lengths(gw_handle *h, uint64_t first, uint64_t n, uint32_t *lens)
{
    if (!h || !lens) return GW_ERR_ARG;
    if (!h->walkers_ready || !h->d_lens) return h->fail(GW_ERR_STATE, "no walk has run");
    if (first + n > h->nwalkers) return h->fail(GW_ERR_ARG, "walker range out of bounds");
    cudaSetDevice(h->cfg.device);
    touch_pages(lens, n * sizeof(uint32_t));
    return h->cuda(cudaMemcpy(lens, h->d_lens + first, n * sizeof(uint32_t), cudaMemcpyDeviceToHost), "lengths D2H");
}

extern "C" int gw_get_paths(gw_handle *h, uint64_t first, uint64_t n, uint32_t *out, uint32_t *lens)
{
    if (!h) return GW_ERR_ARG;
    if (h->cfg.record_paths != GW_PATHS_FULL || !h->d_paths)
        return h->fail(GW_ERR_STATE, "paths were not recorded (record_paths = GW_PATHS_FULL)");
    if (first + n > h->nwalkers) return h->fail(GW_ERR_ARG, "walker range out of bounds");
    cudaSetDevice(h->cfg.device);
    int st;
    if (out && n) {
        // rows end with zeros past the walk's length: padded on the device,
        // then one copy
        k_zero_tails<<<h->num_sms * 8, 256, 0, h->s_compute>>>(h->d_paths + first * h->path_stride, h->d_lens + first,
                                                              n, h->path_stride);
        if ((st = h->cuda(cudaGetLastError(), "path padding"))) return st;
        touch_pages(out, n * h->path_stride * sizeof(uint32_t));
        if ((st = h->cuda(cudaMemcpyAsync(out, h->d_paths + first * h->path_stride,
                                          n * h->path_stride * sizeof(uint32_t), cudaMemcpyDeviceToHost, h->s_compute),
                          "paths D2H")))
            return st;
    }
    if (lens && n) {
        touch_pages(lens, n * sizeof(uint32_t));
        if ((st = h->cuda(cudaMemcpyAsync(lens, h->d_lens + first, n * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                          h->s_compute),
                          "lengths D2H")))
            return st;
    }
    return h->cuda(cudaStreamSynchronize(h->s_compute), "paths D2H");
}

extern "C" int gw_path_hashes(gw_handle *h, uint64_t first, uint64_t n, uint64_t *out)
{
    if (!h || !out) return GW_ERR_ARG;
    if (first + n > h->nwalkers) return h->fail(GW_ERR_ARG, "walker range out of bounds");
    cudaSetDevice(h->cfg.device);
    touch_pages(out, n * sizeof(uint64_t));
    return h->cuda(cudaMemcpy(out, h->d_hashes + first, n * sizeof(uint64_t), cudaMemcpyDeviceToHost),
                   "hashes D2H");
}

extern "C" int gw_checksum(gw_handle *h, uint64_t *hash_sum, uint64_t *steps)
{
    if (!h) return GW_ERR_ARG;
    if (hash_sum) *hash_sum = h->last_hash_sum;
    if (steps) *steps = h->last_steps;
    return GW_OK;
}
