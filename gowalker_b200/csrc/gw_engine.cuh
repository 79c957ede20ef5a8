// The engine handle (internal).  One per host thread; owns its device memory
// and streams.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>
#include "gw_kernels.cuh"
#include "gw_weighted.cuh"
#include "../../include/gowalker.h"

namespace gw {
struct OocState;
// Step constants of a configuration (fp32 thresholds computed as the
// reference writes them, engine/engine.hpp:169-172).
void consts_from_config(const gw_config &c, StepConsts &k);
}

struct gw_handle {
    gw_config cfg{};
    int num_sms = 0;
    cudaStream_t s_compute = nullptr;  // step kernels, bucketing, scheduler
    cudaStream_t s_copy = nullptr;     // block copies host -> device slots
    cudaEvent_t ev_start = nullptr, ev_kernel0 = nullptr, ev_kernel1 = nullptr, ev_stop = nullptr;
    std::string err;

    // graph (graph_block, engine/cache.hpp:144-193)
    uint32_t nverts = 0;
    uint64_t nedges = 0;
    uint32_t nblocks = 0;
    std::vector<uint32_t> vblocks;
    std::vector<uint64_t> eblocks;
    std::vector<const uint64_t *> host_beg;  // borrowed host blocks
    std::vector<const uint32_t *> host_csr;

    // whole graph on the device (in-core)
    const uint64_t *dev_beg = nullptr;
    const uint32_t *dev_csr = nullptr;
    uint64_t *own_beg = nullptr;  // offsets, with the neighbours behind them or, small ones, apart
    uint32_t *own_csr = nullptr, *own_csr_apart = nullptr;
    bool resident = false;
    bool device_graph = false;
    bool validated = false;
    // index of the resident CSR, built by the run that wants it: one allocation,
    // the parts of tables on 256-byte boundaries
    static constexpr uint64_t kSmallIndex = 256ull << 20;
    char *d_index = nullptr;
    uint64_t index_cap = 0;
    int index_search = gw::kQuarter;  // what is built: kTable, kLevels or none
    bool index_refused = false;       // the last attempt had no memory, or the index gave way
    double index_steps = 0.0;         // run_steps() of the runs on this graph so far
    uint4 *d_verts = nullptr;
    uint32_t *d_heads_hi = nullptr;  // null: every offset is below 2^32
    uint32_t *d_table = nullptr;
    gw::Levels levels{};
    uint64_t index_sum = 0;  // borrowed CSR: sum of the contents the index was built from

    // edge weights (weighted Node2vec, in-core): per host block, or resident
    std::vector<const float *> host_w;
    const float *dev_w = nullptr;
    float *own_w = nullptr;
    bool weighted = false;
    gw::AliasEntry *d_alias = nullptr;  // alias tables, rebuilt when the graph or weights change
    bool alias_ready = false;

    // walker population
    uint64_t nwalkers = 0;      // walkers of the population: ids wid_first .. wid_first + nwalkers - 1
    uint32_t wid_first = 0;     // first walker id (a shard of the whole population)
    uint32_t numwalks_eff = 0;  // walkers of the whole population (SOSR's single-source split uses it)
    bool walkers_ready = false;
    bool ooc_walkers_stale = true;

    // per-walker outputs
    uint32_t *d_paths = nullptr;
    uint64_t *d_hashes = nullptr;  // one allocation: hashes, then lengths
    uint32_t *d_lens = nullptr;
    uint64_t cap_walkers = 0;
    uint64_t cap_path_words = 0;
    uint64_t cap_path_walkers = 0;
    uint32_t path_stride = 0;

    // counters
    unsigned long long *d_ctr = nullptr;  // kCtrWords: counters, error word, graph sum
    uint32_t *d_err = nullptr;            // that word
    unsigned long long *h_ctr = nullptr;  // pinned, the same
    uint64_t last_hash_sum = 0;
    uint64_t last_steps = 0;

    // out-of-core state (gw_ooc.cu)
    gw::OocState *ooc = nullptr;

    int fail(int status, const char *fmt, ...);
    int cuda(cudaError_t e, const char *what);
    bool in_call = false;  // a run of this engine, which may read its index
    // Device memory (device_malloc): all that a handle allocates but its index,
    // which gives way.
    int dev_alloc(void **p, uint64_t bytes, const char *what);
    template <class T>
    int dev_alloc(T *&p, uint64_t bytes, const char *what)
    {
        return dev_alloc((void **)&p, bytes, what);
    }
    int init_device();
    void release();
    uint64_t graph_bytes() const;
    void free_own_graph();
    bool host_graph_complete() const;
    int upload_whole_graph(cudaStream_t s, uint64_t *h2d);
    int ensure_outputs();
    struct IndexLayout {
        uint64_t bytes, buckets, heads_hi, table;  // kTable: offsets behind the records
        uint64_t level[gw::kIdxLevels];            // kLevels: entries
        uint32_t nlevels;
    };
    IndexLayout index_layout(int search) const;
    bool reserve_index(int search);
    void drop_index();
    double run_steps() const;
    int wanted_search(bool sopr, bool sure) const;
    int validate_graph(cudaStream_t s, int search);
    int build_alias(cudaStream_t s);
    int run_incore(gw_stats *stats);
    int run_ooc(uint32_t policy, gw_stats *stats);
    void ooc_release();
    void ooc_invalidate(bool blocks_changed);
};
