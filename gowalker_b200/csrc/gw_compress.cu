// Compressed neighbour lists of out-of-core blocks: host encoder, device decoder.
// The format is described in gw_compress.cuh.
#include <algorithm>
#include <cstring>
#include <thread>
#include <vector>
#include "gw_compress.cuh"
#include "gw_kernels.cuh"

namespace gw {

static inline uint32_t zigzag(uint32_t d) { return (d << 1) ^ (uint32_t)((int32_t)d >> 31); }
static inline uint32_t bit_length(uint32_t x) { return x ? 32u - (uint32_t)__builtin_clz(x) : 0u; }

// Code byte of the chunk ids[0, k): the deltas as they are when that is
// narrower (a sorted list: one bit less; at most 31 bits then), else
// zigzag-coded -- an OR has the same bit length as the maximum -- and the
// first id in as few bytes as hold it.
static inline uint32_t chunk_code(const uint32_t *ids, uint32_t k)
{
    uint32_t mz = 0, mr = 0;
    for (uint32_t i = 1; i < k; ++i) {
        mz |= zigzag(ids[i] - ids[i - 1]);
        mr |= ids[i] - ids[i - 1];
    }
    const uint32_t c = bit_length(mr) < bit_length(mz) ? 32u + bit_length(mr) : bit_length(mz);
    const uint32_t fb = std::max(1u, (bit_length(ids[0]) + 7u) / 8u);
    return c | ((fb - 1u) << 6);
}

// Bytes of a vertex's chunks; with `group` non-null, also the byte offset
// (from the vertex's first chunk) of every 32nd chunk.
static uint64_t vertex_bytes(const uint32_t *ids, uint64_t d, uint64_t *group)
{
    uint64_t s = 0, c = 0;
    for (uint64_t j = 0; j < d; j += kChunkIds, ++c) {
        if (group && c % kChunkIds == 0) group[c / kChunkIds] = s;
        const uint32_t k = (uint32_t)std::min<uint64_t>(kChunkIds, d - j);
        s += chunk_bytes(chunk_code(ids + j, k), k);
    }
    return s;
}

static inline uint64_t nchunks(uint64_t d) { return (d + kChunkIds - 1) / kChunkIds; }
static inline uint64_t ngroups(uint64_t d) { return nchunks(d) > kChunkIds ? (nchunks(d) + kChunkIds - 1) / kChunkIds : 0; }

static void encode_vertex(const uint32_t *ids, uint64_t d, uint8_t *p)
{
    for (uint64_t j = 0; j < d; j += kChunkIds) {
        const uint32_t k = (uint32_t)std::min<uint64_t>(kChunkIds, d - j);
        const uint32_t *c = ids + j;
        const uint32_t code = chunk_code(c, k), w = chunk_width(code);
        const bool plain = chunk_plain(code);
        *p++ = (uint8_t)code;
        for (uint32_t b = 0; b < chunk_first_bytes(code); ++b) *p++ = (uint8_t)(c[0] >> (8 * b));
        uint64_t acc = 0;
        uint32_t nbits = 0;
        for (uint32_t i = 1; i < k; ++i) {
            const uint32_t dl = c[i] - c[i - 1];
            acc |= (uint64_t)(plain ? dl : zigzag(dl)) << nbits;
            nbits += w;
            while (nbits >= 8) {
                *p++ = (uint8_t)acc;
                acc >>= 8;
                nbits -= 8;
            }
        }
        if (nbits) *p++ = (uint8_t)acc;
    }
}

bool compress_block(const uint64_t *beg, const uint32_t *csr, uint32_t nv, uint64_t e0, uint64_t e1,
                    unsigned threads, CompressedBlock &out, std::string &why)
{
    if (beg[0] != e0 || beg[nv] != e1) {
        why = "block offsets do not start and end at the block's first and last edge";
        return false;
    }
    for (uint32_t v = 0; v < nv; ++v)
        if (beg[v + 1] < beg[v]) {
            why = "block offsets are not non-decreasing";
            return false;
        }
    threads = std::max(1u, std::min(threads, 64u));
    // vertex ranges of about equal edge count
    std::vector<uint32_t> cut(threads + 1, nv);
    cut[0] = 0;
    for (unsigned t = 1; t < threads; ++t) {
        const uint64_t target = e0 + (e1 - e0) * t / threads;
        cut[t] = (uint32_t)(std::lower_bound(beg, beg + nv, target) - beg);
        cut[t] = std::max(cut[t], cut[t - 1]);
    }
    std::vector<uint64_t> off(nv + 1, 0), gstart(nv + 1, 0);
    for (uint32_t v = 0; v < nv; ++v) gstart[v + 1] = gstart[v] + ngroups(beg[v + 1] - beg[v]);
    const uint64_t nsplit = gstart[nv];
    std::vector<uint64_t> gofs(nsplit);  // byte offset of each group, from its vertex's first chunk
    auto run = [&](auto &&fn) {
        std::vector<std::thread> pool;
        for (unsigned t = 0; t < threads; ++t) pool.emplace_back(fn, cut[t], cut[t + 1]);
        for (auto &th : pool) th.join();
    };
    run([&](uint32_t a, uint32_t b) {
        for (uint32_t v = a; v < b; ++v) {
            const uint64_t d = beg[v + 1] - beg[v];
            off[v + 1] = vertex_bytes(csr + (beg[v] - e0), d, ngroups(d) ? gofs.data() + gstart[v] : nullptr);
        }
    });
    for (uint32_t v = 0; v < nv; ++v) off[v + 1] += off[v];
    const uint64_t payload = off[nv];
    if (payload >= (1ull << 32) || nsplit >= (1ull << 30)) {
        why = "block too large to compress (payload of 4 GB or more)";
        return false;
    }
    out.split_off = ((uint64_t)(nv + 1) * 4 + 15) & ~15ull;
    out.nsplit = (uint32_t)nsplit;
    out.payload_off = (out.split_off + nsplit * 12 + 15) & ~15ull;
    out.payload_bytes = payload;
    out.bytes = (out.payload_off + payload + 8 + 15) & ~15ull;
    if (cudaHostAlloc((void **)&out.host, out.bytes, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        out.host = nullptr;
        why = "pinned allocation for a compressed block failed";
        return false;
    }
    memset(out.host, 0, out.payload_off);
    memset(out.host + out.payload_off + payload, 0, out.bytes - out.payload_off - payload);
    uint32_t *voff = (uint32_t *)out.host;
    for (uint32_t v = 0; v <= nv; ++v) voff[v] = (uint32_t)off[v];
    uint32_t *split = (uint32_t *)(out.host + out.split_off);
    for (uint32_t v = 0; v < nv; ++v)
        for (uint64_t g = gstart[v]; g < gstart[v + 1]; ++g) {
            split[3 * g] = v;
            split[3 * g + 1] = (uint32_t)((g - gstart[v]) * kChunkIds);
            split[3 * g + 2] = (uint32_t)(off[v] + gofs[g]);
        }
    uint8_t *pay = out.host + out.payload_off;
    run([&](uint32_t a, uint32_t b) {
        for (uint32_t v = a; v < b; ++v) encode_vertex(csr + (beg[v] - e0), beg[v + 1] - beg[v], pay + off[v]);
    });
    // pieces of about equal payload, cut at multiples of 32 vertices
    const uint32_t pieces = (uint32_t)std::clamp<uint64_t>(payload / kPieceBytes, 1, kPieces);
    out.piece_v[0] = 0;
    for (uint32_t k = pieces; k <= kPieces; ++k) out.piece_v[k] = nv;
    for (uint32_t k = 1; k < pieces; ++k) {
        const uint64_t target = payload * k / pieces;
        uint32_t v = (uint32_t)(std::lower_bound(off.begin(), off.begin() + nv, target) - off.begin());
        v &= ~31u;
        out.piece_v[k] = std::max(v, out.piece_v[k - 1]);
    }
    for (uint32_t k = 0; k <= kPieces; ++k) {
        out.piece_g[k] = (uint32_t)gstart[out.piece_v[k]];
        out.piece_e[k] = beg[out.piece_v[k]] - e0;
    }
    return true;
}

// Up to kBatchChunks chunks, `left` ids, from byte `pos` of the payload, decoded
// by the warp from its shared-memory window of the payload words
// [base, base + kWindowWords): lane 0 takes a chunk's first id, lane i < 32 delta
// i (its bits read straight from the window), and a warp prefix sum (mod 2^32)
// rebuilds the ids.  `end` is the byte past the chunks this task may read; a
// chunk reaching past it is malformed.  A chunk's place follows from the width
// byte of the one before, but nothing else does: four at a time take 0.1 us each,
// one by one 0.35.
constexpr uint32_t kBatchChunks = 4;
__device__ __forceinline__ uint64_t decode_chunks_sm(const uint32_t *sm, uint64_t base, uint64_t pos, uint64_t end,
                                                     uint64_t left, uint32_t lane, uint32_t *__restrict__ row,
                                                     uint32_t nverts, bool &bad_id, bool &bad)
{
    uint32_t x[kBatchChunks], ids[kBatchChunks];
#pragma unroll
    for (uint32_t i = 0; i < kBatchChunks; ++i) {
        const uint32_t k = left > kChunkIds * i ? (uint32_t)min((uint64_t)kChunkIds, left - kChunkIds * i) : 0u;
        x[i] = ids[i] = 0;
        if (k == 0 || bad) continue;
        if (pos + 2 > end) {
            bad = true;
            continue;
        }
        const uint32_t off = (uint32_t)((pos >> 2) - base);
        const uint32_t sh = (uint32_t)(pos & 3u) * 8u;
        const uint64_t head = (((uint64_t)sm[off + 1] << 32) | sm[off]) >> sh;
        const uint32_t code = (uint32_t)head & 0xFFu, w = chunk_width(code), fb = chunk_first_bytes(code);
        const uint32_t zz = chunk_plain(code) ? 0u : 1u;  // zigzag-coded deltas
        const uint64_t size = chunk_bytes(code, k);
        if (pos + size > end) {
            bad = true;
            continue;
        }
        ids[i] = k;
        pos += size;
        const uint32_t bo = sh + 8u + 8u * fb + (lane ? (lane - 1) * w : 0u);
        const uint32_t q = off + (bo >> 5);
        if (lane == 0) {
            x[i] = (uint32_t)((head >> 8) & (0xFFFFFFFFull >> (32u - 8u * fb)));
        } else if (lane < k && w != 0) {
            const uint64_t acc = ((uint64_t)sm[q + 1] << 32) | sm[q];
            const uint64_t mask = (w == 32) ? 0xFFFFFFFFull : ((1ull << w) - 1);
            const uint32_t z = (uint32_t)((acc >> (bo & 31u)) & mask);
            x[i] = zz ? (z >> 1) ^ (0u - (z & 1u)) : z;
        }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (uint32_t i = 0; i < kBatchChunks; ++i) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x[i], o);
            if (lane >= (uint32_t)o) x[i] += y;
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < kBatchChunks; ++i)
        if (lane < ids[i]) {
            row[kChunkIds * i + lane] = x[i];
            bad_id |= x[i] >= nverts;
        }
    return pos;
}

// A warp's shared-memory window of the payload (4.3 KB), filled 16 bytes a lane.
// A chunk spans at most 5 + 124 bytes, so kBatchChunks of them from byte `pos`
// on lie in the 131 words from pos / 4, and one word more is read: kSlideAt is
// the last word of the window that they may start in.
constexpr uint32_t kWindowWords = 1088;
constexpr uint32_t kSlideAt = kWindowWords - 132;
// Payload words [base, base + n) to the window; base and n are multiples of 4.
// Three loads of a lane in flight: one after another, 33 of a word each were
// 24 us of a 34 us decode.
__device__ __forceinline__ void fill_window(uint32_t *sm, const uint32_t *__restrict__ pay_words, uint64_t base,
                                            uint32_t n, uint64_t limit, uint32_t lane)
{
    constexpr uint32_t R = 3;
    for (uint32_t i0 = 4 * lane; i0 < n; i0 += 128 * R) {
        uint4 r[R];
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint32_t i = i0 + 128 * k;
            r[k] = make_uint4(0u, 0u, 0u, 0u);
            if (i < n && base + i < limit) r[k] = __ldg(reinterpret_cast<const uint4 *>(pay_words + base + i));
        }
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint32_t i = i0 + 128 * k;
            if (i < n) *reinterpret_cast<uint4 *>(sm + i) = r[k];
        }
    }
}
constexpr uint32_t kDecodeThreads = 256;
constexpr uint32_t kDecodeCtas = 3;  // of an SM

// Vertex v of a block lies at beg[v] + kVertexWeight * v on the line that tasks
// cut: a batch of 32 vertices weighs what 128 ids do, whether it has ids or not.
constexpr uint32_t kVertexWeight = 4;

// First vertex v in [lo, hi) at or past t on that line (hi if none), by the
// whole warp: 32 probes a round.
__device__ __forceinline__ uint32_t warp_first_vertex(const uint64_t *__restrict__ beg, uint32_t lo, uint32_t hi,
                                                      uint64_t t, uint32_t lane)
{
    auto past = [&](uint32_t v) { return __ldg(beg + v) + (uint64_t)kVertexWeight * v >= t; };
    while (hi - lo > 32) {
        const uint32_t q = lo + (uint32_t)((uint64_t)(hi - lo) * (lane + 1) / 33);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, past(q));
        const uint32_t below = (uint32_t)__popc(~m);  // places increase: the first `below` probes are before t
        const uint32_t q_lo = __shfl_sync(0xFFFFFFFFu, q, below ? below - 1 : 0);
        const uint32_t q_hi = __shfl_sync(0xFFFFFFFFu, q, below < 32 ? below : 31);
        if (below) lo = q_lo + 1;
        if (below < 32) hi = q_hi;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, lo + lane < hi && past(lo + lane));
    return m ? lo + (uint32_t)__ffs(m) - 1 : hi;
}

// The vertices [v_lo, v_hi) of a block, whose ids are [e_lo, e_hi) of the
// block's, and the split groups [g_lo, g_hi).
//
// Warp tasks: task t < nbt takes the vertices of at most 32 chunks that lie in
// the t-th stretch of `per` on the line of ids and vertices above, 32 at a time
// (lane i loads a vertex's payload offset and neighbour range, coalesced); the
// tasks behind those each decode one split group (32 chunks of a larger
// vertex).  A task's chunks are
// read from a window of the payload in shared memory, filled by the warp with
// coalesced, independent loads and slid forward when the next chunk would
// run past it, so the only dependent chain -- each chunk's position follows
// from the previous chunk's width byte -- runs through shared memory.  Every
// id written is checked against nverts (the validation of a plain block
// copy, done here in the same pass).
//
// What bounds it is the longest task: a vertex's chunks follow one another, and
// so do a task's batches.  Cut by vertices alone, 32 vertices of up to 32 chunks
// each were one warp's work, a chain of 1,024 chunks, about 80 us for each of a
// block's four pieces whatever its size; by ids alone, 27 us, a few ids spread
// over hundreds of vertices without any; by both, 22 us.
__global__ void __launch_bounds__(kDecodeThreads, 4)
    k_decode_block(const uint8_t *__restrict__ src, uint64_t split_off, uint64_t payload_off, uint64_t payload_bytes,
                   uint32_t nv, const uint64_t *__restrict__ beg, uint32_t v0, uint64_t e0, uint64_t ne,
                   uint32_t nverts, uint32_t *__restrict__ out, uint32_t *err, uint32_t v_lo, uint32_t v_hi,
                   uint64_t e_lo, uint64_t e_hi, uint32_t per, uint32_t g_lo, uint32_t g_hi)
{
    __shared__ __align__(16) uint32_t s_win[kDecodeThreads / 32][kWindowWords];
    uint32_t *sm = s_win[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t *voff = reinterpret_cast<const uint32_t *>(src);
    const uint32_t *split = reinterpret_cast<const uint32_t *>(src + split_off);
    const uint32_t *pay_words = reinterpret_cast<const uint32_t *>(src + payload_off);
    const uint64_t limit = (payload_bytes + 8) >> 2;  // whole words of payload and padding
    const uint64_t line0 = e0 + e_lo + (uint64_t)kVertexWeight * v_lo;
    const uint64_t nbt = (e_hi - e_lo + (uint64_t)kVertexWeight * (v_hi - v_lo) + per - 1) / per;
    const uint64_t ntasks = nbt + (g_hi - g_lo);
    bool bad_id = false, bad = false;
    uint64_t base = ~0ull;  // first payload word in the window (~0: empty)
    // make the window hold the chunks from byte `pos` on (warp-uniform)
    auto cover = [&](uint64_t pos) {
        const uint64_t w = pos >> 2;
        if (base != ~0ull && w >= base && w - base <= kSlideAt) return;
        __syncwarp();  // every lane is done with the old window
        base = w & ~3ull;
        fill_window(sm, pay_words, base, kWindowWords, limit, lane);
        __syncwarp();
    };
    for (uint64_t task = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < ntasks; task += nwarps) {
        if (task >= nbt) {
            const uint64_t g = g_lo + (task - nbt);
            const uint32_t v = __ldg(split + 3 * g), c0 = __ldg(split + 3 * g + 1);
            uint64_t pos = __ldg(split + 3 * g + 2);
            if (v >= nv) {
                bad = true;
                continue;
            }
            const uint64_t b0 = __ldg(beg + v0 + v), b1 = __ldg(beg + v0 + v + 1);
            if (b1 < b0 || b0 < e0 || b1 - e0 > ne) {
                bad = true;
                continue;
            }
            const uint64_t d = b1 - b0;
            const uint64_t nch = (d + kChunkIds - 1) / kChunkIds;
            const uint64_t c1 = min(nch, (uint64_t)c0 + kChunkIds);
            bool vbad = false;
            const uint64_t ids_end = min(d, c1 * kChunkIds);
            for (uint64_t i = (uint64_t)c0 * kChunkIds; i < ids_end && !vbad; i += kBatchChunks * kChunkIds) {
                cover(pos);
                pos = decode_chunks_sm(sm, base, pos, payload_bytes, ids_end - i, lane, out + (b0 - e0) + i, nverts,
                                       bad_id, vbad);
            }
            bad |= vbad;
            continue;
        }
        const uint64_t t_end = line0 + (task + 1) * per;
        uint32_t vb = warp_first_vertex(beg + v0, v_lo, v_hi, line0 + task * per, lane);
        for (; vb < v_hi; vb += 32) {
            const uint32_t nvt = min(32u, v_hi - vb);
            uint64_t mpos = 0, mnext = 0, mb0 = 0, mb1 = 0;
            if (lane < nvt) {
                mpos = __ldg(voff + vb + lane);
                mnext = __ldg(voff + vb + lane + 1);
                mb0 = __ldg(beg + v0 + vb + lane);
                mb1 = __ldg(beg + v0 + vb + lane + 1);
            }
            // lanes of the task's vertices; the others belong to the next task
            const bool mine = lane < nvt && mb0 + (uint64_t)kVertexWeight * (vb + lane) < t_end;
            const unsigned ours = __ballot_sync(0xFFFFFFFFu, mine);
            if (ours == 0) break;
            if (__ballot_sync(0xFFFFFFFFu, mine && mb1 != mb0) == 0) continue;  // no ids in the batch
            // the batch's payload: [first vertex's offset, past its last vertex's)
            const uint32_t last = 31u - (uint32_t)__clz((int)ours);
            const uint64_t p0 = __shfl_sync(0xFFFFFFFFu, mpos, 0);
            const uint64_t p1 = __shfl_sync(0xFFFFFFFFu, mnext, last);
            if (p1 < p0 || p1 > payload_bytes) {
                bad = true;
                continue;
            }
            // every chunk of the batch reads words [p0 / 4, p1 / 4 + 2)
            const uint64_t b_base = (p0 >> 2) & ~3ull, nwords = (((p1 + 3) >> 2) - b_base + 2 + 3) & ~3ull;
            if (nwords <= kWindowWords) {
                // ---- the whole batch in the window: one fill, then each lane
                // decodes its own vertex when it has one chunk (most do), and
                // the warp decodes the chunks of the batch's larger vertices
                __syncwarp();
                base = b_base;
                fill_window(sm, pay_words, base, (uint32_t)nwords, limit, lane);
                __syncwarp();
                const bool range_ok = !mine || (mb1 >= mb0 && mb0 >= e0 && mb1 - e0 <= ne);
                bad |= !range_ok;
                const uint64_t d = (mine && range_ok) ? mb1 - mb0 : 0;
                if (d >= 1 && d <= kChunkIds) {
                    if (mpos < p0 || mpos + 2 > p1) {
                        bad = true;
                    } else {
                        const uint32_t off = (uint32_t)((mpos >> 2) - base);
                        const uint32_t sh = (uint32_t)(mpos & 3u) * 8u;
                        const uint64_t head = (((uint64_t)sm[off + 1] << 32) | sm[off]) >> sh;
                        const uint32_t code = (uint32_t)head & 0xFFu, w = chunk_width(code);
                        const uint32_t fb = chunk_first_bytes(code);
                        const bool zz = !chunk_plain(code);
                        if (mpos + chunk_bytes(code, (uint32_t)d) > p1) {
                            bad = true;
                        } else {
                            uint32_t *row = out + (mb0 - e0);
                            uint32_t x = (uint32_t)((head >> 8) & (0xFFFFFFFFull >> (32u - 8u * fb)));
                            row[0] = x;
                            bool over = x >= nverts;
                            const uint64_t mask = (w == 32) ? 0xFFFFFFFFull : ((1ull << w) - 1);
                            uint32_t bit = sh + 8u + 8u * fb;  // from word `off`
                            for (uint32_t i = 1; i < (uint32_t)d; ++i, bit += w) {
                                const uint32_t q = off + (bit >> 5);
                                const uint64_t acc = ((uint64_t)sm[q + 1] << 32) | sm[q];
                                const uint32_t z = (uint32_t)((acc >> (bit & 31u)) & mask);
                                x += zz ? (z >> 1) ^ (0u - (z & 1u)) : z;
                                row[i] = x;
                                over |= x >= nverts;
                            }
                            bad_id |= over;
                        }
                    }
                }
                // vertices of 2..32 chunks, one after another, a chunk per warp step
                for (unsigned mm = __ballot_sync(0xFFFFFFFFu, d > kChunkIds && d <= (uint64_t)kChunkIds * kChunkIds);
                     mm; mm &= mm - 1) {
                    const int j = __ffs(mm) - 1;
                    uint64_t pos = __shfl_sync(0xFFFFFFFFu, mpos, j);
                    const uint64_t b0 = __shfl_sync(0xFFFFFFFFu, mb0, j);
                    const uint64_t dj = __shfl_sync(0xFFFFFFFFu, d, j);
                    bool vbad = pos < p0;
                    for (uint64_t i = 0; i < dj && !vbad; i += kBatchChunks * kChunkIds)
                        pos = decode_chunks_sm(sm, base, pos, p1, dj - i, lane, out + (b0 - e0) + i, nverts, bad_id,
                                               vbad);
                    bad |= vbad;
                }
                base = ~0ull;  // the window holds this batch's words only
                continue;
            }
            // ---- a batch larger than the window: vertex by vertex, sliding it
            for (uint32_t j = 0; j <= last; ++j) {
                uint64_t pos = __shfl_sync(0xFFFFFFFFu, mpos, j);
                const uint64_t b0 = __shfl_sync(0xFFFFFFFFu, mb0, j), b1 = __shfl_sync(0xFFFFFFFFu, mb1, j);
                if (b1 < b0 || b0 < e0 || b1 - e0 > ne) {
                    bad = true;
                    continue;
                }
                const uint64_t d = b1 - b0;
                const uint64_t nch = (d + kChunkIds - 1) / kChunkIds;
                if (nch > kChunkIds) continue;  // decoded by its split groups
                bool vbad = pos < p0;
                for (uint64_t i = 0; i < d && !vbad; i += kBatchChunks * kChunkIds) {
                    cover(pos);
                    pos = decode_chunks_sm(sm, base, pos, p1, d - i, lane, out + (b0 - e0) + i, nverts, bad_id, vbad);
                }
                bad |= vbad;
            }
        }
    }
    if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicOr(err, kErrBlock);
    if (__any_sync(0xFFFFFFFFu, bad_id) && lane == 0) atomicOr(err, kErrVertexRange);
}

cudaError_t launch_decode_block(const uint8_t *src, const CompressedBlock &cb, uint32_t nv, const uint64_t *beg,
                                uint32_t v0, uint64_t e0, uint64_t ne, uint32_t nverts, uint32_t *out, uint32_t *err,
                                int num_sms, cudaStream_t s, int piece)
{
    if (nv == 0) return cudaSuccess;
    const int k0 = piece < 0 ? 0 : piece, k1 = piece < 0 ? (int)kPieces : piece + 1;
    const uint64_t ids = cb.piece_e[k1] - cb.piece_e[k0];
    const uint32_t groups = cb.piece_g[k1] - cb.piece_g[k0];
    if (ids == 0) return cudaSuccess;
    // one task a warp as far as they go: a task of 128 ids costs its search
    // for the first vertex and little more
    const uint64_t all = (uint64_t)num_sms * kDecodeCtas * (kDecodeThreads / 32);
    const uint64_t warps = all - std::min<uint64_t>(groups, all / 2);  // the others take a split group each
    const uint64_t line = ids + (uint64_t)kVertexWeight * (cb.piece_v[k1] - cb.piece_v[k0]);
    const uint32_t per = (uint32_t)std::min<uint64_t>(1024, std::max<uint64_t>(128, (line + warps - 1) / warps));
    const uint64_t tasks = (line + per - 1) / per + groups;
    const uint64_t need = (tasks + kDecodeThreads / 32 - 1) / (kDecodeThreads / 32);
    k_decode_block<<<(int)std::min<uint64_t>(need, (uint64_t)num_sms * kDecodeCtas), kDecodeThreads, 0, s>>>(
        src, cb.split_off, cb.payload_off, cb.payload_bytes, nv, beg, v0, e0, ne, nverts, out, err, cb.piece_v[k0],
        cb.piece_v[k1], cb.piece_e[k0], cb.piece_e[k1], per, cb.piece_g[k0], cb.piece_g[k1]);
    return cudaGetLastError();
}

}  // namespace gw
