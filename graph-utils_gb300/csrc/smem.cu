// smem.cu -- per-source BFS with the search state in shared memory: AUTO's engine
// for small graphs and few sources.
//
// The batched engine (msbfs.cu) shares every level among 64 W sources and pays a
// grid barrier and a dozen dependent L2 accesses per level whatever the graph's
// size: a level with almost no work takes about 10 us.  Here one thread-block
// cluster of S CTAs (1 .. 16) runs one source.  The frontier and visited bitmaps
// are kept whole in every CTA's shared memory, so that a neighbour costs one
// global load (its id in the adjacency list) and one shared-memory bit; a level
// ends with a CTA or cluster barrier.  CTA r of the cluster owns a slice of the
// vertices: it searches them bottom-up, expands them top-down, and keeps their
// levels (16 bits each) until the row is written, whole and coalesced, at the end.
//
// Level j, from the frontier F_{j-1}:
//   top-down   each CTA expands the frontier vertices of its slice (a queue built
//              when they were discovered) into its own whole-graph bitmap nxt;
//              after a cluster barrier the owner of a slice ORs the S copies and
//              drops the visited bits
//   bottom-up  each CTA scans the in-neighbours of its unvisited vertices, hubs
//              first, until one is in the frontier
// Then the owner records the level of the new vertices, queues them, counts them
// and their out-edges; after a cluster barrier every CTA gathers all slices' new
// bits as the next frontier.  Direction after Beamer, Asanovic, Patterson (SC'12), by the
// work that each would be.  Vertices without in-edges are never scanned: they start out
// visited.
#include "device_utils.cuh"
#include "gu_internal.h"
#include "kernel_fit.h"

#include <algorithm>
#include <climits>
#include <cstdlib>

namespace gu {

constexpr int SB_MAX_THREADS = 1024;
constexpr int SB_MAX_CLUSTER = 16;
constexpr int SB_QCAP = 8192;   // queued frontier vertices per CTA; a wider level is searched bottom-up
constexpr int SB_BIG = 512;     // out-degree from which the whole CTA expands a vertex
constexpr int SB_BIGCAP = 512;  // such vertices per level and CTA; the rest are left to their warps
constexpr int SB_BYTES_MAX_N = 8192;  // up to here nxt is a byte per vertex: plain stores, no atomics on a few words
constexpr int SB_LIST = 4096;   // unvisited vertices per CTA whose first four in-neighbours miss the frontier
constexpr int SB_MAX_LEVEL = 65533;
constexpr int SB_MAX_N = 262144;          // vertices whose state fits a cluster of sixteen CTAs
constexpr int64_t SB_MAX_M = 1 << 30;     // edge indices plus a step stay within 32 bits
constexpr size_t SB_MAX_SMEM = 223 * 1024;
constexpr unsigned SB_UNREACHED = 0xFFFFu;

// What a cluster reports, one word each in pinned host memory: no accumulator to
// clear before a launch, no copy after it.
constexpr int SB_MAX_CLUSTERS = 4096;
union SbStatus {
    struct {
        uint16_t err, td_levels, bu_levels, max_level;
    };
    unsigned long long word;
};

struct SbArgs {
    const int32_t *__restrict__ R;
    const int32_t *__restrict__ C;
    const int32_t *__restrict__ RT;
    const int32_t *__restrict__ CT;
    int32_t n;
    int64_t m;
    const int32_t *__restrict__ sources;
    int32_t k;
    int32_t *dist;  // k x ld rows, or null
    int64_t ld;
    unsigned long long *reach;  // k counts of reached vertices, or null
    const int4 *__restrict__ head;      // [n] first four in-neighbours (-1: none)
    const uint32_t *__restrict__ none;  // bitmap of the vertices without in-edges, padded with ones
    int slice;  // bitmap words per CTA of a cluster
    int32_t live;  // vertices with in-edges
    float alpha, beta;
    SbStatus *status;  // [clusters], pinned host memory
};

// Shared memory: cur, vis, nxt ([S * slice] words each), fresh[2][slice], queue, list,
// levels of the slice.
__host__ __device__ inline size_t sb_smem_bytes(int slice, int S, bool bytes)
{
    return (size_t)slice * S * (bytes ? 10 : 3) * sizeof(uint32_t) + 2 * (size_t)slice * sizeof(uint32_t) +
           (SB_QCAP + SB_LIST) * sizeof(int32_t) +
           (size_t)slice * 32 * sizeof(uint16_t);
}

struct SbCounts {
    int vertices, overflow;
    long long edges;
};

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_ctas()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Word at the same shared-memory offset as p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t ld_cluster_u32(const void *p, unsigned rank)
{
    uint32_t v;
    asm volatile("{\n\t.reg .u32 a, b;\n\tcvt.u32.u64 a, %1;\n\tmapa.shared::cluster.u32 b, a, %2;\n\t"
                 "ld.shared::cluster.u32 %0, [b];\n\t}"
                 : "=r"(v) : "l"(__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return v;
}

__device__ __forceinline__ uint4 ld_cluster_v4(const void *p, unsigned rank)
{
    uint4 v;
    asm volatile("{\n\t.reg .u32 a, b;\n\tcvt.u32.u64 a, %4;\n\tmapa.shared::cluster.u32 b, a, %5;\n\t"
                 "ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [b];\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(__cvta_generic_to_shared(p)), "r"(rank) : "memory");
    return v;
}

// MODE: one CTA per source with nxt a byte per vertex, one CTA, a cluster.
enum : int { SB_BYTES = 0, SB_CTA = 1, SB_CLUSTER = 2 };
template <int MODE>
__global__ void __launch_bounds__(SB_MAX_THREADS, 1) smem_bfs_kernel(SbArgs a)
{
    constexpr bool CLUSTER = MODE == SB_CLUSTER;
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ SbCounts s_cnt[2];  // new vertices of this slice and their out-edges, by parity
    __shared__ SbCounts s_tot;
    __shared__ int s_nbig, s_qn, s_nlist;
    __shared__ int32_t s_big[SB_BIGCAP];
    const int S = CLUSTER ? (int)cluster_ctas() : 1;
    const int r = CLUSTER ? (int)cluster_rank() : 0;
    const int cid = (int)blockIdx.x / S, nclusters = (int)gridDim.x / S;
    const int words = a.slice * S;
    uint32_t *cur = sm, *vis = cur + words, *nxt = vis + words;
    uint32_t *fresh2 = nxt + (MODE == SB_BYTES ? 8 : 1) * words;  // [2][slice]
    int32_t *queue = reinterpret_cast<int32_t *>(fresh2 + 2 * a.slice);
    int32_t *list = queue + SB_QCAP;
    uint16_t *lev = reinterpret_cast<uint16_t *>(list + SB_LIST);
    const int lane = lane_id(), warp = warp_in_block(), nw = blockDim.x >> 5, T = blockDim.x;
    const int w0 = r * a.slice;       // first word of the slice
    const int32_t v0 = w0 * 32;       // first vertex
    auto sync = [&] {
        if (CLUSTER) cluster_sync();
        else __syncthreads();
    };
    int par = 0, n_td = 0, n_bu = 0, deepest = 0, err = 0;
    // every CTA checks all sources: a call with a bad one is refused and writes nothing
    bool bad = false;
    for (int i = threadIdx.x; i < a.k; i += T) bad |= (unsigned)__ldg(a.sources + i) >= (unsigned)a.n;
    for (int si = cid; si < a.k; si += nclusters) {
        const int32_t src = __ldg(a.sources + si);
        for (int i = threadIdx.x; i < words; i += T) {
            const uint32_t bit = (src >> 5) == i ? 1u << (src & 31) : 0u;
            cur[i] = bit;
            vis[i] = __ldg(a.none + i) | bit;
        }
        for (int i = threadIdx.x; i < (MODE == SB_BYTES ? 8 : 1) * words; i += T) nxt[i] = 0;
        for (int i = threadIdx.x; i < a.slice * 16; i += T) reinterpret_cast<uint32_t *>(lev)[i] = 0xFFFFFFFFu;
        const bool mine = src >= v0 && src < v0 + a.slice * 32;
        if (__syncthreads_or(bad)) {  // (with a barrier that is there anyway; the same for every CTA)
            err = DEV_ERR_BAD_SOURCE;
            break;
        }
        if (threadIdx.x == 0) {
            s_qn = mine ? 1 : 0;
            s_nbig = 0;
            if (mine) {
                queue[0] = src;
                lev[src - v0] = 0;
            }
        }
        __syncthreads();
        long long fe = 0;  // out-edges and vertices of the frontier
        int nf = 1, reached = 1;
        bool bu = false, wide = false;
        int level = 1;
        for (;; ++level) {
            // ---- direction ----
            const bool was_bu = bu;
            if (level > 1) {
                // (32-bit floats: FP64 runs at two lanes a cycle per SM on this part, and a
                // few such instructions in every warp cost more than the rest of the level end)
                // Bottom-up, each of the vertices not reached tries its in-neighbours until one
                // is in the frontier, m / fe of them at random: fewer than the frontier's fe
                // out-edges if fe^2 > alpha x vertices left x m.  A frontier of few edges is
                // one round of loads top-down, whatever the graph.
                if (!bu)
                    bu = wide || ((float)fe * (float)fe > a.alpha * (float)(a.live - reached) * (float)a.m &&
                                  fe > (long long)(4 * S) * T);
                else bu = (float)nf * a.beta > (float)a.n || nf > SB_QCAP;
            }
            if (threadIdx.x == 0) {
                s_cnt[par].vertices = 0;
                s_cnt[par].overflow = 0;
                s_cnt[par].edges = 0;
            }
            uint32_t *fresh = fresh2 + par * a.slice;
            long long edges = 0;
            int found_n = 0;
            // the queue of the slice's frontier: of x, the new bits of word i (per lane)
            auto enqueue = [&](uint32_t x, int i, bool discovered) {
                const int c = __popc(x);
                int inc = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(FULL_MASK, inc, o);
                    if (lane >= o) inc += y;
                }
                const int total = __shfl_sync(FULL_MASK, inc, 31);
                if (!total) return;
                int pos = 0;
                if (lane == 0) pos = atomicAdd(&s_qn, total);
                pos = __shfl_sync(FULL_MASK, pos, 0) + inc - c;
                for (; x; x &= x - 1, ++pos) {
                    const int32_t v = v0 + 32 * i + __ffs(x) - 1;
                    if (discovered) lev[v - v0] = (uint16_t)level;
                    if (pos < SB_QCAP) queue[pos] = v;
                }
            };
            if (!bu) {
                // ---- top-down: the queued frontier vertices of the slice ----
                auto discover = [&](int32_t w) {
                    const uint32_t bit = 1u << (w & 31);
                    if (MODE == SB_BYTES) {
                        if (!(vis[w >> 5] & bit)) reinterpret_cast<unsigned char *>(nxt)[w] = 1;
                    } else if (!((vis[w >> 5] | nxt[w >> 5]) & bit)) {
                        atomicOr(nxt + (w >> 5), bit);
                    }
                };
                if (was_bu) {  // the last level's new bits of the slice (still in the other buffer)
                    const uint32_t *last = fresh2 + (par ^ 1) * a.slice;
                    if (threadIdx.x == 0) s_qn = 0;
                    __syncthreads();
                    for (int i0 = 32 * warp; i0 < a.slice; i0 += 32 * nw)
                        enqueue(i0 + lane < a.slice ? last[i0 + lane] : 0u, i0 + lane, false);
                    __syncthreads();
                }
                const int qn = s_qn;
                const int chunk = min(32, (qn + nw - 1) / nw);  // vertices per warp step: every warp gets some
                for (int base = warp * chunk; base < qn; base += nw * chunk) {  // warp-uniform
                    int32_t e0 = 0, deg = 0;
                    if (lane < chunk && base + lane < qn) {
                        const int32_t v = queue[base + lane];
                        e0 = __ldg(a.R + v);
                        deg = __ldg(a.R + v + 1) - e0;
                        if (deg >= SB_BIG) {
                            const int b = atomicAdd(&s_nbig, 1);
                            if (b < SB_BIGCAP) {
                                s_big[b] = v;
                                deg = 0;
                            }
                        }
                    }
                    int inc = deg;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(FULL_MASK, inc, o);
                        if (lane >= o) inc += y;
                    }
                    const int start = e0 - (inc - deg);  // edge slot t of the warp is C[start(owner) + t]
                    const int total = __shfl_sync(FULL_MASK, inc, 31);
                    for (int t0 = 0; t0 < total; t0 += 128) {
                        int32_t w[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int t = t0 + 32 * u + lane;
                            int lo = 0;  // owner: lanes whose inclusive prefix is <= t
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1)
                                if (__shfl_sync(FULL_MASK, inc, lo + o - 1) <= t) lo += o;
                            const int st = __shfl_sync(FULL_MASK, start, lo & 31);
                            w[u] = t < total ? __ldg(a.C + st + t) : -1;
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (w[u] >= 0) discover(w[u]);
                        }
                    }
                }
                __syncthreads();
                const int nbig = min(s_nbig, SB_BIGCAP);
                for (int b = 0; b < nbig; ++b) {
                    const int32_t v = s_big[b], e1 = __ldg(a.R + v + 1);
                    for (int32_t e = __ldg(a.R + v) + threadIdx.x; e < e1; e += 2 * T) {
                        const int32_t x = __ldg(a.C + e), y = e + T < e1 ? __ldg(a.C + e + T) : -1;
                        discover(x);
                        if (y >= 0) discover(y);
                    }
                }
                sync();
                if (threadIdx.x == 0) {
                    s_qn = 0;
                    s_nbig = 0;
                }
                __syncthreads();
                // ---- the slice's new vertices: the S copies together, less the visited ones ----
                if (CLUSTER) {
                    // 16 lanes per four words, one CTA's copy each, all loads in flight at once
                    for (int i = threadIdx.x >> 4; i < ((a.slice >> 2) + 1 & ~1); i += T >> 4) {
                        uint4 x = make_uint4(0u, 0u, 0u, 0u);
                        const int o = threadIdx.x & 15;
                        if (o < S && 4 * i < a.slice) x = ld_cluster_v4(nxt + w0 + 4 * i, o);
#pragma unroll
                        for (int d = 1; d < 16; d <<= 1) {
                            x.x |= __shfl_xor_sync(FULL_MASK, x.x, d);
                            x.y |= __shfl_xor_sync(FULL_MASK, x.y, d);
                            x.z |= __shfl_xor_sync(FULL_MASK, x.z, d);
                            x.w |= __shfl_xor_sync(FULL_MASK, x.w, d);
                        }
                        if (o == 0 && 4 * i < a.slice) *reinterpret_cast<uint4 *>(fresh + 4 * i) = x;
                    }
                    __syncthreads();
                }
                if (MODE == SB_BYTES) {  // bytes to bits
                    for (int i = warp; i < words; i += nw) {
                        const unsigned x = __ballot_sync(FULL_MASK, reinterpret_cast<unsigned char *>(nxt)[32 * i + lane]);
                        if (lane == 0) fresh[i] = x;
                    }
                    __syncthreads();
                }
                for (int i0 = 32 * warp; i0 < a.slice; i0 += 32 * nw) {  // warp-uniform, a word per lane
                    const int i = i0 + lane;
                    uint32_t x = 0;
                    if (i < a.slice) {
                        x = (MODE == SB_CTA ? nxt[i] : fresh[i]) & ~vis[w0 + i];
                        fresh[i] = x;
                        found_n += __popc(x);
                    }
                    enqueue(x, i, true);
                }
                __syncthreads();
                // their out-edges (a wider level is searched bottom-up whatever they are)
                for (int i = threadIdx.x; i < min(s_qn, SB_QCAP); i += T) {
                    const int32_t v = queue[i];
                    edges += __ldg(a.R + v + 1) - __ldg(a.R + v);
                }
            } else {
                if (threadIdx.x == 0) s_nlist = 0;
                __syncthreads();
                // ---- bottom-up, a lane per unvisited vertex: the first four in-neighbours
                // (the hubs; one coalesced load) against the frontier; vertices they do not
                // decide are listed with their remaining in-edges left to the second pass
                auto in_frontier = [&](int32_t c) { return (cur[c >> 5] >> (c & 31)) & 1u; };
                // in-neighbours [e, e1) of one vertex per lane: aligned 16-byte pieces, then, for
                // what is left of long lists, the warp together
                auto scan = [&](int32_t e, int32_t e1) {
                    bool hit = false;
#pragma unroll 1
                    for (int step = 0; step < 4; ++step) {
                        const bool go = e < e1 && !hit;
                        if (!__any_sync(FULL_MASK, go)) return hit;
                        if (go) {  // two 16-byte pieces in flight
                            const int32_t b = e & ~3;
                            const int4 *p = reinterpret_cast<const int4 *>(a.CT) + (b >> 2);
                            const int4 c = __ldg(p);
                            int4 d = make_int4(0, 0, 0, 0);
                            if (b + 4 < e1) d = __ldg(p + 1);
                            if (b >= e) hit = in_frontier(c.x);
                            if (b + 1 >= e && b + 1 < e1) hit |= in_frontier(c.y);
                            if (b + 2 >= e && b + 2 < e1) hit |= in_frontier(c.z);
                            if (b + 3 < e1) hit |= in_frontier(c.w);
                            if (!hit && b + 4 < e1) {
                                hit = in_frontier(d.x);
                                if (b + 5 < e1) hit |= in_frontier(d.y);
                                if (b + 6 < e1) hit |= in_frontier(d.z);
                                if (b + 7 < e1) hit |= in_frontier(d.w);
                            }
                            e = b + 8;
                        }
                    }
                    unsigned todo = __ballot_sync(FULL_MASK, e < e1 && !hit);
                    while (todo) {
                        const int l = __ffs(todo) - 1;
                        todo &= todo - 1;
                        const int32_t be = __shfl_sync(FULL_MASK, e, l), en = __shfl_sync(FULL_MASK, e1, l);
                        bool any = false;
#pragma unroll 1
                        for (int32_t b = be; b < en && !any; b += 128) {
                            int32_t c[4];
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                c[t] = b + 32 * t + lane < en ? __ldg(a.CT + b + 32 * t + lane) : -1;
                            bool h = false;
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (c[t] >= 0) h |= in_frontier(c[t]);
                            any = __any_sync(FULL_MASK, h);
                        }
                        if (lane == l) hit = any;
                    }
                    return hit;
                };
#pragma unroll 1
                for (int i0 = warp; i0 < a.slice; i0 += 4 * nw) {  // warp-uniform; four words in flight
                    int4 h[4];
                    bool more[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int i = i0 + u * nw;
                        h[u].x = -1;
                        if (i < a.slice && !((vis[w0 + i] >> lane) & 1u)) h[u] = __ldg(a.head + v0 + 32 * i + lane);
                    }
                    int nmore = 0;  // lanes of the four words with more, this one's place among them
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int i = i0 + u * nw;
                        bool hit = false;
                        if (h[u].x >= 0) {
                            hit = in_frontier(h[u].x);
                            if (!hit && h[u].y >= 0) hit = in_frontier(h[u].y);
                            if (!hit && h[u].z >= 0) hit = in_frontier(h[u].z);
                            if (!hit && h[u].w >= 0) hit = in_frontier(h[u].w);
                        }
                        more[u] = h[u].x >= 0 && !hit && h[u].y >= 0 && h[u].z >= 0 && h[u].w >= 0;
                        if (hit) lev[32 * i + lane] = (uint16_t)level;
                        found_n += hit;
                        const unsigned x = __ballot_sync(FULL_MASK, hit);
                        if (lane == 0 && i < a.slice) fresh[i] = x;
                        nmore += __popc(__ballot_sync(FULL_MASK, more[u]));
                    }
                    if (!nmore) continue;  // warp-uniform
                    int pos = 0;
                    if (lane == 0) pos = atomicAdd(&s_nlist, nmore);
                    pos = __shfl_sync(FULL_MASK, pos, 0);
#pragma unroll 1
                    for (int u = 0; u < 4; ++u) {
                        const bool m = u == 0 ? more[0] : u == 1 ? more[1] : u == 2 ? more[2] : more[3];
                        const unsigned y = __ballot_sync(FULL_MASK, m);
                        const int at = pos + __popc(y & ((1u << lane) - 1u)), i = i0 + u * nw;
                        const int32_t v = v0 + 32 * i + lane;
                        if (m && at < SB_LIST) list[at] = v;
                        if (pos + __popc(y) > SB_LIST) {  // a full list: the rest at once (warp-uniform)
                            const bool late = m && at >= SB_LIST;
                            const bool hit = scan(late ? __ldg(a.RT + v) + 4 : 0, late ? __ldg(a.RT + v + 1) : 0);
                            if (hit) lev[v - v0] = (uint16_t)level;
                            found_n += hit;
                            const unsigned z = __ballot_sync(FULL_MASK, hit);
                            if (lane == 0 && z) fresh[i] |= z;
                        }
                        pos += __popc(y);
                    }
                }
                __syncthreads();
                const int nl = min(s_nlist, SB_LIST);
#pragma unroll 1
                for (int i0 = warp * 32; i0 < nl; i0 += nw * 32) {  // warp-uniform
                    const bool on = i0 + lane < nl;
                    const int32_t v = on ? list[i0 + lane] : 0;
                    const int32_t e = on ? __ldg(a.RT + v) + 4 : 0, e1 = on ? __ldg(a.RT + v + 1) : 0;
                    if (scan(e, e1)) {
                        lev[v - v0] = (uint16_t)level;
                        ++found_n;
                        atomicOr(fresh + ((v - v0) >> 5), 1u << (v & 31));
                    }
                }
            }
            // ---- counts of the slice ----
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) edges += __shfl_xor_sync(FULL_MASK, edges, o);
            found_n = __reduce_add_sync(FULL_MASK, found_n);
            // (vertices are counted by bitmap word, their edges by place in the queue: a warp
            // may have either without the other)
            if (lane == 0) {
                if (found_n) atomicAdd(&s_cnt[par].vertices, found_n);
                if (edges) atomicAdd(reinterpret_cast<unsigned long long *>(&s_cnt[par].edges), (unsigned long long)edges);
            }
            __syncthreads();
            if (threadIdx.x == 0) s_cnt[par].overflow = !bu && s_qn > SB_QCAP;
            sync();
            // ---- the next frontier, from all slices ----
            if (bu) ++n_bu;
            else ++n_td;
            const int quads = a.slice >> 2;
            for (int i = threadIdx.x; i < words >> 2; i += T) {
                uint4 x;
                if (CLUSTER) {
                    const int o = i / quads;
                    x = ld_cluster_v4(fresh + 4 * (i - o * quads), o);
                } else {
                    x = reinterpret_cast<const uint4 *>(fresh)[i];
                }
                reinterpret_cast<uint4 *>(cur)[i] = x;
                uint4 y = reinterpret_cast<uint4 *>(vis)[i];
                y.x |= x.x;
                y.y |= x.y;
                y.z |= x.z;
                y.w |= x.w;
                reinterpret_cast<uint4 *>(vis)[i] = y;
                if (MODE != SB_BYTES) reinterpret_cast<uint4 *>(nxt)[i] = make_uint4(0u, 0u, 0u, 0u);
            }
            if (MODE == SB_BYTES)
                for (int i = threadIdx.x; i < 2 * words; i += T) reinterpret_cast<uint4 *>(nxt)[i] = make_uint4(0u, 0u, 0u, 0u);
            if (warp == 0) {
                int nv = 0, ov = 0;
                long long ne = 0;
                if (CLUSTER) {
                    if (lane < S) {
                        nv = (int)ld_cluster_u32(&s_cnt[par].vertices, lane);
                        ov = (int)ld_cluster_u32(&s_cnt[par].overflow, lane);
                        const char *pe = reinterpret_cast<const char *>(&s_cnt[par].edges);
                        ne = (long long)(((u64)ld_cluster_u32(pe + 4, lane) << 32) | ld_cluster_u32(pe, lane));
                    }
                    nv = __reduce_add_sync(FULL_MASK, nv);
                    ov = __reduce_or_sync(FULL_MASK, ov);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ne += __shfl_xor_sync(FULL_MASK, ne, o);
                } else if (lane == 0) {
                    nv = s_cnt[par].vertices;
                    ov = s_cnt[par].overflow;
                    ne = s_cnt[par].edges;
                }
                if (lane == 0) {
                    s_tot.vertices = nv;
                    s_tot.overflow = ov;
                    s_tot.edges = ne;
                }
            }
            __syncthreads();
            nf = s_tot.vertices;
            fe = s_tot.edges;
            wide = s_tot.overflow != 0;
            reached += nf;
            par ^= 1;
            if (nf == 0) break;
            if (level >= SB_MAX_LEVEL) {  // levels beyond 16 bits: the call reruns on the batched engine
                err = max(err, (int)DEV_ERR_QUEUE_OVERFLOW);
                break;
            }
        }
        deepest = max(deepest, level - 1);
        // ---- the slice of the row ----
        if (a.reach && r == 0 && threadIdx.x == 0) a.reach[si] = (unsigned long long)reached;
        const int32_t nv = min(a.slice * 32, a.n - v0);
        if (a.dist && nv > 0) {
            int32_t *row = a.dist + (int64_t)si * a.ld + v0;
            if ((((uintptr_t)row) & 15) == 0) {
                const int32_t nv4 = nv >> 2;
                for (int i = threadIdx.x; i < nv4; i += T) {
                    const uint2 p = reinterpret_cast<const uint2 *>(lev)[i];
                    int4 o;
                    o.x = (p.x & 0xFFFFu) == SB_UNREACHED ? INT_MAX : (int32_t)(p.x & 0xFFFFu);
                    o.y = (p.x >> 16) == SB_UNREACHED ? INT_MAX : (int32_t)(p.x >> 16);
                    o.z = (p.y & 0xFFFFu) == SB_UNREACHED ? INT_MAX : (int32_t)(p.y & 0xFFFFu);
                    o.w = (p.y >> 16) == SB_UNREACHED ? INT_MAX : (int32_t)(p.y >> 16);
                    __stcs(reinterpret_cast<int4 *>(row) + i, o);
                }
                for (int i = 4 * nv4 + threadIdx.x; i < nv; i += T) row[i] = lev[i] == SB_UNREACHED ? INT_MAX : (int32_t)lev[i];
            } else {
                for (int i = threadIdx.x; i < nv; i += T) row[i] = lev[i] == SB_UNREACHED ? INT_MAX : (int32_t)lev[i];
            }
        }
        __syncthreads();
    }
    // no CTA leaves while another may still read its shared memory
    if (CLUSTER) cluster_sync();
    if (r == 0 && threadIdx.x == 0) {
        SbStatus st;
        st.err = (uint16_t)err;
        st.td_levels = (uint16_t)min(n_td, 65535);
        st.bu_levels = (uint16_t)min(n_bu, 65535);
        st.max_level = (uint16_t)deepest;
        a.status[cid].word = st.word;
    }
}

// head and none of the graph (padded to whole clusters' slices).
__global__ void smem_head_kernel(const int32_t *__restrict__ RT, const int32_t *__restrict__ CT, int32_t n, int pad_words,
                                 int4 *__restrict__ head, uint32_t *__restrict__ none)
{
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < 32 * pad_words; v += gridDim.x * blockDim.x) {  // whole warps
        const int32_t e = v < n ? __ldg(RT + v) : 0, d = v < n ? __ldg(RT + v + 1) - e : 0;
        int4 h;
        h.x = d > 0 ? __ldg(CT + e) : -1;
        h.y = d > 1 ? __ldg(CT + e + 1) : -1;
        h.z = d > 2 ? __ldg(CT + e + 2) : -1;
        h.w = d > 3 ? __ldg(CT + e + 3) : -1;
        if (v < n) head[v] = h;
        const unsigned b = __ballot_sync(FULL_MASK, d == 0);
        if ((v & 31) == 0) none[v >> 5] = b;
    }
}

static const void *sb_kernel(int mode)
{
    return mode == SB_CLUSTER ? (const void *)smem_bfs_kernel<SB_CLUSTER>
           : mode == SB_CTA   ? (const void *)smem_bfs_kernel<SB_CTA>
                              : (const void *)smem_bfs_kernel<SB_BYTES>;
}

struct SbConfig {
    int S = 0, threads = 0, mode = 0, slice = 0;
    size_t smem = 0;
    int resident = 0;  // clusters
};

// A launch with clusters of S CTAs on the graph; resident = 0 where it does not fit.
static SbConfig sb_config(const DeviceGraph &g, int S, int threads)
{
    SbConfig c;
    c.S = S;
    c.threads = threads;
    const int words = std::max(1, (int)(((int64_t)g.n + 31) / 32));
    c.slice = ((words + S - 1) / S + 3) & ~3;
    c.mode = S > 1 ? SB_CLUSTER : g.n <= SB_BYTES_MAX_N ? SB_BYTES : SB_CTA;
    c.smem = sb_smem_bytes(c.slice, S, c.mode == SB_BYTES);
    if (c.smem > SB_MAX_SMEM) return c;
    c.resident = kernel_fit(g.device, sb_kernel(c.mode), threads, c.smem, SB_MAX_SMEM, S) * (S > 1 ? 1 : g.sm_count);
    return c;
}

// Whether AUTO takes this engine for k sources, and how.  Call times in us, this
// engine / the engine AUTO took before, k sources:
//   n <= 16384, always: one CTA per source keeps its advantage at any k (R-MAT 12
//     k = 300 50 / 360, R-MAT 14 k = 150 59 / 154, k = 1500 279 / 919, ER 2000
//     k = 512 71 / 180).  Out-degrees up to 16 have an engine of their own (local.cu),
//     which is level from n = 6400, k = 256 (524 / 488) down and behind elsewhere
//     (128 x 128 grid k = 1 507 / 649, k = 256 665 / 784); above, it is ahead
//     (256 x 256 grid 1477 / 1277).
//   n <= 32768: up to one source per SM and k m = 140 M (R-MAT 15 k = 150 90 / 174,
//     ER 30000 k = 150 101 / 143; k = 300 196 / 254, but behind on denser graphs).
//   above, by k m, the work that the batched engine shares among the sources: up to
//     60 M (R-MAT 16 k = 32 70 / 143, ER 100000 k = 30 98 / 143; ER 65000 k = 80 226 /
//     157), with four CTAs a source at least (a DAG of 60000 vertices and 26 levels,
//     counts, k = 100, one CTA a source: 451 / 305), and beyond 131072 vertices, where
//     a source needs eight CTAs, up to 8 sources (R-MAT 18 k = 8 115 / 153, k = 16 179 /
//     167).
// Out-degrees up to four go to the mesh form of the per-source engine (rows, this engine
// / that one: 48 x 48 grid k = 1 183 / 128 us, 100 x 100 k = 150 488 / 313, 128 x 128
// k = 256 718 / 410); with out-degrees of 5 to 16 this one is ahead (random graph of 10000
// vertices, k = 64, 75 / 139).
// Cluster size: as many CTAs per source as all k keep resident at once, while a CTA
// has at least 4096 vertices (R-MAT 17 k = 1: S = 4 83 us, 8 65, 16 58; R-MAT 14
// k = 1: S = 1 47, 4 43, 16 43).
static SbConfig sb_choose(const DeviceGraph &g, int32_t k)
{
    const char *e = std::getenv("GU_AUTO_LOCAL");
    if (e && e[0] == '0') return SbConfig();  // AUTO kept on the batched engine
    const double km = (double)k * (double)g.m;
    const bool low = g.max_degree <= LOCAL_MAX_DEGREE, many = k > g.sm_count;
    if (k < 1 || g.n < 1 || g.m > SB_MAX_M || g.max_degree <= LOCAL_MESH_DEGREE) return SbConfig();
    if (g.n <= 16384) {
        if (low && many && g.n <= 8192) return SbConfig();
    } else if (low) {
        return SbConfig();
    } else if (g.n <= 32768) {
        if (many || km > 140e6) return SbConfig();
    } else if (g.n > SB_MAX_N || km > 60e6 || (g.n > 131072 && k > 8)) {
        return SbConfig();
    }
    if (g.n >= 16384 && !low)
        for (int S = SB_MAX_CLUSTER; S > (g.n > 32768 ? 2 : 1); S /= 2) {
            if (g.n / S < 4096) continue;
            const SbConfig c = sb_config(g, S, g.n / S <= (S == SB_MAX_CLUSTER ? 4096 : 8192) ? 512 : 1024);
            if (c.resident >= k) return c;
        }
    if (g.n > 32768) return SbConfig();
    const int threads = g.n <= 4096 ? (many ? 256 : 512) : g.n <= 16384 ? (many || low ? 512 : 1024) : 1024;
    SbConfig c = sb_config(g, 1, threads);
    return c.resident > 0 ? c : SbConfig();
}

bool smem_bfs_takes(const DeviceGraph &g, int32_t k) { return sb_choose(g, k).S > 0; }

// Rows (dist) and / or counts (reach) of k sources; false if AUTO does not take this
// engine here, its tables cannot be allocated or a level does not fit 16 bits (the caller
// runs another engine).
// Synchronises stream.
bool launch_smem_bfs(DeviceGraph &g, const int32_t *sources, int32_t k, int32_t *dist, int64_t ld,
                     unsigned long long *reach, int *max_level, cudaStream_t stream)
{
    const SbConfig c = sb_choose(g, k);
    if (c.S == 0) return false;
    // an allocation that fails: the other engines run the search in the memory they have
    auto got = [](cudaError_t e) {
        if (e == cudaErrorMemoryAllocation) {
            (void)cudaGetLastError();
            return false;
        }
        GU_CUDA_CHECK(e);
        return true;
    };
    if (!g.sb_status && !got(pinned_alloc(&g.sb_status, sizeof(SbStatus) * SB_MAX_CLUSTERS))) return false;
    const int pad_words = (int)(((int64_t)g.n + 31) / 32) + 4 * SB_MAX_CLUSTER;  // slices are multiples of four words
    const size_t head_bytes = (size_t)g.n * sizeof(int4);
    if (!g.sb_head) {
        void *p = nullptr;
        const size_t bytes = head_bytes + (size_t)pad_words * sizeof(uint32_t);
        if (!got(dev_malloc(&p, bytes))) return false;
        g.extra_allocs.push_back(p);
        g.bytes += bytes;
        g.sb_head = p;
        smem_head_kernel<<<std::min(g.sm_count * 4, (pad_words + 7) / 8), 256, 0, stream>>>(
            g.RT, g.CT, g.n, pad_words, static_cast<int4 *>(p),
            reinterpret_cast<uint32_t *>(static_cast<char *>(p) + head_bytes));
        GU_CUDA_CHECK(cudaGetLastError());
    }
    SbArgs a;
    a.R = g.R;
    a.C = g.C;
    a.RT = g.RT;
    a.CT = g.CT;
    a.n = g.n;
    a.m = g.m;
    a.sources = sources;
    a.k = k;
    a.dist = dist;
    a.ld = ld;
    a.reach = reach;
    a.head = static_cast<const int4 *>(g.sb_head);
    a.none = reinterpret_cast<const uint32_t *>(static_cast<const char *>(g.sb_head) + head_bytes);
    a.slice = c.slice;
    a.live = g.nlight + g.nmid + g.nwide + g.nheavy;
    // The first in-neighbours are the hubs, so a skewed graph needs fewer tries.  Call times
    // in us, alpha 0.4 / 0.55 / 0.7 / 1: R-MAT 14 k = 150 74 / 77 / 79 / 80, R-MAT 18 (ef 10)
    // k = 4 90 / 90 / 104 / 106, R-MAT 15 k = 120 91 / 92 / 92 / 110; ER 100000 (24 entries a
    // vertex) k = 8 105 / 98 / 86 / 86, k = 20 152 / 146 / 137 / 119.  (Frontier edges x 8 >
    // m, the batched engine's form of the rule: ER 2000, k = 64 42, R-MAT 14 k = 150 73, but
    // ER 100000, k = 20 146 and ER 8000 with 1000 entries a vertex, k = 1024 1758, 280 now.)
    // Of a directed graph part of what is left may be out of reach, and its lists are tried in
    // vain: DAG 20000 (60 entries a vertex) k = 100, alpha 1 / 4 417 / 325 us, DAG 16000 (40)
    // k = 300 387 / 283; random directed graph of 30000 (24) k = 100 104 / 117.
    const bool skewed = (double)g.max_in_degree * a.live > 8.0 * (double)g.m;
    a.alpha = skewed ? 0.5f : g.directed ? 2.f : 1.f;
    a.beta = 24.f;
    a.status = static_cast<SbStatus *>(g.sb_status);
    const int nclusters = std::min(std::min(k, c.resident), SB_MAX_CLUSTERS);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c.S;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nclusters * c.S));
    cfg.blockDim = dim3((unsigned)c.threads);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = c.S > 1 ? 1 : 0;
    void *params[] = {&a};
    g.timeline = 2;
    g.sb_clusters = nclusters;
    g.mark_start(stream);
    GU_CUDA_CHECK(cudaLaunchKernelExC(&cfg, sb_kernel(c.mode), params));
    g.mark_stop(stream);
    GU_CUDA_CHECK(cudaStreamSynchronize(stream));
    int err = 0;
    for (int i = 0; i < nclusters; ++i) err = std::max(err, (int)a.status[i].err);
    if (err == DEV_ERR_BAD_SOURCE) throw gu_error(GU_ERR_INVALID_ARGUMENT, "source vertex out of range");
    if (max_level) smem_bfs_stats(g, nullptr, nullptr, max_level);
    return err == 0;
}

// Levels of the last launch: the most any cluster ran, and the deepest level.
void smem_bfs_stats(const DeviceGraph &g, int *td_levels, int *bu_levels, int *max_level)
{
    const SbStatus *st = static_cast<const SbStatus *>(g.sb_status);
    int td = 0, bu = 0, ml = 0;
    for (int i = 0; i < g.sb_clusters; ++i) {
        td = std::max(td, (int)st[i].td_levels);
        bu = std::max(bu, (int)st[i].bu_levels);
        ml = std::max(ml, (int)st[i].max_level);
    }
    if (td_levels) *td_levels = td;
    if (bu_levels) *bu_levels = bu;
    if (max_level) *max_level = ml;
}

}  // namespace gu
