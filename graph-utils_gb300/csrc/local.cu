// local.cu -- per-source BFS for low-degree (mesh-like, high-diameter) graphs,
// and AUTO's choice between the search engines.
//
// The batched bit-matrix engine shares a level among 64 W sources, which pays off
// when the sources' frontiers overlap (small-world graphs reach most vertices in a
// handful of levels).  On meshes (a 2048 x 2048 grid has a diameter near 4000)
// every source reaches a vertex at a different level, the union frontier holds
// each vertex once per distinct level, and every visit moves whole source words.
// There the reference's own decomposition -- one CTA per source, level-
// synchronous (multi_search/shuffle_based.cuh:81-286, the atomicCAS visit of
// multi_search/linear_with_atomics.cu:130) -- is the right one, provided a level
// costs little: here the level queues and a table of the vertices claimed lately
// live in shared memory, a thread expands the whole adjacency list of a low-degree
// vertex with four claims in flight, and appends are warp-aggregated shared
// atomics.  A frontier larger than the shared queue ends the launch with a flag and
// the caller reruns the search on the batched engine.  Rows mode claims vertices in the
// distance row itself; the counting modes (diameter, reachability) claim them in a
// per-CTA visited bitmap and write no rows.
//
// The adjacency is read from a padded copy (ELL: the neighbours of v in CSR
// order at v * width, width 4, 8 or 16, padded with -1), built on the graph's
// first per-source search: one 16-byte load brings a grid vertex's whole list,
// where the CSR form needs the offsets first and then a second, dependent load.
// With a few hundred sources' frontiers spread over the graph the adjacency does
// not stay in L2, so the halved sector count matters as much as the shorter
// chain.
#include "device_utils.cuh"
#include "gu_internal.h"
#include "kernel_fit.h"
#include "recent.h"

#include <algorithm>
#include <climits>
#include <cstdlib>

namespace gu {

// One 1024-thread CTA per source, two per SM: 256 sources fill the GPU, and a
// level's frontier (a few thousand vertices on a 2048 x 2048 mesh) takes one or
// two dependent load chains per thread (768 threads 38.6 ms, 512 44.0 ms against 37.1
// on that grid with 256 sources, rows).
constexpr int LOCAL_THREADS = 1024;
// Vertices of two consecutive levels in local_bfs_kernel's ring.  Shared memory the
// queues do not use is L1, and lines in flight there are what a wide level waits for:
// 32 KiB of queues 35.0 ms, 40 KiB 37.3, 48 KiB 37.1, 70 KiB 83 (the grid above).  A
// search that overflows the small ring runs again with the wide one, and so does every
// later search of that graph; one that overflows that as well goes back to the caller.
constexpr int LOCAL_RING = 8192, LOCAL_WIDE_RING = 12288;

struct LocalArgs {
    const int4 *__restrict__ ell;  // [n][width / 4]
    int32_t n;
    const int32_t *sources;
    int32_t k;
    int32_t *dist;  // rows mode: k x ld
    int64_t ld;
    uint32_t *vis;  // counting modes: [gridDim.x][vis_words]
    int64_t vis_words;
    unsigned long long *reach;  // counting: per-source reachable count (null: none)
    int *max_level;             // atomicMax of the deepest level reached (null: none)
    int *overflow;              // set when a frontier exceeds the queue
    int ring;                   // entries of local_bfs_kernel's ring
    bool alone;                 // one CTA per SM: local_bfs_kernel keeps adjacency pieces in L1
};

__global__ void build_ell_kernel(const int32_t *__restrict__ R, const int32_t *__restrict__ C, int32_t n, int width,
                                 int32_t *__restrict__ ell)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)n * width;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)(i / width), t = (int32_t)(i % width);
        const int32_t e = __ldg(R + v) + t;
        ell[i] = e < __ldg(R + v + 1) ? __ldg(C + e) : -1;
    }
}

// Vertices claimed lately by the CTA's search: a direct-mapped table of 16-bit tags in
// shared memory.  The hash is a bijection of the ids below 2^30, slot its upper and tag
// its lower bits, so a tag that matches is this vertex and no other; a tag that was
// overwritten only sends the vertex to the global claim again, and an id from 2^30 up
// always goes there.  A mesh vertex's
// neighbours lie on the levels before and after its own, so nearly all that are
// claimed already were claimed within two levels and are found here: a shared-memory
// read whose lanes meet a few bank conflicts, where a read of the distance row or the
// bitmap is a line of its own for every lane (2048 x 2048 grid, 256 sources: rows 40.6 ->
// 37.1 ms, counts 34.9 -> 30.2; 2^13 slots 37.6, 2^12 42).
// (The constants and the hash: recent.h.)

// A piece of an adjacency row, kept out of L1: every lane reads another line, and with
// two CTAs on an SM lines in flight that fill the L1 hold up the claims (2048 x 2048
// grid, 256 sources: 35.0 -> 34.2 ms; with 8 KiB more shared memory, so less L1, 37.1).
// A CTA alone on its SM keeps them: a line's other vertices come up on the next levels
// (1024 x 1024, 64 sources, counts 6.4 ms past L1, 6.2 through it).
__device__ __forceinline__ int4 ld_row(const int4 *p)
{
    int4 q;
    asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "l"(p));
    return q;
}

// Wide levels: bound by the SM's rate of scattered accesses (2048 x 2048 grid, 256
// sources, depth 4013: rows 34.9 ms, counts 28.0; 40.6 and 34.9 without the table of
// recent claims and with a wider queue).
template <bool ROWS, int WIDTH>
__global__ void __launch_bounds__(LOCAL_THREADS, 2) local_bfs_kernel(LocalArgs a)
{
    extern __shared__ int32_t sq[];  // [a.ring] ring of two levels, then recent
    uint16_t *recent = reinterpret_cast<uint16_t *>(sq + a.ring);
    __shared__ int s_len[2];
    __shared__ int s_stop;
    uint32_t *vis = ROWS ? nullptr : a.vis + (size_t)blockIdx.x * a.vis_words;
    const int lane = lane_id();
    auto wrap = [&](int i) { return i < a.ring ? i : i - a.ring; };
    for (int si = blockIdx.x; si < a.k; si += gridDim.x) {
        if (threadIdx.x == 0) s_stop = ld_volatile_i32(a.overflow);  // another CTA overflowed: the caller reruns
        __syncthreads();
        if (s_stop) return;
        const int32_t src = __ldg(a.sources + si);
        int32_t *d = ROWS ? a.dist + (int64_t)si * a.ld : nullptr;
        if (ROWS) {
            for (int32_t v = threadIdx.x; v < a.n; v += blockDim.x) d[v] = (v == src) ? 0 : INT_MAX;
        } else {
            for (int64_t w = threadIdx.x; w < a.vis_words; w += blockDim.x)
                vis[w] = (w == (src >> 5)) ? (1u << (src & 31)) : 0u;
        }
        for (int i = threadIdx.x; i < RECENT_SLOTS / 2; i += blockDim.x)
            reinterpret_cast<uint32_t *>(recent)[i] = 0x10001u * RECENT_EMPTY;
        __syncthreads();
        if (threadIdx.x == 0) {
            sq[0] = src;
            s_len[0] = 1;
            s_len[1] = 0;
            const uint32_t h = recent_hash(src);
            recent[h >> 16] = (uint16_t)h;
        }
        __syncthreads();
        int cur = 0, head = 0, level = 0, maxl = 0;
        long long reached = 1;
        while (true) {
            const int qlen = s_len[cur];
            if (qlen == 0) break;
            maxl = level;
            // this level's vertices are entries [head, head + qlen) of the ring, the next
            // level's follow
            const int tail = head + qlen < a.ring ? head + qlen : head + qlen - a.ring;
            int *nlen = &s_len[cur ^ 1];
            for (int i0 = threadIdx.x - lane; i0 < qlen; i0 += blockDim.x) {  // warp-uniform
                const bool on = i0 + lane < qlen;
                const int4 *row = a.ell + (size_t)(on ? sq[wrap(head + i0 + lane)] : 0) * (WIDTH / 4);
                bool go = on;
#pragma unroll
                for (int c = 0; c < WIDTH / 4; ++c) {
                    const int4 q4 = go ? (a.alone ? __ldg(row + c) : ld_row(row + c)) : make_int4(-1, -1, -1, -1);
                    const int32_t w[4] = {q4.x, q4.y, q4.z, q4.w};
                    go = w[0] >= 0;  // padding: the list ended
                    if (!__any_sync(FULL_MASK, go)) break;
                    bool ok[4];
                    uint32_t h[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        h[t] = recent_hash(w[t]);
                        ok[t] = w[t] >= 0 && ((uint16_t)h[t] == RECENT_EMPTY || recent[h[t] >> 16] != (uint16_t)h[t]);
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t) {  // four claims in flight
                        if (!ok[t]) continue;
                        if (ROWS) {
                            ok[t] = atomicCAS(d + w[t], INT_MAX, level + 1) == INT_MAX;
                        } else {
                            const uint32_t bit = 1u << (w[t] & 31);
                            ok[t] = !(atomicOr(vis + (w[t] >> 5), bit) & bit);
                        }
                        // claimed now or before: either way it need not be asked for again
                        recent[h[t] >> 16] = (uint16_t)h[t];
                    }
                    unsigned m[4];
                    int cnt = 0;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        m[t] = __ballot_sync(FULL_MASK, ok[t]);
                        cnt += __popc(m[t]);
                    }
                    if (!cnt) continue;
                    int pos = 0;
                    if (lane == 0) pos = atomicAdd(nlen, cnt);
                    pos = __shfl_sync(FULL_MASK, pos, 0);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int at = pos + __popc(m[t] & ((1u << lane) - 1u));
                        if (ok[t] && at < a.ring - qlen) sq[wrap(tail + at)] = w[t];
                        pos += __popc(m[t]);
                    }
                }
            }
            __syncthreads();
            const int nl = *nlen;
            if (nl > a.ring - qlen) {  // two levels too large for the ring: hand back to the caller
                if (threadIdx.x == 0) atomicExch(a.overflow, 1);
                return;
            }
            reached += nl;
            if (threadIdx.x == 0) s_len[cur] = 0;  // the queue just read is the next level's target
            cur ^= 1;
            head = tail;
            ++level;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            if (a.reach) a.reach[si] = (unsigned long long)reached;
            if (a.max_level) atomicMax(a.max_level, maxl);
        }
        __syncthreads();  // shared queues reused by the next source
    }
}

// ---- out-degree up to four ---------------------------------------------------------
// Searches whose levels are mostly narrow are bound by a level's dependent chain.  Up to
// MESH_NARROW vertices the queue holds the frontier's adjacency rows themselves (int4),
// fetched while their claims are in flight, so that the chain is: row from shared memory
// -> recent table -> claim -> barrier.  A slot is reserved as soon as the table lets a
// vertex through, the row is copied there asynchronously and struck out if the claim
// fails (a vertex visited earlier whose entry was overwritten).  The exchange on the
// table also settles which of a vertex's parents on this level asks first, so nearly
// every claim succeeds.  Wider levels, bound by the rate of scattered accesses, queue ids
// after the claims and only read the table.  Rows, before -> now: 512 x 512 grid, 64
// sources 3.21 -> 1.81 ms (local_bfs_kernel: 2.42); 128 x 2000, 64 sources 6.43 -> 3.13
// (4.80); 90 x 90, 256 sources 0.53 -> 0.27 (0.40).
constexpr int MESH_ROWS = 1536;                 // rows per shared queue (two: 48 KiB)
constexpr int MESH_QCAP = 4 * MESH_ROWS;        // ids in the same space; wider levels go back to the caller
constexpr int MESH_NARROW = MESH_ROWS / 4;      // every neighbour reserved: no overflow of the rows
constexpr int MESH_RECENT_BITS = 12;
// Meshes on which two CTAs share an SM and most levels are wide take local_bfs_kernel.
// Rows, here / there: 1024 x 1024 grid, 1 / 64 / 256 sources 4.8 / 5.6 / 8.4 ms and 6.0 /
// 7.6 / 9.2; 876 x 1763, 64 / 256 sources 7.5 / 11.6 and 10.2 / 13.3; 2048 x 2048, 64 /
// 150 / 256 sources 20.3 / 22.0 / 40.6 and 23.2 / 25.7 / 35.7.  Counts, where a claim is
// in a small bitmap and the chain is shorter: 600 x 1000, 1 / 64 / 256 sources 3.6 / 3.7 /
// 5.2 and 3.4 / 4.2 / 5.0; 863 x 642 2.9 / 3.4 / 4.7 and 3.2 / 4.2 / 4.7; 1024 x 1024 6.7
// / 6.8 / 9.7 and 5.7 / 6.2 / 7.5.  (A long narrow mesh of this size would do better here:
// 300 x 6000, 64 sources, counts 12.2 and 17.6.)
constexpr int MESH_MAX_N_SHARED = 1 << 21, MESH_MAX_N_COUNT = 5 << 17;
static bool mesh_form(const DeviceGraph &g, int32_t k, bool rows)
{
    if (g.ell_width != LOCAL_MESH_DEGREE) return false;
    return rows ? k <= g.sm_count || g.n <= MESH_MAX_N_SHARED : g.n <= MESH_MAX_N_COUNT;
}
constexpr size_t MESH_SMEM = 2 * MESH_ROWS * sizeof(int4) + sizeof(int32_t) * (1 << MESH_RECENT_BITS);

__device__ __forceinline__ void copy16_async(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <bool ROWS>
__global__ void __launch_bounds__(LOCAL_THREADS, 2) mesh_bfs_kernel(LocalArgs a)
{
    extern __shared__ __align__(16) int4 mq[];  // [2][MESH_ROWS] rows or [2][MESH_QCAP] ids, then the recent table
    int32_t *recent = reinterpret_cast<int32_t *>(mq + 2 * MESH_ROWS);
    __shared__ int s_len[3];
    __shared__ int s_stop;
    __shared__ unsigned s_reached;
    uint32_t *vis = ROWS ? nullptr : a.vis + (size_t)blockIdx.x * a.vis_words;
    const int lane = lane_id();
    const int4 none = make_int4(-1, -1, -1, -1);
    auto slot_of = [](int32_t v) { return ((uint32_t)v * 0x9E3779B1u) >> (32 - MESH_RECENT_BITS); };
    for (int si = blockIdx.x; si < a.k; si += gridDim.x) {
        if (threadIdx.x == 0) s_stop = ld_volatile_i32(a.overflow);  // another CTA overflowed: the caller reruns
        __syncthreads();
        if (s_stop) return;
        const int32_t src = __ldg(a.sources + si);
        int32_t *d = ROWS ? a.dist + (int64_t)si * a.ld : nullptr;
        if (ROWS) {
            for (int32_t v = threadIdx.x; v < a.n; v += LOCAL_THREADS) d[v] = (v == src) ? 0 : INT_MAX;
        } else {
            for (int64_t w = threadIdx.x; w < a.vis_words; w += LOCAL_THREADS)
                vis[w] = (w == (src >> 5)) ? (1u << (src & 31)) : 0u;
        }
        for (int i = threadIdx.x; i < (1 << MESH_RECENT_BITS); i += LOCAL_THREADS) recent[i] = -1;
        __syncthreads();
        if (threadIdx.x == 0) {
            mq[0] = __ldg(a.ell + src);
            s_len[0] = 1;
            s_len[1] = 0;
            s_reached = 1;
            recent[slot_of(src)] = src;
        }
        __syncthreads();
        int cur = 0, li = 0, level = 0;
        bool as_rows = true;  // the frontier is queued as rows
        unsigned reached = 0;
        while (true) {
            const int qlen = s_len[li];
            if (qlen > MESH_QCAP) {  // too wide for the queue: hand back to the caller
                if (threadIdx.x == 0) atomicExch(a.overflow, 1);
                return;
            }
            const int ln = li == 2 ? 0 : li + 1;
            if (threadIdx.x == 0) s_len[ln == 2 ? 0 : ln + 1] = 0;  // collects the level after the next
            const int4 *rows = mq + cur * MESH_ROWS;
            int4 *rows2 = mq + (cur ^ 1) * MESH_ROWS;
            const int32_t *ids = reinterpret_cast<const int32_t *>(rows);
            int32_t *ids2 = reinterpret_cast<int32_t *>(rows2);
            const bool narrow = qlen <= MESH_NARROW;
            bool any = false;
            for (int i0 = threadIdx.x - lane; i0 < qlen; i0 += LOCAL_THREADS) {  // warp-uniform
                const int i = i0 + lane;
                const int4 q4 = i >= qlen ? none : as_rows ? rows[i] : ld_row(a.ell + ids[i]);
                const int32_t w[4] = {q4.x, q4.y, q4.z, q4.w};
                unsigned ok = 0, won = 0;  // bit t: neighbour t goes to the claim, is claimed
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (w[t] < 0) continue;
                    int32_t *r = recent + slot_of(w[t]);
                    if ((narrow ? atomicExch(r, w[t]) : *r) != w[t]) ok |= 1u << t;
                }
                if (!__any_sync(FULL_MASK, ok)) continue;
                int32_t old[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {  // four claims in flight
                    if (!((ok >> t) & 1u)) continue;
                    if (ROWS) old[t] = atomicCAS(d + w[t], INT_MAX, level + 1);
                    else old[t] = (int32_t)atomicOr(vis + (w[t] >> 5), 1u << (w[t] & 31));
                    if (!narrow) recent[slot_of(w[t])] = w[t];  // claimed now or before
                }
                auto results = [&] {
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (((ok >> t) & 1u) && (ROWS ? old[t] == INT_MAX : !(((uint32_t)old[t] >> (w[t] & 31)) & 1u)))
                            won |= 1u << t;
                };
                auto reserve = [&](unsigned take) {  // this lane's first slot
                    unsigned below = 0, total = 0;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const unsigned m = __ballot_sync(FULL_MASK, (take >> t) & 1u);
                        below += __popc(m & ((1u << lane) - 1u));
                        total += __popc(m);
                    }
                    int pos = 0;
                    if (lane == 0 && total) pos = atomicAdd(&s_len[ln], (int)total);
                    return __shfl_sync(FULL_MASK, pos, 0) + (int)below;
                };
                if (narrow) {
                    const int pos = reserve(ok);
                    int at = pos;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if ((ok >> t) & 1u) copy16_async(rows2 + at++, a.ell + w[t]);
                    results();
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    at = pos;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if ((ok >> t) & 1u) {
                            if (!((won >> t) & 1u)) rows2[at] = none;
                            ++at;
                        }
                } else {
                    results();
                    int at = reserve(won);
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if ((won >> t) & 1u) {
                            if (at < MESH_QCAP) ids2[at] = w[t];
                            ++at;
                        }
                }
                reached += __popc(won);
                any |= won != 0;
            }
            if (!__syncthreads_or(any)) break;
            cur ^= 1;
            li = ln;
            as_rows = narrow;
            ++level;
        }
        reached = __reduce_add_sync(FULL_MASK, reached);
        if (lane == 0 && reached) atomicAdd(&s_reached, reached);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (a.reach) a.reach[si] = (unsigned long long)s_reached;
            if (a.max_level) atomicMax(a.max_level, level);
        }
        __syncthreads();  // the shared state is reused by the next source
    }
}

// AUTO's choice where the shared-memory engine (smem.cu) does not apply: the
// per-source engine for low-degree graphs (its thread-per-vertex expansion wants
// short adjacency lists), the batched bit-matrix engine otherwise.
// GU_AUTO_LOCAL=0 in the environment keeps AUTO on the batched engine (tests use
// it to cover every engine on the same graphs).
AutoEngine auto_engine(const DeviceGraph &g)
{
    const char *e = std::getenv("GU_AUTO_LOCAL");
    if (e && e[0] == '0') return AutoEngine::BATCHED;
    return g.max_degree <= LOCAL_MAX_DEGREE ? AutoEngine::LOCAL : AutoEngine::BATCHED;
}

// Returns false if a frontier overflowed the shared queues (the caller reruns the
// search on the batched engine).  Synchronises `stream`.
bool launch_local_bfs(DeviceGraph &g, const int32_t *sources, int32_t k, int32_t *dist, int64_t ld,
                      unsigned long long *reach, int *max_level_host, cudaStream_t stream)
{
    if (!g.ell) {  // the padded adjacency, once per graph
        const int width = g.max_degree <= 4 ? 4 : g.max_degree <= 8 ? 8 : 16;
        if (g.max_degree > 16) throw gu_error(GU_ERR_INTERNAL, "per-source engine on a graph of out-degree > 16");
        const size_t bytes = (size_t)(g.n > 0 ? g.n : 1) * width * sizeof(int32_t);
        GU_CUDA_CHECK(dev_malloc((void **)&g.ell, bytes));
        g.extra_allocs.push_back(g.ell);
        g.bytes += bytes;
        g.ell_width = width;
        const int64_t total = (int64_t)g.n * width;
        const int blocks = (int)std::min<int64_t>((total + 255) / 256, (int64_t)g.sm_count * 8);
        if (total > 0) build_ell_kernel<<<blocks > 0 ? blocks : 1, 256, 0, stream>>>(g.R, g.C, g.n, width, g.ell);
        GU_CUDA_CHECK(cudaGetLastError());
    }
    const bool rows = dist != nullptr;
    const int wi = g.ell_width == 8 ? 1 : g.ell_width == 16 ? 2 : mesh_form(g, k, rows) ? 3 : 0;
    const bool mesh = wi == 3;
    void (*const kerns[2][4])(LocalArgs) = {{local_bfs_kernel<false, 4>, local_bfs_kernel<false, 8>,
                                             local_bfs_kernel<false, 16>, mesh_bfs_kernel<false>},
                                            {local_bfs_kernel<true, 4>, local_bfs_kernel<true, 8>,
                                             local_bfs_kernel<true, 16>, mesh_bfs_kernel<true>}};
    auto kern = kerns[rows][wi];
    auto smem_for = [&](int ring) { return mesh ? MESH_SMEM : ring * sizeof(int32_t) + RECENT_SLOTS * sizeof(uint16_t); };
    const int ring = g.local_wide ? LOCAL_WIDE_RING : LOCAL_RING;
    const size_t smem = smem_for(ring);
    const int per_sm = kernel_fit(g.device, (const void *)kern, LOCAL_THREADS, smem, smem_for(LOCAL_WIDE_RING));
    if (per_sm < 1) throw gu_error(GU_ERR_INTERNAL, "per-source BFS kernel cannot be resident");
    int grid = g.sm_count * per_sm;
    if (grid > k) grid = k;
    const int64_t vis_words = rows ? 0 : ((int64_t)g.n + 31) / 32;
    const size_t need = WS_CONTROL_BYTES + (size_t)grid * (size_t)vis_words * sizeof(uint32_t);
    char *ws = (char *)g.ws.get(need);
    GU_CUDA_CHECK(cudaMemsetAsync(ws, 0, 64, stream));
    LocalArgs a;
    a.ell = reinterpret_cast<const int4 *>(g.ell);
    a.n = g.n;
    a.sources = sources;
    a.k = k;
    a.dist = dist;
    a.ld = ld;
    a.vis = reinterpret_cast<uint32_t *>(ws + WS_CONTROL_BYTES);
    a.vis_words = vis_words;
    a.reach = reach;
    a.max_level = reinterpret_cast<int *>(ws);
    a.overflow = reinterpret_cast<int *>(ws) + 1;
    a.ring = ring;
    a.alone = grid <= g.sm_count;
    g.timeline = 0;
    g.mark_start(stream);
    kern<<<grid, LOCAL_THREADS, smem, stream>>>(a);
    GU_CUDA_CHECK(cudaGetLastError());
    g.mark_stop(stream);
    int flags[2] = {0, 0};
    GU_CUDA_CHECK(cudaMemcpyAsync(flags, ws, sizeof(flags), cudaMemcpyDeviceToHost, stream));
    GU_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (max_level_host) *max_level_host = flags[0];
    if (flags[1] != 0 && !mesh && !g.local_wide) {  // once more, and from now on, with the wider ring
        g.local_wide = true;
        return launch_local_bfs(g, sources, k, dist, ld, reach, max_level_host, stream);
    }
    return flags[1] == 0;
}

}  // namespace gu
