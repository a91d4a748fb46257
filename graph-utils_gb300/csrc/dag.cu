// dag.cu -- reachable sets of every vertex of a DAG (the all-roots closure of
// graph-utils/dag_reachability.cpp:36-65), as per-vertex set sizes.
//
// The reference recurses from the roots with a std::set per vertex, each set the
// union of its successors' sets.  The same recurrence runs here on bit rows, level
// by level of the longest path to a sink: the row of a vertex is the OR of its
// successors' rows and its own bit, and its set size is the row's population count
// less one.  Rows are indexed by topological position in both directions, so the
// row of position p ends at bit p and a closure of n vertices moves about
// m n / 24 bytes of rows (successors of a random DAG sit at a third of n on
// average) instead of the m n / 8 of full rows.
//
// A multi-source search from every vertex (256 sources per batch, one pass over
// the graph per batch and level) is the form for a directed graph with a cycle.
#include "device_utils.cuh"
#include "gu_internal.h"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <string>

namespace gu {

constexpr int TOPO_THREADS = 512;
constexpr int TOPO_MIN_BLOCKS = 3;
constexpr int64_t TOPO_MAX_N = (int64_t)1 << 26;  // positions fit the packed append counter
constexpr int CLOSURE_CHUNK = 4096;               // columns per warp step: 16 bytes per lane
// Reachable counts by levels of the order: up to this many levels (about 3.5 us each;
// a search takes about 10 us a level of its own, of which it may have far fewer), and
// lists short enough for eight lanes.
constexpr int REACH_MAX_LEVELS = 96;
constexpr int32_t REACH_MAX_IN_DEGREE = 2048;
constexpr int REACH_LEVEL_VERTICES = 1000;  // vertices per level at least, where out-degrees are low
// Rows kept at once: the closure runs in column blocks of at most this many bytes
// of rows (n = 65536 fits one block; a block costs one pass over the levels, about
// 3 us each, so narrower blocks that would stay in L2 cost more than they save).
constexpr size_t CLOSURE_ROWS_BYTES = (size_t)512 << 20;

// The first words match the batched engine's control block (barrier, error), so
// that the launch statistics read after a closure show no levels.
struct TopoCtl {
    unsigned bar;
    int err;
    int pad[4];
    int nlevels, total;
    u64 pack[4];  // appended vertices of a level, (count << 38) | out-edges
    u64 ins[4];   // ... and their in-edges
    int top;      // reach_kernel: highest level of the batch's sources
    int deep;     // topo_plan_kernel stopped at its level limit
};
constexpr int TOPO_PACK = 38;

struct TopoArgs {
    const int32_t *__restrict__ R;
    const int32_t *__restrict__ C;
    const int32_t *__restrict__ RT;
    const int32_t *__restrict__ CT;
    int32_t n;
    int64_t m;
    int32_t *cnt;  // successors not yet placed
    int2 *in;      // in-list ends (RT) by position
    int32_t *pos;  // position of a vertex (kept)
    int32_t *order, *lvl, *PR, *PC, *IC;
    int2 *IR;
    TopoCtl *ctl;
    unsigned long long wait_ns;
    int max_levels;  // an order of more is not completed
};

// All lanes of the warp call it; lanes with pred place their vertex (out-degree deg,
// in-list ends in) at the end of the level being collected: one 64-bit atomic per warp
// reserves the positions and the out-edge range, another, by a second lane at once, the
// in-edge range.  (In-edge ranges are then not in position order: both ends are kept.)
__device__ __forceinline__ void topo_place(const TopoArgs &a, int slot, long long base_p, long long base_e, long long base_i,
                                           bool pred, int32_t v, unsigned deg, int2 in)
{
    const unsigned mask = __ballot_sync(FULL_MASK, pred);
    if (!mask) return;
    const int lane = lane_id();
    const unsigned ind = pred ? (unsigned)(in.y - in.x) : 0u;
    if (!pred) deg = 0;
    unsigned inc = deg, inci = ind;  // (sums over distinct vertices: at most m)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(FULL_MASK, inc, o), z = __shfl_up_sync(FULL_MASK, inci, o);
        if (lane >= o) {
            inc += y;
            inci += z;
        }
    }
    const unsigned toti = __shfl_sync(FULL_MASK, inci, 31);
    u64 r = 0;
    if (lane == 31) r = atomicAdd(&a.ctl->pack[slot], ((u64)__popc(mask) << TOPO_PACK) | inc);
    if (lane == 30) r = atomicAdd(&a.ctl->ins[slot], (u64)toti);
    const u64 old = __shfl_sync(FULL_MASK, r, 31), oldi = __shfl_sync(FULL_MASK, r, 30);
    if (pred) {
        const int32_t p = (int32_t)(base_p + (long long)(old >> TOPO_PACK) + __popc(mask & ((1u << lane) - 1u)));
        a.order[p] = v;
        a.pos[v] = p;
        a.PR[p] = (int32_t)(base_e + (long long)(old & ((1ull << TOPO_PACK) - 1ull)) + (long long)(inc - deg));
        const int32_t i0 = (int32_t)(base_i + (long long)oldi + (long long)(inci - ind));
        a.IR[p] = make_int2(i0, i0 + (int32_t)ind);
        a.in[p] = in;
    }
}

// Levels by removing sinks: level 0 holds the vertices without successors, level
// j + 1 those whose last successor was placed in level j.  A vertex on a cycle is
// never placed (total < n).  The order inside a level depends on scheduling; no
// result does.
__global__ void __launch_bounds__(TOPO_THREADS, TOPO_MIN_BLOCKS) topo_plan_kernel(TopoArgs a)
{
    __shared__ u64 s_pack[8];  // pack and ins
    unsigned epoch = 0;
    TopoCtl *ctl = a.ctl;
    auto barrier = [&] { return grid_barrier(&ctl->bar, &ctl->err, epoch, a.wait_ns, ctl->pack, s_pack, 8); };
    const long long rank = (long long)blockIdx.x * blockDim.x + threadIdx.x, size = (long long)gridDim.x * blockDim.x;
    const long long ngrp = size >> 3;
    const int sub = lane_id() & 7;
    for (long long b = rank & ~31ll; b < a.n; b += size) {  // warp-uniform
        const long long v = b + lane_id();
        int32_t d = 1;
        int2 in = make_int2(0, 0);
        if (v < a.n) {
            d = __ldg(a.R + v + 1) - __ldg(a.R + v);
            in = make_int2(__ldg(a.RT + v), __ldg(a.RT + v + 1));
            a.cnt[v] = d;
        }
        topo_place(a, 0, 0, 0, 0, d == 0, (int32_t)v, 0, in);
    }
    if (!barrier()) return;
    long long ls = 0, ebase = 0, ibase = 0;
    int level = 0;
    for (;; ++level) {
        const u64 pk = s_pack[level & 3];
        const long long le = ls + (long long)(pk >> TOPO_PACK);
        if (le == ls) break;
        if (level == a.max_levels) {
            if (rank == 0) ctl->deep = 1;
            return;
        }
        const long long enext = ebase + (long long)(pk & ((1ull << TOPO_PACK) - 1ull));
        const long long inext = ibase + (long long)s_pack[4 + (level & 3)];
        if (rank == 0) {
            a.lvl[level] = (int32_t)ls;
            ctl->ins[(level + 2) & 3] = 0;
            ctl->pack[(level + 2) & 3] = 0;  // collects level + 2; last read two levels ago
        }
        // eight lanes per vertex of the level, their in-lists' ends kept when it was placed
        for (long long p0 = ls + (rank >> 5) * 4; p0 < le; p0 += ngrp) {  // warp-uniform
            const long long p = p0 + (lane_id() >> 3);
            const int2 r = p < le ? __ldcg(a.in + p) : make_int2(0, 0);
            for (int32_t e = r.x + sub; __any_sync(FULL_MASK, e < r.y); e += 8) {
                int32_t u = 0;
                bool last = false;
                int2 in = make_int2(0, 0);
                unsigned d = 0;
                if (e < r.y) {
                    u = __ldg(a.CT + e);
                    // (the degrees in case it is placed, with the decrement and not after it)
                    d = (unsigned)(__ldg(a.R + u + 1) - __ldg(a.R + u));
                    in = make_int2(__ldg(a.RT + u), __ldg(a.RT + u + 1));
                    last = atomicSub(a.cnt + u, 1) == 1;
                }
                topo_place(a, (level + 1) & 3, le, enext, inext, last, u, d, in);
            }
        }
        if (!barrier()) return;
        ls = le;
        ebase = enext;
        ibase = inext;
    }
    if (rank == 0) {
        a.lvl[level] = (int32_t)ls;
        ctl->nlevels = level;
        ctl->total = (int)ls;
    }
    if (ls != a.n) return;
    if (rank == 0) a.PR[a.n] = (int32_t)a.m;
    // neighbours in position space, eight lanes per vertex
    for (long long p = rank >> 3; p < a.n; p += size >> 3) {
        const int32_t v = __ldcg(a.order + p);
        const int32_t e0 = __ldg(a.R + v), d = __ldg(a.R + v + 1) - e0, o = __ldcg(a.PR + p);
        for (int32_t i = sub; i < d; i += 8) a.PC[o + i] = __ldcg(a.pos + __ldg(a.C + e0 + i));
        const int32_t f0 = __ldg(a.RT + v);
        const int2 r = __ldcg(a.IR + p);
        for (int32_t i = sub; i < r.y - r.x; i += 8) a.IC[r.x + i] = __ldcg(a.pos + __ldg(a.CT + f0 + i));
    }
}

struct ClosureArgs {
    const int32_t *__restrict__ order;
    const int32_t *__restrict__ lvl;
    const int32_t *__restrict__ PR;
    const int32_t *__restrict__ PC;
    int32_t n, nlevels;
    int64_t block;       // columns per block, a multiple of CLOSURE_CHUNK
    unsigned char *rows;  // [n][block / 8]
    unsigned long long *counts;
    TopoCtl *ctl;
    unsigned long long wait_ns;
};

// One column block after another, and in each the levels from the sinks up, one
// grid barrier per level.  A warp takes (position, 4096-column chunk): it ORs the
// chunk of every successor whose row reaches it, four 512-byte loads in flight,
// adds its own bit, stores the chunk and adds its population to the vertex's count.
// Rows are read through L2 (__ldcg): a row is read by about m / n vertices of
// other SMs, never twice by one warp.  Bound: the row bytes plus the levels'
// barriers.  Random DAG, n = 65536, m = 8 n (45 levels): 0.56 ms per call for
// about 1.5 GB of rows, against 92.8 ms for the search from every vertex.
__global__ void __launch_bounds__(TOPO_THREADS, TOPO_MIN_BLOCKS) closure_kernel(ClosureArgs a)
{
    unsigned epoch = 0;
    TopoCtl *ctl = a.ctl;
    const long long rank = (long long)blockIdx.x * blockDim.x + threadIdx.x, size = (long long)gridDim.x * blockDim.x;
    const long long gw = rank >> 5, nw = size >> 5;
    const int lane = lane_id();
    const size_t stride = (size_t)(a.block / 8);
    for (int64_t c0 = 0; c0 < a.n; c0 += a.block) {
        for (int l = 0; l < a.nlevels; ++l) {
            const int64_t le = __ldg(a.lvl + l + 1);
            if (le <= c0) continue;  // rows that end before the block
            const int64_t ls = max((int64_t)__ldg(a.lvl + l), c0);
            const int64_t maxch = (min(le, c0 + a.block) - c0 + CLOSURE_CHUNK - 1) / CLOSURE_CHUNK;
            for (int64_t u = gw; u < (le - ls) * maxch; u += nw) {
                const int64_t i = u / maxch;
                const int32_t p = (int32_t)(ls + i);
                const int64_t cb = c0 + (u - i * maxch) * CLOSURE_CHUNK;  // the chunk's first column
                if (p < cb) continue;
                const unsigned char *col = a.rows + (cb - c0) / 8 + 16 * lane;
                uint4 acc = make_uint4(0u, 0u, 0u, 0u);
                const int own = (int)(p - cb) - 128 * lane;  // the own bit, in this lane's 128 columns
                if (own >= 0 && own < 128) {
                    const unsigned bit = 1u << (own & 31);
                    if (own < 32) acc.x = bit;
                    else if (own < 64) acc.y = bit;
                    else if (own < 96) acc.z = bit;
                    else acc.w = bit;
                }
                const int32_t e1 = __ldg(a.PR + p + 1);
                for (int32_t eb = __ldg(a.PR + p); eb < e1; eb += 32) {
                    const int32_t q = eb + lane < e1 ? __ldg(a.PC + eb + lane) : -1;
                    unsigned todo = __ballot_sync(FULL_MASK, q >= cb);
                    while (todo) {  // warp-uniform
                        uint4 x[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            x[t] = make_uint4(0u, 0u, 0u, 0u);
                            if (todo) {
                                const int32_t s = __shfl_sync(FULL_MASK, q, __ffs(todo) - 1);
                                todo &= todo - 1;
                                x[t] = __ldcg(reinterpret_cast<const uint4 *>(col + (size_t)(s - c0) * stride));
                            }
                        }
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            acc.x |= x[t].x;
                            acc.y |= x[t].y;
                            acc.z |= x[t].z;
                            acc.w |= x[t].w;
                        }
                    }
                }
                *reinterpret_cast<uint4 *>(const_cast<unsigned char *>(col) + (size_t)(p - c0) * stride) = acc;
                const int pc = __reduce_add_sync(FULL_MASK, __popc(acc.x) + __popc(acc.y) + __popc(acc.z) + __popc(acc.w));
                if (lane == 0 && pc) atomicAdd(a.counts + __ldg(a.order + p), (unsigned long long)pc);
            }
            if (!grid_barrier(&ctl->bar, &ctl->err, epoch, a.wait_ns)) return;
        }
    }
}

// ---- reachable counts of k sources -------------------------------------------------
struct ReachArgs {
    const int32_t *__restrict__ pos;
    const int32_t *__restrict__ lvl;
    const int2 *__restrict__ IR;
    const int32_t *__restrict__ IC;
    int32_t n, nlevels;
    const int32_t *__restrict__ sources;
    int32_t k;
    u64 *rows;  // [n][W] by position: the sources that reach the vertex
    unsigned long long *counts;
    TopoCtl *ctl;
    unsigned long long wait_ns;
};

// Vertices reached by each source of the batch: a thread adds up to 15 of the rows'
// words in bit slices (four 64-bit planes: a count of four bits for each of 64
// sources), the lanes that hold the same word add their slices, and each lane then
// reads its share of the sources' counts.
template <int W>
__device__ void count_rows(const u64 *rows, size_t words, unsigned *s_cnt, long long rank, long long size)
{
    constexpr int PER = 2 * W;  // sources per lane: 64 among the 32 / W lanes of a word
    constexpr int PLANES = W == 1 ? 9 : W == 2 ? 8 : 7;  // 15 words x 32 / W lanes
    const int lane = lane_id();
    unsigned sum[PER] = {};
    for (size_t i0 = 0; i0 < words; i0 += 15 * (size_t)size) {  // warp-uniform
        u64 c[PLANES] = {};
#pragma unroll 5
        for (int j = 0; j < 15; ++j) {
            const size_t i = i0 + (size_t)j * size + rank;
            u64 x = i < words ? __ldcg(rows + i) : 0ull;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const u64 y = c[b] & x;
                c[b] ^= x;
                x = y;
            }
        }
#pragma unroll
        for (int r = 0, o = W; o < 32; ++r, o <<= 1) {
            u64 carry = 0;
#pragma unroll
            for (int b = 0; b < PLANES; ++b) {
                if (b > 4 + r) break;
                const u64 y = __shfl_xor_sync(FULL_MASK, c[b], o), z = c[b] ^ y;
                const u64 s = z ^ carry;
                carry = (c[b] & y) | (z & carry);
                c[b] = s;
            }
        }
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const int bit = (lane / W) * PER + s;
#pragma unroll
            for (int b = 0; b < PLANES; ++b) sum[s] += (unsigned)((c[b] >> bit) & 1ull) << b;
        }
    }
#pragma unroll
    for (int s = 0; s < PER; ++s)
        if (sum[s]) atomicAdd(s_cnt + 64 * (lane % W) + (lane / W) * PER + s, sum[s]);
}

// Levels from the highest source's down: a vertex's row is its own sources' bits and
// the OR of its predecessors' rows, eight lanes per vertex, one grid barrier per level.
// Every vertex is visited once, where the level-synchronous search expands it at each
// distance at which a source first meets it.  The next level's lists are asked for
// before the barrier, so that only the rows are waited for after it.  Bound: the levels'
// chain (rows, barrier), about 2.7 us each.  DAG of 200,003 vertices, m = 8 n, 200
// sources: 151 us (0.19 ms a call), the search 377 us (0.42 ms).
template <int W>
__global__ void __launch_bounds__(TOPO_THREADS, 2) reach_kernel(ReachArgs a)
{
    __shared__ unsigned s_cnt[64 * W];
    __shared__ int s_top;
    unsigned epoch = 0;
    TopoCtl *ctl = a.ctl;
    auto barrier = [&] { return grid_barrier(&ctl->bar, &ctl->err, epoch, a.wait_ns); };
    const long long rank = (long long)blockIdx.x * blockDim.x + threadIdx.x, size = (long long)gridDim.x * blockDim.x;
    const long long grp = rank >> 3, ngrp = size >> 3;
    const int sub = threadIdx.x & 7;
    const size_t words = (size_t)a.n * W;
    for (int32_t row0 = 0; row0 < a.k; row0 += 64 * W) {
        const int nb = min(64 * W, a.k - row0);
        for (size_t i = (size_t)rank; i < words; i += (size_t)size) a.rows[i] = 0ull;
        if (rank == 0) ctl->top = 0;
        if (!barrier()) return;
        if (rank < nb) {
            const int32_t p = __ldg(a.pos + __ldg(a.sources + row0 + rank));
            atomicOr(a.rows + (size_t)p * W + (rank >> 6), 1ull << (rank & 63));
            int lo = 0, hi = a.nlevels - 1;  // the level of position p
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (__ldg(a.lvl + mid) <= p) lo = mid;
                else hi = mid - 1;
            }
            atomicMax(&ctl->top, lo);
        }
        if (!barrier()) return;
        if (threadIdx.x == 0) s_top = ld_volatile_i32(&ctl->top);
        __syncthreads();
        // this group's first vertex of a level: its list's ends and this lane's first entry
        int32_t ls = 0, le = 0, e = 0, e1 = 0, q = 0;
        auto first = [&](int l) {
            ls = __ldg(a.lvl + l);
            le = __ldg(a.lvl + l + 1);
            e = e1 = 0;
            if (ls + grp < le) {
                const int2 r = __ldg(a.IR + ls + grp);
                e = r.x + sub;
                e1 = r.y;
                if (e < e1) q = __ldg(a.IC + e);
            }
        };
        if (s_top > 0) first(s_top - 1);
        for (int l = s_top - 1; l >= 0; --l) {
            for (long long p = ls + grp; __any_sync(FULL_MASK, p < le); p += ngrp) {  // warp-uniform trips
                if (p != ls + grp) {
                    e = e1 = 0;
                    if (p < le) {
                        const int2 r = __ldg(a.IR + p);
                        e = r.x + sub;
                        e1 = r.y;
                        if (e < e1) q = __ldg(a.IC + e);
                    }
                }
                u64 acc[W] = {};
                if (p < le && sub == 0) {  // its own sources
#pragma unroll
                    for (int w = 0; w < W; ++w) acc[w] = __ldcg(a.rows + (size_t)p * W + w);
                }
                while (e < e1) {
                    const int32_t qn = e + 8 < e1 ? __ldg(a.IC + e + 8) : 0;
                    const u64 *r = a.rows + (size_t)q * W;
                    if constexpr (W == 4) {
                        u64 x0, x1, x2, x3;
                        asm volatile("ld.global.cg.v4.u64 {%0, %1, %2, %3}, [%4];"
                                     : "=l"(x0), "=l"(x1), "=l"(x2), "=l"(x3) : "l"(r) : "memory");
                        acc[0] |= x0, acc[1] |= x1, acc[2] |= x2, acc[3] |= x3;
                    } else {
#pragma unroll
                        for (int w = 0; w < W; ++w) acc[w] |= __ldcg(r + w);
                    }
                    q = qn;
                    e += 8;
                }
                u64 any = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) acc[w] |= __shfl_xor_sync(FULL_MASK, acc[w], o);
                    any |= acc[w];
                }
                if (p < le && sub < W && any) {
                    u64 mine = acc[0];
#pragma unroll
                    for (int w = 1; w < W; ++w)
                        if (sub == w) mine = acc[w];
                    a.rows[(size_t)p * W + sub] = mine;
                }
            }
            if (l > 0) first(l - 1);  // static lists: loads in flight across the barrier
            if (!barrier()) return;
        }
        for (int i = threadIdx.x; i < 64 * W; i += blockDim.x) s_cnt[i] = 0;
        __syncthreads();
        count_rows<W>(a.rows, words, s_cnt, rank, size);
        __syncthreads();
        for (int i = threadIdx.x; i < nb; i += blockDim.x)
            if (s_cnt[i]) atomicAdd(a.counts + row0 + i, (unsigned long long)s_cnt[i]);
        if (row0 + 64 * W < a.k && !barrier()) return;  // the rows are cleared for the next batch
    }
}

template <class K>
static int topo_grid(K kern, int sms)
{
    int per_sm = 0;
    GU_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TOPO_THREADS, 0));
    if (per_sm < 1) throw gu_error(GU_ERR_INTERNAL, "topological kernel cannot be resident");
    return sms * per_sm;
}

static void check_topo(const TopoCtl &c)
{
    if (c.err == DEV_ERR_BARRIER_TIMEOUT) throw gu_error(GU_ERR_TIMEOUT, "a device-side wait exceeded its limit");
    if (c.err != 0) throw gu_error(GU_ERR_INTERNAL, "device reported error code " + std::to_string(c.err));
}

// Builds the graph's topological order once (synchronises st); false if the graph has a
// cycle or its order more than max_levels levels.  Only a completed order is kept: what
// is known of the others is their state.  ws_bytes: workspace that the caller takes next
// (allocated at once).
static bool ensure_topo(DeviceGraph &g, int max_levels, size_t ws_bytes, cudaStream_t st)
{
    TopoPlan &t = g.topo;
    if (t.state == TopoPlan::CYCLIC || (t.state == TopoPlan::DEEP && max_levels <= REACH_MAX_LEVELS)) return false;
    if (t.state == TopoPlan::ACYCLIC) return t.nlevels <= max_levels;
    const size_t n = (size_t)g.n, m = (size_t)g.m;
    char *ws = (char *)g.ws.get(std::max(ws_bytes, WS_CONTROL_BYTES + 3 * n * sizeof(int32_t)));
    const size_t ints = 2 * n + 2 * n + (n + 2) + (n + 1) + 2 * m;
    struct Buffer {
        int32_t *p = nullptr;
        ~Buffer()
        {
            if (p) cudaFree(p);
        }
    } buf;
    const cudaError_t e = dev_malloc((void **)&buf.p, ints * sizeof(int32_t));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        throw gu_error(GU_ERR_OUT_OF_MEMORY, "topological order allocation failed");
    }
    TopoArgs a;
    a.R = g.R;
    a.C = g.C;
    a.RT = g.RT;
    a.CT = g.CT;
    a.n = g.n;
    a.m = g.m;
    a.in = reinterpret_cast<int2 *>(ws + WS_CONTROL_BYTES);
    a.cnt = reinterpret_cast<int32_t *>(a.in + n);
    a.IR = reinterpret_cast<int2 *>(buf.p);
    a.order = buf.p + 2 * n;
    a.pos = a.order + n;
    a.lvl = a.pos + n;
    a.PR = a.lvl + n + 2;
    a.PC = a.PR + n + 1;
    a.IC = a.PC + m;
    a.ctl = reinterpret_cast<TopoCtl *>(ws);
    a.wait_ns = wait_limit_ns();
    a.max_levels = max_levels;
    GU_CUDA_CHECK(cudaMemsetAsync(ws, 0, WS_CONTROL_BYTES, st));
    void *params[] = {&a};
    GU_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)topo_plan_kernel, dim3(g.sm_count), dim3(TOPO_THREADS), params, 0, st));
    TopoCtl c;
    GU_CUDA_CHECK(cudaMemcpyAsync(&c, ws, sizeof(c), cudaMemcpyDeviceToHost, st));
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    check_topo(c);
    t.state = c.deep ? TopoPlan::DEEP : c.total == g.n ? TopoPlan::ACYCLIC : TopoPlan::CYCLIC;
    if (t.state != TopoPlan::ACYCLIC) return false;
    g.extra_allocs.push_back(buf.p);
    buf.p = nullptr;
    g.bytes += ints * sizeof(int32_t);
    t.order = a.order;
    t.lvl = a.lvl;
    t.pos = a.pos;
    t.PR = a.PR;
    t.PC = a.PC;
    t.IR = reinterpret_cast<int32_t *>(a.IR);
    t.IC = a.IC;
    t.nlevels = c.nlevels;
    return true;
}

// The closure on bit rows; false where it does not apply (a cycle, too many
// vertices, no memory for the rows): the caller searches from every vertex instead.
// Queues the launch on st.
static bool launch_closure(DeviceGraph &g, unsigned long long *counts, cudaStream_t st)
{
    if (g.n > TOPO_MAX_N) return false;
    const size_t n = (size_t)g.n;
    char *ws = nullptr;
    int64_t block = 0;
    try {
        // equal column blocks within the row budget, at least one chunk wide
        const int64_t fit = std::max<int64_t>(1, (int64_t)(CLOSURE_ROWS_BYTES / (n * (CLOSURE_CHUNK / 8))));
        const int64_t chunks = ((int64_t)n + CLOSURE_CHUNK - 1) / CLOSURE_CHUNK;
        const int64_t nblocks = (chunks + fit - 1) / fit;
        block = (chunks + nblocks - 1) / nblocks * CLOSURE_CHUNK;
        // One warp ORs the rows of a vertex's successors in each block, about 0.18 us a row:
        // where there is little but a hub's list, the search (30 us for every 256 sources) is
        // faster.  Star of 60000 vertices 7.3 ms by the search, 11.2 by the closure; of
        // 150000, in six blocks, 19.5 and 100.
        if (g.m < 2 * (int64_t)g.n && 0.18 * g.max_degree * nblocks > 30.0 / 256.0 * g.n) return false;
        const size_t need = WS_CONTROL_BYTES + n * (size_t)(block / 8);
        const bool known = g.topo.state == TopoPlan::CYCLIC;
        if (!ensure_topo(g, INT_MAX, need, st)) {
            if (!known) g.ws.release();  // sized for the rows: the search takes what it needs
            return false;
        }
        ws = (char *)g.ws.get(need);
    } catch (const gu_error &e) {
        if (e.code == GU_ERR_OUT_OF_MEMORY) return false;
        throw;
    }
    ClosureArgs a;
    a.order = g.topo.order;
    a.lvl = g.topo.lvl;
    a.PR = g.topo.PR;
    a.PC = g.topo.PC;
    a.n = g.n;
    a.nlevels = g.topo.nlevels;
    a.block = block;
    a.rows = reinterpret_cast<unsigned char *>(ws + WS_CONTROL_BYTES);
    a.counts = counts;
    a.ctl = reinterpret_cast<TopoCtl *>(ws);
    a.wait_ns = wait_limit_ns();
    GU_CUDA_CHECK(cudaMemsetAsync(ws, 0, WS_CONTROL_BYTES, st));
    g.timeline = 0;
    g.mark_start(st);
    void *params[] = {&a};
    GU_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)closure_kernel, dim3(topo_grid(closure_kernel, g.sm_count)),
                                              dim3(TOPO_THREADS), params, 0, st));
    g.mark_stop(st);
    return true;
}

// Reachable counts of k sources (themselves included) on an acyclic graph; false where
// this does not apply.  Synchronises st.
bool launch_dag_reach(DeviceGraph &g, const int32_t *sources, int32_t k, unsigned long long *counts, cudaStream_t st)
{
    const char *env = std::getenv("GU_AUTO_LOCAL");
    if (env && env[0] == '0') return false;
    if (!g.directed || g.n < 1 || g.n > TOPO_MAX_N || g.max_in_degree > REACH_MAX_IN_DEGREE) return false;
    // Graphs of low out-degree have the per-source engine, which runs two sources per SM at
    // about a level's cost here each: the order pays where there is more to a level than
    // that.  Call times in us, by the order / that engine, k = 100 and 600: binary out-tree of
    // 60000 vertices 77 / 51 and 159 / 64; DAG of 20000, m = n 69 / 50 and 130 / 72, of
    // 50000, m = 2 n 89 / 80 and 194 / 96; 90 layers of 500, m = 4 n 337 / 287 and 878 / 574.
    const bool low = g.max_degree <= LOCAL_MAX_DEGREE;
    if (low && g.m < 3 * (int64_t)g.n) return false;
    const int max_levels = low ? std::min(REACH_MAX_LEVELS, g.n / REACH_LEVEL_VERTICES) : REACH_MAX_LEVELS;
    char *ws = nullptr;
    const int W = msbfs_words_for(k);
    // The order costs about as much to build as the searches that it replaces save in one
    // call (n = 200,003: 0.55 ms; 0.42 -> 0.19 ms a call): a graph that is asked once is
    // searched, and the order is built when it is asked again.
    if (g.topo.state == TopoPlan::UNBUILT && g.topo.asked++ == 0) return false;
    try {
        const size_t need = WS_CONTROL_BYTES + sizeof(u64) * (size_t)g.n * W;
        if (!ensure_topo(g, max_levels, need, st)) return false;
        ws = (char *)g.ws.get(need);
    } catch (const gu_error &e) {
        if (e.code == GU_ERR_OUT_OF_MEMORY) return false;
        throw;
    }
    ReachArgs a;
    a.pos = g.topo.pos;
    a.lvl = g.topo.lvl;
    a.IR = reinterpret_cast<const int2 *>(g.topo.IR);
    a.IC = g.topo.IC;
    a.n = g.n;
    a.nlevels = g.topo.nlevels;
    a.sources = sources;
    a.k = k;
    a.rows = reinterpret_cast<u64 *>(ws + WS_CONTROL_BYTES);
    a.counts = counts;
    a.ctl = reinterpret_cast<TopoCtl *>(ws);
    a.wait_ns = wait_limit_ns();
    GU_CUDA_CHECK(cudaMemsetAsync(ws, 0, WS_CONTROL_BYTES, st));
    GU_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int64_t) * (size_t)k, st));
    g.timeline = 0;
    g.mark_start(st);
    const void *kern = W == 1 ? (const void *)reach_kernel<1> : W == 2 ? (const void *)reach_kernel<2> : (const void *)reach_kernel<4>;
    void *params[] = {&a};
    // one CTA per SM: a level's vertices seldom need more groups, and the barrier is cheaper
    GU_CUDA_CHECK(cudaLaunchCooperativeKernel(kern, dim3(g.sm_count), dim3(TOPO_THREADS), params, 0, st));
    g.mark_stop(st);
    TopoCtl c = {};
    GU_CUDA_CHECK(cudaMemcpyAsync(&c, ws, sizeof(c), cudaMemcpyDeviceToHost, st));
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    check_topo(c);
    return true;
}

__global__ void iota_kernel(int32_t *v, int32_t n)
{
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

// counts[v] -= 1 (the source itself) and their sum into *total.
__global__ void reach_finish_kernel(long long *counts, int32_t n, unsigned long long *total)
{
    unsigned long long s = 0;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const long long c = counts[i] - 1;
        counts[i] = c;
        s += (unsigned long long)c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
    if (lane_id() == 0 && s) atomicAdd(total, s);
}

// Search from every vertex, counting in the kernel (counts zeroed by the caller).
static void reach_by_search(DeviceGraph &g, unsigned long long *cnt, char *io, cudaStream_t st, int blocks)
{
    int32_t *src = reinterpret_cast<int32_t *>(io + 256);
    iota_kernel<<<blocks, 256, 0, st>>>(src, g.n);
    GU_CUDA_CHECK(cudaGetLastError());
    if (auto_engine(g) == AutoEngine::LOCAL && launch_local_bfs(g, src, g.n, nullptr, g.n, cnt, nullptr, st)) return;
    GU_CUDA_CHECK(cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (size_t)g.n, st));
    MsOptions opt;
    opt.variant = GU_BFS_AUTO;
    opt.reach = cnt;
    launch_msbfs(g, src, g.n, nullptr, g.n, opt, st, nullptr);
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    int err = 0;
    msbfs_read_status(g, &err, nullptr, nullptr, nullptr);
    if (err == DEV_ERR_BARRIER_TIMEOUT) throw gu_error(GU_ERR_TIMEOUT, "a device-side wait exceeded its limit");
    if (err != 0) throw gu_error(GU_ERR_INTERNAL, "device reported error code " + std::to_string(err));
}

void dag_reach(DeviceGraph &g, int64_t *counts, int64_t *total_host, cudaStream_t st)
{
    if (!g.directed) throw gu_error(GU_ERR_INVALID_ARGUMENT, "DAG reachability needs a directed graph");
    *total_host = 0;
    if (g.n == 0) return;
    char *io = (char *)g.io.get(256 + sizeof(int32_t) * (size_t)g.n);
    auto *total = reinterpret_cast<unsigned long long *>(io);
    const int blocks = std::min(g.sm_count * 8, (g.n + 255) / 256);
    GU_CUDA_CHECK(cudaMemsetAsync(total, 0, sizeof(unsigned long long), st));
    GU_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int64_t) * (size_t)g.n, st));
    auto *cnt = reinterpret_cast<unsigned long long *>(counts);
    // GU_AUTO_LOCAL=0 keeps this call, as AUTO, on the batched engine
    const char *env = std::getenv("GU_AUTO_LOCAL");
    const bool closed = !(env && env[0] == '0') && launch_closure(g, cnt, st);
    if (!closed) reach_by_search(g, cnt, io, st, blocks);
    reach_finish_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<long long *>(counts), g.n, total);
    GU_CUDA_CHECK(cudaGetLastError());
    unsigned long long t = 0;
    TopoCtl c = {};
    if (closed) GU_CUDA_CHECK(cudaMemcpyAsync(&c, g.ws.ptr, sizeof(c), cudaMemcpyDeviceToHost, st));
    GU_CUDA_CHECK(cudaMemcpyAsync(&t, total, sizeof(t), cudaMemcpyDeviceToHost, st));
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    check_topo(c);
    *total_host = (int64_t)t;
}

}  // namespace gu
