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
#include <cstdlib>
#include <string>

namespace gu {

constexpr int TOPO_THREADS = 512;
constexpr int TOPO_MIN_BLOCKS = 3;
constexpr int64_t TOPO_MAX_N = (int64_t)1 << 26;  // positions fit the packed append counter
constexpr int CLOSURE_CHUNK = 4096;               // columns per warp step: 16 bytes per lane
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
    int32_t *pos;  // position of a vertex
    int32_t *order, *lvl, *PR, *PC;
    TopoCtl *ctl;
    unsigned long long wait_ns;
};

// All lanes of the warp call it; lanes with pred place their vertex at the end of
// the level being collected (one 64-bit atomic per warp reserves the positions and
// the out-edge range).
__device__ __forceinline__ void topo_place(const TopoArgs &a, u64 *pack, long long base_p, long long base_e, bool pred,
                                           int32_t v)
{
    const unsigned mask = __ballot_sync(FULL_MASK, pred);
    if (!mask) return;
    const int lane = lane_id();
    const unsigned deg = pred ? (unsigned)(__ldg(a.R + v + 1) - __ldg(a.R + v)) : 0u;
    unsigned long long inc = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += y;
    }
    u64 old = 0;
    if (lane == 31) old = atomicAdd(pack, ((u64)__popc(mask) << TOPO_PACK) | inc);
    old = __shfl_sync(FULL_MASK, old, 31);
    if (pred) {
        const int32_t p = (int32_t)(base_p + (long long)(old >> TOPO_PACK) + __popc(mask & ((1u << lane) - 1u)));
        a.order[p] = v;
        a.pos[v] = p;
        a.PR[p] = (int32_t)(base_e + (long long)(old & ((1ull << TOPO_PACK) - 1ull)) + (long long)(inc - deg));
    }
}

// Levels by removing sinks: level 0 holds the vertices without successors, level
// j + 1 those whose last successor was placed in level j.  A vertex on a cycle is
// never placed (total < n).  The order inside a level depends on scheduling; no
// result does.
__global__ void __launch_bounds__(TOPO_THREADS, TOPO_MIN_BLOCKS) topo_plan_kernel(TopoArgs a)
{
    __shared__ u64 s_pack[4];
    unsigned epoch = 0;
    TopoCtl *ctl = a.ctl;
    auto barrier = [&] { return grid_barrier(&ctl->bar, &ctl->err, epoch, a.wait_ns, ctl->pack, s_pack, 4); };
    const long long rank = (long long)blockIdx.x * blockDim.x + threadIdx.x, size = (long long)gridDim.x * blockDim.x;
    const long long gw = rank >> 5, nw = size >> 5;
    const int lane = lane_id();
    for (long long b = gw * 32; b < a.n; b += nw * 32) {  // warp-uniform
        const long long v = b + lane;
        int32_t d = 1;
        if (v < a.n) {
            d = __ldg(a.R + v + 1) - __ldg(a.R + v);
            a.cnt[v] = d;
        }
        topo_place(a, &ctl->pack[0], 0, 0, d == 0, (int32_t)v);
    }
    if (!barrier()) return;
    long long ls = 0, ebase = 0;
    int level = 0;
    for (;; ++level) {
        const u64 pk = s_pack[level & 3];
        const long long le = ls + (long long)(pk >> TOPO_PACK);
        if (le == ls) break;
        const long long enext = ebase + (long long)(pk & ((1ull << TOPO_PACK) - 1ull));
        if (rank == 0) {
            a.lvl[level] = (int32_t)ls;
            ctl->pack[(level + 2) & 3] = 0;  // collects level + 2; last read two levels ago
        }
        for (long long p = ls + gw; p < le; p += nw) {
            const int32_t v = __ldcg(a.order + p);
            const int32_t e1 = __ldg(a.RT + v + 1);
            for (int32_t eb = __ldg(a.RT + v); eb < e1; eb += 32) {
                int32_t u = 0;
                bool last = false;
                if (eb + lane < e1) {
                    u = __ldg(a.CT + eb + lane);
                    last = atomicSub(a.cnt + u, 1) == 1;
                }
                topo_place(a, &ctl->pack[(level + 1) & 3], le, enext, last, u);
            }
        }
        if (!barrier()) return;
        ls = le;
        ebase = enext;
    }
    if (rank == 0) {
        a.lvl[level] = (int32_t)ls;
        ctl->nlevels = level;
        ctl->total = (int)ls;
    }
    if (ls != a.n) return;
    if (rank == 0) a.PR[a.n] = (int32_t)a.m;
    // successors in position space, eight lanes per vertex
    const int sub = lane & 7;
    for (long long p = rank >> 3; p < a.n; p += size >> 3) {
        const int32_t v = __ldcg(a.order + p);
        const int32_t e0 = __ldg(a.R + v), d = __ldg(a.R + v + 1) - e0, o = __ldcg(a.PR + p);
        for (int32_t i = sub; i < d; i += 8) a.PC[o + i] = __ldcg(a.pos + __ldg(a.C + e0 + i));
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

// Builds the graph's topological order once (synchronises st); false if the graph
// has a cycle.
static bool ensure_topo(DeviceGraph &g, cudaStream_t st)
{
    TopoPlan &t = g.topo;
    if (t.state != TopoPlan::UNBUILT) return t.state == TopoPlan::ACYCLIC;
    const size_t n = (size_t)g.n, m = (size_t)g.m;
    char *ws = (char *)g.ws.get(WS_CONTROL_BYTES + 2 * n * sizeof(int32_t));
    const size_t ints = n + (n + 2) + (n + 1) + m;
    int32_t *buf = nullptr;
    const cudaError_t e = dev_malloc((void **)&buf, ints * sizeof(int32_t));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        throw gu_error(GU_ERR_OUT_OF_MEMORY, "topological order allocation failed");
    }
    g.extra_allocs.push_back(buf);
    g.bytes += ints * sizeof(int32_t);
    TopoArgs a;
    a.R = g.R;
    a.C = g.C;
    a.RT = g.RT;
    a.CT = g.CT;
    a.n = g.n;
    a.m = g.m;
    a.cnt = reinterpret_cast<int32_t *>(ws + WS_CONTROL_BYTES);
    a.pos = a.cnt + n;
    a.order = buf;
    a.lvl = buf + n;
    a.PR = a.lvl + n + 2;
    a.PC = a.PR + n + 1;
    a.ctl = reinterpret_cast<TopoCtl *>(ws);
    a.wait_ns = wait_limit_ns();
    GU_CUDA_CHECK(cudaMemsetAsync(ws, 0, WS_CONTROL_BYTES, st));
    void *params[] = {&a};
    GU_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)topo_plan_kernel, dim3(topo_grid(topo_plan_kernel, g.sm_count)),
                                              dim3(TOPO_THREADS), params, 0, st));
    TopoCtl c;
    GU_CUDA_CHECK(cudaMemcpyAsync(&c, ws, sizeof(c), cudaMemcpyDeviceToHost, st));
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    check_topo(c);
    t.order = a.order;
    t.lvl = a.lvl;
    t.PR = a.PR;
    t.PC = a.PC;
    t.nlevels = c.nlevels;
    t.state = c.total == g.n ? TopoPlan::ACYCLIC : TopoPlan::CYCLIC;
    return t.state == TopoPlan::ACYCLIC;
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
        if (!ensure_topo(g, st)) return false;
        // equal column blocks within the row budget, at least one chunk wide
        const int64_t fit = std::max<int64_t>(1, (int64_t)(CLOSURE_ROWS_BYTES / (n * (CLOSURE_CHUNK / 8))));
        const int64_t chunks = ((int64_t)n + CLOSURE_CHUNK - 1) / CLOSURE_CHUNK;
        const int64_t nblocks = (chunks + fit - 1) / fit;
        block = (chunks + nblocks - 1) / nblocks * CLOSURE_CHUNK;
        ws = (char *)g.ws.get(WS_CONTROL_BYTES + n * (size_t)(block / 8));
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
