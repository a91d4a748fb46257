// smem_bc.cu -- shortest-path counts and Brandes dependencies of small graphs, one CTA
// per source with the state in shared memory.
//
// The batched engine (bc.cu) runs 64 .. 1024 sources through each level together, with
// a grid barrier per step and its state in HBM; on a graph of a few thousand vertices a
// level is then mostly barriers and a hub's serial work items (R-MAT 10, 256 sources:
// 0.75 ms).  Here a CTA keeps one source's counts, levels and BFS order in shared
// memory (14 bytes a vertex) and reads only the adjacency, as 16-bit ids that L1 holds.
//
// Vertices are renumbered by descending out-degree.  A level, kept in id order, then
// starts with its long lists (a warp each, coalesced) and goes on with short ones of
// nearly equal length (a lane each, eight ids a load), and neither needs a search for
// an edge's owner.
//
// Forward, level j: the frontier's out-edges are pushed -- an edge to a vertex on no
// level yet or on level j adds the frontier vertex's count (64-bit integer sums, so
// the order does not matter and the counts are bit-exact).  Backward, from the last
// level: S_w = sum of beta over w's successors (level l + 1), delta = sigma S, beta =
// (1 + delta) / sigma, as in bc.cu; beta takes sigma's place.
//
// The sums S are formed in integers: an SM issues a warp's FP64 instruction over
// sixteen cycles, and one addition per edge was two thirds of the kernel.  The terms
// are positive doubles; a lane keeps their sum as a 64-bit integer in units of 2^-56
// (a warp's lane 2^-55) of its largest term, each term rounded to nearest, where a
// double sum rounds to 2^-53 of the whole at every addition.  A warp's 32 partial sums
// are added in 96 bits.  Against a quadruple-precision oracle betweenness is off by
// 3.4-5.5e-17 (2-norm, ER 198-2500 and R-MAT 10-13), the batched engine's by 6.5e-17 to
// 2.9e-16.
//
// bc: every CTA adds its sources' dependencies, in the order it runs them, to a row of
// its own (sources are dealt to CTAs by number); a second kernel adds the rows in CTA
// order.  The result depends on the grid size, which the graph and k fix, and not on
// scheduling.
#include "device_utils.cuh"
#include "fp64_int.cuh"
#include "gu_internal.h"
#include "kernel_fit.h"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <vector>

namespace gu {

constexpr int SC_MAX_THREADS = 1024;
constexpr int SC_MAX_N = 8192;
constexpr int64_t SC_MAX_M = 1 << 30;
// Dense graphs (smem_bc_takes): above so many vertices, up to so many sources, above so
// many entries.
constexpr int SC_DENSE_N = 2500, SC_FEW = 16;
constexpr int64_t SC_DENSE_M = 820000;
constexpr int SC_LONG = 64;  // out-degree from which a warp takes a vertex
constexpr unsigned SC_NONE = 0xFFFFu;

struct ScArgs {
    const int32_t *__restrict__ R;      // offsets by new id
    const uint16_t *__restrict__ C;     // 16-bit new ids, readable in whole 16-byte pieces
    const uint16_t *__restrict__ newid;
    const uint16_t *__restrict__ oldid;
    int32_t n, nlong;                   // new ids below nlong have long lists
    const int32_t *__restrict__ RT;     // in-edge offsets by old id
    int32_t live;                       // vertices with in-edges
    const int32_t *__restrict__ sources;
    int32_t k;
    u64 *sigma_rows;     // k x ld, or null
    int32_t *dist_rows;  // k x ld, or null
    double *delta_rows;  // k x ld, or null
    int64_t ld;
    double *part;        // [CTAs][n] dependencies by new id (backward)
    int *err;            // [CTAs] device copy of the report's error
    u64 *report;         // [CTAs] pinned: error, deepest level << 32
};

__host__ __device__ inline size_t sc_smem_bytes(int n)
{
    const size_t v = ((size_t)n + 8) & ~(size_t)7;  // one more than n at least: level starts
    return v * (sizeof(u64) + 4 * sizeof(uint16_t));
}

constexpr int SC_GUARD_LANE = 4;  // up to 127 terms: a short list
constexpr int SC_GUARD_WARP = 3;  // up to 255: a lane's share of a list of 32 x 255
constexpr int SC_MAX_DEGREE = 32 * 255;
// IntSum::e from which a term was infinite or NaN (a count that wrapped to zero: beta is
// 1 / 0): the sum is then formed by FP64 additions, which have a result for those.
constexpr int SC_NOT_FINITE = 2047;

__device__ __forceinline__ void shared_add_u64(u64 *p, u64 x)
{
    // two 32-bit additions with the carry between them (the 64-bit form is a
    // compare-and-swap loop in shared memory); the halves' sums commute
    unsigned *q = reinterpret_cast<unsigned *>(p);
    const unsigned lo = (unsigned)x, old = atomicAdd(q, lo);
    const unsigned hi = (unsigned)(x >> 32) + (old + lo < lo);
    if (hi) atomicAdd(q + 1, hi);
}

// ROWS: per-source rows are written (always without BACKWARD).
template <bool BACKWARD, bool ROWS>
__global__ void __launch_bounds__(SC_MAX_THREADS, 1) smem_bc_kernel(ScArgs a)
{
    extern __shared__ __align__(16) u64 sc_mem[];
    __shared__ int s_cnt[SC_MAX_THREADS / 32], s_long[SC_MAX_THREADS / 32];
    const int32_t n = a.n;
    const int vpad = (n + 8) & ~7;
    u64 *val = sc_mem;  // sigma, then beta
    // levels; vertices level by level, ids ascending; first vertex of a level; its long lists
    uint16_t *lev = reinterpret_cast<uint16_t *>(val + vpad), *ord = lev + vpad, *lstart = ord + vpad;
    uint16_t *llong = lstart + vpad;
    const int lane = lane_id(), warp = warp_in_block(), T = blockDim.x, nw = T >> 5;
    double *part = BACKWARD ? a.part + (size_t)blockIdx.x * n : nullptr;
    if (BACKWARD)
        for (int v = threadIdx.x; v < n; v += T) part[v] = 0.0;
    int err = 0, deepest = 0;
    // A call with a source out of range is refused and writes nothing: bc is written by the
    // next kernel, but rows source by source, so every CTA looks at all sources first.
    bool refused = false;
    if (ROWS) {
        for (int i = threadIdx.x; i < a.k; i += T) refused |= (unsigned)__ldg(a.sources + i) >= (unsigned)n;
        refused = __syncthreads_or(refused);
        if (refused) err = DEV_ERR_BAD_SOURCE;
    }
    for (int si = blockIdx.x; si < a.k && !refused; si += gridDim.x) {
        const int32_t given = __ldg(a.sources + si);
        if ((unsigned)given >= (unsigned)n) {
            err = DEV_ERR_BAD_SOURCE;
            continue;
        }
        const int src = __ldg(a.newid + given);
        for (int v = threadIdx.x; v < vpad; v += T) {
            val[v] = v == src ? 1ull : 0ull;
            lev[v] = v == src ? 0 : (uint16_t)SC_NONE;
        }
        if (threadIdx.x == 0) {
            ord[0] = (uint16_t)src;
            lstart[0] = 0;
            llong[0] = src < a.nlong;
        }
        __syncthreads();
        int fs = 0, fe = 1, flong = src < a.nlong, level = 1;
        for (;; ++level) {
            // ---- push the frontier's counts ----
            auto visit = [&](unsigned w, u64 sg) {
                unsigned l = lev[w];
                if (l == SC_NONE) lev[w] = (uint16_t)(l = level);
                if (l == (unsigned)level) shared_add_u64(val + w, sg);
            };
            const int cnt = fe - fs, byw = cnt < 4 * nw ? cnt : flong;  // vertices that a warp takes
            for (int i = warp; i < byw; i += nw) {
                const int v = ord[fs + i];
                const int32_t e1 = __ldg(a.R + v + 1);
                const u64 sg = val[v];
                int32_t e = __ldg(a.R + v) + lane;
                for (; e + 32 < e1; e += 64) {
                    const unsigned x = __ldg(a.C + e), y = __ldg(a.C + e + 32);
                    visit(x, sg);
                    visit(y, sg);
                }
                if (e < e1) visit(__ldg(a.C + e), sg);
            }
            for (int i = byw + threadIdx.x; i < cnt; i += T) {
                const int v = ord[fs + i];
                const int32_t e0 = __ldg(a.R + v), e1 = __ldg(a.R + v + 1);
                const u64 sg = val[v];
#pragma unroll 1
                for (int32_t e = e0 & ~7; e < e1; e += 8) {  // eight ids a load
                    const uint4 p = __ldg(reinterpret_cast<const uint4 *>(a.C + e));
                    const unsigned x[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (e + t >= e0 && e + t < e1) visit((x[t >> 1] >> (16 * (t & 1))) & 0xFFFFu, sg);
                }
            }
            __syncthreads();
            // ---- the new vertices in id order: each warp counts its share, then places it ----
            const unsigned *lev2 = reinterpret_cast<const unsigned *>(lev);  // two levels a word
            const int words = (n + 1) / 2, share = ((words + nw - 1) / nw + 31) & ~31;
            const int wb = warp * share, we = min(words, wb + share);
            int mine = 0, mlong = 0;
            for (int i0 = wb; i0 < we; i0 += 32) {  // warp-uniform
                const int i = i0 + lane;
                const unsigned two = i < we ? lev2[i] : 0u;
                const bool p = (two & 0xFFFFu) == (unsigned)level, q = (two >> 16) == (unsigned)level;
                mine += __popc(__ballot_sync(FULL_MASK, p)) + __popc(__ballot_sync(FULL_MASK, q));
                mlong += __popc(__ballot_sync(FULL_MASK, p && 2 * i < a.nlong)) +
                         __popc(__ballot_sync(FULL_MASK, q && 2 * i + 1 < a.nlong));
            }
            if (lane == 0) {
                s_cnt[warp] = mine;
                s_long[warp] = mlong;
            }
            __syncthreads();
            const int c = lane < nw ? s_cnt[lane] : 0;
            const int total = __reduce_add_sync(FULL_MASK, c);
            int pos = fe + __reduce_add_sync(FULL_MASK, lane < warp ? c : 0);
            const int tlong = __reduce_add_sync(FULL_MASK, lane < nw ? s_long[lane] : 0);
            if (mine)
                for (int i0 = wb; i0 < we; i0 += 32) {  // warp-uniform
                    const int i = i0 + lane;
                    const unsigned two = i < we ? lev2[i] : 0u;
                    const bool p = (two & 0xFFFFu) == (unsigned)level, q = (two >> 16) == (unsigned)level;
                    const unsigned bp = __ballot_sync(FULL_MASK, p), bq = __ballot_sync(FULL_MASK, q);
                    const unsigned lt = (1u << lane) - 1u;
                    const int at = pos + __popc(bp & lt) + __popc(bq & lt);
                    if (p) ord[at] = (uint16_t)(2 * i);
                    if (q) ord[at + p] = (uint16_t)(2 * i + 1);
                    pos += __popc(bp) + __popc(bq);
                }
            if (threadIdx.x == 0) {
                lstart[level] = (uint16_t)fe;
                llong[level] = (uint16_t)tlong;
            }
            __syncthreads();
            if (!total) break;
            // Nothing is left to reach (but the vertices with in-edges and the source): the
            // level is the last and is not pushed.
            if (fe + total >= a.live && fe + total >= a.live + (__ldg(a.RT + given) == __ldg(a.RT + given + 1))) {
                ++level;
                if (threadIdx.x == 0) lstart[level] = (uint16_t)(fe + total);
                break;
            }
            fs = fe;
            fe += total;
            flong = tlong;
        }
        const int L = level - 1;  // the deepest level; level l is ord[lstart[l] .. lstart[l + 1])
        deepest = max(deepest, L);
        if (ROWS && (a.dist_rows || a.sigma_rows))
            for (int v = threadIdx.x; v < n; v += T) {
                const int x = __ldg(a.newid + v);
                if (a.dist_rows) __stcs(a.dist_rows + (int64_t)si * a.ld + v, lev[x] == SC_NONE ? INT_MAX : (int32_t)lev[x]);
                if (a.sigma_rows) __stcs(a.sigma_rows + (int64_t)si * a.ld + v, val[x]);
            }
        if (BACKWARD) {
            double *drow = ROWS && a.delta_rows ? a.delta_rows + (int64_t)si * a.ld : nullptr;
            if (drow)  // 0 at the source, where unreached and on the last level
                for (int v = threadIdx.x; v < n; v += T) drow[v] = 0.0;
            __syncthreads();
            const double *beta = reinterpret_cast<const double *>(val);
            auto finish = [&](int w, double S) {
                const double sg = u64_to_double(val[w]), d = sg * S;
                reinterpret_cast<double *>(val)[w] = quotient(1.0 + d, sg);
                __stcg(part + w, __ldcg(part + w) + d);
                if (drow) drow[__ldg(a.oldid + w)] = d;
            };
            for (int i = lstart[L] + threadIdx.x; L > 0 && i < lstart[L + 1]; i += T) {  // no successors
                const int w = ord[i];
                reinterpret_cast<double *>(val)[w] = quotient(1.0, u64_to_double(val[w]));
            }
            __syncthreads();
            for (int l = L - 1; l >= 1; --l) {
                const int b0 = lstart[l], cnt = lstart[l + 1] - b0, byw = cnt < 4 * nw ? cnt : llong[l];
                const unsigned next = l + 1;
                // a warp per vertex, up to 32 of them before their dependencies are
                // finished together: lane j keeps the sum of the j-th
                for (int i0 = warp; i0 < byw; i0 += 32 * nw) {  // warp-uniform
                    u64 khi = 0;
                    unsigned klo = 0;
                    int ke = 0, kw = -1;
                    for (int j = 0; j < 32 && i0 + j * nw < byw; ++j) {
                        const int w = ord[b0 + i0 + j * nw];
                        const int32_t e1 = __ldg(a.R + w + 1);
                        IntSum<SC_GUARD_WARP> s;
                        for (int32_t e = __ldg(a.R + w) + lane; e < e1; e += 32) {
                            const unsigned v = __ldg(a.C + e);
                            if (lev[v] == next) s.add(beta[v]);
                        }
                        const int em = __reduce_max_sync(FULL_MASK, s.e), d = em - s.e;
                        if (em >= SC_NOT_FINITE) {  // warp-uniform
                            double p = 0.0;
                            for (int32_t e = __ldg(a.R + w) + lane; e < e1; e += 32) {
                                const unsigned v = __ldg(a.C + e);
                                if (lev[v] == next) p += beta[v];
                            }
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(FULL_MASK, p, o);
                            if (lane == j) {
                                khi = (u64)__double_as_longlong(p);
                                ke = em;
                                kw = w;
                            }
                            continue;
                        }
                        // acc 2^24, shifted to the largest exponent: 96 bits, 32 of them add up
                        u64 hi = d < 56 ? s.acc >> (d + 8) : 0ull;
                        unsigned lo = d <= 24 ? (unsigned)(s.acc << (24 - d)) : d < 88 ? (unsigned)(s.acc >> (d - 24)) : 0u;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) {
                            const u64 h2 = __shfl_xor_sync(FULL_MASK, hi, o);
                            const unsigned l2 = __shfl_xor_sync(FULL_MASK, lo, o), sum = lo + l2;
                            hi += h2 + (sum < l2);
                            lo = sum;
                        }
                        if (lane == j) {
                            khi = hi;
                            klo = lo;
                            ke = em;
                            kw = w;
                        }
                    }
                    if (kw >= 0 && ke >= SC_NOT_FINITE) {
                        finish(kw, __longlong_as_double((long long)khi));
                    } else if (kw >= 0) {
                        const double x = (double)khi * 4294967296.0 + (double)klo;
                        finish(kw, x == 0.0 ? 0.0 : scalbn(x, ke - 1023 - 52 - SC_GUARD_WARP - 24));
                    }
                }
                for (int i = byw + threadIdx.x; i < cnt; i += T) {  // a lane per vertex
                    const int w = ord[b0 + i];
                    const int32_t e0 = __ldg(a.R + w), e1 = __ldg(a.R + w + 1);
                    IntSum<SC_GUARD_LANE> s;
#pragma unroll 1
                    for (int32_t e = e0 & ~7; e < e1; e += 8) {  // eight ids a load
                        const uint4 p = __ldg(reinterpret_cast<const uint4 *>(a.C + e));
                        const unsigned x[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            const unsigned v = (x[t >> 1] >> (16 * (t & 1))) & 0xFFFFu;
                            if (e + t >= e0 && e + t < e1 && lev[v] == next) s.add(beta[v]);
                        }
                    }
                    double S = s.value();
                    if (s.e >= SC_NOT_FINITE) {
                        S = 0.0;
                        for (int32_t e = e0; e < e1; ++e) {
                            const unsigned v = __ldg(a.C + e);
                            if (lev[v] == next) S += beta[v];
                        }
                    }
                    finish(w, S);
                }
                __syncthreads();
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.err[blockIdx.x] = err;
        a.report[blockIdx.x] = (u64)(unsigned)err | ((u64)(unsigned)deepest << 32);
    }
}

// x added to the pair (t, c): t rounded, c what the roundings dropped (Knuth's two-sum).
__device__ __forceinline__ void add_exactly(double &t, double &c, double x)
{
    const double s = t + x, y = s - t;
    c += (t - (s - y)) + (x - y);
    t = s;
}

// bc[v] = the CTAs' rows added in CTA order by eight threads per vertex, each a
// contiguous run of rows, and then the eight runs in order; the roundings' errors are
// carried along, so that the sum over a few hundred rows adds none of its own.  Nothing
// is written when a source was out of range.
__global__ void __launch_bounds__(256) smem_bc_reduce_kernel(const double *__restrict__ part, const int *__restrict__ err,
                                                             const uint16_t *__restrict__ oldid, int rows, int32_t n,
                                                             double *__restrict__ bc)
{
    __shared__ double s[8][33], sc[8][33];
    bool bad = false;
    for (int i = threadIdx.x; i < rows; i += 256) bad |= __ldcg(err + i) != 0;
    if (__syncthreads_or(bad)) return;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, per = (rows + 7) / 8;
    const int32_t v = blockIdx.x * 32 + x;
    double t = 0.0, c = 0.0;
    if (v < n)
        for (int r = y * per; r < min(rows, (y + 1) * per); ++r) add_exactly(t, c, __ldcg(part + (size_t)r * n + v));
    s[y][x] = t;
    sc[y][x] = c;
    __syncthreads();
    if (y == 0 && v < n) {
        for (int i = 1; i < 8; ++i) {
            add_exactly(t, c, s[i][x]);
            c += sc[i][x];
        }
        bc[__ldg(oldid + v)] = isfinite(t) ? t + c : t;  // (the roundings' errors of an infinite sum are NaN)
    }
}

// The adjacency by new id: eight lanes per vertex.
__global__ void renumber_kernel(const int32_t *__restrict__ R, const int32_t *__restrict__ C, int32_t n,
                                const uint16_t *__restrict__ newid, const uint16_t *__restrict__ oldid,
                                const int32_t *__restrict__ R2, uint16_t *__restrict__ C2)
{
    const int sub = threadIdx.x & 7;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; v < n; v += (gridDim.x * blockDim.x) >> 3) {
        const int o = __ldg(oldid + v);
        const int32_t e0 = __ldg(R + o), d = __ldg(R + o + 1) - e0, at = __ldg(R2 + v);
        for (int32_t i = sub; i < d; i += 8) C2[at + i] = __ldg(newid + __ldg(C + e0 + i));
    }
}

// One buffer: R by new id, newid, oldid, C by new id.
static void ensure_renumbered(DeviceGraph &g, cudaStream_t stream)
{
    if (g.sc_graph) return;
    const size_t n = (size_t)g.n;
    const size_t r_bytes = (sizeof(int32_t) * (n + 1) + 15) & ~(size_t)15, id_bytes = (2 * n + 15) & ~(size_t)15;
    const size_t head = r_bytes + 2 * id_bytes, bytes = head + ((sizeof(uint16_t) * ((size_t)g.m + 8) + 15) & ~(size_t)15);
    std::vector<char> host(head);
    int32_t *R2 = reinterpret_cast<int32_t *>(host.data());
    uint16_t *newid = reinterpret_cast<uint16_t *>(host.data() + r_bytes);
    uint16_t *oldid = reinterpret_cast<uint16_t *>(host.data() + r_bytes + id_bytes);
    const std::vector<int32_t> &R = g.host_R;
    // counting sort by descending out-degree (longer lists than top together first); with
    // parallel edges a list can be longer than n, and the long ones still come first
    const int32_t top = std::max((int32_t)n, SC_LONG);
    std::vector<int32_t> at((size_t)top + 2, 0);
    auto key = [&](size_t v) { return top - std::min(R[v + 1] - R[v], top); };
    for (size_t v = 0; v < n; ++v) ++at[(size_t)key(v) + 1];
    for (size_t i = 1; i < at.size(); ++i) at[i] += at[i - 1];
    for (size_t v = 0; v < n; ++v) newid[v] = (uint16_t)at[(size_t)key(v)]++;
    for (size_t v = 0; v < n; ++v) oldid[newid[v]] = (uint16_t)v;
    R2[0] = 0;
    for (size_t i = 0; i < n; ++i) R2[i + 1] = R2[i] + (R[oldid[i] + 1] - R[oldid[i]]);
    char *p = nullptr;
    GU_CUDA_CHECK(dev_malloc((void **)&p, bytes));
    g.extra_allocs.push_back(p);
    g.bytes += bytes;
    GU_CUDA_CHECK(cudaMemcpyAsync(p, host.data(), head, cudaMemcpyHostToDevice, stream));
    GU_CUDA_CHECK(cudaMemsetAsync(p + head, 0, bytes - head, stream));
    const uint16_t *dn = reinterpret_cast<uint16_t *>(p + r_bytes), *dold = reinterpret_cast<uint16_t *>(p + r_bytes + id_bytes);
    renumber_kernel<<<std::min(g.sm_count * 8, (g.n + 31) / 32), 256, 0, stream>>>(
        g.R, g.C, g.n, dn, dold, reinterpret_cast<int32_t *>(p), reinterpret_cast<uint16_t *>(p + head));
    GU_CUDA_CHECK(cudaGetLastError());
    GU_CUDA_CHECK(cudaStreamSynchronize(stream));  // host goes out of scope
    g.sc_graph = p;
}

// Whether gu_bc / gu_sigma take this engine.  Call times in us, this engine / the
// batched one: ER 198 k = 198 60 / 225, ER 4000 k = 256 156 / 299, R-MAT 10 k = 256
// 107 / 756, R-MAT 12 k = 1024 664 / 1360 (1024 sources per pass; 3980 at the default
// 256), R-MAT 13 k = 1024 1474 / 1676 (4335).  Above 8192 vertices the state does not
// fit an SM.  A batch narrower than the request asks for passes, which only the batched
// engine has.
// Where most lists are long a source reads nearly the whole adjacency here, once on the
// way out and once on the way back, and a pass's sources share it there -- unless all is
// reached within two levels (m / n squared over 12 n), where the way out ends early.
// Times as fast as the batched engine, bc k = 1 / 40 / 1000: ER 8000 with 80 entries a
// vertex 0.5 / 0.7 / 0.9, with 150 (1.2 M) 0.3 / 0.5 / 0.6, with 1000 0.8 / 2.0 / 2.4; ER
// 4000 with 90 0.6 / 0.8 / 0.8, with 150 0.6 / 0.8 / 0.8 (k = 150 and 300, whole waves of
// CTAs: 1.3), with 300 2.3 / 2.7 / 3.5; and with nearly all possible entries ER 1000 0.5 /
// 0.7 / 1.3.
bool smem_bc_takes(DeviceGraph &g, int32_t k, int32_t batch)
{
    if (g.n < 1 || g.n > SC_MAX_N || g.m > SC_MAX_M || g.max_degree > SC_MAX_DEGREE || (batch != 0 && k > batch)) return false;
    if (g.sc_nlong < 0) {
        g.sc_nlong = 0;
        for (int32_t v = 0; v < g.n; ++v) g.sc_nlong += g.host_R[v + 1] - g.host_R[v] >= SC_LONG;
    }
    const double n = (double)g.n, m = (double)g.m;
    if (g.n > SC_DENSE_N) {
        if (2 * g.sc_nlong > g.n && m * m < 12.0 * n * n * n &&
            (k <= SC_FEW || g.m > SC_DENSE_M || (m > 100.0 * n && (k <= 100 || k > 400))))
            return false;
    } else if (m > 550.0 * n && 8.0 * k * n < m) {
        return false;
    }
    for (const char *name : {"GU_BC_WORDS", "GU_BC_LEVEL_BUDGET_MB"}) {  // settings of the batched engine
        const char *s = std::getenv(name);
        if (s && *s) return false;
    }
    return true;
}

// sigma / dist rows and, with bc, the betweenness and optional delta rows; synchronises.
void launch_smem_bc(DeviceGraph &g, const int32_t *sources, int32_t k, double *bc, int32_t *dist_rows,
                    uint64_t *sigma_rows, double *delta_rows, int64_t ld, cudaStream_t stream)
{
    ensure_renumbered(g, stream);
    const bool back = bc != nullptr;
    const void *kern = !back        ? (const void *)smem_bc_kernel<false, true>
                       : delta_rows ? (const void *)smem_bc_kernel<true, true> : (const void *)smem_bc_kernel<true, false>;
    const size_t smem = sc_smem_bytes(g.n);
    // Threads per source: wide where a source has an SM to itself (by shared memory, or
    // because there are few), narrow where several share one.  Call times with 128 / 256 /
    // 512 / 1024 threads: R-MAT 10 k = 256 117 / 95 / 90 / 144 us, k = 1000 137 / 170 /
    // 215 / 328; ER 4000 k = 32 386 / 219 / 140 / 114, k = 1024 1113 / 645 / 526 / 650;
    // R-MAT 13 k = 1024 6357 / 3460 / 2081 / 1487.
    const int sms = g.sm_count;
    const int threads = g.n > 4096   ? 1024
                        : g.n > 1024 ? (k <= sms ? 1024 : 512)
                                     : (k <= 2 * sms ? 512 : k <= 4 * sms ? 256 : 128);
    const int per_sm = kernel_fit(g.device, kern, threads, smem, sc_smem_bytes(SC_MAX_N));
    if (per_sm < 1) throw gu_error(GU_ERR_INTERNAL, "shared-memory BC kernel cannot be resident");
    const int grid = std::min(k, g.sm_count * per_sm);
    if (!g.sc_report) GU_CUDA_CHECK(pinned_alloc(&g.sc_report, sizeof(u64) * 4096));
    const size_t err_bytes = sizeof(int) * 4096;
    if (grid > 4096) throw gu_error(GU_ERR_INTERNAL, "shared-memory BC grid too large");
    char *ws = (char *)g.ws.get(WS_CONTROL_BYTES + err_bytes + (back ? sizeof(double) * (size_t)grid * (size_t)g.n : 0));
    ScArgs a;
    const size_t n = (size_t)g.n;
    const size_t r_bytes = (sizeof(int32_t) * (n + 1) + 15) & ~(size_t)15, id_bytes = (2 * n + 15) & ~(size_t)15;
    const char *sg = static_cast<const char *>(g.sc_graph);
    a.R = reinterpret_cast<const int32_t *>(sg);
    a.newid = reinterpret_cast<const uint16_t *>(sg + r_bytes);
    a.oldid = reinterpret_cast<const uint16_t *>(sg + r_bytes + id_bytes);
    a.C = reinterpret_cast<const uint16_t *>(sg + r_bytes + 2 * id_bytes);
    a.n = g.n;
    a.nlong = g.sc_nlong;
    a.RT = g.RT;
    a.live = g.nlight + g.nmid + g.nwide + g.nheavy;
    a.sources = sources;
    a.k = k;
    a.sigma_rows = reinterpret_cast<u64 *>(sigma_rows);
    a.dist_rows = dist_rows;
    a.delta_rows = delta_rows;
    a.ld = ld;
    a.err = reinterpret_cast<int *>(ws + WS_CONTROL_BYTES);
    a.part = reinterpret_cast<double *>(ws + WS_CONTROL_BYTES + err_bytes);
    a.report = static_cast<u64 *>(g.sc_report);
    g.timeline = 3;
    g.sc_levels = 0;
    void *params[] = {&a};
    g.mark_start(stream);
    GU_CUDA_CHECK(cudaLaunchKernel(kern, dim3(grid), dim3(threads), params, smem, stream));
    if (back) {
        smem_bc_reduce_kernel<<<(g.n + 31) / 32, 256, 0, stream>>>(a.part, a.err, a.oldid, grid, g.n, bc);
        GU_CUDA_CHECK(cudaGetLastError());
    }
    g.mark_stop(stream);
    GU_CUDA_CHECK(cudaStreamSynchronize(stream));
    int err = 0;
    for (int i = 0; i < grid; ++i) {
        err = std::max(err, (int)(unsigned)a.report[i]);
        g.sc_levels = std::max(g.sc_levels, (int)(a.report[i] >> 32));
    }
    if (err) throw gu_error(GU_ERR_INVALID_ARGUMENT, "source vertex out of range");
}

}  // namespace gu
