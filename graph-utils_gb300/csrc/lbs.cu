// lbs.cu -- load-balanced search and warp race-and-resolve on sm_103a.
//
// Load-balanced search (load_balanced_search.cu:123-192, example lbs.cu:18-31):
// given per-item work counts, scanned = exclusive prefix sum (int32), total =
// sum, and result[i] for every work slot i < total = the item owning it
// (upper_bound(scanned, i) - 1).  The reference runs it in ONE CTA whose threads
// each walk the scanned array from the start (quadratic in the item count);
// here three kernels:
//   1. lbs_tile_sums: the sum of every tile of 4096 counts, and whether one of them is
//      negative.
//   2. lbs_scan_expand: each tile adds the sums of the tiles before it (all final, so
//      no tile waits on another) and of all tiles, which gives its prefix, the total
//      and the verdict on the call (no negative count, total within int32 and within
//      the result capacity, a result buffer when the total is positive); scans its
//      counts in registers, writes its part of scanned, and each warp writes the
//      owners of its 256 items' slots (lbs_fill: found by binary search among the items;
//      short lists by way of shared memory and a bulk copy).
//   3. lbs_expand_rest: the slots of warps whose items own many, listed by kernel 2 in
//      pieces of 2048, a warp each.  With no such warp it ends at once.
//   Kernels 2 and 3 are launched as programmatic dependents of their predecessor, so
//   that their launch overlaps its tail.  The total and the verdict go to pinned host
//   memory; the host waits once, at the end.
// Bound: HBM, 4 N (counts) + 4 N (scanned) + 4 total (owners).  Degree array of a
// 2048 x 2048 grid (97 MB): see lbs_scan_expand.
// race_and_resolve (race_and_resolve.cuh:13-25) is exposed as a warp-level
// kernel over an array of predicates for testing the device primitive.
#include "device_utils.cuh"
#include "gu_internal.h"

#include <algorithm>

namespace gu {

constexpr int LBS_THREADS = 512;
constexpr int LBS_WARPS = LBS_THREADS / 32;
constexpr int LBS_ITEMS = 8;                          // consecutive counts per thread
constexpr int LBS_TILE = LBS_THREADS * LBS_ITEMS;     // counts per tile
constexpr int LBS_WARP_ITEMS = 32 * LBS_ITEMS;
constexpr int LBS_LOCAL = 4096;                       // slots that a warp of kernel 2 always writes itself
constexpr int LBS_SHARE = 13;                         // ... or 2^-13 of the total, if that is more
constexpr int LBS_PIECE = 2048;                       // slots of a piece of kernel 3
constexpr int LBS_KEYS = LBS_WARP_ITEMS + 4;
constexpr int LBS_SHORT = 4;                          // counts up to which a warp's lists are short
constexpr int LBS_CROWD = 8;                          // lanes that may start in one bank then
constexpr int LBS_STAGE = LBS_WARP_ITEMS * LBS_SHORT + 8;
constexpr int LBS_RTHREADS = 256;                     // kernel 3
constexpr int LBS_REST_CTAS = 5;                      // ... CTAs per SM
constexpr int LBS_DIRECT_TILES = 4096;                // tile sums that every tile adds up itself

struct LbsHead {  // device scratch
    long long total;
    unsigned pieces;  // entries in kernel 3's list
    int pad;
};
struct LbsReport {  // pinned
    long long total;
    int neg;
};

// Programmatic dependent launch: a kernel launched with programmatic stream
// serialization may start while its predecessor is still running; it waits
// here for the predecessor's completion (and its memory) before reading its
// results.  A kernel lets its successor start launching once all of its own
// CTAs have started (every CTA calls launch_dependents first): the successor's
// CTAs then only take SM room that this kernel's CTAs no longer need.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// A thread's eight consecutive counts from i (16-byte loads where the array allows).
__device__ __forceinline__ void lbs_load(const int32_t *__restrict__ counts, long long i, long long N, int32_t (&c)[LBS_ITEMS])
{
    if (i + LBS_ITEMS <= N && (((uintptr_t)counts) & 15) == 0) {
        const int4 x = __ldg(reinterpret_cast<const int4 *>(counts + i)), y = __ldg(reinterpret_cast<const int4 *>(counts + i) + 1);
        c[0] = x.x, c[1] = x.y, c[2] = x.z, c[3] = x.w;
        c[4] = y.x, c[5] = y.y, c[6] = y.z, c[7] = y.w;
    } else {
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j) c[j] = i + j < N ? __ldg(counts + i + j) : 0;
    }
}

__device__ __forceinline__ long long warp_sum_ll(long long x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL_MASK, x, o);
    return x;
}

// Pass 1: twice the sum of each tile's counts, plus one if a count is negative.  The
// counts are read with the default caching so that they are still in L2 for pass 2.
__global__ void __launch_bounds__(LBS_THREADS) lbs_tile_sums(const int32_t *__restrict__ counts, int32_t N,
                                                            long long *__restrict__ sums, LbsHead *head)
{
    griddep_launch_dependents();
    __shared__ long long s_part[LBS_WARPS];
    int32_t c[LBS_ITEMS];
    lbs_load(counts, (long long)blockIdx.x * LBS_TILE + (long long)threadIdx.x * LBS_ITEMS, N, c);
    long long sum = 0;
    bool bad = false;
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j) {
        bad |= c[j] < 0;
        sum += c[j];
    }
    sum = warp_sum_ll(sum);
    if (lane_id() == 0) s_part[warp_in_block()] = sum;
    const int neg = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        long long t = 0;
#pragma unroll
        for (int w = 0; w < LBS_WARPS; ++w) t += s_part[w];
        sums[blockIdx.x] = 2 * t + (neg ? 1 : 0);
        if (blockIdx.x == 0) head->pieces = 0;
    }
}

// Above LBS_DIRECT_TILES tiles: the prefix of every tile sum in place (doubled, as the
// sums are), the total with the negative flag after the last.  One CTA.
__global__ void __launch_bounds__(1024) lbs_scan_sums(long long *__restrict__ sums, int32_t ntiles)
{
    griddep_launch_dependents();
    griddep_wait();
    __shared__ long long s_warp[32];
    __shared__ long long s_run;
    __shared__ int s_neg;
    if (threadIdx.x == 0) {
        s_run = 0;
        s_neg = 0;
    }
    __syncthreads();
    for (int b = 0; b < ntiles; b += 1024) {
        const int i = b + threadIdx.x;
        const long long raw = i < ntiles ? __ldcg(sums + i) : 0, x = raw & ~1ll;
        if (raw & 1) s_neg = 1;
        long long inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(FULL_MASK, inc, o);
            if (lane_id() >= o) inc += y;
        }
        if (lane_id() == 31) s_warp[warp_in_block()] = inc;
        __syncthreads();
        long long before = s_run;
        for (int w = 0; w < warp_in_block(); ++w) before += s_warp[w];
        if (i < ntiles) sums[i] = before + inc - x;
        __syncthreads();
        if (threadIdx.x == 1023) s_run = before + inc;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[ntiles] = s_run | (s_neg ? 1 : 0);
}

__device__ __forceinline__ void bulk_store(void *dst, const void *src, unsigned bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"((unsigned)__cvta_generic_to_shared(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// The items of a warp that own slots, in order, as keys: first slot (from the first of the
// slots to be written on) << 8 | item's number among the 256.  A lane comes with eight
// consecutive items: the first slots and whether it owns any.
__device__ __forceinline__ void lbs_keys(uint32_t *key, const uint32_t (&slot)[LBS_ITEMS], const bool (&owns)[LBS_ITEMS])
{
    const int lane = lane_id();
#pragma unroll
    for (int j = lane; j < LBS_KEYS; j += 32) key[j] = UINT32_MAX;
    int n = 0;
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j) n += owns[j];
    int at = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL_MASK, at, o);
        if (lane >= o) at += y;
    }
    at -= n;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j)
        if (owns[j]) key[at++] = slot[j] << 8 | (uint32_t)(LBS_ITEMS * lane + j);
    __syncwarp();
}

// The owners of n slots from `lo` on, by the warp's keys; its items start with `first`.
// 128 slots at a time, four per lane from a 16-byte boundary of result on: a binary
// search finds the first one's owner, and the others' owners are among the next three
// keys, since every one of them owns a slot.  Two such steps are in flight.
__device__ __forceinline__ void lbs_fill(const uint32_t *key, int32_t first, uint32_t lo, int n, int32_t *__restrict__ result)
{
    int32_t *dst = result + (long long)lo;
    const int skip = (int)(((uintptr_t)dst >> 2) & 3);  // elements from a 16-byte boundary to dst
    for (int t0 = -skip; t0 < n; t0 += 256) {           // warp-uniform
        int t[2], l[2];
        uint32_t x[2];  // keys below it: items whose first slot is at or before t
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            t[u] = t0 + 128 * u + 4 * lane_id();
            x[u] = (uint32_t)(max(t[u], 0) + 1) << 8;
            l[u] = 0;
        }
#pragma unroll
        for (int step = LBS_WARP_ITEMS / 2; step > 0; step >>= 1)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (key[l[u] + step] < x[u]) l[u] += step;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t k0 = key[l[u]], k1 = key[l[u] + 1], k2 = key[l[u] + 2], k3 = key[l[u] + 3];
            const uint32_t x1 = (uint32_t)(t[u] + 2) << 8, x2 = x1 + 256, x3 = x2 + 256;
            int4 o;
            o.x = (int)k0;
            o.y = (int)(k1 < x1 ? k1 : k0);
            o.z = (int)(k2 < x2 ? k2 : k1 < x2 ? k1 : k0);
            o.w = (int)(k3 < x3 ? k3 : k2 < x3 ? k2 : k1 < x3 ? k1 : k0);
            o.x = first + (o.x & 255);
            o.y = first + (o.y & 255);
            o.z = first + (o.z & 255);
            o.w = first + (o.w & 255);
            if (t[u] >= 0 && t[u] + 4 <= n) {
                *reinterpret_cast<int4 *>(dst + t[u]) = o;
            } else {
                if (t[u] >= 0 && t[u] < n) dst[t[u]] = o.x;
                if (t[u] + 1 >= 0 && t[u] + 1 < n) dst[t[u] + 1] = o.y;
                if (t[u] + 2 >= 0 && t[u] + 2 < n) dst[t[u] + 2] = o.z;
                if (t[u] + 3 >= 0 && t[u] + 3 < n) dst[t[u] + 3] = o.w;
            }
        }
    }
}

// Pass 2 (see the head of the file).  summed: sums holds prefixes (lbs_scan_sums).
//
// A warp's slots.  Lists of up to four (a mesh's degrees): every lane stores its items'
// ids to shared memory, and the warp's slots leave as one bulk copy.  Longer lists, and
// equal ones whose lanes would store into the same few banks: by search.  Storing longer
// lists item by item left most lanes idle and met conflicts of up to 32 lanes, and the
// warps above 4096 slots were left to a kernel 3 of two CTAs per SM.  Calls in us, that
// form / this one / with the owners found by marks and a running maximum over merge-path
// tiles in a kernel of its own, N = 2^22: degrees of a grid with 5 % of its edges deleted
// 43 / 41 / 75; all counts 4: 99 / 49 / 90, 16: 267 / 77 / 152, 20: 829 / 89 / 173; counts
// 0 .. 8 60 / 50 / 89, 0 .. 32 532 / 80 / 154; heavy-tailed (exponent 1.4, mean 2.8) 60 /
// 54 / 79; N = 262144, counts 0 .. 400 249 / 85 / 120.
//
// On the grid the three kernels take about 28 us, 0.5 of measured HBM: without the stores
// of the owners they take as long, so the bound is the tiles' dependent chain (counts,
// sums, scan, slots).  Three CTAs per SM: two 41.8 us a call, three 40.5; lists of up to
// three as short ones 46.8.  What a warp writes itself: 4096 slots or 2^-13 of the total;
// with 2^-11 heavy tails wait for single warps (mean 56, N = 2^22: 119 us, 96).
__global__ void __launch_bounds__(LBS_THREADS, 3) lbs_scan_expand(const int32_t *__restrict__ counts, int32_t N, int32_t ntiles,
                                                              const long long *__restrict__ sums, int summed,
                                                              int32_t *__restrict__ scanned, LbsHead *head,
                                                              LbsReport *report, int32_t *total_out, long long capacity,
                                                              int32_t *__restrict__ result, int2 *__restrict__ list)
{
    extern __shared__ __align__(16) int32_t s_stage[];  // [LBS_WARPS][LBS_STAGE]
    __shared__ long long s_part[LBS_WARPS], s_all[LBS_WARPS], s_warp[LBS_WARPS];
    griddep_launch_dependents();
    const int lane = lane_id(), warp = warp_in_block(), t = blockIdx.x;
    const long long i0 = (long long)t * LBS_TILE + (long long)threadIdx.x * LBS_ITEMS;
    int32_t c[LBS_ITEMS];
    lbs_load(counts, i0, N, c);  // (an input: no need to wait for pass 1)
    long long sum = 0;
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j) sum += c[j];
    long long inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    griddep_wait();
    long long before = 0, all = 0;
    bool neg = false;
    if (!summed) {
        for (int i = threadIdx.x; i < ntiles; i += LBS_THREADS) {
            const long long x = __ldcg(sums + i);
            neg |= x & 1;
            all += x >> 1;
            if (i < t) before += x >> 1;
        }
        before = warp_sum_ll(before);
        all = warp_sum_ll(all);
        if (lane == 0) {
            s_part[warp] = before;
            s_all[warp] = all;
        }
    }
    neg = __syncthreads_or(neg);
    long long P = 0, total = 0;
    if (summed) {
        const long long x = __ldcg(sums + ntiles);
        P = __ldcg(sums + t) >> 1;
        total = x >> 1;
        neg = x & 1;
    } else {
#pragma unroll
        for (int w = 0; w < LBS_WARPS; ++w) {
            P += s_part[w];
            total += s_all[w];
        }
    }
    for (int w = 0; w < warp; ++w) P += s_warp[w];  // of the warp's first item
    long long at = P + inc - sum;                     // of the thread's
    uint32_t off[LBS_ITEMS];
    {
        long long x = at;
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j) {
            off[j] = (uint32_t)x;
            x += c[j];
        }
    }
    if (i0 + LBS_ITEMS <= N && (((uintptr_t)scanned) & 15) == 0) {
        int4 *p = reinterpret_cast<int4 *>(scanned + i0);
        p[0] = make_int4((int)off[0], (int)off[1], (int)off[2], (int)off[3]);
        p[1] = make_int4((int)off[4], (int)off[5], (int)off[6], (int)off[7]);
    } else {
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j)
            if (i0 + j < N) scanned[i0 + j] = (int32_t)off[j];
    }
    const bool good = !neg && total <= INT32_MAX && total <= capacity && (total == 0 || result);
    if (t == ntiles - 1 && threadIdx.x == 0) {
        head->total = total;
        report->total = total;
        report->neg = neg;
        if (good && total_out) *total_out = (int32_t)total;
    }
    if (!good || total == 0) return;
    // ---- the warp's slots [P, P + R) ----
    const long long R = __shfl_sync(FULL_MASK, inc, 31);
    if (R == 0) return;  // warp-uniform, no barrier below
    const int32_t first = (int32_t)((long long)t * LBS_TILE + warp * LBS_WARP_ITEMS);
    if (R > max((long long)LBS_LOCAL, total >> LBS_SHARE)) {
        const unsigned n = (unsigned)((R + LBS_PIECE - 1) / LBS_PIECE);
        unsigned pos = 0;
        if (lane == 0) pos = atomicAdd(&head->pieces, n);
        pos = __shfl_sync(FULL_MASK, pos, 0);
        for (unsigned j = lane; j < n; j += 32) list[pos + j] = make_int2(first, (int)(P + (long long)j * LBS_PIECE));
        return;
    }
    int32_t *stage = s_stage + warp * LBS_STAGE;
    int most = 0;
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j) {
        most = max(most, c[j]);
        off[j] -= (uint32_t)P;
    }
    int32_t *dst = result + P;
    // Short lists: every lane stores its items' ids to the warp's slots in shared memory,
    // which leave as one bulk copy -- unless equal lists put the lanes' stores into the
    // same few banks (lists of four: 32 lanes in one).
    if (!__any_sync(FULL_MASK, most > LBS_SHORT) &&
        !__any_sync(FULL_MASK, __popc(__match_any_sync(FULL_MASK, off[0] & 31u)) > LBS_CROWD)) {
        const int x0 = (int)(((uintptr_t)dst >> 2) & 3), x1 = x0 + (int)R;  // from dst's 16-byte boundary on
        const int m0 = (x0 + 3) & ~3, m1 = x1 & ~3;                        // ... the whole 16-byte pieces
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j)
#pragma unroll
            for (int q = 0; q < LBS_SHORT; ++q)
                if (q < c[j]) stage[x0 + (int)off[j] + q] = (int32_t)(i0 + j);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stores above, before the copy engine reads
        __syncwarp();
        dst -= x0;
        if (m1 > m0 && lane == 0) bulk_store(dst + m0, stage + m0, (unsigned)(m1 - m0) * 4u);
        if (lane < 4) {  // the ends
            const int x = x0 + lane;
            if (x < min(m0, x1)) dst[x] = stage[x];
        } else if (lane < 8) {
            const int x = max(m1, m0) + lane - 4;
            if (x < x1) dst[x] = stage[x];
        }
        if (m1 > m0 && lane == 0) bulk_store_wait_read();
        return;
    }
    bool owns[LBS_ITEMS];
#pragma unroll
    for (int j = 0; j < LBS_ITEMS; ++j) owns[j] = c[j] > 0;
    uint32_t *key = reinterpret_cast<uint32_t *>(stage);
    lbs_keys(key, off, owns);
    lbs_fill(key, first, (uint32_t)P, (int)R, result);
}

// The listed pieces, a warp each: (first item of a warp's 256, first slot).
__global__ void __launch_bounds__(LBS_RTHREADS) lbs_expand_rest(const int32_t *__restrict__ scanned, int32_t N,
                                                               const LbsHead *head, const int2 *__restrict__ list,
                                                               int32_t *__restrict__ result)
{
    __shared__ uint32_t s_key[LBS_RTHREADS / 32][LBS_KEYS];
    griddep_wait();
    const unsigned pieces = head->pieces, nw = gridDim.x * (LBS_RTHREADS / 32);
    const uint32_t total = (uint32_t)head->total;
    uint32_t *key = s_key[warp_in_block()];
    for (unsigned x = blockIdx.x * (LBS_RTHREADS / 32) + warp_in_block(); x < pieces; x += nw) {  // warp-uniform
        const int2 pc = __ldcg(list + x);
        const int32_t first = pc.x;
        const uint32_t lo = (uint32_t)pc.y;
        __syncwarp();
#pragma unroll
        for (int i = lane_id(); i <= LBS_WARP_ITEMS; i += 32)
            key[i] = i < N - first ? (uint32_t)__ldcg(scanned + first + i) : total;
        __syncwarp();
        const uint32_t hi = min(lo + LBS_PIECE, key[LBS_WARP_ITEMS]);
        uint32_t slot[LBS_ITEMS + 1];
        bool owns[LBS_ITEMS];
#pragma unroll
        for (int j = 0; j <= LBS_ITEMS; ++j) slot[j] = key[LBS_ITEMS * lane_id() + j];
        uint32_t from[LBS_ITEMS];
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j) {  // the item's slots within the piece
            const uint32_t a = max(slot[j], lo);
            owns[j] = a < min(slot[j + 1], hi);
            from[j] = a - lo;
        }
        __syncwarp();
        lbs_keys(key, from, owns);
        lbs_fill(key, first, lo, (int)(hi - lo), result);
    }
}

// Winner lane per warp of 32 predicates (race_and_resolve_warp).
__global__ void race_and_resolve_kernel(const int32_t *__restrict__ pred, int32_t nwarps, int32_t *__restrict__ winner)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if ((i >> 5) >= nwarps) return;  // whole warps only (blockDim is a multiple of 32)
    winner[i] = race_and_resolve_warp(pred[i] != 0);
}

// Scratch: the head, one sum per tile and the total, kernel 3's list (a warp with R >
// LBS_LOCAL slots lists at most R / LBS_PIECE + 1 pieces, less than 3 R / LBS_LOCAL).
constexpr size_t LBS_HEAD = 64;
size_t lbs_scratch_bytes(int32_t N, int64_t result_capacity)
{
    const long long n = N > 0 ? N : 0;
    const size_t ntiles = (size_t)((n + LBS_TILE - 1) / LBS_TILE);
    const long long cap = result_capacity < 0 ? 0 : (result_capacity > INT32_MAX ? INT32_MAX : result_capacity);
    return LBS_HEAD + (ntiles + 1) * sizeof(long long) + (3 * (size_t)(cap / LBS_LOCAL) + 4) * sizeof(int2);
}

// Device time of the last call on each device: from before the flags are
// cleared to after the search, CUDA events on the call's stream (the three
// kernels overlap, so their sum would overstate it).  Calls are serialised by
// the caller (one scratch area per device).
static cudaEvent_t g_lbs_ev[128][2];
static double g_lbs_last_ms[128];

double lbs_last_ms(int device) { return device >= 0 && device < 128 ? g_lbs_last_ms[device] : 0.0; }

void launch_lbs(const int32_t *counts, int32_t N, int32_t *scanned, int32_t *result, int64_t result_capacity,
                int32_t *total_dev, int64_t *total_host, void *scratch_ptr, size_t scratch_bytes, cudaStream_t st)
{
    if (N < 0) throw gu_error(GU_ERR_INVALID_ARGUMENT, "N must be >= 0");
    if (N > 0 && (!counts || !scanned)) throw gu_error(GU_ERR_INVALID_ARGUMENT, "null counts or scanned");
    const int32_t ntiles = (int32_t)(((long long)N + LBS_TILE - 1) / LBS_TILE);
    if (scratch_bytes < lbs_scratch_bytes(N, result_capacity)) throw gu_error(GU_ERR_INTERNAL, "lbs scratch too small");
    char *base = reinterpret_cast<char *>(scratch_ptr);
    LbsHead *head = reinterpret_cast<LbsHead *>(base);
    long long *sums = reinterpret_cast<long long *>(base + LBS_HEAD);
    int2 *list = reinterpret_cast<int2 *>(sums + ntiles + 1);
    // all kernels are queued at once; the scan decides on the device whether results may
    // be written, and the host checks the same conditions after one wait
    long long tot = 0;
    int neg = 0, dev = 0;
    GU_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) throw gu_error(GU_ERR_UNSUPPORTED, "device ordinal out of range");
    cudaEvent_t *ev = g_lbs_ev[dev];
    if (!ev[0]) {
        GU_CUDA_CHECK(cudaEventCreate(&ev[0]));
        GU_CUDA_CHECK(cudaEventCreate(&ev[1]));
    }
    static void *reports[128];  // a pinned word per device (calls are serialised by the caller)
    if (!reports[dev]) GU_CUDA_CHECK(pinned_alloc(&reports[dev], sizeof(LbsReport)));
    LbsReport *report = static_cast<LbsReport *>(reports[dev]);
    if (N > 0) {
        GU_CUDA_CHECK(cudaEventRecord(ev[0], st));
        lbs_tile_sums<<<ntiles, LBS_THREADS, 0, st>>>(counts, N, sums, head);
        cudaLaunchAttribute pdl[1];
        pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        pdl[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.stream = st;
        cfg.attrs = pdl;
        cfg.numAttrs = 1;
        const int summed = ntiles > LBS_DIRECT_TILES;
        if (summed) {
            cfg.gridDim = dim3(1);
            cfg.blockDim = dim3(1024);
            GU_CUDA_CHECK(cudaLaunchKernelEx(&cfg, lbs_scan_sums, sums, ntiles));
        }
        constexpr size_t stage_bytes = sizeof(int32_t) * LBS_WARPS * LBS_STAGE;
        static bool attr[128];
        if (!attr[dev]) {
            GU_CUDA_CHECK(cudaFuncSetAttribute((const void *)lbs_scan_expand, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)stage_bytes));
            attr[dev] = true;
        }
        cfg.gridDim = dim3((unsigned)ntiles);
        cfg.blockDim = dim3(LBS_THREADS);
        cfg.dynamicSmemBytes = stage_bytes;
        GU_CUDA_CHECK(cudaLaunchKernelEx(&cfg, lbs_scan_expand, counts, N, ntiles, (const long long *)sums, summed, scanned,
                                         head, report, total_dev, (long long)result_capacity, result, list));
        static int sms_of[128];
        int &sms = sms_of[dev];
        if (!sms) GU_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        cfg.dynamicSmemBytes = 0;
        cfg.gridDim = dim3((unsigned)sms * LBS_REST_CTAS);
        cfg.blockDim = dim3(LBS_RTHREADS);
        GU_CUDA_CHECK(cudaLaunchKernelEx(&cfg, lbs_expand_rest, (const int32_t *)scanned, N, (const LbsHead *)head,
                                         (const int2 *)list, result));
        GU_CUDA_CHECK(cudaGetLastError());
        GU_CUDA_CHECK(cudaEventRecord(ev[1], st));
    } else if (total_dev) {
        GU_CUDA_CHECK(cudaMemsetAsync(total_dev, 0, sizeof(int32_t), st));
    }
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
    if (N > 0) {
        float ms = 0.f;
        GU_CUDA_CHECK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
        g_lbs_last_ms[dev] = ms;
        tot = report->total;
        neg = report->neg;
    }
    if (total_host) *total_host = tot;
    if (neg) throw gu_error(GU_ERR_INVALID_ARGUMENT, "work counts must be >= 0");
    if (tot > INT32_MAX) throw gu_error(GU_ERR_OVERFLOW, "total work exceeds INT32_MAX (int32 scanned offsets)");
    if (tot > result_capacity)
        throw gu_error(GU_ERR_CAPACITY, "result buffer holds " + std::to_string(result_capacity) + " slots, need " +
                                            std::to_string(tot));
    if (tot > 0 && !result) throw gu_error(GU_ERR_INVALID_ARGUMENT, "null result");
}

void launch_race_and_resolve(const int32_t *pred, int32_t nwarps, int32_t *winner, cudaStream_t st)
{
    if (nwarps <= 0) return;
    const long long threads = (long long)nwarps * 32;
    race_and_resolve_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(pred, nwarps, winner);
    GU_CUDA_CHECK(cudaGetLastError());
    GU_CUDA_CHECK(cudaStreamSynchronize(st));
}

}  // namespace gu
