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
//      owners of its 256 items' slots: lanes store their items' ids into a window of
//      1024 slots in shared memory and the window leaves as one bulk copy.
//   3. lbs_expand_rest: the slots of warps whose items own more than 4096 slots, listed
//      by kernel 2 in pieces of 4096; persistent CTAs find each slot's owner among the
//      256 items by binary search.  With no such warp it ends at once.
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
constexpr int LBS_WINDOW = 1024;                      // slots staged at once by a warp
constexpr int LBS_LOCAL = 4096;                       // slots that a warp of kernel 2 writes itself; piece of kernel 3
constexpr int LBS_BIG = 32;                           // count from which the warp fills an item's slots together
constexpr int LBS_RTHREADS = 256;                     // kernel 3
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

// Pass 2 (see the head of the file).  summed: sums holds prefixes (lbs_scan_sums).
// Degree array of a 2048 x 2048 grid (N = 4.2 M, 15.9 M slots, 97 MB): the three
// kernels take 30 us on the device, 0.48 of measured HBM; with the owners found by marks
// and a running maximum over merge-path tiles, in a kernel of its own, they took 45 us
// (the shared-memory pipe was the bound: three passes over every slot's mark; here a
// slot is stored once and the window is read by the copy engine).  The call: 71 -> 44
// us, also for want of two copies into pageable memory.  Counts of 0.1-density 1 .. 39:
// device 44.5 -> 39 us; heavy-tailed counts (exponent 1.4): 43.6 -> 46 us, call 71 -> 60.
// Two CTAs per SM: three, with 42 registers, took 32.5 us, six of 256 threads 33.1.
// Filling items together from counts of 8 up: 46 and 54 us on the last two.
__global__ void __launch_bounds__(LBS_THREADS, 2) lbs_scan_expand(const int32_t *__restrict__ counts, int32_t N, int32_t ntiles,
                                                              const long long *__restrict__ sums, int summed,
                                                              int32_t *__restrict__ scanned, LbsHead *head,
                                                              LbsReport *report, int32_t *total_out, long long capacity,
                                                              int32_t *__restrict__ result, int2 *__restrict__ list)
{
    extern __shared__ __align__(16) int32_t s_stage[];  // [LBS_WARPS][LBS_WINDOW]
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
    if (R > LBS_LOCAL) {
        const unsigned n = (unsigned)((R + LBS_LOCAL - 1) / LBS_LOCAL);
        unsigned pos = 0;
        if (lane == 0) pos = atomicAdd(&head->pieces, n);
        pos = __shfl_sync(FULL_MASK, pos, 0);
        for (unsigned j = lane; j < n; j += 32) list[pos + j] = make_int2(first, (int)(P + (long long)j * LBS_LOCAL));
        return;
    }
    int32_t *stage = s_stage + warp * LBS_WINDOW;
    const int ra = (int)(((uintptr_t)result >> 2) & 3);  // result's element offset from a 16-byte boundary
    const long long s1 = P + R;
    // windows start at 16-byte boundaries of result (the first one at or below P)
    for (long long a = P - ((P + ra) & 3); a < s1; a += LBS_WINDOW) {
        const uint32_t lo = (uint32_t)max(a, P), hi = (uint32_t)min(a + LBS_WINDOW, s1);
        const int32_t base = (int32_t)a;  // (a >= -3; differences to it stay small)
#pragma unroll
        for (int j = 0; j < LBS_ITEMS; ++j) {
            const uint32_t b = max(off[j], lo), e = min(off[j] + (uint32_t)c[j], hi);
            const bool big = c[j] >= LBS_BIG && b < e;
            const int cnt = big || e <= b ? 0 : (int)(e - b);
            int32_t *p0 = stage + ((int32_t)b - base);
#pragma unroll
            for (int q = 0; q < 4; ++q)  // short counts without a loop
                if (q < cnt) p0[q] = (int32_t)(i0 + j);
            for (int q = 4; q < cnt; ++q) p0[q] = (int32_t)(i0 + j);
            unsigned todo = __ballot_sync(FULL_MASK, big);
            while (todo) {
                const int l = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t bb = __shfl_sync(FULL_MASK, b, l), ee = __shfl_sync(FULL_MASK, e, l);
                const int32_t id = first + l * LBS_ITEMS + j;
                for (uint32_t p = bb + lane; p < ee; p += 32) stage[(int32_t)p - base] = id;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stores above, before the copy engine reads
        __syncwarp();
        const int x0 = (int)(lo - (uint32_t)base), x1 = (int)(hi - (uint32_t)base);  // the window's slots, by position
        const int m0 = (x0 + 3) & ~3, m1 = x1 & ~3;           // ... in whole 16-byte pieces
        int32_t *dst = result + a;
        if (m1 > m0 && lane == 0) bulk_store(dst + m0, stage + m0, (unsigned)(m1 - m0) * 4u);
        if (lane < 4) {  // the ends
            const int x = x0 + lane;
            if (x < min(m0, x1)) dst[x] = stage[x];
        } else if (lane < 8) {
            const int x = max(m1, m0) + lane - 4;
            if (x < x1) dst[x] = stage[x];
        }
        if (m1 > m0 && lane == 0) bulk_store_wait_read();
        __syncwarp();
    }
}

// The listed pieces: (first item of a warp's 256, first slot).
__global__ void __launch_bounds__(LBS_RTHREADS) lbs_expand_rest(const int32_t *__restrict__ scanned, int32_t N,
                                                               const LbsHead *head, const int2 *__restrict__ list,
                                                               int32_t *__restrict__ result)
{
    __shared__ uint32_t s_off[LBS_WARP_ITEMS + 1];
    griddep_wait();
    const unsigned pieces = head->pieces;
    const int ra = (int)(((uintptr_t)result >> 2) & 3);
    for (unsigned x = blockIdx.x; x < pieces; x += gridDim.x) {
        const int2 pc = __ldcg(list + x);
        const int32_t first = pc.x, items = min(LBS_WARP_ITEMS, N - first);
        for (int i = threadIdx.x; i <= items; i += LBS_RTHREADS)
            s_off[i] = first + i < N ? (uint32_t)__ldcg(scanned + first + i) : (uint32_t)head->total;
        __syncthreads();
        const uint32_t lo = (uint32_t)pc.y, hi = min(lo + LBS_LOCAL, s_off[items]);
        const long long a = (long long)lo - ((lo + ra) & 3);
        for (long long p0 = a + 4 * threadIdx.x; p0 < hi; p0 += 4 * LBS_RTHREADS) {
            const uint32_t p = (uint32_t)max(p0, (long long)lo);
            int l = 0, h = items - 1;  // the last item whose first slot is at or before p
            while (l < h) {
                const int mid = (l + h + 1) >> 1;
                if (s_off[mid] <= p) l = mid;
                else h = mid - 1;
            }
            int32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t q = (uint32_t)max(p0 + j, (long long)lo);
                while (l + 1 < items && s_off[l + 1] <= q) ++l;
                o[j] = first + l;
            }
            if (p0 >= (long long)lo && p0 + 4 <= (long long)hi) {
                *reinterpret_cast<int4 *>(result + p0) = make_int4(o[0], o[1], o[2], o[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (p0 + j >= (long long)lo && p0 + j < (long long)hi) result[p0 + j] = o[j];
            }
        }
        __syncthreads();
    }
}

// Winner lane per warp of 32 predicates (race_and_resolve_warp).
__global__ void race_and_resolve_kernel(const int32_t *__restrict__ pred, int32_t nwarps, int32_t *__restrict__ winner)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if ((i >> 5) >= nwarps) return;  // whole warps only (blockDim is a multiple of 32)
    winner[i] = race_and_resolve_warp(pred[i] != 0);
}

// Scratch: the head, one sum per tile and the total, kernel 3's list (a warp with more
// than LBS_LOCAL slots lists at most twice its slots / LBS_LOCAL pieces).
constexpr size_t LBS_HEAD = 64;
size_t lbs_scratch_bytes(int32_t N, int64_t result_capacity)
{
    const long long n = N > 0 ? N : 0;
    const size_t ntiles = (size_t)((n + LBS_TILE - 1) / LBS_TILE);
    const long long cap = result_capacity < 0 ? 0 : (result_capacity > INT32_MAX ? INT32_MAX : result_capacity);
    return LBS_HEAD + (ntiles + 1) * sizeof(long long) + (2 * (size_t)(cap / LBS_LOCAL) + 2) * sizeof(int2);
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
        constexpr size_t stage_bytes = sizeof(int32_t) * LBS_WARPS * LBS_WINDOW;
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
        cfg.gridDim = dim3((unsigned)sms * 2);
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
