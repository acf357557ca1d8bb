// prims.cuh -- device-wide exclusive scan and stable LSD radix sort.
//
// The reference calls thrust::exclusive_scan in 1e9-element chunks plus a
// carry kernel (include/fgssjoin/scan.cuh:13-105).  Here the scan, and a sort of up
// to kSortLookTiles tiles, are single-pass kernels with decoupled look-back (Merrill
// and Garland, "Single-pass parallel prefix scan with decoupled look-back"; for the
// sort, one pass per 8-bit digit after one histogram of all digits, Adinets and
// Merrill, "Onesweep"): a tile publishes its sums, adds up its predecessors' and goes
// on, so every element is read and written once per pass.  Larger sorts count per
// tile, scan the counts and scatter; up to one tile is one CTA's work.  Tiles are numbered by a counter as they start,
// so a tile only waits for tiles that already run.  Both can take their element
// count from device memory (`d_n`), so a captured CUDA graph can run them on
// data-dependent sizes; `n_cap` sizes the grid.  noalloc.cu keeps the three-phase
// scan (tile scan, one-CTA scan of tile totals, carry add), whose scratch is one
// word per tile.
#pragma once

#include <algorithm>
#include <utility>

#include "common.cuh"
#include "ctx.h"

namespace fgss {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

// `in` may alias `out` (in-place scans): each element is read and written by
// the same thread, the read before the block's barrier and the write after.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const T* in, T* out, T* tile_sums,
                                                              uint64_t n_cap, const uint64_t* d_n) {
    __shared__ T wsum[33];
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint64_t idx = base + i;
        v[i] = idx < n ? in[idx] : T(0);
        s += v[i];
    }
    T total;
    T pre = block_excl_scan<T>(s, wsum, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint64_t idx = base + i;
        T x = v[i];
        if (idx < n) out[idx] = pre;
        pre += x;
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// One CTA scans the tile totals in place (exclusive) and writes the grand total.
template <typename T>
__global__ void __launch_bounds__(1024) k_scan_totals(T* sums, uint64_t ntiles_cap, uint64_t n_cap,
                                                      const uint64_t* d_n, T* grand_total) {
    __shared__ T wsum[33];
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const uint64_t ntiles = n == 0 ? 0 : (n + kScanTile - 1) / kScanTile;
    T carry = 0;
    for (uint64_t b = 0; b < ntiles; b += blockDim.x) {
        uint64_t i = b + threadIdx.x;
        T x = i < ntiles ? sums[i] : T(0);
        T tot;
        T pre = block_excl_scan<T>(x, wsum, &tot);
        if (i < ntiles) sums[i] = pre + carry;
        carry += tot;
    }
    if (threadIdx.x == 0 && grand_total) *grand_total = carry;
    (void)ntiles_cap;
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_add(T* out, const T* __restrict__ sums, uint64_t n_cap,
                                                           const uint64_t* d_n) {
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const T c = sums[blockIdx.x];
    if (c == 0) return;
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads) {
        uint64_t idx = base + i;
        if (idx < n) out[idx] += c;
    }
}

// ------------------------------------------------------- decoupled look-back

// Status word of a tile (or of a tile's digit): 0 = nothing yet, else the sum of
// the tile alone (kLbSum) or of everything up to it (kLbAll).
constexpr uint64_t kLbSum = 1ull << 62, kLbAll = 2ull << 62, kLbValue = (1ull << 62) - 1;

// A tile gives up: the others of its kernel stop waiting (*abort), the kernels that
// follow write nothing by what it leaves and the call fails with FGSS_ERR_TIMEOUT.
__device__ __forceinline__ void lb_give_up(volatile uint64_t* abort, const WaitErr& err) {
    *abort = 1;
    *(volatile uint32_t*)err.word = 1;
    *(volatile uint32_t*)err.host = 1;
}

// Waits for the status word *p, err.polls times at most; 0 when it gave up (or
// another tile did): the caller then returns without writing anything.
__device__ __forceinline__ uint64_t lb_wait(const volatile uint64_t* p, volatile uint64_t* abort, const WaitErr& err) {
    for (uint32_t i = 0; i < err.polls; i++) {
        const uint64_t v = *p;
        if (v) return v;
        if ((i & 255u) == 255u && *abort) return 0;
    }
    lb_give_up(abort, err);
    return 0;
}

// state: u64 [0] tile counter, [1] abort, [2 ..] tile statuses; zero at launch.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) k_scan_pass(const T* in, T* out, uint64_t n_cap, const uint64_t* d_n,
                                                             uint64_t* state, T* grand_total, WaitErr err) {
    __shared__ T wsum[33];
    __shared__ uint64_t s_tile, s_pre;
    __shared__ bool s_stop;
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const uint64_t ntiles = n ? (n + kScanTile - 1) / kScanTile : 1;
    if (threadIdx.x == 0) {
        s_tile = gridDim.x == 1 ? 0 : atomicAdd((unsigned long long*)state, 1ull);
        s_stop = false;
    }
    __syncthreads();
    const uint64_t tile = s_tile;
    if (tile >= ntiles) return;
    volatile uint64_t* st = state + 2;
    const uint64_t base = tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    constexpr int kVec = 16 / sizeof(T);
    const bool vec = base + kScanItems <= n && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    if (vec) {  // a full row of a 16-byte aligned array (the caller's may not be)
#pragma unroll
        for (int i = 0; i < kScanItems; i += kVec)
            *reinterpret_cast<uint4*>(&v[i]) = *reinterpret_cast<const uint4*>(in + base + i);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) v[i] = base + i < n ? in[base + i] : T(0);
    }
    T s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) s += v[i];
    T total;
    T pre = block_excl_scan<T>(s, wsum, &total);
    if (gridDim.x > 1 && threadIdx.x < 32) {
        // warp 0: 32 predecessors at a time, back to the nearest one that knows everything before it
        uint64_t sum = 0;
        bool stop = false;
        if (tile == 0) {
            if (threadIdx.x == 0) st[0] = kLbAll | ((uint64_t)total & kLbValue);
        } else {
            if (threadIdx.x == 0) st[tile] = kLbSum | ((uint64_t)total & kLbValue);
            for (int64_t b = (int64_t)tile - 1; b >= 0 && !stop; b -= 32) {
                const int64_t t = b - (int64_t)threadIdx.x;
                const uint64_t w = t >= 0 ? lb_wait(st + t, state + 1, err) : kLbAll;
                stop = __any_sync(kFull, w == 0);
                const uint32_t all = __ballot_sync(kFull, (w & kLbAll) != 0);
                const uint32_t last = all ? __ffs(all) - 1 : 31;
                sum += warp_sum(threadIdx.x <= last ? w & kLbValue : 0ull);
                if (all) break;
            }
            if (threadIdx.x == 0 && !stop) st[tile] = kLbAll | ((sum + (uint64_t)total) & kLbValue);
        }
        if (threadIdx.x == 0) {
            s_pre = sum;
            s_stop = stop;
        }
    } else if (gridDim.x == 1 && threadIdx.x == 0) {
        s_pre = 0;
    }
    __syncthreads();
    if (s_stop) return;
    pre += (T)s_pre;
    if (grand_total && tile == ntiles - 1 && threadIdx.x == 0) *grand_total = (T)s_pre + total;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const T x = v[i];
        v[i] = pre;
        pre += x;
    }
    if (vec) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += kVec)
            *reinterpret_cast<uint4*>(out + base + i) = *reinterpret_cast<const uint4*>(&v[i]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++)
            if (base + i < n) out[base + i] = v[i];
    }
}

// Exclusive scan of n_cap (or *d_n) elements (out may alias in); optional grand
// total to `total` (device).  Sums below 2^62 (of 32-bit elements: any, modulo 2^32).
// polls: see WaitErr.
template <typename T>
void exclusive_scan(Ctx& c, const T* in, T* out, uint64_t n_cap, const uint64_t* d_n, T* total,
                    const char* tag = "scan", uint32_t polls = WaitErr::kPolls) {
    const uint64_t ntiles = n_cap == 0 ? 1 : (n_cap + kScanTile - 1) / kScanTile;
    uint64_t* state = nullptr;
    if (ntiles > 1) {
        state = c.devT<uint64_t>(std::string(tag) + ".lb", ntiles + 2);
        FGSS_CK(cudaMemsetAsync(state, 0, (ntiles + 2) * 8, c.stream));
    }
    k_scan_pass<T><<<(unsigned)ntiles, kScanThreads, 0, c.stream>>>(in, out, n_cap, d_n, state, total, c.waits(polls));
    FGSS_LAUNCH_CK();
}

// ------------------------------------------------------------- radix sort

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;  // per thread; item i of a warp's lane l is the warp's 32 i + l
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortWarps = kSortThreads / 32;
// Tiles up to which a pass looks back instead of scanning per-tile histograms: a
// look-back pass is one launch where the other is three (1 M elements, 244 tiles:
// 22 us a pass), but beyond one wave of CTAs it waits on a longer chain (14 M
// elements, five passes: 1182 us with look-back, 1060 us without; 27 M: 2127 and
// 1926 us; both 1982 and 3749 us before).
constexpr uint32_t kSortLookTiles = 512;

template <typename K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift) {
    return (uint32_t)((k >> shift) & 0xffu);
}

// Histograms of all `passes` 8-bit digits from bit `begin`: hist[256 p + d].
template <typename K>
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const K* __restrict__ keys, unsigned long long* hist,
                                                            uint64_t n_cap, const uint64_t* d_n, int begin, int passes) {
    __shared__ uint32_t h[sizeof(K)][256];
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    for (int i = threadIdx.x; i < passes * 256; i += kSortThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * kSortThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kSortThreads + threadIdx.x; i < n; i += stride) {
        const K k = keys[i];
        for (int p = 0; p < passes; p++) atomicAdd(&h[p][digit_of(k, begin + 8 * p)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += kSortThreads)
        if (const uint32_t x = (&h[0][0])[i]) atomicAdd(hist + i, (unsigned long long)x);
}

// The lanes that hold the same 8-bit digit: eight ballots (a __match_any_sync
// over 32 different values is slower by far: 14 M elements, 245 us a pass).
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
    uint32_t peers = kFull;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const bool on = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(kFull, on);
        peers &= on ? m : ~m;
    }
    return peers;
}

struct SortShared {
    uint32_t wcnt[kSortWarps][256];  // per warp: items of each digit so far, then of the earlier warps
    uint32_t start[256];             // first position of each digit in the tile
    uint32_t wsum[33];
};

// Stable ranks of a tile's keys by one digit (rank[i]: position in the sorted
// tile), the tile's digit starts in sh.start; returns the count of digit
// threadIdx.x.  Items past the end take digit 255, so they rank last.
template <typename K>
__device__ __forceinline__ uint32_t rank_tile(SortShared& sh, const K (&key)[kSortItems], uint32_t n_tile, int shift,
                                              uint32_t (&rank)[kSortItems]) {
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, lt = lanemask_lt();
    for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortThreads) (&sh.wcnt[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = wid * 32 * kSortItems + i * 32 + lane;
        const uint32_t d = at < n_tile ? digit_of(key[i], shift) : 255u;
        const uint32_t peers = same_digit(d);
        const uint32_t before = sh.wcnt[wid][d];
        __syncwarp();
        if ((peers & lt) == 0) sh.wcnt[wid][d] = before + __popc(peers);
        __syncwarp();
        rank[i] = before + __popc(peers & lt);
    }
    __syncthreads();
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
        const uint32_t x = sh.wcnt[w][threadIdx.x];
        sh.wcnt[w][threadIdx.x] = cnt;
        cnt += x;
    }
    uint32_t total;
    sh.start[threadIdx.x] = block_excl_scan<uint32_t>(cnt, sh.wsum, &total);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = wid * 32 * kSortItems + i * 32 + lane;
        const uint32_t d = at < n_tile ? digit_of(key[i], shift) : 255u;
        rank[i] += sh.start[d] + sh.wcnt[wid][d];
    }
    return cnt - (threadIdx.x == 255 ? (uint32_t)kSortTile - n_tile : 0u);
}

// Digit counts of every tile, digit-major: cnt[d ntiles + tile].
template <typename K>
__global__ void __launch_bounds__(kSortThreads) k_sort_tile_hist(const K* __restrict__ keys, uint32_t* __restrict__ cnt,
                                                                 uint64_t n_cap, const uint64_t* d_n, int shift) {
    __shared__ uint32_t h[kSortWarps][256];
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const uint32_t wid = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kSortTile + threadIdx.x;
#pragma unroll
    for (int i = 0; i < kSortItems; i++)
        if (base + i * kSortThreads < n) atomicAdd(&h[wid][digit_of(keys[base + i * kSortThreads], shift)], 1u);
    __syncthreads();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) s += h[w][threadIdx.x];
    cnt[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
}

// One digit's pass.  LOOK: hist holds the digit's 256 counts over all keys and
// state is as in k_scan_pass with 256 statuses per tile; else offs holds the
// exclusive scan of k_sort_tile_hist's counts.  Keys and values go through shared
// memory in sorted order, so a digit's run is written contiguously.
template <typename K, typename V, bool LOOK>
__global__ void __launch_bounds__(kSortThreads, 3) k_sort_pass(const K* __restrict__ kin, K* __restrict__ kout,
                                                            const V* __restrict__ vin, V* __restrict__ vout,
                                                            const unsigned long long* __restrict__ hist,
                                                            const uint32_t* __restrict__ offs, uint64_t n_cap,
                                                            const uint64_t* d_n, int shift, uint64_t* state,
                                                            WaitErr err) {
    constexpr size_t kElem = sizeof(K) > sizeof(V) ? sizeof(K) : sizeof(V);
    extern __shared__ __align__(16) unsigned char s_buf[];  // kSortTile x kElem
    (void)kElem;
    __shared__ SortShared sh;
    __shared__ unsigned long long s_dst[256];  // where a digit's items of this tile go, less their tile position
    __shared__ unsigned long long s_wsum[33];
    __shared__ uint64_t s_tile;
    const uint64_t n = d_n ? min(*d_n, n_cap) : n_cap;
    // Nothing is written by counts or positions of a scan, or of this sort's earlier passes, that
    // gave up.  (One thread looks where tiles of this kernel may give up: the same for its block.)
    if (LOOK) {
        if (threadIdx.x == 0) s_tile = gave_up(err.word) ? ~0ull : atomicAdd((unsigned long long*)state, 1ull);
        __syncthreads();
    }
    if (LOOK ? s_tile == ~0ull : gave_up(err.word)) return;
    const uint64_t tile = LOOK ? s_tile : blockIdx.x, base = tile * kSortTile;
    if (base >= n) return;
    const uint32_t n_tile = (uint32_t)min((uint64_t)kSortTile, n - base);
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, w0 = wid * 32 * kSortItems;
    K key[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = w0 + i * 32 + lane;
        key[i] = at < n_tile ? kin[base + at] : K(0);
    }
    const uint32_t cnt = rank_tile<K>(sh, key, n_tile, shift, rank);
    // thread d: the items of digit d in earlier tiles, and of smaller digits anywhere
    if (LOOK) {
        volatile uint64_t* st = state + 2 + threadIdx.x;
        unsigned long long total;
        const unsigned long long below = block_excl_scan<unsigned long long>(hist[threadIdx.x], s_wsum, &total);
        uint64_t sum = 0;
        bool stop = false;
        if (tile == 0) {
            st[0] = kLbAll | cnt;
        } else {
            st[tile * 256] = kLbSum | cnt;
            // eight predecessors' words per round trip: a tile of the first wave would else walk
            // back over half the wave one L2 latency at a time (14 M elements: 260 us a pass)
            uint32_t polls = 0;
            bool done = false;
            for (int64_t t = (int64_t)tile - 1; !done;) {
                uint64_t w[8];
    #pragma unroll
                for (int i = 0; i < 8; i++) w[i] = t - i >= 0 ? (uint64_t)st[(t - i) * 256] : (uint64_t)kLbAll;
                int got = 0;
    #pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (done || got != i || w[i] == 0) continue;
                    sum += w[i] & kLbValue;
                    done = (w[i] & kLbAll) != 0;
                    got = i + 1;
                }
                t -= got;
                if (got == 0) {
                    polls++;
                    if (polls > err.polls || ((polls & 255u) == 0 && *(volatile uint64_t*)(state + 1))) {
                        stop = true;
                        lb_give_up(state + 1, err);
                        break;
                    }
                }
            }
            if (!stop) st[tile * 256] = kLbAll | ((sum + cnt) & kLbValue);
        }
        s_dst[threadIdx.x] = below + sum - sh.start[threadIdx.x];
        if (__syncthreads_or(stop)) return;
    } else {
        s_dst[threadIdx.x] = (unsigned long long)offs[(uint64_t)threadIdx.x * gridDim.x + tile] - sh.start[threadIdx.x];
        __syncthreads();
    }
    (void)cnt;
    K* sk = reinterpret_cast<K*>(s_buf);
#pragma unroll
    for (int i = 0; i < kSortItems; i++) sk[rank[i]] = key[i];
    __syncthreads();
    uint8_t dig[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = i * kSortThreads + threadIdx.x;
        const K k = sk[at];
        dig[i] = (uint8_t)digit_of(k, shift);
        if (at < n_tile) kout[s_dst[dig[i]] + at] = k;
    }
    if (!vin) return;
    __syncthreads();
    V* sv = reinterpret_cast<V*>(s_buf);
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = w0 + i * 32 + lane;
        if (at < n_tile) sv[rank[i]] = vin[base + at];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = i * kSortThreads + threadIdx.x;
        if (at < n_tile) vout[s_dst[dig[i]] + at] = sv[at];
    }
}

// At most kSortTile elements: every pass in one CTA, in place.
template <typename K, typename V>
__global__ void __launch_bounds__(kSortThreads) k_sort_small(K* keys, V* vals, uint64_t n_cap, const uint64_t* d_n,
                                                             int begin, int end) {
    extern __shared__ __align__(16) unsigned char s_buf[];
    __shared__ SortShared sh;
    const uint32_t n = (uint32_t)(d_n ? min(*d_n, n_cap) : n_cap);
    const uint32_t w0 = (threadIdx.x >> 5) * 32 * kSortItems + lane_id();
    K key[kSortItems];
    V val[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = w0 + i * 32;
        key[i] = at < n ? keys[at] : K(0);
        val[i] = vals && at < n ? vals[at] : V(0);
    }
    K* sk = reinterpret_cast<K*>(s_buf);
    V* sv = reinterpret_cast<V*>(s_buf);
    for (int shift = begin; shift < end; shift += 8) {
        rank_tile<K>(sh, key, n, shift, rank);
#pragma unroll
        for (int i = 0; i < kSortItems; i++) sk[rank[i]] = key[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSortItems; i++) key[i] = sk[w0 + i * 32];
        __syncthreads();
        if (!vals) continue;
#pragma unroll
        for (int i = 0; i < kSortItems; i++) sv[rank[i]] = val[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSortItems; i++) val[i] = sv[w0 + i * 32];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const uint32_t at = w0 + i * 32;
        if (at < n) {
            keys[at] = key[i];
            if (vals) vals[at] = val[i];
        }
    }
}

// Stable sort of (keys, values) by the 8-bit digits from begin_bit up to the one
// that holds end_bit - 1.  Ping-pongs between the given arrays and pool scratch;
// the sorted data ends in the given arrays.  `values` may be null.  Element count
// below 2^32.
template <typename K, typename V>
void radix_sort(Ctx& c, K* keys, V* values, uint64_t n_cap, const uint64_t* d_n, int begin_bit, int end_bit,
                const char* tag = "sort") {
    if (n_cap == 0 || end_bit <= begin_bit) return;
    if (n_cap >= (1ull << 32)) fail(FGSS_ERR_UNSUPPORTED, "radix sort of 2^32 or more elements");
    const size_t smem = kSortTile * std::max(sizeof(K), values ? sizeof(V) : size_t(0));
    if (n_cap <= (uint64_t)kSortTile) {
        k_sort_small<K, V><<<1, kSortThreads, smem, c.stream>>>(keys, values, n_cap, d_n, begin_bit, end_bit);
        FGSS_LAUNCH_CK();
        return;
    }
    const uint32_t ntiles = (uint32_t)((n_cap + kSortTile - 1) / kSortTile);
    const int passes = (end_bit - begin_bit + 7) / 8;
    std::string t(tag);
    K* k2 = c.devT<K>(t + ".k", n_cap);
    V* v2 = values ? c.devT<V>(t + ".v", n_cap) : nullptr;
    K* ka = keys;
    K* kb = k2;
    V* va = values;
    V* vb = v2;
    const uint64_t per = 2 + 256ull * ntiles;
    if (ntiles <= kSortLookTiles) {
        // one cleared block: histograms of every pass, then the passes' states
        uint64_t* work = c.devT<uint64_t>(t + ".lb", passes * (256 + per));
        FGSS_CK(cudaMemsetAsync(work, 0, passes * (256 + per) * 8, c.stream));
        unsigned long long* hist = reinterpret_cast<unsigned long long*>(work);
        k_sort_hist<K><<<grid_for(n_cap, kSortTile, c.num_sms * 8), kSortThreads, 0, c.stream>>>(
            keys, hist, n_cap, d_n, begin_bit, passes);
        FGSS_LAUNCH_CK();
        for (int p = 0; p < passes; p++) {
            k_sort_pass<K, V, true><<<ntiles, kSortThreads, smem, c.stream>>>(
                ka, kb, va, vb, hist + 256 * p, nullptr, n_cap, d_n, begin_bit + 8 * p, work + passes * 256 + p * per,
                c.waits());
            FGSS_LAUNCH_CK();
            std::swap(ka, kb);
            std::swap(va, vb);
        }
    } else {
        uint32_t* cnt = c.devT<uint32_t>(t + ".hist", 256ull * ntiles);
        for (int p = 0; p < passes; p++) {
            k_sort_tile_hist<K><<<ntiles, kSortThreads, 0, c.stream>>>(ka, cnt, n_cap, d_n, begin_bit + 8 * p);
            FGSS_LAUNCH_CK();
            exclusive_scan<uint32_t>(c, cnt, cnt, 256ull * ntiles, nullptr, (uint32_t*)nullptr, (t + ".hs").c_str());
            k_sort_pass<K, V, false><<<ntiles, kSortThreads, smem, c.stream>>>(
                ka, kb, va, vb, nullptr, cnt, n_cap, d_n, begin_bit + 8 * p, nullptr, c.waits());
            FGSS_LAUNCH_CK();
            std::swap(ka, kb);
            std::swap(va, vb);
        }
    }
    if (passes & 1) {
        // result sits in scratch: copy back (element count from the device when given)
        FGSS_CK(cudaMemcpyAsync(keys, ka, n_cap * sizeof(K), cudaMemcpyDeviceToDevice, c.stream));
        if (values) FGSS_CK(cudaMemcpyAsync(values, va, n_cap * sizeof(V), cudaMemcpyDeviceToDevice, c.stream));
    }
}

}  // namespace fgss
