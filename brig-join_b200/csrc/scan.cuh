// scan.cuh - device-wide exclusive scan of uint32 counts into int64 offsets, one kernel (k_scan_one or
// k_scan_grid). Included by kernels.cu inside its namespace; ld_acquire and kThreads come from there.
#pragma once

// Block-wide exclusive scan of one int64 value per thread; returns this thread's prefix.
__device__ int64_t block_scan_excl_i64(int64_t v, int64_t* tmp /* kThreads/32 */, int64_t* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int kWarps = kThreads / 32;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int64_t w = lane < kWarps ? tmp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kWarps) tmp[lane] = w;
    }
    __syncthreads();
    int64_t excl = x - v + (wid > 0 ? tmp[wid - 1] : 0);
    *total = tmp[kWarps - 1];
    __syncthreads();
    return excl;
}

// A run scans seven small arrays (513 to 1.5M counts), each between two kernels that need all of it, so a
// scan costs its launches and little else. Up to kScanOne counts one CTA walks them; above that a
// grid of at most one CTA per SM sums its shares, waits for the sums before each and writes it.
// With three launches per scan instead (sums, their scan, the rest) and the level-2 plan in a kernel of
// its own, a 16M x 16M join took 765 us against 722 us, a 4M x 16M join 909 against 856 us.
constexpr int kScanItems = 8;
constexpr int kScanTile = kThreads * kScanItems;
constexpr int64_t kScanOne = 2 * kScanTile;

// Exclusive scan of tiles [t0, t1) of `in`, starting from `carry`; returns the sum with it.
__device__ int64_t scan_tiles(const uint32_t* __restrict__ in, int64_t n, int64_t t0, int64_t t1, int64_t carry,
                              int64_t* __restrict__ out, int64_t* tmp) {
    for (int64_t t = t0; t < t1; ++t) {
        const int64_t i0 = t * kScanTile + (int64_t)threadIdx.x * kScanItems;
        uint32_t v[kScanItems];
        int64_t s = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = i0 + k < n ? in[i0 + k] : 0u;
            s += v[k];
        }
        int64_t total;
        int64_t run = block_scan_excl_i64(s, tmp, &total) + carry;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (i0 + k < n) out[i0 + k] = run;
            run += v[k];
        }
        carry += total;
    }
    return carry;
}

__global__ void __launch_bounds__(kThreads) k_scan_one(const uint32_t* __restrict__ in, int64_t n,
                                                        int64_t* __restrict__ out, int64_t* __restrict__ grand) {
    __shared__ int64_t tmp[kThreads / 32];
    const int64_t total = scan_tiles(in, n, 0, (n + kScanTile - 1) / kScanTile, 0, out, tmp);
    if (threadIdx.x == 0 && grand) *grand = total;
}

// A share's sum is published in sums[blockIdx.x] under the scan's tag (a run's scans count up from 1, and the
// run starts with cleared words), and thread t of a later CTA waits for share t. Every CTA publishes before it
// waits, and for lower CTAs only, which the hardware starts first: the grid need not be resident together. The
// wait is bounded by *polls; a CTA whose wait runs out adds up the counts before its share itself (at most a few
// MB from L2), so its share is written, and right, however long the others take.
constexpr int kScanTagShift = 48;  // sums are below 2^48
__global__ void __launch_bounds__(kThreads) k_scan_grid(const uint32_t* __restrict__ in, int64_t n,
                                                         unsigned long long* sums, int64_t* __restrict__ out,
                                                         int64_t* __restrict__ grand, unsigned long long tag,
                                                         const unsigned long long* polls) {
    __shared__ int64_t tmp[kThreads / 32];
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    const int64_t t0 = tiles * blockIdx.x / gridDim.x, t1 = tiles * (blockIdx.x + 1) / gridDim.x;
    int64_t s = 0;
    for (int64_t i = t0 * kScanTile + threadIdx.x; i < t1 * kScanTile && i < n; i += kThreads) s += in[i];
    int64_t total;
    block_scan_excl_i64(s, tmp, &total);
    if (threadIdx.x == 0) atomicExch(sums + blockIdx.x, (tag << kScanTagShift) | (unsigned long long)total);
    bool ok = true;
    int64_t before = 0;
    if (threadIdx.x < blockIdx.x) {  // at most kThreads CTAs
        const uint32_t bound = (uint32_t)*polls;
        ok = false;
        for (uint32_t it = 0; it < bound && !ok; ++it) {
            const unsigned long long v = ld_acquire(sums + threadIdx.x);
            ok = v >> kScanTagShift == tag;
            before = (int64_t)(v & ((1ull << kScanTagShift) - 1));
            if (!ok && it > 64) __nanosleep(100);
        }
    }
    if (!__syncthreads_and(ok)) {
        before = 0;
        for (int64_t i = threadIdx.x; i < t0 * kScanTile; i += kThreads) before += in[i];
    }
    int64_t carry;
    block_scan_excl_i64(before, tmp, &carry);
    const int64_t end = scan_tiles(in, n, t0, t1, carry, out, tmp);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0 && grand) *grand = end;
}
