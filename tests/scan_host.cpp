// The scan kernels (scan.cuh) on the host: a CTA's threads are fibers and the CTAs run one after another: in
// order, each with the sums that it waits for already there, or in reverse, where no wait succeeds.
// argv: n, grid, polls, reverse. Prints "ok" when every offset and the total are right.
#include <ucontext.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <vector>

#define __global__
#define __device__
#define __restrict__
#define __shared__ static
#define __launch_bounds__(...)
constexpr int kThreads = 512;
struct Dim { unsigned x; };
static Dim gridDim, blockIdx;
static std::vector<ucontext_t> fibers(kThreads);
static std::vector<char> done(kThreads);
static ucontext_t scheduler;
static int now, barrier_count;
static unsigned long barrier_gen;
static int64_t lanes[kThreads];
static void yield() { swapcontext(&fibers[now], &scheduler); }
static Dim thread_dim() { return {(unsigned)now}; }
#define threadIdx thread_dim()
static void __syncthreads() {
    const unsigned long gen = barrier_gen;
    if (++barrier_count == kThreads) {
        barrier_count = 0;
        ++barrier_gen;
    }
    while (gen == barrier_gen) yield();
}
// A warp's fibers run in thread order, so once each has stored its value and yielded all 32 values are there.
static int64_t __shfl_up_sync(unsigned, int64_t v, int d) {
    const int me = now;
    lanes[me] = v;
    yield();
    const int64_t x = lanes[(me & 31) >= d ? me - d : me];
    yield();
    return x;
}
static bool votes;
static bool __syncthreads_and(bool v) {
    __syncthreads();
    votes = true;
    __syncthreads();
    votes = votes && v;
    __syncthreads();
    return votes;
}
static void __nanosleep(int) {}
static unsigned long long ld_acquire(const unsigned long long* p) { return *p; }
static void atomicExch(unsigned long long* p, unsigned long long v) { *p = v; }

#include "scan.cuh"

static std::function<void()> body;
static void entry() {
    body();
    done[now] = 1;
    yield();
}
static void run_cta() {
    static std::vector<char> stacks((size_t)kThreads * 65536);
    for (int t = 0; t < kThreads; ++t) {
        done[t] = 0;
        getcontext(&fibers[t]);
        fibers[t].uc_stack.ss_sp = &stacks[(size_t)t * 65536];
        fibers[t].uc_stack.ss_size = 65536;
        makecontext(&fibers[t], entry, 0);
    }
    for (bool left = true; left;) {
        left = false;
        for (now = 0; now < kThreads; ++now)
            if (!done[now]) {
                swapcontext(&scheduler, &fibers[now]);
                left = true;
            }
    }
}

int main(int, char** argv) {
    const int64_t n = atoll(argv[1]);
    gridDim.x = (unsigned)atoi(argv[2]);
    std::vector<uint32_t> in(n);
    std::vector<int64_t> out(n, -1);
    std::vector<unsigned long long> sums(512, (1ull << kScanTagShift) | 5);  // of an earlier scan
    int64_t total = -1, want = 0;
    const unsigned long long polls = strtoull(argv[3], nullptr, 10);
    for (int64_t i = 0; i < n; ++i) in[i] = (uint32_t)((i * 2654435761ull) >> 7) % 1000;
    for (unsigned b = 0; b < gridDim.x; ++b) {
        blockIdx.x = atoi(argv[4]) ? gridDim.x - 1 - b : b;
        body = [&] {
            if (gridDim.x == 1) k_scan_one(in.data(), n, out.data(), &total);
            else k_scan_grid(in.data(), n, sums.data(), out.data(), &total, 2, &polls);
        };
        run_cta();
    }
    int64_t wrong = 0;
    for (int64_t i = 0; i < n; ++i) {
        wrong += out[i] != want;
        want += in[i];
    }
    if (wrong || total != want) printf("%lld of %lld offsets wrong, total %lld of %lld\n", (long long)wrong, (long long)n, (long long)total, (long long)want);
    else puts("ok");
}
