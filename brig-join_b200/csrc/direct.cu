// direct.cu - the unpartitioned join: one cooperative kernel over tables that stay in L2.
//
// On the B200 a random 8-byte L2 read costs 1/280 ns, a random L2 atomic 1/190 ns and a random 8-byte
// L2 store 1/188 ns while the table holds at most 64 MB (64M operations, 512-thread CTAs, two per SM;
// 155, 120 and 116 G/s at 96 MB). Two partition levels cost 1/95 ns per tuple of either relation. So a
// join whose smaller side fits L2 as a hash table runs faster without partitioning it: per build tuple
// one atomic (its rank in its bucket) and one store, per tuple of the other side one directory read,
// and table reads only where the bucket holds the key's tag.
//
// Phases, with a grid barrier (1.2-1.5 us) between them:
//   clear    filter and bucket directory
//   filter   (filtered joins) every R key sets its bits with one 64-bit atomicOr; then every S key reads
//            its word pair and survivors are compacted. The filter's bits are those of the partitioned
//            join (same segments, blocks and masks), so the survivor count is the same
//   count    directory[bucket] += 1 and its tag; the atomic's result is the tuple's rank
//   scan     counts -> start, count and tags present; a tile of the directory takes its table space with
//            one atomic on a cursor, so tiles need no order and no second barrier
//   place    table[start + rank] = tuple
//   probe    the other side streams through the directory and the table
//   long     (only when a bucket exceeds kLockstep) the listed long buckets, spread over the grid in pieces:
//            neighbouring rows of the streamed side often share their skew (Zipf ranks in row order), and a
//            warp that walked its own rows' buckets held up the whole grid. Rows that the list has no room
//            for are walked by warps that have done little or marked and listed in further rounds, two
//            barriers each, so a round's work is bounded and even however many pairs the join has
// A filtered join whose R is the build side (`fused`) builds R's table beside the filter and probes S's
// survivors on the spot: four barriers instead of seven, and no survivors written.
//
// Repeated keys: a bucket keeps all its tuples and is walked by whole warps above kLockstep of them. Hot
// keys on the build side would serialise the atomics on their bucket (0.65 ns each): warps whose lanes
// share a bucket add once per distinct bucket, and the filter build skips keys its CTA has just set.
#include <algorithm>
#include "direct.h"

namespace brig {
namespace {

constexpr int kU = 4;                        // rows per lane and step
constexpr uint32_t kStep = kU * 32;          // rows a warp takes per step
constexpr int kWarps = kThreads / 32;
constexpr int kLockstep = 8;                 // longest bucket the lanes walk in lock step; others are listed
constexpr uint32_t kLongPiece = 256;         // entries of a listed bucket that are walked together
constexpr uint32_t kLongPieces = 1 << 22;    // most pieces of a round (10 ms of walking)
constexpr uint32_t kWalkAhead = 65536;       // entries a warp may walk itself beyond its share (1 ms)
constexpr uint32_t kWalkHere = 64;           // longest bucket that a warp beyond it walks all the same
constexpr int kStage = 128;                  // pairs staged per warp
constexpr int kQueue = 160;                  // streamed rows queued per warp for the table: 31 and a step's
constexpr int kPacked = 256;                 // survivors queued per warp: 127 and a step's
constexpr int kSeen = 1024;                  // keys a CTA remembers while it builds a filter
static_assert(32ull * (kDirectMaxBuild / kLongPiece + 1) <= kLongPieces, "a warp's buckets fit an empty list");
static_assert(kQueue >= 31 + (int)kStep && kPacked >= 127 + (int)kStep, "a step's rows fit");
constexpr uint32_t kBarrierPolls = 1u << 25; // bound of a grid barrier's wait (each poll 0.2 us or more)

// Directory entries. While counting: tuples in the low half, and in the high half 16 two-bit counters
// of the tuples per tag (the key's mix mod 16), which one 64-bit atomicAdd raises together; a bucket of
// at most three tuples overflows none of them. After the scan: low half the bucket's start, high half
// min(count, 255) and a bit per tag present (all of them above three tuples). So a streamed key reads
// table entries only when its bucket holds its tag.
constexpr uint32_t kCntMask = 255;
// Buckets for n build tuples: 1.25 to 1 over n, in whole tiles.
__host__ __device__ __forceinline__ uint32_t dir_entries(uint32_t n) { return ((n + n / 4) / kDirTile + 1) * kDirTile; }
__device__ __forceinline__ uint32_t tag_of(uint32_t m) { return m & 15u; }
__device__ __forceinline__ unsigned long long count_one(uint32_t m) { return 1ull | (1ull << (32 + 2 * tag_of(m))); }
__device__ __forceinline__ uint2 entry_of(uint2 counted, uint32_t start) {
    const uint32_t pairs = counted.y | (counted.y >> 1);  // bit 2t: tag t present
    uint32_t tags = pairs & 0x55555555u;                  // to bit t
    tags = (tags | (tags >> 1)) & 0x33333333u;
    tags = (tags | (tags >> 2)) & 0x0f0f0f0fu;
    tags = (tags | (tags >> 4)) & 0x00ff00ffu;
    tags = (tags | (tags >> 8)) & 0xffffu;
    if (counted.x > 3) tags = 0xffffu;
    return make_uint2(start, min(counted.x, kCntMask) | (tags << 8));
}
__device__ __forceinline__ bool entry_has(uint2 e, uint32_t m) { return (e.y >> (8 + tag_of(m))) & 1u; }

// State words beyond GlobalWord.
enum DirectWord : int {
    kDBarrier = 8,    // arrivals of all barriers so far
    kDExit = 9,       // CTAs that have finished
    kDLong = 10,      // some bucket is long
    kDWalked = 11,    // entries of long buckets walked by the warps that met them
    // In turn by round, so that the next round's are reset while this round's are read:
    kDLongCount = 12, // buckets (high half) and pieces asked of the long list
    kDLongEnd = 14,   // complement of the count at which the list was full (0: it was not)
    kDLeft = 16,      // rows are marked for a further round
};
static_assert(kDLeft + 2 <= kDirectWords, "state words");
// Counters of a join that only this kernel uses.
enum DirectCounter : int { kCntCursor = 6 };  // table space handed out

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Roles and sizes of the join once they are known.
struct Role {
    uint32_t bn, pn;     // build and streamed tuples
    uint32_t bs;         // 1: the build side is S
    uint32_t nb;         // buckets (a multiple of kDirTile)
};

// Per warp: the pairs waiting to be written, and the queue of a phase.
struct WarpShared {
    uint2 pair[kStage];
    uint32_t pair_key[kStage];
    // of long buckets that the warp meets once the list is full: entries walked, of those reported to the
    // grid's count, and the most it may walk as of its last report
    unsigned long long walked, reported, may_walk;
    uint32_t list_full;
    union {
        struct {
            uint32_t key[kQueue], row[kQueue], entry[kQueue];  // entry: start << 8 | min(count, 255)
        } q;
        uint2 packed[kPacked];  // (key, row) of survivors
    };
};
struct Shared {
    WarpShared w[kWarps];
    uint32_t seen[kSeen];
    uint2 pat[kPatterns];                  // pattern table (k != 7)
    Role role;
    uint32_t tmp[kWarps];
    uint32_t base;
    int ok;
};

// One warp's position in the run.
struct Ctx {
    const DirectArgs& a;
    Shared& s;
    uint32_t gw, nw;      // warp index in the grid, warps in the grid
    uint32_t bars;        // barriers passed
    int lane, wid;
};

// Waits until every CTA has arrived; everything written before is visible after. Bounded: when the
// wait runs out, or another CTA's has, an error is counted and every CTA leaves.
__device__ bool grid_barrier(Ctx& c) {
    ++c.bars;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* g = c.a.gwords;
        __threadfence();
        atomicAdd(&g[kDBarrier], 1ull);
        const unsigned long long want = (unsigned long long)c.bars * gridDim.x;
        uint32_t it = 0;
        bool ok = false;
        for (; it < kBarrierPolls; ++it) {
            if (ld_acquire(&g[kDBarrier]) >= want) { ok = true; break; }
            if (it > 64) {
                __nanosleep(100);
                if ((it & 1023u) == 0 && ld_acquire(&g[kGQueue]) != 0) break;
            }
        }
        if (!ok) {
            atomicAdd(&g[kGErrors], 1ull);
            atomicExch(&g[kGQueue], 1ull);  // tells the other CTAs to leave
        }
        c.s.ok = ok ? 1 : 0;
        __threadfence();
    }
    __syncthreads();
    return c.s.ok != 0;
}

// A side of a join: the caller's key and value arrays, or packed filter survivors.
template <bool kPacked>
struct Side {
    const uint32_t* k;
    const uint32_t* v;
    const uint2* kv;
    __device__ __forceinline__ uint32_t load(uint32_t i) const {
        if constexpr (kPacked) return __ldcg(&kv[i].x);
        else return __ldcs(k + i);
    }
    __device__ __forceinline__ uint32_t value(uint32_t i) const {
        if constexpr (kPacked) return __ldcg(&kv[i].y);
        else return __ldcs(v + i);
    }
};
template <bool kPacked>
__device__ __forceinline__ Side<kPacked> side_of(const DirectJoin& d, int rel) {
    return Side<kPacked>{d.key[rel], d.val[rel], d.cmp};
}

// Loads this lane's rows row0 + 32 * u + lane below n (zeros at or past it).
template <class S>
__device__ __forceinline__ void load_step(const S& side, uint64_t row0, uint32_t n, int lane, uint32_t (&t)[kU]) {
#pragma unroll
    for (int u = 0; u < kU; ++u) {
        const uint64_t i = row0 + 32u * u + lane;
        t[u] = i < n ? side.load((uint32_t)i) : 0u;
    }
}

// The rows of a phase are dealt to the warps of the grid in steps of kStep, round robin. Streams this
// warp's steps of a side, the next step's rows loaded before f runs: f(row, keys)
// with key u of this lane at row `row` + 32 * u.
template <class S, class F>
__device__ __forceinline__ void stream(const Ctx& c, const S& side, uint32_t row0, uint32_t n, F&& f) {
    const uint64_t stride = (uint64_t)c.nw * kStep;
    uint32_t t[kU];
    load_step(side, row0, n, c.lane, t);
    for (uint64_t r = row0; r < n; r += stride) {
        uint32_t nt[kU];
        load_step(side, r + stride, n, c.lane, nt);
        f((uint32_t)r + c.lane, t);
#pragma unroll
        for (int u = 0; u < kU; ++u) t[u] = nt[u];
    }
}

// Counts the tuple with mix m in bucket b for the lanes with `on`; lanes of a warp that share a bucket
// and a tag add once together. Returns the tuple's rank.
__device__ __forceinline__ uint32_t bucket_add(uint2* dir, uint32_t b, uint32_t m, bool on, int lane) {
    const uint32_t key = on ? m : ~m;
    // neighbours with the same key: probably a hot key
    const uint32_t next = __shfl_xor_sync(0xffffffffu, key, 1);
    unsigned long long* p = reinterpret_cast<unsigned long long*>(dir + b);
    if (__any_sync(0xffffffffu, on && next == key)) {
        const unsigned long long tagged = on ? (unsigned long long)m : (1ull << 32) + lane;
        const uint32_t peers = __match_any_sync(0xffffffffu, tagged);
        const int leader = __ffs(peers) - 1;
        uint32_t r = 0;
        if (on && lane == leader) {
            // more than three leave the tag counters meaningless; the bucket then counts every tag
            const uint32_t k = (uint32_t)__popc(peers);
            r = (uint32_t)atomicAdd(p, k + ((unsigned long long)min(k, 3u) << (32 + 2 * tag_of(m))));
        }
        r = __shfl_sync(0xffffffffu, r, leader);
        return r + __popc(peers & lanemask_lt());
    }
    return on ? (uint32_t)atomicAdd(p, count_one(m)) : 0u;
}

// The warp's staging buffer of pairs (r, s) or of survivors (key, value).
struct Stage {
    uint2* buf;
    uint32_t* keys;
    int count;
};

__device__ __noinline__ void flush_staged(const DirectJoin* dp, const uint2* buf, const uint32_t* keys, int count, int lane) {
    const DirectJoin& d = *dp;
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0)
        base = atomicAdd(reinterpret_cast<unsigned long long*>(&d.counters[kCntMatches]), (unsigned long long)count);
    base = __shfl_sync(0xffffffffu, base, 0);
    const int64_t cap = d.cap;
    uint32_t* __restrict__ orr = d.out_r;
    uint32_t* __restrict__ oss = d.out_s;
    uint32_t* __restrict__ okk = d.out_k;
#pragma unroll 1
    for (int i = lane; i < count; i += 32) {
        const int64_t dst = (int64_t)base + i;
        if (dst < cap) {
            const uint2 p = buf[i];
            orr[dst] = p.x;
            oss[dst] = p.y;
            if (okk) okk[dst] = keys[i];
        }
    }
    __syncwarp();
}
__device__ __forceinline__ void flush_pairs(const DirectJoin& d, Stage& st, int lane) {
    flush_staged(&d, st.buf, st.keys, st.count, lane);
    st.count = 0;
}

__device__ __forceinline__ void stage_pair(const DirectJoin& d, Stage& st, bool m, uint32_t r, uint32_t s, uint32_t key,
                                           int lane) {
    const uint32_t mm = __ballot_sync(0xffffffffu, m);
    if (!mm) return;
    const int n = __popc(mm);
    if (st.count + n > kStage) flush_pairs(d, st, lane);
    if (m) {
        const int p = st.count + __popc(mm & lanemask_lt());
        st.buf[p] = make_uint2(r, s);
        if (d.out_k) st.keys[p] = key;
    }
    st.count += n;
    __syncwarp();
}

// Writes queued survivors [0, n), n <= 128, with their values, which are read here: four per lane in
// flight and one atomic on the survivor count.
__device__ __forceinline__ void flush_survivors(const DirectJoin& d, const uint2* q, int n, int lane, unsigned long long* errors) {
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0)
        base = atomicAdd(reinterpret_cast<unsigned long long*>(&d.counters[kCntSurvivors]), (unsigned long long)n);
    const uint32_t* val = d.val[1];
    uint2 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = 32 * u + lane;
        if (i < n) {
            x[u] = q[i];
            x[u].y = __ldcs(val + x[u].y);
        }
    }
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = 32 * u + lane;
        if (i < n) {
            if (base + i < d.n[1]) d.cmp[base + i] = x[u];
            else atomicAdd(errors, 1ull);
        }
    }
    __syncwarp();
}

// The entries of lanes with long or uneven buckets: the warp walks the concatenation of its lanes'
// bucket remainders [lo, lo + len), 32 entries at a time. Out of line: few warps come here.
__device__ __noinline__ int walk_spread(const DirectJoin* d, uint32_t key, uint32_t val, uint32_t lo, uint32_t len,
                                        uint32_t bs, int lane, uint2* buf, uint32_t* keys, int count) {
    Stage st{buf, keys, count};
    uint32_t inc = len;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, s);
        if (lane >= s) inc += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t base = 0; base < total; base += 64) {  // two steps of 32 entries in flight
        uint32_t ck[2], cv[2];
        uint2 x[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t g = base + 32u * h + (uint32_t)lane;
            int c = 0;  // the first lane with inc > g owns entry g
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                const uint32_t v = __shfl_sync(0xffffffffu, inc, c + s - 1);
                if (v <= g) c += s;
            }
            const uint32_t c_lo = __shfl_sync(0xffffffffu, lo, c);
            const uint32_t c_start = __shfl_sync(0xffffffffu, inc - len, c);
            ck[h] = __shfl_sync(0xffffffffu, key, c);
            cv[h] = __shfl_sync(0xffffffffu, val, c);
            x[h] = make_uint2(~ck[h], 0u);
            if (g < total) x[h] = __ldcg(d->table + c_lo + (g - c_start));
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            stage_pair(*d, st, x[h].x == ck[h], bs ? cv[h] : x[h].y, bs ? x[h].y : cv[h], ck[h], lane);
    }
    return st.count;
}

// Length of the bucket that starts at `start` and holds at least kCntMask tuples: the first position whose
// tuple is of another bucket, or the end of the placed tuples. A bucket's tuples are adjacent and the
// buckets of a directory tile are in order, so the test is monotone up to the end of the bucket.
__device__ __noinline__ uint32_t long_length(const uint2* table, uint32_t start, uint32_t end, uint32_t b, uint32_t nb) {
    auto inside = [&](uint32_t p) { return p < end && fastrange32(mix32(__ldcg(&table[p].x)), nb) == b; };
    uint32_t lo = start + kCntMask - 1, step = 64;  // lo is inside
    while (inside(lo + step) && step < (1u << 30)) {
        lo += step;
        step <<= 1;
    }
    uint32_t hi = lo + step;  // outside
    while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (inside(mid)) lo = mid; else hi = mid;
    }
    return lo + 1 - start;
}

// Lists the buckets of the lanes with len > 0 for phase_long; false when the list has no room for all of
// them (an empty list has). One atomic takes list entries and piece numbers together, so the first piece
// numbers of the entries ascend.
__device__ __noinline__ bool list_long(const DirectArgs* a, int round, uint32_t key, uint32_t val, uint32_t start,
                                       uint32_t len, int lane) {
    const uint32_t pieces = (len + kLongPiece - 1) / kLongPiece, on = __ballot_sync(0xffffffffu, len > 0);
    uint32_t inc = pieces;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, s);
        if (lane >= s) inc += y;
    }
    const unsigned long long add = ((unsigned long long)__popc(on) << 32) | __shfl_sync(0xffffffffu, inc, 31);
    auto room = [&](unsigned long long to) { return (to >> 32) <= a->long_cap && (uint32_t)to <= kLongPieces; };
    unsigned long long base = 0;
    int fits = 0;
    if (lane == 0) {
        unsigned long long* count = &a->gwords[kDLongCount + (round & 1)];
        if (room(__ldcg(count))) {  // a full list's count stays: at most one addition a warp goes beyond it
            base = atomicAdd(count, add);
            fits = room(base + add);
            if (!fits) atomicMax(&a->gwords[kDLongEnd + (round & 1)], ~base);
        }
    }
    fits = __shfl_sync(0xffffffffu, fits, 0);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (fits && len > 0) {
        const uint32_t at = (uint32_t)(base >> 32) + __popc(on & lanemask_lt());
        a->longs[at] = DirectLong{key, val, start, len};
        a->first[at] = (uint32_t)base + inc - pieces;
    }
    __syncwarp();
    return fits;
}

// The bucket [start, + cnt) of each lane beyond its first three tuples (already compared), in lock step; lanes with
// more than kLockstep or at most three: none. Returns the staging count.
__device__ __noinline__ int probe_rest(const DirectJoin* dp, uint32_t key, uint32_t val, uint32_t start, uint32_t cnt,
                                       uint32_t bs, int lane, uint2* buf, uint32_t* keys, int count) {
    const DirectJoin& d = *dp;
    Stage st{buf, keys, count};
    if (cnt > kLockstep) cnt = 0;
    const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
    for (uint32_t t = 3; t < most; ++t) {
        uint2 x = make_uint2(0u, 0u);
        const bool in = t < cnt;
        if (in) x = __ldcg(d.table + start + t);
        stage_pair(d, st, in && x.x == key, bs ? val : x.y, bs ? x.y : val, key, lane);
    }
    return st.count;
}

// The same for the lanes with more than kLockstep tuples. row: index of the lane's row in the streamed side.
// Long buckets are listed. Once the list is full, a warp walks its buckets itself while it stays within
// kWalkAhead entries of twice what the grid's warps have walked so on average; a warp that holds more of them,
// as where hot rows lie side by side, marks them for the next round. Marking all of them instead cost 1M x 1M
// rows of 100 copies a key 2.2 ms against 0.75 ms; walking all of them, 200 neighbours that match 100K tuples
// each 269 ms against 0.22 ms.
__device__ __noinline__ int probe_long(const DirectArgs* ap, WarpShared* wp, uint32_t key, uint32_t val, uint32_t row,
                                       uint32_t start, uint32_t cnt, uint32_t nb, uint32_t bs, int lane, int count) {
    const DirectArgs& a = *ap;
    const DirectJoin& d = a.join;
    WarpShared& ws = *wp;
    uint32_t len = cnt > kLockstep ? cnt - 3 : 0u;
    if (cnt == kCntMask)
        len = long_length(d.table, start, (uint32_t)__ldcg(&d.counters[kCntCursor]), fastrange32(mix32(key), nb), nb) - 3;
    __syncwarp();
    if (!ws.list_full && list_long(&a, 0, key, val, start + 3, len, lane)) return count;
    const uint32_t total = __reduce_add_sync(0xffffffffu, len);
    int here = 0;
    if (lane == 0) {
        ws.list_full = 1;
        const unsigned long long walked = ws.walked + total;
        if (walked > ws.may_walk || walked - ws.reported > kWalkAhead / 4) {
            const unsigned long long all = atomicAdd(&a.gwords[kDWalked], ws.walked - ws.reported);
            ws.reported = ws.walked;
            ws.may_walk = kWalkAhead + 2 * (all / (gridDim.x * kWarps));
        }
        here = walked <= ws.may_walk;
        if (here) ws.walked = walked;
    }
    here = __shfl_sync(0xffffffffu, here, 0);
    if (!here && len > kWalkHere) {
        atomicOr(&a.left[row >> 5], 1u << (row & 31));
        a.gwords[kDLeft] = 1ull;
        len = 0;
    }
    __syncwarp();
    return walk_spread(&d, key, val, start + 3, len, bs, lane, ws.pair, ws.pair_key, count);
}

// ---- phases ------------------------------------------------------------------------------------------

__device__ __forceinline__ void clear16(void* p, size_t bytes) {
    uint4* q = reinterpret_cast<uint4*>(p);
    const size_t n = bytes / 16;
    for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads)
        q[i] = make_uint4(0u, 0u, 0u, 0u);
}

template <int M>
__device__ __forceinline__ uint32_t fine_index(const PartFn& f, uint32_t key, uint32_t m) {
    if constexpr (M == 0) return top_bits(m, f.b1 + f.b2);
    else return fastmod(key, f.M1, f.P1) * f.P2 + fastmod(key, f.M2, f.P2);
}

template <int M, int K>
__device__ __noinline__ void phase_filter_build(Ctx& c, const uint2* pat) {
    // seen[m mod kSeen]: the mix that the CTA has set last; a mix of another slot to start with
    for (int i = threadIdx.x; i < kSeen; i += kThreads) c.s.seen[i] = (uint32_t)i + 1;
    __syncthreads();
    const DirectJoin& d = c.a.join;
    const uint32_t n = d.n[0], row0 = c.gw * kStep;
    if (row0 >= n) return;
    const PartFn pf = d.pf;
    const uint32_t seg = d.seg_blocks;
    uint32_t* bloom = d.bloom;
    auto insert = [&](uint32_t key, bool on) {
        const uint32_t m = mix32(key);
        const uint32_t f = fine_index<M>(pf, key, m);
        uint32_t& seen = c.s.seen[m & (kSeen - 1)];
        if (on && seen != m) {
            seen = m;
            const BloomSlot sl = bloom_slot(m, f, seg);
            const uint2 mk = slot_masks<K>(pat, sl);
            atomicOr(reinterpret_cast<unsigned long long*>(bloom + sl.widx),
                     (unsigned long long)mk.x | ((unsigned long long)mk.y << 32));
        }
        return m;
    };
    if (d.fused) {
        const uint32_t nb = c.s.role.nb;
        uint2* dir = d.dir;
        uint32_t* rank = d.rank;
        stream(c, side_of<false>(d, 0), row0, n, [&](uint32_t row, const uint32_t (&t)[kU]) {
            uint32_t q[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const uint32_t m = insert(t[u], row + 32u * u < n);
                q[u] = bucket_add(dir, fastrange32(m, nb), m, row + 32u * u < n, c.lane);
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (row + 32u * u < n) rank[row + 32u * u] = q[u];
        });
    } else {
        stream(c, side_of<false>(d, 0), row0, n, [&](uint32_t row, const uint32_t (&t)[kU]) {
#pragma unroll
            for (int u = 0; u < kU; ++u) insert(t[u], row + 32u * u < n);
        });
    }
}

template <int M, int K>
__device__ __noinline__ void phase_filter_probe(Ctx& c, const uint2* pat) {
    const DirectJoin& d = c.a.join;
    const uint32_t n = d.n[1], row0 = c.gw * kStep;
    if (row0 >= n) return;
    const PartFn pf = d.pf;
    const uint32_t seg = d.seg_blocks;
    const uint32_t* bloom = d.bloom;
    uint2* q = c.s.w[c.wid].packed;
    int qn = 0;
    const Side<false> side = side_of<false>(d, 1);
    const uint64_t stride = (uint64_t)c.nw * kStep;
    uint32_t t[kU], nt[kU];
    uint2 w[kU];
    auto words = [&](uint64_t row) {  // the filter words of the rows in t
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t m = mix32(t[u]);
            const uint32_t f = fine_index<M>(pf, t[u], m);
            w[u] = make_uint2(0u, 0u);  // fails every mask
            if (row + 32u * u < n)
                w[u] = __ldcg(reinterpret_cast<const uint2*>(bloom + bloom_slot(m, f, seg).widx));
        }
    };
    load_step(side, row0, n, c.lane, t);
    words((uint64_t)row0 + c.lane);
    load_step(side, row0 + stride, n, c.lane, nt);
    for (uint64_t r = row0; r < n; r += stride) {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const bool pass = bloom_pass(w[u], slot_masks<K>(pat, bloom_slot(mix32(t[u]), 0u, seg)));
            const uint32_t b = __ballot_sync(0xffffffffu, pass);
            if (pass) q[qn + __popc(b & lanemask_lt())] = make_uint2(t[u], (uint32_t)r + 32u * u + c.lane);
            qn += __popc(b);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) t[u] = nt[u];
        words(r + stride + c.lane);  // on their way while survivors are written
        load_step(side, r + 2 * stride, n, c.lane, nt);
        if (qn >= 128) {
            qn -= 128;
            flush_survivors(d, q + qn, 128, c.lane, &c.a.gwords[kGErrors]);
        }
    }
    if (qn > 0) flush_survivors(d, q, qn, c.lane, &c.a.gwords[kGErrors]);
}

// The build side is the smaller one; of a filtered join R, or the survivors of an S below R.
__device__ __noinline__ void set_roles(Ctx& c, bool filter) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const DirectJoin& d = c.a.join;
        const uint32_t nr = d.n[0];
        Role r;
        uint32_t ns = d.n[1];
        if (filter && !d.fused) ns = (uint32_t)__ldcg(&d.counters[kCntSurvivors]);
        r.bs = filter ? (d.fused ? 0u : 1u) : (ns < nr ? 1u : 0u);
        r.bn = r.bs ? ns : nr;
        r.pn = r.bs ? nr : ns;
        r.nb = min(d.dir_cap, dir_entries(r.bn));
        c.s.role = r;
    }
    __syncthreads();
}

template <bool kPacked>
__device__ __forceinline__ void count_run(const Ctx& c, const DirectJoin& d, const Role& r, int rel, uint32_t row0,
                                          uint32_t n) {
    uint2* dir = d.dir;
    uint32_t* rank = d.rank;
    const uint32_t nb = r.nb;
    stream(c, side_of<kPacked>(d, rel), row0, n, [&](uint32_t row, const uint32_t (&t)[kU]) {
        uint32_t q[kU];
        bool on[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t m = mix32(t[u]);
            on[u] = row + 32u * u < n;
            q[u] = bucket_add(dir, fastrange32(m, nb), m, on[u], c.lane);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (on[u]) rank[row + 32u * u] = q[u];
    });
}

template <bool kPacked>
__device__ __forceinline__ void place_run(const Ctx& c, const DirectJoin& d, const Role& r, int rel, uint32_t row0,
                                          uint32_t n) {
    const uint2* dir = d.dir;
    const uint32_t* rank = d.rank;
    uint2* table = d.table;
    const uint32_t nb = r.nb, cap = d.build_cap;
    const Side<kPacked> side = side_of<kPacked>(d, rel);
    stream(c, side, row0, n, [&](uint32_t row, const uint32_t (&t)[kU]) {
        uint32_t pos[kU], v[kU];
        bool on[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t i = row + 32u * u;
            on[u] = i < n;
            pos[u] = v[u] = 0;
            if (on[u]) {
                pos[u] = __ldcg(&dir[fastrange32(mix32(t[u]), nb)].x) + __ldcg(rank + i);
                v[u] = side.value(i);
            }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (!on[u]) continue;
            if (pos[u] < cap) table[pos[u]] = make_uint2(t[u], v[u]);
            else atomicAdd(&c.a.gwords[kGErrors], 1ull);
        }
    });
}

// The build side's tuples: counted (kPlace false) or placed.
template <bool kFilter, bool kPlace>
__device__ __noinline__ void phase_build(Ctx& c) {
    const DirectJoin& d = c.a.join;
    const Role r = c.s.role;
    const uint32_t row0 = c.gw * kStep;
    if (row0 >= r.bn) return;
    if (kFilter && r.bs) {
        if constexpr (kPlace) place_run<true>(c, d, r, 1, row0, r.bn);
        else count_run<true>(c, d, r, 1, row0, r.bn);
    } else {
        if constexpr (kPlace) place_run<false>(c, d, r, r.bs ? 1 : 0, row0, r.bn);
        else count_run<false>(c, d, r, r.bs ? 1 : 0, row0, r.bn);
    }
}

// Counts to entries: each tile of kDirTile buckets is scanned by one CTA and takes its table space from
// the join's cursor.
__device__ __noinline__ void phase_scan(Ctx& c) {
    constexpr int kPer = kDirTile / kThreads;  // entries per thread
    static_assert(kPer % 2 == 0, "16-byte accesses");
    const DirectJoin& d = c.a.join;
    const uint32_t tiles = c.s.role.nb / kDirTile;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint4* p = reinterpret_cast<uint4*>(d.dir + (size_t)t * kDirTile + threadIdx.x * kPer);
        uint4 v[kPer / 2];  // two entries each
        uint32_t sum = 0, most = 0;
#pragma unroll
        for (int k = 0; k < kPer / 2; ++k) {
            v[k] = __ldcg(p + k);
            sum += v[k].x + v[k].z;
            most = max(most, max(v[k].x, v[k].z));
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (c.lane >= o) x += y;
        }
        __syncthreads();  // the previous tile is done with tmp and base
        if (c.lane == 31) c.s.tmp[c.wid] = x;
        if (most > kLockstep) c.a.gwords[kDLong] = 1ull;
        __syncthreads();
        uint32_t w = c.lane < kWarps ? c.s.tmp[c.lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (c.lane >= o) w += y;
        }
        if (threadIdx.x == kThreads - 1)
            c.s.base = (uint32_t)atomicAdd(reinterpret_cast<unsigned long long*>(&d.counters[kCntCursor]),
                                           (unsigned long long)w);
        const uint32_t before = __shfl_sync(0xffffffffu, w, c.wid > 0 ? c.wid - 1 : 0);
        __syncthreads();
        uint32_t run = c.s.base + x - sum + (c.wid > 0 ? before : 0u);
#pragma unroll
        for (int k = 0; k < kPer / 2; ++k) {
            const uint2 e0 = entry_of(make_uint2(v[k].x, v[k].y), run);
            run += v[k].x;
            const uint2 e1 = entry_of(make_uint2(v[k].z, v[k].w), run);
            run += v[k].z;
            p[k] = make_uint4(e0.x, e0.y, e1.x, e1.y);
        }
    }
}

// Compares queued rows [0, n) of the streamed side with their buckets, up to kPer per lane: the row's
// value and the bucket's first three tuples are read together, the rest of longer buckets in probe_rest or
// probe_long.
template <int kPer, bool kPacked>
__device__ __forceinline__ void probe_queued(const Ctx& c, const DirectJoin& d, const Side<kPacked>& side, uint32_t bs,
                                             uint32_t nb, const uint32_t* qkey, const uint32_t* qrow, const uint32_t* qent,
                                             int n, Stage& st) {
    __syncwarp();
    uint32_t key[kPer], val[kPer], e[kPer];
    uint2 x[kPer][3];
    uint32_t more = 0;
#pragma unroll
    for (int h = 0; h < kPer; ++h) {
        const int i = 32 * h + c.lane;
        key[h] = val[h] = e[h] = 0;
        if (i < n) {
            key[h] = qkey[i];
            e[h] = qent[i];
            val[h] = side.value(qrow[i]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[h][k] = make_uint2(~key[h], 0u);
            if ((e[h] & kCntMask) > (uint32_t)k) x[h][k] = __ldcg(d.table + (e[h] >> 8) + k);
        }
        const uint32_t cnt = e[h] & kCntMask;
        more |= cnt > kLockstep ? 1u << (kPer + h) : cnt > 3 ? 1u << h : 0u;
    }
#pragma unroll
    for (int h = 0; h < kPer; ++h)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            stage_pair(d, st, x[h][k].x == key[h], bs ? val[h] : x[h][k].y, bs ? x[h][k].y : val[h], key[h], c.lane);
    more = __reduce_or_sync(0xffffffffu, more);
    if (more) {
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
            const uint32_t start = e[h] >> 8, cnt = e[h] & kCntMask;
            if ((more >> h) & 1u)
                st.count = probe_rest(&d, key[h], val[h], start, cnt, bs, c.lane, st.buf, st.keys, st.count);
            if ((more >> (kPer + h)) & 1u)
                st.count = probe_long(&c.a, &c.s.w[c.wid], key[h], val[h], 32 * h + c.lane < n ? qrow[32 * h + c.lane] : 0u,
                                      start, cnt, nb, bs, c.lane, st.count);
        }
    }
    __syncwarp();
}

// Streams a run of the probe side through the directory; rows whose bucket holds their tag are queued
// and compared with the table 64 at a time. The directory entries of a step are read while the queue of
// the last one is worked off. Few values live across the two parts: with a step's table entries held
// beside its rows, 64 registers spilled, and two CTAs' spills do not fit L1 (16.8M rows, 2M-tuple table:
// 322 us). Of the 230 to 250 bytes of spill stores that remain, all but 12 to 28 save registers across the
// calls out of line (flush_staged, probe_rest, probe_long), which few warps' steps make. kFilter: rows are
// tested against the filter first (S of a fused join). Returns this lane's rows that passed.
template <bool kPacked, bool kFilter, int M, int K>
__device__ __noinline__ uint32_t probe_run(const Ctx& c, const DirectJoin& d, const Role& r, int rel,
                                           uint32_t row0, uint32_t n, const uint2* pat) {
    WarpShared& ws = c.s.w[c.wid];
    Stage st{ws.pair, ws.pair_key, 0};
    if (c.lane == 0) {
        ws.walked = ws.reported = 0;
        ws.may_walk = kWalkAhead;
        ws.list_full = 0;
    }
    const uint32_t nb = r.nb, bs = r.bs;
    const uint2* dir = d.dir;
    const Side<kPacked> side = side_of<kPacked>(d, rel);
    const uint64_t stride = (uint64_t)c.nw * kStep;
    uint32_t passed = 0;
    uint32_t t[kU], nt[kU];
    uint2 e[kU];
    auto entries = [&](uint64_t row) {  // the directory entries of the rows in t
        uint32_t on = 0;
        if constexpr (kFilter) {
            uint2 w[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const uint32_t m = mix32(t[u]);
                const BloomSlot sl = bloom_slot(m, fine_index<M>(d.pf, t[u], m), d.seg_blocks);
                w[u] = make_uint2(0u, 0u);
                if (row + 32u * u < n) w[u] = __ldcg(reinterpret_cast<const uint2*>(d.bloom + sl.widx));
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (bloom_pass(w[u], slot_masks<K>(pat, bloom_slot(mix32(t[u]), 0u, d.seg_blocks)))) on |= 1u << u;
            passed += __popc(on);
        } else {
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (row + 32u * u < n) on |= 1u << u;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            e[u] = make_uint2(0u, 0u);
            if ((on >> u) & 1u) e[u] = __ldcg(dir + fastrange32(mix32(t[u]), nb));
        }
    };
    int qn = 0;
    load_step(side, row0, n, c.lane, t);
    entries((uint64_t)row0 + c.lane);
    load_step(side, row0 + stride, n, c.lane, nt);
    for (uint64_t r0 = row0; r0 < n; r0 += stride) {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const bool has = entry_has(e[u], mix32(t[u]));
            const uint32_t b = __ballot_sync(0xffffffffu, has);
            if (has) {
                const int at = qn + __popc(b & lanemask_lt());
                ws.q.key[at] = t[u];
                ws.q.row[at] = (uint32_t)r0 + 32u * u + c.lane;
                ws.q.entry[at] = (e[u].x << 8) | (e[u].y & kCntMask);
            }
            qn += __popc(b);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) t[u] = nt[u];
        entries(r0 + stride + c.lane);
        load_step(side, r0 + 2 * stride, n, c.lane, nt);
        while (qn >= 32) {  // the queue's end first: its order does not matter
            const int k = min(qn, 64);
            qn -= k;
            probe_queued<2>(c, d, side, bs, nb, ws.q.key + qn, ws.q.row + qn, ws.q.entry + qn, k, st);
        }
    }
    if (qn > 0) probe_queued<1>(c, d, side, bs, nb, ws.q.key, ws.q.row, ws.q.entry, qn, st);
    if (st.count > 0) flush_pairs(d, st, c.lane);
    return passed;
}

template <int M, int K, bool kFilter>
__device__ __noinline__ void phase_probe(Ctx& c, const uint2* pat) {
    const DirectJoin& d = c.a.join;
    const Role r = c.s.role;
    const uint32_t row0 = c.gw * kStep;
    if (row0 >= r.pn || r.bn == 0) return;
    if constexpr (kFilter) {
        if (d.fused) {
            uint32_t p = probe_run<false, true, M, K>(c, d, r, 1, row0, r.pn, pat);
            p = __reduce_add_sync(0xffffffffu, p);
            if (c.lane == 0 && p)
                atomicAdd(reinterpret_cast<unsigned long long*>(&d.counters[kCntSurvivors]), (unsigned long long)p);
        } else {  // S's survivors are the build side
            probe_run<false, false, M, K>(c, d, r, 0, row0, r.pn, pat);
        }
    } else {
        probe_run<false, false, M, K>(c, d, r, r.bs ? 0 : 1, row0, r.pn, pat);
    }
}

// The long list: each warp takes up to 32 pieces at a time.
__device__ __noinline__ void phase_long(Ctx& c, int round) {
    const DirectJoin& d = c.a.join;
    const unsigned long long full = __ldcg(&c.a.gwords[kDLongEnd + (round & 1)]);
    const unsigned long long end = full ? ~full : __ldcg(&c.a.gwords[kDLongCount + (round & 1)]);
    const uint32_t n = (uint32_t)(end >> 32), pieces = (uint32_t)end;
    const uint32_t per = min(32u, (pieces + c.nw - 1) / c.nw), bs = c.s.role.bs;
    const uint32_t* first = c.a.first;
    Stage st{c.s.w[c.wid].pair, c.s.w[c.wid].pair_key, 0};
    for (uint32_t g0 = c.gw * per; g0 < pieces; g0 += c.nw * per) {
        // e0: the entry of piece g0, the last whose first piece is not beyond it
        uint32_t e0 = 0;
        if (pieces == n) {
            e0 = g0;
        } else {
            for (uint32_t span = n; span > 1;) {
                const uint32_t step = (span + 31) / 32, at = step * c.lane;
                const uint32_t b = __ballot_sync(0xffffffffu, at < span && __ldcg(first + e0 + min(at, span - 1)) <= g0);
                const uint32_t k = step * (31 - __clz(b));
                e0 += k;
                span = min(step, span - k);
            }
        }
        // every entry has a piece, so those of the 32 pieces are among the next 32 entries
        const uint32_t f = e0 + c.lane < n ? __ldcg(first + e0 + c.lane) : 0xffffffffu, g = g0 + c.lane;
        int i = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            if (__shfl_sync(0xffffffffu, f, i + s) <= g) i += s;
        const uint32_t fi = __shfl_sync(0xffffffffu, f, i);
        uint4 p = make_uint4(0u, 0u, 0u, 0u);  // key, value, start, length
        if (c.lane < per && g < pieces) {
            p = __ldcg(reinterpret_cast<const uint4*>(c.a.longs + e0 + i));
            const uint32_t k = (g - fi) * kLongPiece;
            p.z += k;
            p.w = min(kLongPiece, p.w - k);
        }
        __syncwarp();
        st.count = walk_spread(&d, p.x, p.y, p.z, p.w, bs, c.lane, st.buf, st.keys, st.count);
    }
    if (st.count > 0) flush_pairs(d, st, c.lane);
}

// Lists the marked rows, 32 neighbours at a time, until the list has no room; those that it takes are
// unmarked. The first 32 that a round lists always fit, so every round makes progress.
__device__ __noinline__ void phase_relist(Ctx& c, int round) {
    const DirectArgs& a = c.a;
    const DirectJoin& d = a.join;
    const Role r = c.s.role;
    const Side<false> side = side_of<false>(d, r.bs ? 0 : 1);  // the streamed side is never packed
    const uint32_t words = (r.pn + 31) / 32, end = (uint32_t)__ldcg(&d.counters[kCntCursor]);
    for (uint32_t w0 = c.gw * 32; w0 < words; w0 += c.nw * 32) {
        const uint32_t mine = w0 + c.lane < words ? __ldcg(a.left + w0 + c.lane) : 0u;
        for (uint32_t todo = __ballot_sync(0xffffffffu, mine != 0); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const uint32_t bits = __shfl_sync(0xffffffffu, mine, src);
            const uint32_t row = (w0 + src) * 32 + c.lane;
            uint32_t key = 0, val = 0, start = 0, len = 0;
            if ((bits >> c.lane) & 1u) {
                key = side.load(row);
                val = side.value(row);
                const uint32_t b = fastrange32(mix32(key), r.nb);
                const uint2 e = __ldcg(d.dir + b);
                start = e.x;
                len = e.y & kCntMask;
                if (len == kCntMask) len = long_length(d.table, start, end, b, r.nb);
                start += 3;
                len -= 3;
            }
            __syncwarp();
            if (!list_long(&a, round, key, val, start, len, c.lane)) {
                if (c.lane == 0) a.gwords[kDLeft + (round & 1)] = 1ull;
                return;  // what is still marked waits for the next round
            }
            if (c.lane == 0) a.left[w0 + src] = 0u;
        }
    }
}

// Walks what the probe has listed, then lists and walks the marked rows until none is left. Returns false when
// a barrier ran out.
__device__ __noinline__ bool long_rounds(Ctx& c) {
    const DirectArgs& a = c.a;
    for (int round = 0;; ++round) {
        if (!grid_barrier(c)) return false;
        const bool left = __ldcg(&a.gwords[kDLeft + (round & 1)]) != 0;
        if (blockIdx.x == 0 && threadIdx.x == 0)  // the next round's words, last read a round ago
            for (int w : {kDLongCount, kDLongEnd, kDLeft}) a.gwords[w + (~round & 1)] = 0ull;
        phase_long(c, round);
        if (!left) return true;
        if (!grid_barrier(c)) return false;
        phase_relist(c, round + 1);
    }
}

// Returns false when a barrier ran out.
template <int M, int K, bool kFilter>
__device__ bool run_join(Ctx& c, const uint2* pat) {
    const DirectArgs& a = c.a;
    const DirectJoin& d = a.join;
    const bool fused = kFilter && d.fused;
    if (!kFilter || fused) set_roles(c, kFilter);
    if constexpr (kFilter) {
        clear16(d.bloom, (size_t)d.nfine * d.seg_blocks * 32);
        if (fused) clear16(d.dir, (size_t)c.s.role.nb * 8);
        if (!grid_barrier(c)) return false;
        phase_filter_build<M, K>(c, pat);
        if (!grid_barrier(c)) return false;
        if (!fused) {
            phase_filter_probe<M, K>(c, pat);
            if (!grid_barrier(c)) return false;
        }
        if (!fused) set_roles(c, kFilter);
    }
    if (!fused) {
        clear16(d.dir, (size_t)c.s.role.nb * 8);
        if (!grid_barrier(c)) return false;
        phase_build<kFilter, false>(c);
        if (!grid_barrier(c)) return false;
    }
    phase_scan(c);
    if (!grid_barrier(c)) return false;
    const bool longs = __ldcg(&a.gwords[kDLong]) != 0;
    if (longs) clear16(a.left, ((size_t)c.s.role.pn + 127) / 128 * 16);
    phase_build<kFilter, true>(c);
    if (!grid_barrier(c)) return false;
    phase_probe<M, K, kFilter>(c, pat);
    if (longs && !long_rounds(c)) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!kFilter) d.counters[kCntSurvivors] = d.n[1];
        d.counters[kCntTasks] = 1;
    }
    return true;
}

template <int M, int K, bool kFilter>
__global__ void __launch_bounds__(kThreads, 2) k_direct(const __grid_constant__ DirectArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared& s = *reinterpret_cast<Shared*>(smem);
    if (kFilter && K != kBloomFastK) fill_patterns(s.pat, a.pat_k);
    __syncthreads();
    Ctx c{a, s, 0, 0, 0, (int)(threadIdx.x & 31), (int)(threadIdx.x >> 5)};
    // consecutive warps of the grid sit on different SMs, so a few steps still use many of them
    c.gw = c.wid * gridDim.x + blockIdx.x;
    c.nw = gridDim.x * kWarps;
    run_join<M, K, kFilter>(c, s.pat);
    // the last CTA to finish publishes the count
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&a.gwords[kDExit], 1ull) + 1 == gridDim.x && a.join.user_count) {
            __threadfence();
            const bool failed = __ldcg(&a.gwords[kGErrors]) != 0;
            *a.join.user_count = failed ? -1 : (int64_t)__ldcg(&a.join.counters[kCntMatches]);
        }
    }
}

const void* kernel_of(bool filter, int mode, int k) {
    if (!filter) return reinterpret_cast<const void*>(&k_direct<0, 0, false>);
    const bool fast = k == kBloomFastK;
    if (mode == 0)
        return fast ? reinterpret_cast<const void*>(&k_direct<0, kBloomFastK, true>)
                    : reinterpret_cast<const void*>(&k_direct<0, 0, true>);
    return fast ? reinterpret_cast<const void*>(&k_direct<1, kBloomFastK, true>)
                : reinterpret_cast<const void*>(&k_direct<1, 0, true>);
}

}  // namespace

cudaError_t direct_residency(bool filter, int mode, int k, int* ctas_per_sm) {
    const void* fn = kernel_of(filter, mode, k);
    const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared));
    if (err != cudaSuccess) return err;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, kThreads, sizeof(Shared));
}

cudaError_t enqueue_direct(const DirectArgs& a, bool filter, int mode, int k, int grid, cudaStream_t st) {
    void* args[] = {const_cast<DirectArgs*>(&a)};
    const cudaError_t err =
        cudaLaunchCooperativeKernel(kernel_of(filter, mode, k), dim3(grid), dim3(kThreads), args, sizeof(Shared), st);
    if (err == cudaSuccess) note_launches(1);
    return err;
}

bool direct_eligible(const brig_join_config& cfg, const JoinPlan& p, int64_t capacity) {
    // A caller that sets fan-outs, table sizes or wait bounds gets the partitioned join that has them.
    if (cfg.partition_size || cfg.second_partition_size || cfg.table_capacity || cfg.s_chunk || cfg.bloom_probe_level ||
        cfg.max_level1_bits || cfg.wait_poll_limit || cfg.partition_fill || cfg.slices_per_sm)
        return false;
    const int64_t small = std::min(p.nr, p.ns), large = std::max(p.nr, p.ns);
    if (small < 1 || small > kDirectMaxBuild || (p.bloom && p.bloom_bits / 8 > kDirectMaxFilter)) return false;
    // room for the pairs of many rows: half of them, of a small table a quarter
    const bool many = capacity >= (small < kDirectSmallTable ? large / 4 : large / 2), few_rows = small < kDirectFewRows;
    int64_t limit = kDirectMaxStream;
    if (p.ns > p.nr) {
        if (many || few_rows || (p.bloom && small < kDirectFewFilterKeys)) limit = kDirectMidStream;
        if (few_rows && (many || p.bloom)) limit = kDirectLowStream;
    } else if (many && few_rows) {
        limit = kDirectMidStream;
    }
    return large <= limit;
}

void direct_layout(const JoinPlan& p, int ctas, DirectShape& sh) {
    sh = DirectShape{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        off = (off + 255) & ~(size_t)255;
        const size_t o = off;
        off += bytes;
        return o;
    };
    sh.counters = take(kCntWords * 8);
    sh.gwords = take(kDirectWords * 8);
    sh.fused = p.bloom && p.nr <= kDirectMaxBuild ? 1 : 0;
    const int64_t build = sh.fused ? p.nr : std::min(p.nr, p.ns);
    sh.build_cap = (uint32_t)build;
    sh.dir_cap = dir_entries(sh.build_cap);
    if (p.bloom) sh.bloom = take((size_t)p.nfine * p.seg_blocks * 32);
    sh.dir = take((size_t)sh.dir_cap * 8);
    sh.table = take((size_t)build * 8);
    sh.rank = take((size_t)build * 4);
    if (p.bloom && !sh.fused) sh.cmp = take((size_t)p.ns * 8);
    // One streamed row per bucket above kLockstep. A round over a full list costs two barriers and a look at
    // the marks (10-20 us), so small build sides get up to 32768.
    const int64_t stream = std::max(p.nr, p.ns);
    sh.long_cap = (uint32_t)std::max(build / kLockstep + 64, std::min<int64_t>(stream / 4, 32768));
    sh.longs = take((size_t)sh.long_cap * sizeof(DirectLong));
    sh.first = take((size_t)sh.long_cap * 4);
    sh.left = take((size_t)(stream + 127) / 128 * 16);
    sh.total = off + 256;
    // Every resident CTA, fewer while the longer side gives each warp less than one step.
    const int64_t want = (std::max(p.nr, p.ns) + kStep * kWarps - 1) / (kStep * kWarps);
    sh.grid = (int)std::min<int64_t>(want, ctas);
}

void direct_fill(const JoinPlan& p, const JoinIO& io, const DirectShape& sh, char* ws, DirectArgs& a) {
    a = DirectArgs{};
    DirectJoin& d = a.join;
    d.key[0] = io.rk;
    d.key[1] = io.sk;
    d.val[0] = io.rv;
    d.val[1] = io.sv;
    d.n[0] = (uint32_t)io.nr;
    d.n[1] = (uint32_t)io.ns;
    d.out_r = io.out.r_val;
    d.out_s = io.out.s_val;
    d.out_k = io.out.key;
    d.cap = io.out.capacity;
    d.counters = reinterpret_cast<int64_t*>(ws + sh.counters);
    d.user_count = io.out.d_count;
    d.pf = p.pf;
    d.nfine = (uint32_t)p.nfine;
    d.seg_blocks = p.seg_blocks;
    d.fused = sh.fused;
    d.bloom = reinterpret_cast<uint32_t*>(ws + sh.bloom);
    d.cmp = reinterpret_cast<uint2*>(ws + sh.cmp);
    d.dir = reinterpret_cast<uint2*>(ws + sh.dir);
    d.rank = reinterpret_cast<uint32_t*>(ws + sh.rank);
    d.table = reinterpret_cast<uint2*>(ws + sh.table);
    d.dir_cap = sh.dir_cap;
    d.build_cap = sh.build_cap;
    a.gwords = reinterpret_cast<unsigned long long*>(ws + sh.gwords);
    a.longs = reinterpret_cast<DirectLong*>(ws + sh.longs);
    a.long_cap = sh.long_cap;
    a.first = reinterpret_cast<uint32_t*>(ws + sh.first);
    a.left = reinterpret_cast<uint32_t*>(ws + sh.left);
    a.pat_k = p.bloom && p.k != kBloomFastK ? p.k : 0;
}

}  // namespace brig
