// direct.h - the unpartitioned join (direct.cu): descriptors and host-side planning.
#pragma once

#include <cstdint>
#include "engine.h"

namespace brig {

// The join of a launch. Device addresses.
struct DirectJoin {
    const uint32_t* key[2];   // inputs: 0 = R, 1 = S
    const uint32_t* val[2];
    uint32_t n[2];
    uint32_t* out_r;
    uint32_t* out_s;
    uint32_t* out_k;          // may be nullptr
    int64_t cap;
    int64_t* counters;        // [kCntWords]
    int64_t* user_count;      // may be nullptr
    PartFn pf;                // filter segments: one per finest partition, as in the partitioned join
    uint32_t nfine;
    uint32_t seg_blocks;
    int32_t fused;            // R is the build side and S is filtered while it is probed
    uint32_t* bloom;          // filter words
    uint2* cmp;               // filter survivors of S [n[1]] (not fused)
    uint2* dir;               // bucket directory [dir_cap]
    uint32_t* rank;           // [build_cap] rank of each build tuple in its bucket
    uint2* table;             // [build_cap] build tuples in bucket order
    uint32_t dir_cap;         // a multiple of kDirTile
    uint32_t build_cap;       // most build tuples
};

// A long bucket [start, start + len) and the streamed tuple that it is compared with.
struct DirectLong {
    uint32_t key, val, start, len;
};
static_assert(sizeof(DirectLong) == 16, "read as one vector");

struct DirectArgs {
    DirectJoin join;
    unsigned long long* gwords; // [kDirectWords], zero at launch
    DirectLong* longs;          // [long_cap]
    uint32_t long_cap;
    uint32_t* first;            // [long_cap] first piece number of each
    uint32_t* left;             // a bit per streamed row: listed in a later round
    int32_t pat_k;              // k of the pattern table (0: none)
};

constexpr int kDirectWords = 18;
constexpr uint32_t kDirTile = 4096;          // directory entries per scan tile
// Limits of the direct path. Engine time in us, partitioned / direct, 10% matches unless noted (|R| x |S|
// in millions; "f": filter of 10 bits per key): 0.1 x 0.1 155 / 45, 0.3 x 1.2 f 219 / 65, 1 x 16 434 / 224,
// 3 x 3 f 292 / 185, 3 x 20 f with all rows matching 926 / 836, 12 x 2 449 / 209, 48 x 3 839 / 529.
// Beyond them the tables leave L2 (6 x 24 with 30% matches 735 / 846, 8 x 8 512 / 639) or the longer side's
// per-row cost outweighs the partitioned join's fixed one (3 x 100 f 1173 / 1279, 0.01 x 100 942 / 1053).
// A row that matches costs the direct join more, and rows that share few table lines wait for one another,
// so the longer side's limit depends on how many pairs are asked for and on the smaller side:
//   S streamed, all rows matching: 3 x 24 791 / 820, 3 x 48 1268 / 1526, 0.1 x 32 695 / 802, 0.1 x 48 943 / 1178,
//     1 x 48 1167 / 1201; 40%: 3 x 48 1037 / 1060, 1 x 32 712 / 553, 0.1 x 48 679 / 769; 10%: 3 x 48 911 / 670,
//     1 x 48 733 / 549, 0.1 x 48 534 / 524
//   filter of few keys: 0.01 x 24 f 395 / 419, 0.01 x 48 f 497 / 1169, 0.1 x 48 f 545 / 541
//   few rows: 0.004 x 8 f 311 / 398, 0.004 x 24 359 / 296, 0.004 x 32 406 / 442; 40%: 0.0003 x 24 480 / 582;
//     all matching: 0.0003 x 4 300 / 206, 0.001 x 8 365 / 411
//   R streamed, all rows matching: 24 x 0.0003 992 / 1054, 48 x 0.0003 1423 / 2058, 48 x 0.01 1149 / 1141
constexpr int64_t kDirectMaxBuild = 3 << 20;     // smaller side
constexpr int64_t kDirectMaxStream = 48 << 20;   // larger side
constexpr int64_t kDirectMidStream = 24 << 20;   // larger side where many rows match or share a small filter
constexpr int64_t kDirectLowStream = 4 << 20;    // larger side where most rows read the same few lines
constexpr int64_t kDirectSmallTable = 256 << 10; // smaller side
constexpr int64_t kDirectFewFilterKeys = 64 << 10;
constexpr int64_t kDirectFewRows = 8 << 10;
// Smaller side of a join whose S is still being copied from the host when it starts (whole call in us,
// partitioned / direct): S the smaller 12 x 2 f 2369 / 2475, 20 x 3 f 3728 / 3955, 30 x 1 5097 / 4907;
// R the smaller 3 x 6 f 1829 / 1893, 3 x 16 f 3820 / 3923, 2 x 7 1906 / 1876, 1 x 8 f 2045 / 1919.
constexpr int64_t kDirectMaxLateR = 1 << 20;     // S, of a larger R
constexpr int64_t kDirectMaxLateS = 2 << 20;     // R, of a larger S
constexpr int64_t kDirectMaxFilter = 56ll << 20; // filter bytes (random accesses slow down above 64 MB)

// Workspace of one join (byte offsets).
struct DirectShape {
    size_t counters = 0, gwords = 0, bloom = 0, cmp = 0, dir = 0, rank = 0, table = 0, longs = 0, first = 0, left = 0;
    size_t total = 0;
    uint32_t dir_cap = 0, build_cap = 0, long_cap = 0;
    int32_t fused = 0;
    int grid = 1;
};

// Whether the join takes the direct path (see direct.cu for the rule). capacity: its output slots; what some
// capacity makes eligible is eligible with 0.
bool direct_eligible(const brig_join_config& cfg, const JoinPlan& p, int64_t capacity);
// ctas: the most CTAs the launch may have (all resident together).
void direct_layout(const JoinPlan& p, int ctas, DirectShape& sh);
void direct_fill(const JoinPlan& p, const JoinIO& io, const DirectShape& sh, char* ws, DirectArgs& a);
// CTAs of the kernel that fit one SM together on the current device. Also sets the kernel's shared-memory
// limit there: called before the first launch.
cudaError_t direct_residency(bool filter, int mode, int k, int* ctas_per_sm);
// Launches the kernel; its counters and state words must be zero.
cudaError_t enqueue_direct(const DirectArgs& a, bool filter, int mode, int k, int grid, cudaStream_t st);

}  // namespace brig
