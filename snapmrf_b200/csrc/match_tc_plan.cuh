// Work units, candidate lists and launch interface of the tensor-core scoring
// kernel (match_tc.cu), shared with the FP32 form that screens with it
// (match_fp32_tc.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"

namespace snapmrf {
namespace tc {

constexpr int BM = 128;                 // voxels per tile (TMEM lanes)
constexpr int BA = 128;                 // atoms per tile
constexpr int BN = 2 * BA;              // B rows per tile
constexpr int BK = 64;                  // bf16 per 128-byte swizzled row
constexpr int BK8 = 128;                // e4m3 per 128-byte swizzled row
constexpr float E4M3_MAX = 448.f;       // largest finite E4M3 value
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK * 2;    // 16 KB
constexpr int B_BYTES = BN * BK * 2;    // 32 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int TOPK_MAX = 16;
constexpr int NLISTS = 2;               // top-k lists per voxel (one per half tile)
constexpr int MAX_PARTS = 8;            // parts an item of the last round may be split into
constexpr int THREADS = 320;
// Scores that pass the epilogue's threshold wait in shared memory, HOLD per
// epilogue thread, until some thread of the warp has no room for four more.
constexpr int HOLD = 12, EPI_THREADS = 256;
constexpr int HOLD_BYTES = HOLD * EPI_THREADS * 8;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + HOLD_BYTES + 1024;
static_assert(SMEM_BYTES + 2 * BM * 8 + 512 <= 227 * 1024, "shared memory of one CTA");
constexpr uint32_t TMEM_COLS = 512;

// What the FP32 form's screen knows of its operands.  v = hi + lo + rest, hi
// and lo its BF16 parts; with c = k / 32 the chunk of element k of nk chunks,
// forward: sum of (nk - c) v_k^2, backward: of (c + 1) v_k^2.  Atoms: the largest
// value of any (the bits of floats >= 0 order as integers); voxels: of the
// slot's voxel at unit norm.
struct AtomStats {
    unsigned norm2, forward2, backward2, lo2, rest2;
};
struct VoxelStats {
    float norm2;                          // 0: nothing scores above 0; < 0: left to the FP32 kernel
    float forward, backward, lo, rest;    // square roots
};
// Twice a bound of |approximate score - FP32 score| (the argument: match_fp32_tc.cu).
__device__ __forceinline__ float screen_margin(const AtomStats &a, const VoxelStats &v, int nk) {
    auto root = [](unsigned bits) { return sqrtf(__uint_as_float(bits)); };
    const float sums = 0x1p-24f * (1.f + (float)nk * 0x1p-17f) *
                       (32.f * root(a.forward2) * v.forward + 61.f * root(a.backward2) * v.backward);
    const float parts = root(a.lo2) * v.lo + root(a.rest2) + root(a.norm2) * (v.rest + 0x1p-20f);
    return 2.002f * (sums + parts);
}

struct Args {
    const long long *tile_start;  // [nbins + 1], in work items
    int nbins;
    int bin_lo, bin_hi;           // bins of this launch
    long long bin_natoms;         // atoms per bin
    int atom0;                    // atoms [atom0, atom0 + chunk_natoms) of each bin are in the operand
    int chunk_natoms;
    int plan_tiles;               // atom tiles that tail_plan splits: of the first chunk
    struct TailPlan *plan;        // out: the launch's plan, for the rescoring
    int nk;                       // K chunks of BK
    int tile_stride;              // atom tiles visited in the order (at * tile_stride) % natiles
    uint32_t idesc;               // tcgen05 instruction descriptor
    const float *ascale2;         // E4M3: [NATOMS] 1 / (atom scale)^2
    long long cap;                // voxel slots; the split items' lists start there
    float *top_s;                 // [slots][NLISTS][TOPK_MAX]; SPLIT: lists at list_offset
    int *top_i;
    int *err;
    // SPLIT: candidates within screen_margin of the best score
    int list_cap;                 // entries per list
    const AtomStats *atom_stats;  // of the atoms packed so far
    const VoxelStats *vox_stats;  // [slots]
    int *list_n;                  // [slots][lists] entries, LIST_OVER: more than the list holds
    float *list_best;             // [slots][lists] the best score the list's thread has seen
    int resume;                   // the lists continue those of an earlier launch (atom0 > 0)
};
constexpr int LIST_OVER = 1 << 30;
// SPLIT: lists per voxel slot (one per epilogue thread of the voxel)
__host__ __device__ constexpr int split_lists(bool imag) { return imag ? 4 : 2; }

// How the items of a launch fall on its CTAs.  Whole rounds run one CTA per
// item; the `rem` items past the last whole round would leave most CTAs idle for a full item's time, so each is split into `parts` by its
// atom tiles (part p takes every parts-th tile from p on), each part with
// lists of its own that the rescoring joins.  parts: the fewest (up to
// MAX_PARTS and the tiles there are) whose last rounds take the least time, if
// that is at most 3/4 of the unsplit item's.  240 x 240 voxels over 41 B1
// blocks, BF16 top-16 (921 items on 148 CTAs): 6.33 rounds instead of 7.
// 16,384 voxels against 111,008 complex atoms (128 items, 0.875 of an item's
// time in 8 parts) measured slower split, 6.22 against 6.01 ms: the chip is
// at its power limit either way, and the rescoring joins 16 lists.
// (A bin larger than the operand is scored in chunks whose launches go on with
// the same lists, so they share the plan of the first chunk.)
struct TailPlan {
    long long item0;       // the launch's first item; the numbers below count from it
    long long bulk, work;  // items before the split ones; CTA work units
    int parts;
};
__device__ __forceinline__ TailPlan tail_plan(long long item0, long long items, int grid, int natiles) {
    TailPlan t;
    t.item0 = item0;
    t.bulk = items / grid * grid;
    const int rem = (int)(items - t.bulk);
    t.parts = 1;
    int best = rem ? natiles : 0;  // tile times of the last rounds
    for (int s = 2; rem && s <= min(MAX_PARTS, natiles); s++) {
        const int c = ((rem * s + grid - 1) / grid) * ((natiles + s - 1) / s);
        if (c < best && 4 * c <= 3 * natiles) {
            best = c;
            t.parts = s;
        }
    }
    t.work = t.bulk + (long long)rem * t.parts;
    return t;
}
// Work unit w: its item (from 0), its part of that item's atom tiles and the
// tile step, and the item whose list slots it writes.
struct WorkUnit {
    long long item, list_item;
    int part, step;
};
__device__ __forceinline__ WorkUnit work_unit(const TailPlan &t, long long w, long long cap_items) {
    WorkUnit u;
    if (w < t.bulk || t.parts == 1) {
        u.item = u.list_item = w;
        u.part = 0;
        u.step = 1;
    } else {
        const long long q = w - t.bulk;
        u.item = t.bulk + q / t.parts;
        u.part = (int)(q % t.parts);
        u.step = t.parts;
        u.list_item = cap_items + q;
    }
    return u;
}

// The tiles of a work unit: (at * stride) % natiles for at = part, part +
// step, .., without a division per tile.
struct TileWalk {
    int at, by, n;
    __device__ __forceinline__ TileWalk(const WorkUnit &u, int stride, int natiles)
        : at((int)((long long)u.part * stride % natiles)), by((int)((long long)u.step * stride % natiles)),
          n(natiles) {}
    __device__ __forceinline__ void next() {
        at += by;
        if (at >= n) at -= n;
    }
};

// Where a voxel slot's lists are: its own list slot, or one per part of its
// item when the item was split (tail_plan).
struct Lists {
    const float *top_s;
    const int *top_i;
    const TailPlan *plan;  // of the scoring launch
    long long cap;
    int vt;
};
struct ListSlots {
    long long first;  // list slots first, first + vt, ..
    int n;
};
__device__ __forceinline__ ListSlots list_slots(const Lists &l, long long slot) {
    const TailPlan t = *l.plan;
    const long long item = slot / l.vt - t.item0;
    if (item < t.bulk || t.parts == 1) return {slot, 1};
    return {l.cap + (item - t.bulk) * t.parts * l.vt + slot % l.vt, t.parts};
}

// SPLIT: entries of a list of an item in `parts` parts.  A part sees every
// parts-th tile; near atoms share tiles, so its share may be twice the average.
__host__ __device__ inline int part_cap(int cap, int parts) {
    if (parts == 1) return cap;
    const int share = (2 * cap / parts + 31) / 32 * 32;
    return share > 64 ? share : 64;
}
// Where list `lid` (list slot x lists + list) begins: the slots' own lists
// first (`own` of them), then those of the split items.
__device__ __forceinline__ long long list_offset(long long lid, long long own, int cap, int parts) {
    return lid < own ? lid * cap : own * cap + (lid - own) * part_cap(cap, parts);
}
// Entries of one of a split voxel slot's lists over its parts, at most.
inline long long split_entries(int cap) {
    long long most = 0;
    for (int parts = 2; parts <= MAX_PARTS; parts++)
        most = std::max(most, (long long)parts * part_cap(cap, parts));
    return most;
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// List slots of split items (in items): at most MAX_PARTS parts of the items
// of one partial round.
inline long long split_slots(long long items, int grid) {
    return MAX_PARTS * std::min<long long>(items, std::max(0, grid - 1));
}

// One launch of the scoring kernel over packed operands.
struct ScoreLaunch {
    const void *A, *B;
    long long arows, brows, Kp;  // operand rows and their pitch in elements
    int fmt;                     // 0 bf16, 1 fp16, 2 e4m3
    bool imag, split;
    int topk;
    Args a;                      // (nk, tile_stride and idesc are set here)
};

int launch_scores(ScoreLaunch &l, int grid, cudaStream_t st);

// The tensor-core forms' bins (match_tc.cu).
__global__ void scan_padded_kernel(const int *counts, long long *tile_start, long long *cursor, int nbins, int vt);
__global__ void global_bin_kernel(long long *tile_start, long long *perm, long long nvox, long long cap, int vt);
__global__ void publish_error_kernel(const int *err);

}  // namespace tc
}  // namespace snapmrf
