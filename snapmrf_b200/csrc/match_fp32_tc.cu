// FP32 matching screened on the tensor cores.
//
// The FP32 form's answer is the first argmax of |s|^2 over the atoms of a
// voxel's block, s being the FP32 sums of match_fp32_kernel in its own order.
// Nearly all of its work goes into atoms that are far from the best.  Here
// tcgen05 scores every pair from BF16 pairs (v = hi + lo, three products each,
// FP32 accumulation), the epilogue lists every atom whose approximate |s| is
// within twice the error bound of the best one, and
//   - the listed atoms are scored again in FP32, in match_fp32_kernel's order
//     (the same chain of FMAs, bit for bit), and their first argmax wins;
//   - a voxel with more such atoms than a list holds, or whose input is not
//     finite or out of range, goes to match_fp32_kernel itself.
// So the approximate scores only decide what need not be looked at, and the
// chosen atom is the one that the FP32 kernel alone chooses: maps and indices
// are the same bit for bit (tests/test_match_screen_gpu.py).
//
// The bound of the difference between an atom's two scores (as complex
// numbers, for a voxel of unit norm).  With v = hi + lo + rest:
//  - the products left out, lo lo', rest v' and (hi + lo) rest', are inner
//    products: at most ||lo_d|| ||lo_x|| + ||rest_d|| + ||d|| ||rest_x||
//    (Cauchy and Schwarz), the norms summed while packing;
//  - both sides round a running sum, at most ||d|| ||x|| over the elements
//    that it holds.  FP32: 2^-24 of it at each of the 32 elements of a chunk.
//    Tensor core: an MMA adds 16 products to the sum with every addend cut at
//    2^-25 of the largest and the result cut to 24 bits, so (16 / 4 + 1) 2^-23
//    of it at each of a chunk's six MMAs (measured on the device with addends
//    of 2^-22 .. 2^-29 beside a sum of 1, each sign: cut exactly there, never
//    rounded up; NVIDIA documents no bound), 60 2^-24 a chunk, 61 since hi may
//    be 2^-8 longer than v.  Summed over the chunks, by Cauchy and Schwarz
//    again: sqrt(sum_c ||d_1..c||^2) sqrt(sum_c ||x_1..c||^2), the forward norms
//    of both.  The tensor core takes the chunks from the last to the first,
//    so its sum has the backward norms: atoms whose signal is over early
//    (short T1 and T2) set the largest forward norm and have small backward
//    ones, and both sums in one order would bound them a quarter higher;
//  - what is left (the voxel's scaling, the squares and roots of the
//    comparison) is 2^-22 of ||d||; 2^-20 is allowed, and 0.1 % on everything
//    for what the bounds above neglect of second order.
// The largest values of any atom of the dictionary stand for each.  On the
// configurations' dictionaries the bound is 1.1e-4 (T = 1000, imaginary atoms;
// 2.2e-4 complex; 2.8e-5 and 4.9e-5 at T = 200), where the scores were seen to
// differ by 1.6e-5 at most.
//
// 57,600 voxels, 284,458 imaginary atoms in 41 blocks, T = 1000: 36.4 -> 4.8
// ms (packing 0.68, scores 2.9 = three BF16 products at 1.68 PFLOP/s, about
// eight candidates per voxel in FP32 0.8, maps 0.11; the FP32 kernel alone
// runs at 0.61 of the FP32 FMA peak); 4,096 voxels, 837 complex atoms: 0.80 ->
// 0.21 ms; fine grids: see list_cap.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "common.h"
#define SNAPMRF_MATCH_KERNEL_DECLARATION_ONLY
#include "match_kernels.cuh"
#undef SNAPMRF_MATCH_KERNEL_DECLARATION_ONLY
#include "match_fp32_tc.h"
#include "match_tc_plan.cuh"

namespace snapmrf {

// Kernels of the FP32 matching path (match.cu).
__global__ void assign_bins_kernel(int *vox_bin, int *counts, const float *b1map, const float *params,
                                   int nparams, long long natoms, int nblocks, long long nvox);
__global__ void scatter_bins_kernel(long long *perm, long long *cursor, const int *vox_bin,
                                    long long nvox);
__global__ void finalize_maps_kernel(float *maps, long long *index_out, const unsigned long long *keys,
                                     const long long *perm, const int *vox_bin, const float2 *atoms,
                                     long long atom_stride, const float2 *img, long long img_stride,
                                     long long nreps, const float *params, int nparams,
                                     long long natoms_per_bin, long long nslots);
__global__ void poison_maps_kernel(float *maps, long long *index_out, long long nvox, const int *err);

namespace screen {

constexpr int KB = 32;               // elements of K per 64-element row chunk (hi, then lo)
constexpr float kMaxAbs = 1e15f;     // larger samples (or not finite) are left to the FP32 kernel
constexpr float kMinNorm2 = 1e-30f;  // smaller norms of a voxel and squared scores too: squares would lose bits
constexpr float kMinAtom2 = 1e-18f;  // (and of all atoms: the squares of their lo and rest parts would)
constexpr float kMaxNorm2 = 1e30f;
// Operand memory of one pass: larger dictionaries are screened in chunks of
// atoms, larger images in ranges of voxels.
constexpr long long kAtomBytes = 2ll << 30, kVoxelBytes = 1ll << 30;
constexpr long long kListBytes = 1ll << 30;  // and of the candidates' lists

struct State {
    int wait_err;            // a bounded wait of the scoring kernel ran out: the FP32 kernel takes every voxel
    int bad_atoms;           // an atom is not finite or out of range: the FP32 kernel takes every voxel
    int nfall;               // voxels left to the FP32 kernel
    tc::AtomStats atoms;
};

__global__ void init_kernel(unsigned long long *keys, long long nkeys, long long *perm, long long nperm, int *counts,
                            int *fall_counts, int nbins, int wait_err, State *st) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < nkeys) keys[i] = 0ull;
    if (i < nperm) perm[i] = -1;
    if (i < nbins) counts[i] = fall_counts[i] = 0;
    if (i == 0) *st = State{wait_err, 0, 0, {0u, 0u, 0u, 0u, 0u}};
}

// Running sums of a row (see tc::AtomStats).
struct RowSums {
    float norm2 = 0.f, forward2 = 0.f, backward2 = 0.f, lo2 = 0.f, rest2 = 0.f;
};

// hi and lo of two neighbouring elements, packed; the squares of lo and of
// what both leave (exact differences).
__device__ __forceinline__ void split2(float a, float b, uint32_t *hi, uint32_t *lo, RowSums &r) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const float2 f = __bfloat1622float2(h);
    const float da = a - f.x, db = b - f.y;
    const __nv_bfloat162 l = __floats2bfloat162_rn(da, db);
    const float2 g = __bfloat1622float2(l);
    r.lo2 = fmaf(g.x, g.x, fmaf(g.y, g.y, r.lo2));
    const float ra = da - g.x, rb = db - g.y;
    r.rest2 = fmaf(ra, ra, fmaf(rb, rb, r.rest2));
    *hi = *reinterpret_cast<const uint32_t *>(&h);
    *lo = *reinterpret_cast<const uint32_t *>(&l);
}

// Eight elements k0 .. k0 + 7 of a row (k0 a multiple of 8): 16 bytes of hi
// and, 64 bytes further, 16 bytes of lo.
__device__ __forceinline__ void store8(__nv_bfloat16 *row, long long k0, const float *v, RowSums &r) {
    uint4 h, l;
    split2(v[0], v[1], &h.x, &l.x, r);
    split2(v[2], v[3], &h.y, &l.y, r);
    split2(v[4], v[5], &h.z, &l.z, r);
    split2(v[6], v[7], &h.w, &l.w, r);
    __nv_bfloat16 *p = row + (k0 / KB) * (2 * KB) + k0 % KB;
    *reinterpret_cast<uint4 *>(p) = h;
    *reinterpret_cast<uint4 *>(p + KB) = l;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// N samples from t of a row, zeros past nreps (VEC: 16-byte loads).
template <int N, bool VEC>
__device__ __forceinline__ void load_samples(const float2 *x, long long t, long long nreps, float2 *s) {
    if (VEC && t + N <= nreps) {
#pragma unroll
        for (int u = 0; u < N / 2; u++) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(x + t) + u);
            s[2 * u] = make_float2(q.x, q.y);
            s[2 * u + 1] = make_float2(q.z, q.w);
        }
    } else {
#pragma unroll
        for (int u = 0; u < N; u++) s[u] = t + u < nreps ? __ldg(x + t + u) : make_float2(0.f, 0.f);
    }
}

// A rows: the slot's voxel at unit norm, two rows (Re, Im) for purely
// imaginary atoms, else one interleaved row; its VoxelStats.  One warp per slot.
template <bool IMAG, bool VEC>
__global__ void pack_voxels_kernel(__nv_bfloat16 *A, tc::VoxelStats *stats, const float2 *img, long long img_stride,
                                   const long long *perm, long long nslots, long long nreps, long long Kp) {
    const long long slot = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32;
    if (slot >= nslots) return;
    const long long v = perm[slot];
    const float2 *x = img + (v >= 0 ? v : 0) * img_stride;
    float n = 0.f, mx = 0.f;
    if (v >= 0)
        for (long long t = 4 * lane; t < nreps; t += 128) {
            float2 s[4];
            load_samples<4, VEC>(x, t, nreps, s);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                n += s[u].x * s[u].x + s[u].y * s[u].y;
                mx = fmaxf(mx, fmaxf(fabsf(s[u].x), fabsf(s[u].y)));
            }
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n += __shfl_xor_sync(0xffffffffu, n, o);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const bool fit = n >= kMinNorm2 && mx <= kMaxAbs && n <= kMaxNorm2;  // (false for NaN)
    const float inv = fit ? rsqrtf(n) : 0.f;
    const long long K = IMAG ? Kp / 2 : Kp / 4;  // samples, padded
    __nv_bfloat16 *row = A + (IMAG ? 2 * slot : slot) * Kp;
    RowSums sums;
    for (long long t = (IMAG ? 8 : 4) * lane; t < K; t += (IMAG ? 256 : 128)) {
        float2 s[IMAG ? 8 : 4];
        if (inv > 0.f) {
            load_samples<IMAG ? 8 : 4, VEC>(x, t, nreps, s);
        } else {
#pragma unroll
            for (int u = 0; u < (IMAG ? 8 : 4); u++) s[u] = make_float2(0.f, 0.f);
        }
        float a[8], b[8], e = 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (IMAG) {
                a[u] = s[u].x * inv;
                b[u] = s[u].y * inv;
                e = fmaf(b[u], b[u], e);
            } else {
                a[u] = (u & 1 ? s[u / 2].y : s[u / 2].x) * inv;
            }
            e = fmaf(a[u], a[u], e);
        }
        const long long k0 = IMAG ? t : 2 * t;
        sums.forward2 = fmaf((float)(Kp / (2 * KB) - k0 / KB), e, sums.forward2);
        sums.backward2 = fmaf((float)(k0 / KB + 1), e, sums.backward2);
        store8(row, k0, a, sums);
        if (IMAG) store8(row + Kp, t, b, sums);
    }
    const float f2 = warp_sum(sums.forward2), b2 = warp_sum(sums.backward2);
    const float l2 = warp_sum(sums.lo2), r2 = warp_sum(sums.rest2);
    if (lane == 0)
        stats[slot] = {fit ? n : (n == 0.f && mx == 0.f) ? 0.f : -1.f, sqrtf(f2), sqrtf(b2), sqrtf(l2), sqrtf(r2)};
}

// B rows of atoms [a0, a0 + n) (row r of the operand: atom a0 + r): one row
// (Im d) for purely imaginary atoms (a real part sets the error word to 7),
// else two, (Re d, Im d) and (-Im d, Re d); the AtomStats and whether every
// sample is finite and in range.  Atoms of bins without voxels are not looked
// at, as match_fp32_kernel does not (a real part there is no error).  One warp per atom.  Bound by
// its traffic: C1's 284,458 atoms (2.28 GB read, 1.17 GB written) 0.6 ms.
template <bool IMAG, bool VEC>
__global__ void pack_atoms_kernel(__nv_bfloat16 *B, const float2 *atoms, long long atom_stride, long long n,
                                  long long nreps, long long Kp, const long long *tile_start, int bin_lo,
                                  long long per_bin, State *st, int *err) {
    const long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int bin = bin_lo + (int)(min(r, n - 1) / per_bin);
    const bool used = r < n && tile_start[bin] < tile_start[bin + 1];
    __shared__ RowSums srow[8];
    RowSums sums;
    bool real_part = false, bad = false;
    if (used) {
        const float2 *src = atoms + r * atom_stride;
        __nv_bfloat16 *row = B + (IMAG ? r : 2 * r) * Kp;
        const long long K = IMAG ? Kp / 2 : Kp / 4;
        for (long long t = (IMAG ? 8 : 4) * lane; t < K; t += (IMAG ? 256 : 128)) {
            float2 s[IMAG ? 8 : 4];
            load_samples<IMAG ? 8 : 4, VEC>(src, t, nreps, s);
            float a[8], b[8], e = 0.f;
#pragma unroll
            for (int u = 0; u < (IMAG ? 8 : 4); u++) {
                e += s[u].x * s[u].x + s[u].y * s[u].y;
                bad |= !(fabsf(s[u].x) <= kMaxAbs && fabsf(s[u].y) <= kMaxAbs);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (IMAG) {
                    real_part |= s[u].x != 0.f;
                    a[u] = s[u].y;
                } else {
                    a[u] = u & 1 ? s[u / 2].y : s[u / 2].x;
                    b[u] = u & 1 ? s[u / 2].x : -s[u / 2].y;
                }
            }
            const long long k0 = IMAG ? t : 2 * t;
            sums.norm2 += e;
            sums.forward2 = fmaf((float)(Kp / (2 * KB) - k0 / KB), e, sums.forward2);
            sums.backward2 = fmaf((float)(k0 / KB + 1), e, sums.backward2);
            store8(row, k0, a, sums);
            if (!IMAG) {
                RowSums same;  // (the same elements, other signs)
                store8(row + Kp, k0, b, same);
            }
        }
    }
    sums = {warp_sum(sums.norm2), warp_sum(sums.forward2), warp_sum(sums.backward2), warp_sum(sums.lo2),
            warp_sum(sums.rest2)};
    bad |= !(sums.norm2 <= kMaxNorm2);
    if (IMAG && __any_sync(0xffffffffu, real_part) && lane == 0) atomicCAS(err, 0, 7);
    if (__any_sync(0xffffffffu, bad)) {
        sums = RowSums();
        if (lane == 0) atomicExch(&st->bad_atoms, 1);
    }
    if (lane == 0) srow[warp] = sums;
    __syncthreads();
    if (threadIdx.x < sizeof(RowSums) / sizeof(float)) {
        // one value per thread: one atomic per CTA, and only while it raises the value
        const int q = threadIdx.x;
        float mx = 0.f;
        for (int w = 0; w < (int)blockDim.x / 32; w++) mx = fmaxf(mx, reinterpret_cast<const float *>(&srow[w])[q]);
        const unsigned bits = __float_as_uint(mx);
        unsigned *top = reinterpret_cast<unsigned *>(&st->atoms) + q;
        if (bits > *reinterpret_cast<volatile unsigned *>(top)) atomicMax(top, bits);
    }
}

// The winners of the voxels of bins [bin_lo, bin_hi): FP32 scores of every
// listed atom within the bound, in match_fp32_kernel's order, or the voxel goes
// to the fall list.  One warp per slot (WIDE: one CTA, whose warps take the
// batches in turn); lane c carries candidate c's chain (kBatch of them at a
// time) through samples that cp.async stages kDepth steps of kSteps ahead.
// The chain is serial by definition: 57,600 voxels of about eight candidates
// 0.77 ms, their rows 4.6 GB from L2 (8-byte copies and reads 0.88, waiting
// for each candidate's load in turn 2.4 ms).
constexpr int kRescoreWarps = 4, kMaxCand = 96, kBatch = 16, kSteps = 16, kDepth = 3;
struct alignas(16) RescoreSmem {
    float2 d[kDepth][kBatch][kSteps + 2];  // (rows padded: the lanes' reads differ in bank)
    float2 x[kDepth][kSteps];
    float2 xi[kSteps];                     // (Im x, -Re x): what Im s multiplies d by
    int cand[kMaxCand];
};

// N samples (1 or 2), of which `have` exist; the rest are filled with zeros.
template <int N>
__device__ __forceinline__ void copy_samples(float2 *dst, const float2 *src, int have) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (N == 2)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(8 * have) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(8 * have) : "memory");
}

// VEC: every row starts 16-byte aligned, so a lane copies two samples at once.
// (7 CTAs per SM, as shared memory allows: 4,096 voxels in one wave)
template <bool IMAG, bool VEC, bool WIDE>
__global__ void __launch_bounds__(kRescoreWarps * 32, 7)
rescore_kernel(unsigned long long *keys, tc::Lists lists, int list_cap, const int *list_n, const float *list_best,
               const long long *perm, const tc::VoxelStats *vstats, const long long *tile_start, int bin_lo, int bin_hi,
               const int *vox_bin, const float2 *atoms, long long atom_stride, const float2 *img,
               long long img_stride, int nreps, long long bin_natoms, int nk, State *st, int *fall,
               int *fall_counts) {
    __shared__ RescoreSmem smem[kRescoreWarps];
    __shared__ float wide_s[kRescoreWarps];
    __shared__ int wide_i[kRescoreWarps];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    RescoreSmem &sm = smem[warp];
    const long long slot = tile_start[bin_lo] * lists.vt +
                           (WIDE ? blockIdx.x : blockIdx.x * (long long)kRescoreWarps + warp);
    const bool first_warp = !WIDE || warp == 0;
    if (slot >= tile_start[bin_hi] * lists.vt) return;
    const long long v = perm[slot];
    const tc::VoxelStats vs = vstats[slot];
    if (v < 0 || vs.norm2 == 0.f) return;
    const int bin = vox_bin ? vox_bin[v] : 0;
    auto leave = [&]() {
        if (first_warp && lane == 0) {
            fall[atomicAdd(&st->nfall, 1)] = (int)v;
            atomicAdd(&fall_counts[bin], 1);
        }
    };
    const tc::AtomStats as = st->atoms;
    const float norm2 = __uint_as_float(as.norm2);
    if (st->wait_err || vs.norm2 < 0.f || st->bad_atoms || norm2 < kMinAtom2 || norm2 * vs.norm2 > kMaxNorm2) return leave();
    // the slot's lists: counts and best scores, one list per lane
    constexpr int LISTS = tc::split_lists(IMAG);
    const tc::ListSlots at = tc::list_slots(lists, slot);
    const int nl = at.n * LISTS;
    static_assert(tc::MAX_PARTS * 4 <= 32, "a lane per list");
    long long lbase = 0;
    int n = 0;
    float best = 0.f;
    if (lane < nl) {
        const long long lid = (at.first + (long long)(lane / LISTS) * lists.vt) * LISTS + lane % LISTS;
        lbase = tc::list_offset(lid, lists.cap * LISTS, list_cap, at.n);
        n = list_n[lid];
        best = list_best[lid];
    }
    const bool over = n == tc::LIST_OVER;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    const float low = sqrtf(best) - tc::screen_margin(as, vs, nk);
    if (__any_sync(0xffffffffu, over) || !(low > 0.f) || best * vs.norm2 < kMinNorm2) return leave();
    const float thr = low * low * (1.f - 0x1p-20f);
    const float2 *x = img + v * img_stride;
    const float2 *d0 = atoms + (long long)bin * bin_natoms * atom_stride;
    // lanes per row and copy, rows per copy instruction
    constexpr int N = VEC ? 2 : 1, LPR = kSteps / N, RPI = 32 / LPR;
    const int steps = (nreps + kSteps - 1) / kSteps, sub = lane % LPR * N, which = lane / LPR;
    float bs = 0.f;
    int bi = -1, seen = 0, l = 0, e0 = 0;
    do {
        // the next candidates (WIDE: this warp's), until the buffer has no room for 32 more
        int count = 0;
        while (l < nl && count <= kMaxCand - 32) {
            const long long base = __shfl_sync(0xffffffffu, lbase, l) + e0;
            const int left = __shfl_sync(0xffffffffu, n, l) - e0;
            const bool in = lane < left && lists.top_s[base + lane] >= thr;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int rank = seen + __popc(m & ((1u << lane) - 1));
            const bool mine = in && (!WIDE || rank / kBatch % kRescoreWarps == warp);
            const unsigned mm = __ballot_sync(0xffffffffu, mine);
            if (mine) sm.cand[count + __popc(mm & ((1u << lane) - 1))] = lists.top_i[base + lane];
            seen += __popc(m);
            count += __popc(mm);
            e0 += 32;
            if (left <= 32) {
                l++;
                e0 = 0;
            }
        }
        __syncwarp();
        if (seen == 1 && l == nl) {
            // no other atom can win (|s| > 0: it is above the bound)
            if (first_warp && lane == 0) keys[v] = pack_key(best, (unsigned)sm.cand[0]);
            return;
        }
        for (int c0 = 0; c0 < count; c0 += kBatch) {
            const int nb = min(kBatch, count - c0);
            const float2 *row[kBatch / RPI];
#pragma unroll
            for (int q = 0; q < kBatch / RPI; q++)
                row[q] = d0 + (long long)sm.cand[min(c0 + RPI * q + which, count - 1)] * atom_stride;
            auto stage = [&](int s) {
                if (s < steps) {
                    const int t = s * kSteps + sub, b = s % kDepth;
                    const int have = max(0, min(N, nreps - t)), at = have ? t : 0;
                    if (which == 0) copy_samples<N>(&sm.x[b][sub], x + at, have);
#pragma unroll
                    for (int q = 0; q < kBatch / RPI; q++)
                        if (RPI * q < nb) copy_samples<N>(&sm.d[b][RPI * q + which][sub], row[q] + at, have);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            for (int s = 0; s < kDepth - 1; s++) stage(s);
            // IMAG: both sums of candidate c on lane c.  Complex (four FMAs per
            // sample): Re s on lane c, Im s on lane c + kBatch.
            static_assert(kBatch == 16 && kSteps == 16, "half a warp each");
            const bool im = !IMAG && lane >= kBatch;
            float acc = 0.f, acc2 = 0.f;
            for (int s = 0; s < steps; s++) {
                stage(s + kDepth - 1);
                asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
                __syncwarp();
                if (!IMAG) {
                    if (!im) {
                        const float2 v = sm.x[s % kDepth][lane];
                        sm.xi[lane] = make_float2(v.y, -v.x);
                    }
                    __syncwarp();
                }
                const float4 *dr = reinterpret_cast<const float4 *>(sm.d[s % kDepth][lane % kBatch]);
                const float4 *xr = reinterpret_cast<const float4 *>(im ? sm.xi : sm.x[s % kDepth]);
                if ((IMAG ? lane : lane % kBatch) < nb) {
                    // (samples past nreps are zeros: their products add exact zeros)
#pragma unroll
                    for (int u = 0; u < kSteps / 2; u++) {
                        const float4 d = dr[u], v = xr[u];
                        if (IMAG) {
                            acc = fmaf(d.y, v.y, acc);
                            acc2 = fmaf(-d.y, v.x, acc2);
                            acc = fmaf(d.w, v.w, acc);
                            acc2 = fmaf(-d.w, v.z, acc2);
                        } else {
                            acc = fmaf(d.x, v.x, acc);
                            acc = fmaf(d.y, v.y, acc);
                            acc = fmaf(d.z, v.z, acc);
                            acc = fmaf(d.w, v.w, acc);
                        }
                    }
                }
                __syncwarp();
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            const float ar = acc, ai = IMAG ? acc2 : __shfl_down_sync(0xffffffffu, acc, kBatch);
            const float sc = ar * ar + ai * ai;
            if (lane < nb && sc > 0.f && beats(sc, sm.cand[c0 + lane], bs, bi)) {
                bs = sc;
                bi = sm.cand[c0 + lane];
            }
        }
        __syncwarp();
    } while (l < nl);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float os = __shfl_xor_sync(0xffffffffu, bs, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (beats(os, oi, bs, bi)) {
            bs = os;
            bi = oi;
        }
    }
    if (WIDE) {
        if (lane == 0) {
            wide_s[warp] = bs;
            wide_i[warp] = bi;
        }
        __syncthreads();
        if (threadIdx.x != 0) return;
        for (int w = 1; w < kRescoreWarps; w++)
            if (beats(wide_s[w], wide_i[w], bs, bi)) {
                bs = wide_s[w];
                bi = wide_i[w];
            }
    }
    if (lane == 0 && bi >= 0) keys[v] = pack_key(bs, (unsigned)bi);
}

// Slots and tiles of the voxels left to the FP32 kernel, by bin.  One CTA:
// usually there are none.
__global__ void __launch_bounds__(1024) fall_bins_kernel(const State *st, const int *fall, const int *fall_counts,
                                                         const int *vox_bin, long long *slot_start,
                                                         long long *tile_start, long long *cursor, long long *perm,
                                                         int nbins) {
    const int n = st->nfall;
    if (threadIdx.x == 0) {
        long long s = 0, t = 0;
        if (n)
            for (int b = 0; b < nbins; b++) {
                slot_start[b] = cursor[b] = s;
                tile_start[b] = t;
                s += fall_counts[b];
                t += (fall_counts[b] + kMatchVT - 1) / kMatchVT;
            }
        slot_start[nbins] = s;
        tile_start[nbins] = t;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int v = fall[i], b = vox_bin ? vox_bin[v] : 0;
        perm[atomicAdd(reinterpret_cast<unsigned long long *>(&cursor[b]), 1ull)] = v;
    }
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace screen

int match_fp32_screened(const ScreenRequest &q, cudaStream_t st, bool *done) {
    using namespace screen;
    *done = false;
    const int nbins = q.b1map ? q.nblocks : 1;
    const long long bin_natoms = q.b1map ? q.natoms : q.NATOMS;
    const int vt = q.imag ? tc::BM / 2 : tc::BM, apt = q.imag ? tc::BN : tc::BA, rows = q.imag ? 1 : 2;
    const long long K = (q.imag ? 1 : 2) * q.nreps, nk = (K + KB - 1) / KB, Kp = nk * 2 * KB;
    if (Kp > 0x7fffffffll / 4) return SNAPMRF_OK;
    // SNAPMRF_SCREEN_PASS="atoms,voxels,lists" (bytes) overrides the pass
    // sizes, so that tests reach several passes with small inputs
    long long atom_bytes = kAtomBytes, voxel_bytes = kVoxelBytes, list_room = kListBytes;
    if (const char *e = getenv("SNAPMRF_SCREEN_PASS")) {
        long long pa = 0, pv = 0, pl = 0;
        if (sscanf(e, "%lld,%lld,%lld", &pa, &pv, &pl) == 3 && pa > 0 && pv > 0 && pl > 0) {
            atom_bytes = pa;
            voxel_bytes = pv;
            list_room = pl;
        }
    }
    // atoms per pass: whole bins, or a chunk of one bin's tiles
    const long long row_bytes = rows * Kp * 2, fit = std::max<long long>(apt, atom_bytes / row_bytes);
    const int bins_per = (int)std::min<long long>(nbins, std::max(1ll, fit / bin_natoms));
    const long long chunk = bin_natoms <= fit ? bin_natoms : fit / apt * apt;
    // Entries per list: the atoms within the bound grow in number with the
    // grid's density (T = 1000, imaginary / complex, mean and most of 512
    // voxels: 6,938 atoms 8, 24 / 15, 44; 41,588 45, 136 / 86, 262; 164,551
    // 175, 536 / 340, 1,036; 334,125 356, 1,089 / 690, 2,109), over four / two
    // lists.  Full lists send the voxel to the FP32 kernel after the screen:
    // 4,096 voxels, 164,551 atoms 58.2 / 111 ms by that kernel alone, 63.4 /
    // 121 with lists for 64 entries, 5.8 / 11.2 with these.
    const int nlists = tc::split_lists(q.imag);
    int list_cap = 64;
    while (list_cap < 2048 && list_cap * 256ll < bin_natoms) list_cap *= 2;
    const long long split_list = tc::split_entries(list_cap) * nlists * 8;  // bytes of a split slot's lists
    int num_sms = 0, dev = 0;
    SNAPMRF_CUDA(cudaGetDevice(&dev));
    SNAPMRF_CUDA(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
    // voxels per pass (at most num_sms - 1 items of vt voxels are split)
    const long long own_list = (long long)nlists * list_cap * 8;
    const long long nv_lists = std::max(list_room / (own_list + split_list),
                                        (list_room - (num_sms - 1) * vt * split_list) / own_list);
    const long long nv_fit =
        std::max<long long>(vt, std::min(voxel_bytes / ((q.imag ? 2 : 1) * Kp * 2), nv_lists));
    const long long nv_max = std::min(q.nvox, nv_fit);
    const long long cap = ((nv_max + vt - 1) / vt + nbins) * vt;
    const long long arows = (q.imag ? 2 : 1) * cap, brows = rows * chunk * bins_per;
    if (arows > 0x7fffffffll || brows > 0x7fffffffll) return SNAPMRF_OK;
    // (every block's voxels are padded to vt: thousands of blocks with few
    // voxels each would take many times a pass's room)
    if (cap * ((q.imag ? 2 : 1) * Kp * 2 + own_list) > 2 * (voxel_bytes + list_room)) return SNAPMRF_OK;
    const long long lslots = cap + tc::split_slots(cap / vt, num_sms) * vt;

    size_t bytes = 0;
    auto take = [&](size_t n) {
        size_t off = bytes;
        bytes += (n + 255) & ~size_t(255);
        return off;
    };
    const size_t oA = take((size_t)arows * Kp * 2), oB = take((size_t)brows * Kp * 2);
    const size_t lb = (size_t)cap * nlists * list_cap * 4 +
                      (size_t)std::min<long long>(cap / vt, num_sms - 1) * vt * split_list / 2;
    const size_t hb = (size_t)lslots * nlists * 4;
    const size_t oTs = take(lb), oTi = take(lb), oLn = take(hb), oLb = take(hb), oPlan = take(sizeof(tc::TailPlan));
    const size_t oKey = take((size_t)nv_max * 8);
    const size_t oPerm = take((size_t)cap * 8), oFperm = take((size_t)nv_max * 8), oFall = take((size_t)nv_max * 4);
    const size_t oVb = take((size_t)nv_max * 4), oVs = take((size_t)cap * sizeof(tc::VoxelStats));
    const size_t oBin = take(5 * (size_t)(nbins + 1) * 8), oCnt = take(2 * (size_t)nbins * 4), oSt = take(sizeof(State)), oErr = take(4);
    DeviceScratch s;
    const cudaError_t ae = s.alloc(bytes, st);
    if (ae == cudaErrorMemoryAllocation) {
        // without room for the operands the FP32 kernel takes the whole call
        cudaGetLastError();
        return SNAPMRF_OK;
    }
    SNAPMRF_CUDA(ae);
    unsigned char *b = s.as<unsigned char>();
    __nv_bfloat16 *A = reinterpret_cast<__nv_bfloat16 *>(b + oA), *B = reinterpret_cast<__nv_bfloat16 *>(b + oB);
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(b + oKey);
    long long *perm = reinterpret_cast<long long *>(b + oPerm), *fperm = reinterpret_cast<long long *>(b + oFperm);
    int *fall = reinterpret_cast<int *>(b + oFall), *vox_bin = reinterpret_cast<int *>(b + oVb);
    tc::VoxelStats *vstats = reinterpret_cast<tc::VoxelStats *>(b + oVs);
    long long *tile_start = reinterpret_cast<long long *>(b + oBin), *cursor = tile_start + nbins + 1;
    long long *fslot = cursor + nbins + 1, *ftile = fslot + nbins + 1, *fcursor = ftile + nbins + 1;
    int *counts = reinterpret_cast<int *>(b + oCnt), *fall_counts = counts + nbins;
    State *state = reinterpret_cast<State *>(b + oSt);
    int *err = reinterpret_cast<int *>(b + oErr);  // 7: an atom with a real part, for the whole call
    *done = true;
    SNAPMRF_CUDA(cudaMemsetAsync(err, 0, 4, st));
    // (tests: as if a wait of every scoring launch had run out)
    const int wait_err = getenv("SNAPMRF_SCREEN_WAIT_ERROR") ? 1 : 0;

    auto aligned = [](const void *p, long long stride) {
        return stride % 2 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
    };
    const bool avec = aligned(q.atoms, q.atom_stride);

    for (long long v0 = 0; v0 < q.nvox; v0 += nv_max) {
        const long long nv = std::min(nv_max, q.nvox - v0);
        const float2 *img = q.img + v0 * q.img_stride;
        const float *b1 = q.b1map ? q.b1map + v0 : nullptr;
        const long long ninit = std::max<long long>(std::max(nv, q.b1map ? cap : 0), nbins);
        init_kernel<<<nblk(ninit, 256), 256, 0, st>>>(keys, nv, perm, q.b1map ? cap : 0, counts, fall_counts, nbins,
                                                      wait_err, state);
        SNAPMRF_LAUNCH_CHECK();
        if (b1) {
            assign_bins_kernel<<<nblk(nv, 256), 256, 0, st>>>(vox_bin, counts, b1, q.params, q.nparams, q.natoms,
                                                              nbins, nv);
            SNAPMRF_LAUNCH_CHECK();
            tc::scan_padded_kernel<<<1, 32, 0, st>>>(counts, tile_start, cursor, nbins, vt);
            SNAPMRF_LAUNCH_CHECK();
            scatter_bins_kernel<<<nblk(nv, 256), 256, 0, st>>>(perm, cursor, vox_bin, nv);
        } else {
            tc::global_bin_kernel<<<nblk(cap, 256), 256, 0, st>>>(tile_start, perm, nv, cap, vt);
        }
        SNAPMRF_LAUNCH_CHECK();
        const bool ivec = aligned(img, q.img_stride);
        auto pv = q.imag ? (ivec ? pack_voxels_kernel<true, true> : pack_voxels_kernel<true, false>)
                         : (ivec ? pack_voxels_kernel<false, true> : pack_voxels_kernel<false, false>);
        pv<<<nblk(cap * 32, 256), 256, 0, st>>>(A, vstats, img, q.img_stride, perm, cap, q.nreps, Kp);
        SNAPMRF_LAUNCH_CHECK();

        tc::ScoreLaunch sl;
        sl.A = A;
        sl.B = B;
        sl.arows = arows;
        sl.Kp = Kp;
        sl.fmt = 0;
        sl.imag = q.imag;
        sl.split = true;
        sl.topk = 16;
        tc::Args &a = sl.a;
        a.tile_start = tile_start;
        a.nbins = nbins;
        a.bin_natoms = bin_natoms;
        a.plan_tiles = (int)((chunk + apt - 1) / apt);
        a.ascale2 = nullptr;
        a.cap = cap;
        a.top_s = reinterpret_cast<float *>(b + oTs);
        a.top_i = reinterpret_cast<int *>(b + oTi);
        a.plan = reinterpret_cast<tc::TailPlan *>(b + oPlan);
        a.list_cap = list_cap;
        a.atom_stats = &state->atoms;
        a.vox_stats = vstats;
        a.list_n = reinterpret_cast<int *>(b + oLn);
        a.list_best = reinterpret_cast<float *>(b + oLb);
        a.err = &state->wait_err;
        auto pa = q.imag ? (avec ? pack_atoms_kernel<true, true> : pack_atoms_kernel<true, false>)
                         : (avec ? pack_atoms_kernel<false, true> : pack_atoms_kernel<false, false>);
        tc::Lists lists;
        lists.top_s = a.top_s;
        lists.top_i = a.top_i;
        lists.plan = a.plan;
        lists.cap = cap;
        lists.vt = vt;
        // A CTA per voxel where fine grids (long lists) and long rows (a wide
        // bound) give it several batches.  ms, a warp / a CTA: 4,096 voxels,
        // 18,687 complex atoms, T = 1000 (list_cap nk = 8,064) 1.60 / 1.45,
        // imaginary (4,096) 0.87 / 0.84, 1,024 voxels 0.43 / 0.35; 19,600
        // complex bSSFP atoms, T = 400 (3,200) 0.56 / 0.61.
        const bool wide = (long long)list_cap * nk >= 4096;
        auto pick = [&](auto vec_wide, auto vec, auto wd, auto plain) {
            return avec && ivec ? (wide ? vec_wide : vec) : (wide ? wd : plain);
        };
        auto rk = q.imag ? pick(rescore_kernel<true, true, true>, rescore_kernel<true, true, false>,
                                rescore_kernel<true, false, true>, rescore_kernel<true, false, false>)
                         : pick(rescore_kernel<false, true, true>, rescore_kernel<false, true, false>,
                                rescore_kernel<false, false, true>, rescore_kernel<false, false, false>);
        for (int b0 = 0; b0 < nbins; b0 += bins_per) {
            const int nb = std::min(bins_per, nbins - b0);
            for (long long a0 = 0; a0 < bin_natoms; a0 += chunk) {
                // (several bins only with chunk == bin_natoms)
                const long long ca = std::min(chunk, bin_natoms - a0);
                const long long na = nb * ca;
                pa<<<nblk(na * 32, 256), 256, 0, st>>>(B, q.atoms + (b0 * bin_natoms + a0) * q.atom_stride,
                                                       q.atom_stride, na, q.nreps, Kp, tile_start, b0, ca, state, err);
                SNAPMRF_LAUNCH_CHECK();
                sl.brows = rows * na;
                a.bin_lo = b0;
                a.bin_hi = b0 + nb;
                a.atom0 = (int)a0;
                a.chunk_natoms = (int)ca;
                a.resume = a0 > 0;
                int rc = tc::launch_scores(sl, num_sms, st);
                if (rc) return rc;
            }
            // (the next bins' launch uses the split items' lists again)
            rk<<<nblk(cap, wide ? 1 : kRescoreWarps), kRescoreWarps * 32, 0, st>>>(
                keys, lists, list_cap, a.list_n, a.list_best, perm, vstats, tile_start, b0, b0 + nb, b1 ? vox_bin : nullptr,
                q.atoms, q.atom_stride, img, q.img_stride, (int)q.nreps, bin_natoms, (int)nk, state, fall,
                fall_counts);
            SNAPMRF_LAUNCH_CHECK();
        }
        fall_bins_kernel<<<1, 1024, 0, st>>>(state, fall, fall_counts, b1 ? vox_bin : nullptr, fslot, ftile, fcursor,
                                             fperm, nbins);
        SNAPMRF_LAUNCH_CHECK();
        MatchArgs m;
        m.atoms = q.atoms;
        m.atom_stride = q.atom_stride;
        m.img = img;
        m.img_stride = q.img_stride;
        m.nreps = q.nreps;
        m.nbins = nbins;
        m.bin_natoms = bin_natoms;
        m.nvox = nv;
        m.keys = keys;
        m.key_by_voxel = 1;
        m.err = nullptr;  // (a real part was looked for while packing)
        m.slot_start = fslot;
        m.tile_start = ftile;
        m.perm = fperm;
        m.perm_mod = 0;
        m.atiles_per_split = 0;
        SNAPMRF_CUDA(launch_match_fp32(m, dim3(2 * num_sms), q.imag, st));
        finalize_maps_kernel<<<nblk(nv * 32, 256), 256, 0, st>>>(
            q.maps + v0 * 5, q.index_out ? q.index_out + v0 : nullptr, keys, nullptr, b1 ? vox_bin : nullptr, q.atoms,
            q.atom_stride, img, q.img_stride, q.nreps, q.params, q.nparams, bin_natoms, nv);
        SNAPMRF_LAUNCH_CHECK();
    }
    if (q.imag) {
        // an atom with a real part: NaN maps, indices -1, error word 7
        poison_maps_kernel<<<nblk(q.nvox, 256), 256, 0, st>>>(q.maps, q.index_out, q.nvox, err);
        SNAPMRF_LAUNCH_CHECK();
        tc::publish_error_kernel<<<1, 1, 0, st>>>(err);
        SNAPMRF_LAUNCH_CHECK();
    }
    return SNAPMRF_OK;
}

}  // namespace snapmrf
