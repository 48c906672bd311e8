// EPG / ROA device kernels (reference operation order).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cuda_runtime.h>

#include "common.h"

namespace snapmrf {

enum Echo { ECHO_SSFP = 0, ECHO_ROA = 1, ECHO_SR = 2, ECHO_SE = 3, ECHO_TSE = 4, ECHO_FISP = 5 };

constexpr int kEpgThreads = 128;      // threads per CTA
constexpr int kChunk = 16;            // time steps staged per shared-memory chunk (<= 32)
constexpr int kMaxStatesPerLane = 8;  // register-resident EPG states per lane

struct EpgArgs {
    float2 *atoms;        // out [blocks][natoms][nreps]
    float *norms;         // optional out [blocks][natoms]
    const float *alpha;   // [gen_blocks][nreps] flip angle per block (rad)
    const float *sched;   // [4][nreps] converted schedule (alpha, phi rad; TR, TE ms)
    const float *params;  // [NATOMS][nparams]
    int nparams;
    long long nreps;
    long long natoms;     // atoms per B1 block
    int nstates;          // EPG states w
    int L;                // lanes per atom (power of two)
    int own_params;       // 1: each atom's own row; 0: block-0 row (epg_ssfp)
    int normalize;        // unit-norm each atom (src/functions.cu:670-685)
    int n_iso;            // ROA isochromats
    // initial pulse (init_rf_pulse): angles in degrees, TI in ms.  Passed at
    // run time like the reference's kernel arguments, so that __sincosf is
    // evaluated on the device rather than folded at compile time.
    float init_alpha_deg, init_phi_deg, init_ti;
    // optional 16-bit copy of Im(atom), [blocks][natoms][packed_pitch]
    void *packed;
    int packed_half;      // 1: fp16, 0: bf16
    long long packed_pitch;
    // first atom of each B1 block in the fine tail of the real-valued kernel
    long long fine_first;
    // 16-bit operand of the unit-norm atoms while the atoms stay as generated
    int pack_normalized;
    // 1: that operand is written by a separate pass over the finished atoms
    // and their norms (pack_operand_kernel), not by the recursion's kernel
    int operand_pass;
    // 1: atoms written as Im rows, [blocks][natoms][nreps] float (the
    // real-valued recursion only; its atoms are purely imaginary)
    int imag_rows;
};

// Number of per-(atom, step) factors staged: E1/E2 at TE and at TR-TE, plus
// the B0 precession phasors at TE and TR-TE for SSFP.
__host__ __device__ constexpr int epg_nf(int echo) { return echo == ECHO_SSFP ? 8 : 4; }

// Per-group strides in shared memory, padded so that the groups of a warp
// hit different banks.
__host__ __device__ constexpr int epg_f_stride(int echo) { return kChunk * epg_nf(echo) + 4; }
constexpr int kReadoutStride = kChunk + 1;  // float2 per group

inline size_t epg_ref_smem_bytes(int echo, int L) {
    int apc = kEpgThreads / L;
    return (size_t)kChunk * 9 * sizeof(float2) + (size_t)apc * epg_f_stride(echo) * sizeof(float) +
           (size_t)apc * kReadoutStride * sizeof(float2) + (size_t)apc * 3 * sizeof(float);
}

// RF transition matrix of fill_transition_matrix (src/functions.cu:483-508),
// same float2 expressions; T[3r + l] multiplies state channel l into row r.
__device__ __forceinline__ void rf_matrix(float alpha, float phi, float2 *T) {
    float sa, ca;
    __sincosf(alpha, &sa, &ca);
    float sa2 = (1 - ca) / 2;
    float ca2 = (1 + ca) / 2;
    float sp, cp;
    __sincosf(phi, &sp, &cp);
    float2 z = make_float2(cp, sp);
    float2 zinv = c_conj(z);
    const float2 im = make_float2(0.f, 1.f);
    const float2 mim = make_float2(-im.x, -im.y);
    T[0] = make_float2(ca2, 0.f);
    T[3] = c_mul(c_scale(zinv, sa2), zinv);
    T[6] = c_mul(c_scale(c_scale(mim, 0.5f), sa), zinv);
    T[1] = c_scale(c_mul(z, z), sa2);
    T[4] = make_float2(ca2, 0.f);
    T[7] = c_scale(c_mul(c_scale(im, 0.5f), z), sa);
    T[2] = c_scale(c_mul(mim, z), sa);
    T[5] = c_mul(c_scale(im, sa), zinv);
    T[8] = make_float2(ca, 0.f);
}

// One output row of the 3x3 complex RF product, accumulated with FMAs over
// the three state channels (the in-place cublasCgemm of
// src/functions.cu:510-528).
__device__ __forceinline__ float2 rf_row(float2 a0, float2 a1, float2 a2, float2 o0, float2 o1,
                                         float2 o2) {
    float rx = a0.x * o0.x;
    rx = fmaf(-a0.y, o0.y, rx);
    rx = fmaf(a1.x, o1.x, rx);
    rx = fmaf(-a1.y, o1.y, rx);
    rx = fmaf(a2.x, o2.x, rx);
    rx = fmaf(-a2.y, o2.y, rx);
    float ry = a0.x * o0.y;
    ry = fmaf(a0.y, o0.x, ry);
    ry = fmaf(a1.x, o1.y, ry);
    ry = fmaf(a1.y, o1.x, ry);
    ry = fmaf(a2.x, o2.y, ry);
    ry = fmaf(a2.y, o2.x, ry);
    return make_float2(rx, ry);
}

// Register-resident EPG state of one lane: states k = gl*S + j.
template <int S>
struct LaneState {
    float2 fp[S], fm[S], zz[S];
};

template <int S>
__device__ __forceinline__ void st_rf(LaneState<S> &s, const float2 *T) {
    float2 t0 = T[0], t1 = T[1], t2 = T[2], t3 = T[3], t4 = T[4], t5 = T[5], t6 = T[6], t7 = T[7],
           t8 = T[8];
#pragma unroll
    for (int j = 0; j < S; j++) {
        float2 o0 = s.fp[j], o1 = s.fm[j], o2 = s.zz[j];
        s.fp[j] = rf_row(t0, t1, t2, o0, o1, o2);
        s.fm[j] = rf_row(t3, t4, t5, o0, o1, o2);
        s.zz[j] = rf_row(t6, t7, t8, o0, o1, o2);
    }
}

// decay_signal_stage1/2 (src/functions.cu:544-569): F+- *= E2, Z *= E1, then
// Z0 += 1 - E1 as a separate rounding.
template <int S>
__device__ __forceinline__ void st_relax(LaneState<S> &s, float E1, float E2, bool lane0) {
#pragma unroll
    for (int j = 0; j < S; j++) {
        s.fp[j] = c_scale(s.fp[j], E2);
        s.fm[j] = c_scale(s.fm[j], E2);
        s.zz[j] = c_scale(s.zz[j], E1);
    }
    if (lane0) s.zz[0].x = __fadd_rn(s.zz[0].x, 1 - E1);
}

// shift_phase (EPG, src/functions.cu:585-607): F+ *= e, F- *= conj(e).
template <int S>
__device__ __forceinline__ void st_b0(LaneState<S> &s, float2 e) {
    float2 ec = c_conj(e);
#pragma unroll
    for (int j = 0; j < S; j++) {
        s.fp[j] = c_mul(e, s.fp[j]);
        s.fm[j] = c_mul(ec, s.fm[j]);
    }
}

// dephase_gradients (src/functions.cu:619-668): F+[k] <- F+[k-1] for
// k = w-1..1, F-[k] <- F-[k+1] for k = 0..w-2 (F-[w-1] keeps its value), then
// F+[0] = conj(F-[0]) and F-[w-1] = 0.  With w = 1 nothing shifts and F+[0]
// takes the conjugate of the unshifted F-[0].  Slots k >= w are kept zero.
template <int S>
__device__ __forceinline__ void st_shift(LaneState<S> &s, int gl, int L, int w) {
    const unsigned full = 0xffffffffu;
    float2 top = s.fp[S - 1];
    float2 up;
    up.x = __shfl_up_sync(full, top.x, 1, L);
    up.y = __shfl_up_sync(full, top.y, 1, L);
    float2 bot = s.fm[0];
    float2 dn;
    dn.x = __shfl_down_sync(full, bot.x, 1, L);
    dn.y = __shfl_down_sync(full, bot.y, 1, L);
#pragma unroll
    for (int j = S - 1; j >= 1; j--) s.fp[j] = s.fp[j - 1];
    s.fp[0] = up;
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int k = gl * S + j;
        float2 nxt = (j < S - 1) ? s.fm[j + 1] : ((gl == L - 1) ? make_float2(0.f, 0.f) : dn);
        if (k != w - 1) s.fm[j] = nxt;
    }
    if (gl == 0) s.fp[0] = c_conj(s.fm[0]);
#pragma unroll
    for (int j = 0; j < S; j++) {
        const int k = gl * S + j;
        if (k >= w) s.fp[j] = make_float2(0.f, 0.f);
        if (k == w - 1) s.fm[j] = make_float2(0.f, 0.f);
    }
}

// init_rf_pulse (EPG, src/functions.cu:456-481) into state 0.
template <int S>
__device__ __forceinline__ void st_init(LaneState<S> &s, bool lane0, float t1, float t2,
                                        float alpha_deg, float phi_deg, float TI) {
#pragma unroll
    for (int j = 0; j < S; j++) {
        s.fp[j] = make_float2(0.f, 0.f);
        s.fm[j] = make_float2(0.f, 0.f);
        s.zz[j] = make_float2(0.f, 0.f);
    }
    float alpha = (float)(alpha_deg * M_PI / 180.f);
    float phi = (float)(phi_deg * M_PI / 180.f);
    float e1 = expf(-TI / t1);
    float e2 = expf(-TI / t2);
    float sa, ca, sph, cph;
    __sincosf(alpha, &sa, &ca);
    __sincosf(phi, &sph, &cph);
    float2 tmp2 = c_scale(make_float2(sph, cph), e2 * sa);
    if (lane0) {
        s.fp[0] = c_conj(tmp2);
        s.fm[0] = tmp2;
        s.zz[0] = make_float2(e1 * ca + 1 - e1, 0.f);
    }
}

// B0 phase of shift_phase: cexpf(2*pi*B0*t/1000) with the argument
// evaluated in double like the reference expression.
__device__ __forceinline__ float2 b0_phasor(float B0, float t) {
    float th = (float)(2 * M_PI * B0 * t / 1000.f);
    float s, c;
    __sincosf(th, &s, &c);
    return make_float2(c, s);
}

// The fused EPG recursion, reference operation order.  One CTA handles
// kEpgThreads / L atoms of one B1 block (blockIdx.y).
template <int ECHO, int S>
__global__ void __launch_bounds__(kEpgThreads) epg_ref_kernel(EpgArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NF = epg_nf(ECHO);
    const int L = a.L;
    const int apc = kEpgThreads / L;
    const int tid = threadIdx.x;
    const int g = tid / L;
    const int gl = tid % L;
    const bool lane0 = (gl == 0);
    const long long blk = blockIdx.y;
    const long long nreps = a.nreps;
    const long long atom0 = (long long)blockIdx.x * apc;
    const long long ab = atom0 + g;
    const bool active = ab < a.natoms;
    const long long gatom = blk * a.natoms + ab;

    constexpr int FS = epg_f_stride(ECHO);
    float2 *sT = reinterpret_cast<float2 *>(smem_raw);
    float *sF = reinterpret_cast<float *>(sT + kChunk * 9);
    float2 *sR = reinterpret_cast<float2 *>(sF + apc * FS);
    float *sP = reinterpret_cast<float *>(sR + apc * kReadoutStride);

    for (int i = tid; i < apc; i += kEpgThreads) {
        long long at = atom0 + i;
        float t1 = 1.f, t2 = 1.f, b0 = 0.f;
        if (at < a.natoms) {
            long long row = a.own_params ? blk * a.natoms + at : at;
            const float *p = a.params + row * a.nparams;
            t1 = p[0];
            t2 = p[1];
            b0 = p[2];
        }
        sP[3 * i] = t1;
        sP[3 * i + 1] = t2;
        sP[3 * i + 2] = b0;
    }
    __syncthreads();
    const float T1 = sP[3 * g], T2 = sP[3 * g + 1];

    const float *alpha = a.alpha + blk * nreps;
    const float *phi = a.sched + nreps;
    const float *TR = a.sched + 2 * nreps;
    const float *TE = a.sched + 3 * nreps;
    const int w = a.nstates;

    LaneState<S> s;
    st_init<S>(s, lane0, T1, T2, a.init_alpha_deg, a.init_phi_deg, a.init_ti);
    if (ECHO == ECHO_SE || ECHO == ECHO_TSE) {
        st_shift<S>(s, gl, L, w);
        float te0 = TE[0];
        st_relax<S>(s, expf(-te0 / T1), expf(-te0 / T2), lane0);
    }

    float nrm = 0.f;
    float2 *out = a.atoms + gatom * nreps;
    for (long long t0 = 0; t0 < nreps; t0 += kChunk) {
        const int nch = (int)min((long long)kChunk, nreps - t0);
        __syncthreads();
        for (int i = tid; i < nch; i += kEpgThreads) rf_matrix(alpha[t0 + i], phi[t0 + i], sT + 9 * i);
        for (int idx = tid; idx < apc * nch; idx += kEpgThreads) {
            int ga = idx / nch, i = idx - ga * nch;
            float t1 = sP[3 * ga], t2 = sP[3 * ga + 1];
            float tr = TR[t0 + i], te = TE[t0 + i];
            float ta = te, tb = tr - te;
            float *f = sF + ga * FS + i * NF;
            f[0] = expf(-ta / t1);
            f[1] = expf(-ta / t2);
            f[2] = expf(-tb / t1);
            f[3] = expf(-tb / t2);
            if (ECHO == ECHO_SSFP) {
                float b0 = sP[3 * ga + 2];
                float2 ea = b0_phasor(b0, ta), eb = b0_phasor(b0, tb);
                f[4] = ea.x;
                f[5] = ea.y;
                f[6] = eb.x;
                f[7] = eb.y;
            }
        }
        __syncthreads();
        for (int i = 0; i < nch; i++) {
            const float *f = sF + g * FS + i * NF;
            st_rf<S>(s, sT + 9 * i);
            if (ECHO == ECHO_SR) {
                st_relax<S>(s, f[0], f[1], lane0);
            } else if (ECHO == ECHO_SE || ECHO == ECHO_TSE) {
                st_shift<S>(s, gl, L, w);
                st_relax<S>(s, f[0], f[1], lane0);
            } else if (ECHO == ECHO_FISP) {
                st_relax<S>(s, f[0], f[1], lane0);
            } else {
                st_relax<S>(s, f[0], f[1], lane0);
                st_b0<S>(s, make_float2(f[4], f[5]));
            }
            if (lane0) {
                float2 v = s.fp[0];
                sR[g * kReadoutStride + i] = v;
                nrm += v.x * v.x + v.y * v.y;
            }
            if (ECHO == ECHO_SR) {
                st_relax<S>(s, f[2], f[3], lane0);
            } else if (ECHO == ECHO_SE || ECHO == ECHO_TSE || ECHO == ECHO_FISP) {
                st_shift<S>(s, gl, L, w);
                st_relax<S>(s, f[2], f[3], lane0);
            } else {
                st_b0<S>(s, make_float2(f[6], f[7]));
                st_shift<S>(s, gl, L, w);
                st_relax<S>(s, f[2], f[3], lane0);
            }
        }
        __syncwarp();
        if (active)
            for (int q = gl; q < nch; q += L) out[t0 + q] = sR[g * kReadoutStride + q];
    }
    if (a.normalize || a.norms) {
        nrm = __shfl_sync(0xffffffffu, nrm, 0, L);
        if (a.norms && lane0 && active) a.norms[gatom] = sqrtf(nrm);
        if (a.normalize) {
            __syncwarp();
            float inv = nrm;
            if (inv > 0.f) inv = 1.f / sqrtf(inv);
            if (active)
                for (long long q = gl; q < nreps; q += L) out[q] = c_scale(out[q], inv);
        }
    }
}

// ---------------------------------------------------------------------------
// Real-valued EPG recursion (FISP / SR with every RF phase exactly 0).
//
// With phi = 0 the transition matrix has real F-rows and imaginary Z-column
// (and the converse for the Z-row), the initial state is Z = 1, and
// relaxation, the shift and conj() preserve the form: F+ and F- stay purely
// imaginary and Z real.  The state is then three floats per EPG state
// (f+ = Im F+, f- = Im F-, z = Re Z) instead of six.  The nine real
// coefficients are the entries of the same complex matrix, and the FMA
// chains below are those of rf_row with the terms whose factors are exact
// zeros removed, so the results are bit-identical to the complex recursion.
// ---------------------------------------------------------------------------
constexpr int kMaxRealStatesPerLane = 32;  // even: states are processed in pairs

// Coefficient pairs (c, c) of the real recursion for one step, in the order
// T0.x, T1.x, T2.y | T3.x, T4.x, T5.y | -T6.y, -T7.y, T8.x (float2 each).
__device__ __forceinline__ void rf_real_coeffs2(float alpha, float phi, float2 *c) {
    float2 T[9];
    rf_matrix(alpha, phi, T);
    const float v[9] = {T[0].x, T[1].x, T[2].y, T[3].x, T[4].x, T[5].y, -T[6].y, -T[7].y, T[8].x};
#pragma unroll
    for (int i = 0; i < 9; i++) c[i] = make_float2(v[i], v[i]);
    c[9] = make_float2(0.f, 0.f);
}

// P pairs of EPG states per lane: element h of pair i is state
// k = gl * 2P + h P + i.  Packed two-wide FP32 instructions (__ffma2_rn /
// __fmul2_rn) perform per element exactly the scalar operations of the
// complex recursion with its zero terms removed.
template <int P>
struct RealLane2 {
    float2 fp[P], fm[P], zz[P];
};

template <int P>
__device__ __forceinline__ void rl2_rf_k(RealLane2<P> &s, float2 c0, float2 c1, float2 c2, float2 c3, float2 c4,
                                         float2 c5, float2 c6, float2 c7, float2 c8) {
#pragma unroll
    for (int i = 0; i < P; i++) {
        const float2 p = s.fp[i], m = s.fm[i], z = s.zz[i];
        float2 np = __fmul2_rn(c0, p);
        np = __ffma2_rn(c1, m, np);
        np = __ffma2_rn(c2, z, np);
        float2 nm = __fmul2_rn(c3, p);
        nm = __ffma2_rn(c4, m, nm);
        nm = __ffma2_rn(c5, z, nm);
        float2 nz = __fmul2_rn(c6, p);
        nz = __ffma2_rn(c7, m, nz);
        nz = __ffma2_rn(c8, z, nz);
        s.fp[i] = np;
        s.fm[i] = nm;
        s.zz[i] = nz;
    }
}

// The same RF with the structure of a phi = 0 pulse (c3 = c1, c4 = c0,
// c5 = -c2, c7 = -c6, as rf_real_coeffs2 produces them and the folded
// relaxation keeps them): F-' = (c0 + c1)(F+ + F-) - F+' and
// Z' = c6 (F+ - F-) + c8 Z, 8 packed operations per pair instead of 9.  It
// rounds differently from the reference's order (unit-norm C1 atoms move by
// at most 6e-8) and is used by the folded recursion only, whose s.fm holds
// -F-: no operand of a packed instruction is then negated (a negation is an
// instruction per element), and no value changes but for the sign of zeros.
template <int P>
__device__ __forceinline__ void rl2_rf_k8(RealLane2<P> &s, float2 c0, float2 nc1, float2 c2, float2 c6, float2 c8) {
    const float2 minus = make_float2(-1.f, -1.f);
    const float2 cs = __ffma2_rn(nc1, minus, c0), ncs = __ffma2_rn(c0, minus, nc1);
#pragma unroll
    for (int i = 0; i < P; i++) {
        const float2 p = s.fp[i], n = s.fm[i], z = s.zz[i];
        float2 np = __fmul2_rn(c0, p);
        np = __ffma2_rn(nc1, n, np);
        np = __ffma2_rn(c2, z, np);
        float2 nz = __fmul2_rn(c6, __fadd2_rn(p, n));
        nz = __ffma2_rn(c8, z, nz);
        float2 nn = __ffma2_rn(cs, n, np);
        nn = __ffma2_rn(ncs, p, nn);
        s.fp[i] = np;
        s.fm[i] = nn;
        s.zz[i] = nz;
    }
}

template <int P>
__device__ __forceinline__ void rl2_rf(RealLane2<P> &s, const float2 *c) {
    rl2_rf_k<P>(s, c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8]);
}

// e = (E2, E1) of one interval: F+- *= E2, Z *= E1, then Z0 += 1 - E1.
template <int P>
__device__ __forceinline__ void rl2_relax(RealLane2<P> &s, float E1, float E2, bool lane0) {
    const float2 e2 = make_float2(E2, E2), e1 = make_float2(E1, E1);
#pragma unroll
    for (int i = 0; i < P; i++) {
        s.fp[i] = __fmul2_rn(s.fp[i], e2);
        s.fm[i] = __fmul2_rn(s.fm[i], e2);
        s.zz[i] = __fmul2_rn(s.zz[i], e1);
    }
    if (lane0) s.zz[0].x = __fadd_rn(s.zz[0].x, 1 - E1);
}

// Gradient shift of the paired real state (see st_shift): F+ up one slot,
// F- down one slot, f+[0] = -f-[0] (Im of conj), F-[w-1] = 0, slots k >= w
// zero; with w = 1 the unshifted f-[0] is used.  A pair holds states P apart,
// so a pair moves as a whole: only the pair that takes the neighbour's state
// is put together anew.
//
// Slots k >= w hold zeros before the shift, so F-[w-1] takes the zero of F-[w]
// and only F+[w], which receives F+[w-1], must be cleared: by a multiply per
// pair whose factors the step loop keeps (a compare and a select per slot took
// w = 49, 53 and 61 from 1.45, 1.43 and 1.59 to 2.16, 2.06 and 2.16 ms, 138,760
// atoms, T = 500).
// TAIL: the layout pads at most two slots (w >= 2P L - 2).  That slot is then the
// second of the last lane's last pair (or of the one before it), and
// tail_keep (0 there, 1 elsewhere; .x the pair before the last, .y the last)
// clears it with one multiply.
// NEG: s.fm holds -F-.
template <int P, bool TAIL, bool NEG>
__device__ __forceinline__ void rl2_shift(RealLane2<P> &s, int gl, int L, int w, float2 tail_keep) {
    const unsigned full = 0xffffffffu;
    const float up = __shfl_up_sync(full, s.fp[P - 1].y, 1, L);
    const float dn = __shfl_down_sync(full, s.fm[0].x, 1, L);
    const float old_fm0 = s.fm[0].x, mid_p = s.fp[P - 1].x, mid_m = s.fm[0].y;
#pragma unroll
    for (int i = P - 1; i >= 1; i--) s.fp[i] = s.fp[i - 1];
    s.fp[0] = make_float2(up, mid_p);
#pragma unroll
    for (int i = 0; i < P - 1; i++) s.fm[i] = s.fm[i + 1];
    s.fm[P - 1] = make_float2(mid_m, (gl == L - 1) ? 0.f : dn);
    if (gl == 0) {
        const float f0 = w == 1 ? old_fm0 : s.fm[0].x;
        s.fp[0].x = NEG ? f0 : -f0;
    }
    if (TAIL) {
        s.fp[P - 1].y *= tail_keep.y;
        if (P > 1)
            s.fp[P - 2].y *= tail_keep.x;
        else
            s.fp[0].x *= tail_keep.x;
        return;
    }
    const int j = w - gl * 2 * P;  // slot w in this lane
#pragma unroll
    for (int i = 0; i < P; i++)
        s.fp[i] = __fmul2_rn(s.fp[i], make_float2(j == i ? 0.f : 1.f, j == P + i ? 0.f : 1.f));
}

// The real-valued kernel: one warp per CTA, so that no CTA barrier makes the
// warps of a CTA wait for each other at every chunk (C1: 7.82 ms with 128
// threads, 7.79 with 64, 7.63 with 32; the atoms are bit-identical).  It
// stages 32 steps per chunk, one per lane.
constexpr int kRealThreads = 32;
constexpr int kRealChunk = 32;
// Steps unrolled: the shift only renames registers, and the moves that a
// loop's end needs come once per four steps (C1's dictionary, 284,458 atoms,
// T = 1000, w = 50 as 2 lanes x 13 pairs: 6.12 ms with 1, 5.55 with 2, 5.41
// with 4, 5.36 with 8; 6.60 with pairs of neighbouring states, which every
// shift puts together anew, and 16-byte pieces of rows written per lane).
// 166 instead of 224 instructions per warp and step, 104 of them the packed
// operations: those keep the FP32 pipe 73 % busy, the rest is latency at two
// to three warps per scheduler (the states take the registers; limits of 128
// and 144 registers spill and take 6.2-6.5 ms).
constexpr int kRealUnroll = 4;
// Resident CTAs per SM asked of the compiler (168 registers at 12).  With more
// pairs a lane takes 208 to 255 registers, and still gains: 138,760 atoms, T =
// 500, ms with pairs of neighbours (148 to 180 registers) and now: w = 50 (13
// pairs) 1.63 / 1.28, 53 (14, padded) 2.43 / 1.43, 56 (14) 1.67 / 1.38, 57 (15,
// padded) 2.79 / 1.51, 64 (16) 1.87 / 1.50; 45 and 49 (padded) 2.15 / 1.37 and
// 2.51 / 1.45.
constexpr int real_min_ctas(int P) { return P <= 13 ? 12 : 1; }
constexpr int kRealFS = kRealChunk * 4 + 4;        // floats per atom of relaxation factors
constexpr int kRealReadoutStride = kRealChunk + 1;  // floats per atom
__host__ __device__ constexpr int epg_real_nc(bool fold) { return fold ? 6 : 10; }  // RF coefficient pairs per step

// Byte offsets in a CTA's shared memory (apc atoms).  RF coefficients, factors
// and parameters are read 16 bytes at a time, so each starts on a multiple of
// 16 for any apc; the readouts, single floats in rows of 33, come last.
__host__ __device__ constexpr size_t epg_real_off_factors(bool fold) {
    return (size_t)kRealChunk * epg_real_nc(fold) * sizeof(float2);
}
__host__ __device__ constexpr size_t epg_real_off_params(int apc, bool fold) {
    return epg_real_off_factors(fold) + (size_t)apc * kRealFS * sizeof(float);
}
__host__ __device__ constexpr size_t epg_real_off_readouts(int apc, bool fold) {
    return epg_real_off_params(apc, fold) + (size_t)apc * 4 * sizeof(float);
}
constexpr bool epg_real_aligned() {
    for (int apc = 1; apc <= kRealThreads; apc++)
        for (int fold = 0; fold < 2; fold++)
            if (epg_real_off_factors(fold) % 16 || epg_real_off_params(apc, fold) % 16) return false;
    return epg_real_nc(true) * sizeof(float2) % 16 == 0 && kRealFS % 4 == 0;
}
static_assert(epg_real_aligned(), "16-byte reads of coefficients, factors and parameters");

inline size_t epg_real_smem_bytes(int L, bool fold) {
    const int apc = kRealThreads / L;
    return epg_real_off_readouts(apc, fold) + (size_t)apc * kRealReadoutStride * sizeof(float);
}

// One element of the optional 16-bit copy of Im(atom) (the tensor-core
// matching operand, one row per atom).
__device__ __forceinline__ void store_packed(const EpgArgs &a, long long atom, long long q, float v) {
    if (a.packed_half)
        reinterpret_cast<__half *>(a.packed)[atom * a.packed_pitch + q] = __float2half_rn(v);
    else
        reinterpret_cast<__nv_bfloat16 *>(a.packed)[atom * a.packed_pitch + q] = __float2bfloat16_rn(v);
}

// FOLD: relaxation is diagonal with one factor for F+ and F- (and Z0's
// recovery only touches state 0), so it commutes with the dephasing shift:
// relax(TE), shift, relax(TR - TE) equals shift followed by one relaxation
// over TR, and that relaxation is folded into the next step's RF columns
// (c_j * E_j, plus the recovery (1 - E1) times the RF's Z column on state 0).
// The readout after relax(TE) is E2(TE) f+[0] right after the RF.  Two
// multiplies per state and step fewer, and one exp fewer per atom and step;
// the result differs from the separate relaxations only by rounding.
//
// One CTA's work: atoms atom0 .. atom0 + kRealThreads / L - 1 of B1 block
// blk, L lanes per atom, P pairs of states per lane.
template <int ECHO, int P, bool TAIL, bool FOLD>
__device__ __forceinline__ void epg_real_cta(const EpgArgs &a, const int L, const long long blk,
                                             const long long atom0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int NF = 4;
    constexpr int FS = kRealFS;
    const int apc = kRealThreads / L;
    const int tid = threadIdx.x;
    const int g = tid / L;
    const int gl = tid % L;
    const bool lane0 = (gl == 0);
    const long long nreps = a.nreps;
    const long long ab = atom0 + g;
    const bool active = ab < a.natoms;
    const long long gatom = blk * a.natoms + ab;

    constexpr int NC = epg_real_nc(FOLD);
    float2 *sC = reinterpret_cast<float2 *>(smem_raw);                                        // [kRealChunk][NC]
    float *sF = reinterpret_cast<float *>(smem_raw + epg_real_off_factors(FOLD));             // [apc][FS]
    float *sP = reinterpret_cast<float *>(smem_raw + epg_real_off_params(apc, FOLD));         // [apc][4]
    float *sR = reinterpret_cast<float *>(smem_raw + epg_real_off_readouts(apc, FOLD));  // [apc][kRealReadoutStride]

    if (tid < apc) {
        const long long at = atom0 + tid;
        float t1 = 1.f, t2 = 1.f;
        if (at < a.natoms) {
            const float *p = a.params + (blk * a.natoms + at) * a.nparams;
            t1 = p[0];
            t2 = p[1];
        }
        sP[4 * tid] = t1;
        sP[4 * tid + 1] = t2;
        sP[4 * tid + 2] = 1.f / t1;
        sP[4 * tid + 3] = 1.f / t2;
    }

    const float *alpha = a.alpha + blk * nreps;
    const float *phi = a.sched + nreps;
    const float *TR = a.sched + 2 * nreps;
    const float *TE = a.sched + 3 * nreps;
    __syncwarp();
    const int w = a.nstates;
    // TAIL layouts: 0 at slot w (cleared after each shift), 1 elsewhere
    float2 tail_keep = make_float2(1.f, 1.f);
    if (TAIL && gl == L - 1) {
        const int pad = L * 2 * P - w;
        tail_keep = make_float2(pad == 2 ? 0.f : 1.f, pad >= 1 ? 0.f : 1.f);
    }

    // init_rf_pulse with alpha = phi = 0, TI = 0 (the expression of st_init)
    RealLane2<P> s;
#pragma unroll
    for (int i = 0; i < P; i++) {
        s.fp[i] = make_float2(0.f, 0.f);
        s.fm[i] = make_float2(0.f, 0.f);
        s.zz[i] = make_float2(0.f, 0.f);
    }
    if (lane0) {
        const float T1 = sP[4 * g];
        float e1 = expf(-0.f / T1), sa, ca;
        __sincosf((float)(0.f * M_PI / 180.f), &sa, &ca);
        s.zz[0].x = e1 * ca + 1 - e1;
    }

    float nrm = 0.f;
    const long long row0 = blk * a.natoms + atom0;  // the CTA's first atom
    const int rows = (int)min((long long)apc, a.natoms - atom0);
    float *const atoms_i = reinterpret_cast<float *>(a.atoms);  // (imaginary rows)
    for (long long t0 = 0; t0 < nreps; t0 += kRealChunk) {
        const int nch = (int)min((long long)kRealChunk, nreps - t0);
        __syncwarp();
        // lane i stages step t0 + i of every atom
        if (tid < nch) {
            const long long t = t0 + tid;
            float2 cf[10];
            rf_real_coeffs2(alpha[t], phi[t], cf);
            if (FOLD) {
                float4 *c = reinterpret_cast<float4 *>(sC + NC * tid);
                c[0] = make_float4(cf[0].x, cf[0].y, -cf[1].x, -cf[1].y);
                c[1] = make_float4(cf[2].x, cf[2].y, cf[6].x, cf[6].y);
                c[2] = make_float4(cf[8].x, cf[8].y, 0.f, 0.f);
            } else {
#pragma unroll
                for (int q = 0; q < NC; q++) sC[NC * tid + q] = cf[q];
            }
            const float tr = TR[t], te = TE[t], tb = tr - te;
            const float trp = t > 0 ? TR[t - 1] : 0.f;
            for (int ga = 0; ga < apc; ga++) {
                const float4 tp = *reinterpret_cast<const float4 *>(sP + 4 * ga);
                float4 f;
                if (FOLD) {
                    // (E1, E2) over the previous step's TR (1 before the first
                    // step), E2 over this step's TE, and Z0's recovery 1 - E1;
                    // rates as reciprocals (|t / T| < 1, so the argument's
                    // rounding moves exp by far less than an ulp)
                    const float e1 = t > 0 ? expf(-trp * tp.z) : 1.f, e2 = t > 0 ? expf(-trp * tp.w) : 1.f;
                    f = make_float4(e1, e2, expf(-te * tp.w), 1.f - e1);
                } else {
                    f = make_float4(expf(-te / tp.x), expf(-te / tp.y), expf(-tb / tp.x), expf(-tb / tp.y));
                }
                *reinterpret_cast<float4 *>(sF + ga * FS + tid * NF) = f;
            }
        }
        __syncwarp();
#pragma unroll kRealUnroll
        for (int i = 0; i < nch; i++) {
            const float4 f = *reinterpret_cast<const float4 *>(sF + g * FS + i * NF);
            if (FOLD) {
                const float4 *c = reinterpret_cast<const float4 *>(sC + NC * i);
                const float4 c01 = c[0], c26 = c[1];
                const float2 c8 = *reinterpret_cast<const float2 *>(c + 2);
                const float2 e1 = make_float2(f.x, f.x), e2 = make_float2(f.y, f.y);
                rl2_rf_k8<P>(s, __fmul2_rn(make_float2(c01.x, c01.y), e2), __fmul2_rn(make_float2(c01.z, c01.w), e2),
                             __fmul2_rn(make_float2(c26.x, c26.y), e1), __fmul2_rn(make_float2(c26.z, c26.w), e2),
                             __fmul2_rn(c8, e1));
                if (lane0) {
                    // the recovery term (1 - E1) of Z0 through the RF's Z column
                    s.fp[0].x = fmaf(c26.x, f.w, s.fp[0].x);
                    s.fm[0].x = fmaf(c26.x, f.w, s.fm[0].x);
                    s.zz[0].x = fmaf(c8.x, f.w, s.zz[0].x);
                    const float v = f.z * s.fp[0].x;
                    sR[g * kRealReadoutStride + i] = v;
                    nrm = fmaf(v, v, nrm);
                }
                if (ECHO == ECHO_FISP) rl2_shift<P, TAIL, FOLD>(s, gl, L, w, tail_keep);
            } else {
                rl2_rf<P>(s, sC + NC * i);
                rl2_relax<P>(s, f.x, f.y, lane0);
                if (lane0) {
                    const float v = s.fp[0].x;
                    sR[g * kRealReadoutStride + i] = v;
                    // the complex path adds round(0*0 + v*v) = round(v*v)
                    nrm = __fadd_rn(nrm, __fmul_rn(v, v));
                }
                if (ECHO == ECHO_FISP) rl2_shift<P, TAIL, FOLD>(s, gl, L, w, tail_keep);
                rl2_relax<P>(s, f.z, f.w, lane0);
            }
        }
        __syncwarp();
        // lane i writes sample t0 + i of every atom: 32 samples of a row at once
        if (tid < nch)
            for (int r = 0; r < rows; r++) {
                const long long at = row0 + r, q = t0 + tid;
                const float v = sR[r * kRealReadoutStride + tid];
                if (a.imag_rows)
                    atoms_i[at * nreps + q] = v;
                else
                    a.atoms[at * nreps + q] = make_float2(0.f, v);
                if (a.packed && !a.normalize && !a.pack_normalized) store_packed(a, at, q, v);
            }
    }
    if (a.norms && lane0 && active) a.norms[gatom] = sqrtf(nrm);
    if (a.normalize || (a.pack_normalized && !a.operand_pass)) {
        for (int r = 0; r < rows; r++) {
            const long long at = row0 + r;
            float inv = __shfl_sync(0xffffffffu, nrm, r * L);
            if (inv > 0.f) inv = 1.f / sqrtf(inv);
            float2 *out = a.atoms + at * nreps;
            float *outi = atoms_i + at * nreps;
            // (a lane reads the samples that it wrote)
            if (a.normalize && a.imag_rows) {
                // (the same product as the complex row's imaginary part)
                for (long long q = tid; q < nreps; q += 32) {
                    const float o = outi[q] * inv;
                    outi[q] = o;
                    if (a.packed) store_packed(a, at, q, o);
                }
            } else if (a.normalize) {
                for (long long q = tid; q < nreps; q += 32) {
                    const float2 o = c_scale(out[q], inv);
                    out[q] = o;
                    if (a.packed) store_packed(a, at, q, o.y);
                }
            } else {
                // the operand of the unit-norm atom (the same product as
                // above); the atom itself is not rewritten
                for (long long q = tid; q < nreps; q += 32)
                    store_packed(a, at, q, a.imag_rows ? outi[q] * inv : c_scale(out[q], inv).y);
            }
        }
    }
    if (a.packed && !a.operand_pass)
        for (int r = 0; r < rows; r++)
            for (long long q = nreps + tid; q < a.packed_pitch; q += 32) store_packed(a, row0 + r, q, 0.f);
}

// Fine layout of the real-valued recursion: kFineP pairs of states per lane
// and kFineL = 32 / kFineP lanes per atom (64 states, so w <= 64).  Two
// pairs measured best on C1's tail (one: a lone warp is latency-bound on the
// shuffles; four: more instructions per step).
#ifndef SNAPMRF_EPG_FINE_P
#define SNAPMRF_EPG_FINE_P 2
#endif
constexpr int kFineP = SNAPMRF_EPG_FINE_P;
constexpr int kFineL = 32 / kFineP;
static_assert(kFineP == 1 || kFineP == 2 || kFineP == 4 || kFineP == 8, "fine layout");

// Grid: x = CTA within the B1 block, y = block.  Each CTA signals at once
// that a grid launched after it as a programmatic dependent (the fine tail
// below) may start: that grid then starts when every CTA of this one has
// started, i.e. during its last round.
template <int ECHO, int P, bool TAIL, bool FOLD>
__global__ void __launch_bounds__(kRealThreads, real_min_ctas(P)) epg_real_kernel(EpgArgs a) {
    asm volatile("griddepcontrol.launch_dependents;");
    epg_real_cta<ECHO, P, TAIL, FOLD>(a, a.L, blockIdx.y, (long long)blockIdx.x * (kRealThreads / a.L));
}

// Fine tail: atoms a.fine_first .. natoms - 1 of each B1 block in the fine
// layout.  A CTA carries its atoms through every step whatever its layout,
// and the fine CTAs, a few times shorter than those of the chosen layout,
// fill the slots that the chosen layout's last, partial round of resident
// CTAs leaves free instead of a few full-length CTAs running alone.  Every
// layout performs the same operations on each state in the same order, so
// the atoms do not depend on the split.  Launched as a programmatic
// dependent of the main grid, this grid must not complete before it (work
// after it on the stream reads the whole dictionary), hence the wait at the
// end; launched alone, the wait returns at once.
template <int ECHO, bool FOLD>
__global__ void __launch_bounds__(kRealThreads, 1) epg_real_fine_kernel(EpgArgs a) {
    epg_real_cta<ECHO, kFineP, false, FOLD>(a, kFineL, blockIdx.y,
                                            a.fine_first + (long long)blockIdx.x * (kRealThreads / kFineL));
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ROA (src/functions.cu:1021-1222).  State m = (Mx, My, Mz).  Per step:
// rotation R(alpha, phi), relaxation over the full TR, z-rotation by
// beta = pi*B0*TR/1000, readout Mx + iMy, z-rotation by beta.
struct RoaStep {
    float T[9];
};

// fill_transition_matrix (ROA, src/functions.cu:1049-1075); the Sgemm with
// OP_N reads it column-major: new[i] = sum_l T[i + 3l] * m[l].
__device__ __forceinline__ void roa_matrix(float alpha, float phi, float *T) {
    float s_a, c_a, s_p, c_p;
    __sincosf(alpha, &s_a, &c_a);
    __sincosf(phi, &s_p, &c_p);
    float s2 = 2 * c_p * s_p, c2 = c_p * c_p - s_p * s_p;
    T[0] = c2;
    T[1] = -s2;
    T[2] = 0.f;
    T[3] = s2 * c_a;
    T[4] = c2 * c_a;
    T[5] = -s_a;
    T[6] = s2 * s_a;
    T[7] = c2 * s_a;
    T[8] = c_a;
}

// init_rf_pulse (ROA, src/functions.cu:1022-1047); roa_ssfp calls it with
// alpha 180, phi 0, TI 0 (run-time values, see EpgArgs).
__device__ __forceinline__ void roa_init(float t1, float t2, float &m0, float &m1, float &m2, float alpha_deg,
                                         float phi_deg, float TI) {
    float ia = (float)(alpha_deg * M_PI / 180.f), ip = (float)(phi_deg * M_PI / 180.f);
    float e1 = expf(-TI / t1), e2 = expf(-TI / t2);
    float sa, ca, sph, cph;
    __sincosf(ia, &sa, &ca);
    __sincosf(ip, &sph, &cph);
    float sph2 = 2 * cph * sph, cph2 = cph * cph - sph * sph;
    m0 = e2 * sph2 * sa;
    m1 = e2 * cph2 * sa;
    m2 = e1 * ca + 1 - e1;
}

#ifndef SNAPMRF_EPG_DEVICE_HELPERS_ONLY
// (the non-template kernel below is defined once, in epg.cu; other sources
// that need only the device helpers above define
// SNAPMRF_EPG_DEVICE_HELPERS_ONLY)

// Single isochromat (the reference's roa_ssfp): one thread per atom.
__global__ void __launch_bounds__(kEpgThreads) roa_kernel(EpgArgs a) {
    __shared__ RoaStep sT[kChunk];
    __shared__ float2 sR[kEpgThreads][kChunk + 1];
    __shared__ float sN[kEpgThreads];
    const int tid = threadIdx.x;
    const long long blk = blockIdx.y;
    const long long nreps = a.nreps;
    const long long atom0 = (long long)blockIdx.x * kEpgThreads;
    const long long ab = atom0 + tid;
    const bool active = ab < a.natoms;
    const long long gatom = blk * a.natoms + ab;
    float t1 = 1.f, t2 = 1.f, b0 = 0.f;
    if (active) {
        const float *p = a.params + (blk * a.natoms + ab) * a.nparams;
        t1 = p[0];
        t2 = p[1];
        b0 = p[2];
    }
    const float *alpha = a.alpha + blk * nreps;
    const float *phi = a.sched + nreps;
    const float *TR = a.sched + 2 * nreps;
    const double rate = M_PI * b0 / 1000.0;  // rad / ms over half a TR
    float m0, m1, m2;
    roa_init(t1, t2, m0, m1, m2, a.init_alpha_deg, a.init_phi_deg, a.init_ti);
    float nrm = 0.f;
    const int warp = tid / 32, lane = tid % 32;
    for (long long t0 = 0; t0 < nreps; t0 += kChunk) {
        const int nch = (int)min((long long)kChunk, nreps - t0);
        __syncthreads();
        for (int i = tid; i < nch; i += kEpgThreads) roa_matrix(alpha[t0 + i], phi[t0 + i], sT[i].T);
        __syncthreads();
        for (int i = 0; i < nch; i++) {
            const float *T = sT[i].T;
            // the in-place cublasSgemm of apply_rf_pulse (ROA), accumulated
            // over the three components in order
            float n0 = fmaf(T[6], m2, fmaf(T[3], m1, T[0] * m0));
            float n1 = fmaf(T[7], m2, fmaf(T[4], m1, T[1] * m0));
            float n2 = fmaf(T[8], m2, fmaf(T[5], m1, T[2] * m0));
            float tr = TR[t0 + i];
            float E1 = expf(-tr / t1), E2 = expf(-tr / t2);
            m0 = E2 * n0;
            m1 = E2 * n1;
            m2 = E1 * n2 + (1 - E1);
            float sb, cb;
            __sincosf((float)(rate * tr), &sb, &cb);
            float w1 = m0, w2 = m1;
            m0 = cb * w1 + sb * w2;
            m1 = cb * w2 - sb * w1;
            sR[tid][i] = make_float2(m0, m1);
            nrm += m0 * m0 + m1 * m1;
            w1 = m0;
            w2 = m1;
            m0 = cb * w1 + sb * w2;
            m1 = cb * w2 - sb * w1;
        }
        __syncthreads();
        for (int r = warp; r < kEpgThreads; r += kEpgThreads / 32) {
            long long at = atom0 + r;
            if (at >= a.natoms) continue;
            float2 *o = a.atoms + (blk * a.natoms + at) * nreps + t0;
            for (int q = lane; q < nch; q += 32) o[q] = sR[r][q];
        }
    }
    if (a.norms && active) a.norms[gatom] = sqrtf(nrm);
    if (a.normalize) {
        sN[tid] = nrm > 0.f ? 1.f / sqrtf(nrm) : nrm;
        __syncthreads();
        for (int r = warp; r < kEpgThreads && atom0 + r < a.natoms; r += kEpgThreads / 32) {
            const float inv = sN[r];
            float2 *out = a.atoms + (blk * a.natoms + atom0 + r) * nreps;
            for (long long q = lane; q < nreps; q += 32) out[q] = c_scale(out[q], inv);
        }
    }
}

// Multi-isochromat ROA: a group of G lanes per atom (G = 8, 16 or 32, a
// divisor of the warp), IPL isochromats per lane; lane r of a group holds
// isochromats r*IPL .. r*IPL + IPL - 1 (those past n_iso idle), so that G*IPL
// close above n_iso wastes few slots (n_iso = 100: 8 x 13 = 104, where 32
// lanes x 4 carried 128).  Isochromat j precesses by an extra d_j = pi*j/n_iso
// per half TR (2*pi*j/n_iso per TR, so the n_iso isochromats dephase uniformly
// across 2*pi); the readout is the mean of Mx + iMy over isochromats.
//
// The RF is a rotation about x and one about z (by 2 phi), and all rotations
// about z commute, so a step is one matrix common to the atom's isochromats
// (the flip, relaxation over TR and the z-rotation by 2 phi + 2 beta),
// followed by the isochromat's rotation by 2 d_j:
//   n = M u,  u' = R(2 d_j) n,  readout = R(-beta) sum_j R(d_j) n_j / n_iso:
// 16 operations per isochromat and step (3 + 3 + 2 for n, 4 for the sum, 4 for
// u'), two-wide on pairs of isochromats, instead of 22 scalar ones that added
// the angles for each.  The atom's constants are computed by the group's lanes,
// one step each; the lanes' sums meet in shared memory, once per chunk.  No
// CTA barrier: a warp's groups depend on nothing outside the warp.
// 55,504 atoms, T = 500, 100 isochromats: 2.92 -> 1.90 ms, of which the 16
// operations take 1.28 at the measured FP32 peak with the idle slots (1, 2
// and 4 steps unrolled 1.91, 1.90, 1.92; a limit of 128 registers spills:
// 1.96); error against 64 bits 2.7e-6 (22 operations: 2.8e-6).
struct RoaIsoStep {
    float4 x;  // Mx row: x, y, z; recovery 1 - E1
    float4 y;  // My row: x, y, z; Mz row: y
    float4 z;  // Mz row: z; cos, sin of beta (the readout's way back)
};

template <int IPL>
__global__ void __launch_bounds__(kEpgThreads) roa_iso_kernel(EpgArgs a, int G) {
    constexpr int MAXA = kEpgThreads / 8;  // atoms per CTA at G = 8
    constexpr int NP = IPL / 2;            // pairs; an odd isochromat by itself
    constexpr bool ODD = IPL % 2 != 0;
    // (rows padded by one entry: the groups of a warp read and write
    // different banks)
    __shared__ RoaIsoStep sF[MAXA][kChunk + 1];
    __shared__ float2 sO[kChunk][kEpgThreads + 1];  // each lane's part of the readout
    const int tid = threadIdx.x;
    const int apc = kEpgThreads / G, ga = tid / G, r = tid % G;
    const long long blk = blockIdx.y;
    const long long nreps = a.nreps;
    const long long ab = (long long)blockIdx.x * apc + ga;
    const bool active = ab < a.natoms;
    const long long gatom = blk * a.natoms + ab;
    float t1 = 1.f, t2 = 1.f, b0 = 0.f;
    if (active) {
        const float *p = a.params + gatom * a.nparams;
        t1 = p[0];
        t2 = p[1];
        b0 = p[2];
    }
    const double rate = M_PI * b0 / 1000.0;  // rad / ms over half a TR
    const float *alpha = a.alpha + blk * nreps;
    const float *phi = a.sched + nreps;
    const float *TR = a.sched + 2 * nreps;
    const int n_iso = a.n_iso;
    float i0, i1, i2;
    roa_init(t1, t2, i0, i1, i2, a.init_alpha_deg, a.init_phi_deg, a.init_ti);
    // (a slot past n_iso gets zero rotations: its Mx, My are 0 from the first
    // step on and its readout adds exactly 0)
    float mx[IPL], my[IPL], mz[IPL], cd[IPL], sd[IPL], ce[IPL], se[IPL];
#pragma unroll
    for (int q = 0; q < IPL; q++) {
        const int j = r * IPL + q;
        mx[q] = i0;
        my[q] = i1;
        mz[q] = i2;
        double s1 = 0, c1 = 0;
        if (j < n_iso) sincospi((double)j / (double)n_iso, &s1, &c1);
        cd[q] = (float)c1;
        sd[q] = (float)s1;
        ce[q] = (float)(c1 * c1 - s1 * s1);
        se[q] = (float)(2 * c1 * s1);
    }
    const float inv_n = 1.f / (float)n_iso;
    float nrm = 0.f;
    float2 *out = a.atoms + gatom * nreps;
    for (long long t0 = 0; t0 < nreps; t0 += kChunk) {
        const int nch = (int)min((long long)kChunk, nreps - t0);
        __syncwarp();
        for (int i = r; i < nch; i += G) {
            const float tr = TR[t0 + i];
            float sb, cb, sa, ca, sp, cp;
            __sincosf((float)(rate * tr), &sb, &cb);
            __sincosf(alpha[t0 + i], &sa, &ca);
            __sincosf(phi[t0 + i], &sp, &cp);
            const float s2 = 2 * cp * sp, c2 = cp * cp - sp * sp, sb2 = 2 * cb * sb, cb2 = cb * cb - sb * sb;
            const float E1 = expf(-tr / t1), E2 = expf(-tr / t2);
            const float ec = E2 * (c2 * cb2 - s2 * sb2), es = E2 * (s2 * cb2 + c2 * sb2);
            RoaIsoStep k;
            k.x = make_float4(ec, es * ca, es * sa, 1.f - E1);
            k.y = make_float4(-es, ec * ca, ec * sa, -E1 * sa);
            k.z = make_float4(E1 * ca, cb, sb, 0.f);
            sF[ga][i] = k;
        }
        __syncwarp();
#pragma unroll 2
        for (int i = 0; i < nch; i++) {
            const float4 kx = sF[ga][i].x, ky = sF[ga][i].y;
            const float zz = sF[ga][i].z.x;
            const float2 x0 = make_float2(kx.x, kx.x), x1 = make_float2(kx.y, kx.y), x2 = make_float2(kx.z, kx.z);
            const float2 y0 = make_float2(ky.x, ky.x), y1 = make_float2(ky.y, ky.y), y2 = make_float2(ky.z, ky.z);
            const float2 z1 = make_float2(ky.w, ky.w), z2 = make_float2(zz, zz), rec = make_float2(kx.w, kx.w);
            float2 px = make_float2(0.f, 0.f), py = px, qy = px;
#pragma unroll
            for (int q = 0; q < NP; q++) {
                const float2 x = make_float2(mx[2 * q], mx[2 * q + 1]), y = make_float2(my[2 * q], my[2 * q + 1]);
                const float2 z = make_float2(mz[2 * q], mz[2 * q + 1]);
                const float2 c = make_float2(cd[2 * q], cd[2 * q + 1]), s = make_float2(sd[2 * q], sd[2 * q + 1]);
                const float2 C = make_float2(ce[2 * q], ce[2 * q + 1]), S = make_float2(se[2 * q], se[2 * q + 1]);
                const float2 nx = __ffma2_rn(x2, z, __ffma2_rn(x1, y, __fmul2_rn(x0, x)));
                const float2 ny = __ffma2_rn(y2, z, __ffma2_rn(y1, y, __fmul2_rn(y0, x)));
                const float2 nz = __ffma2_rn(z2, z, __ffma2_rn(z1, y, rec));
                px = __ffma2_rn(s, ny, __ffma2_rn(c, nx, px));
                py = __ffma2_rn(c, ny, py);
                qy = __ffma2_rn(s, nx, qy);
                const float2 ux = __ffma2_rn(S, ny, __fmul2_rn(C, nx));
                const float2 uy = __ffma2_rn(make_float2(-S.x, -S.y), nx, __fmul2_rn(C, ny));
                mx[2 * q] = ux.x;
                mx[2 * q + 1] = ux.y;
                my[2 * q] = uy.x;
                my[2 * q + 1] = uy.y;
                mz[2 * q] = nz.x;
                mz[2 * q + 1] = nz.y;
            }
            float sx = px.x + px.y, sy = (py.x - qy.x) + (py.y - qy.y);
            if (ODD) {
                constexpr int q = IPL - 1;
                const float x = mx[q], y = my[q], z = mz[q];
                const float nx = fmaf(kx.z, z, fmaf(kx.y, y, kx.x * x));
                const float ny = fmaf(ky.z, z, fmaf(ky.y, y, ky.x * x));
                mz[q] = fmaf(zz, z, fmaf(ky.w, y, kx.w));
                sx = fmaf(sd[q], ny, fmaf(cd[q], nx, sx));
                sy = fmaf(-sd[q], nx, fmaf(cd[q], ny, sy));
                mx[q] = fmaf(se[q], ny, ce[q] * nx);
                my[q] = fmaf(-se[q], nx, ce[q] * ny);
            }
            sO[i][tid] = make_float2(sx, sy);
        }
        __syncwarp();
        // the group's sums (a group never straddles a warp)
        for (int i = r; i < nch; i += G) {
            float sx = 0.f, sy = 0.f;
            for (int q = 0; q < G; q++) {
                const float2 o = sO[i][tid - r + q];
                sx += o.x;
                sy += o.y;
            }
            const float4 k = sF[ga][i].z;
            const float2 v = make_float2((k.y * sx - k.z * sy) * inv_n, (k.y * sy + k.z * sx) * inv_n);
            nrm = fmaf(v.x, v.x, fmaf(v.y, v.y, nrm));
            if (active) out[t0 + i] = v;
        }
    }
    for (int o = G / 2; o; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (a.norms && active && r == 0) a.norms[gatom] = sqrtf(nrm);
    // (with G = 32 a lane rescales samples another lane of the group wrote)
    __syncwarp();
    if (a.normalize && active) {
        float inv = nrm;
        if (inv > 0.f) inv = 1.f / sqrtf(inv);
        for (long long q = r; q < nreps; q += G) out[q] = c_scale(out[q], inv);
    }
}

// Isochromats per lane and lanes per atom of roa_iso_kernel: the fewest
// slots G * IPL >= n_iso (n_iso <= 256), then the most isochromats per lane.
inline void roa_iso_layout(int n_iso, int *G, int *ipl) {
    static const int ipls[] = {13, 8, 7, 4, 2, 1};
    int best = 1 << 30;
    for (int g : {8, 16, 32})
        for (int i : ipls)
            if (g * i >= n_iso && (g * i < best || (g * i == best && i > *ipl))) {
                best = g * i;
                *G = g;
                *ipl = i;
            }
}

inline cudaError_t launch_roa(const EpgArgs &a, long long natoms, unsigned gen_blocks,
                              cudaStream_t st) {
    if (a.n_iso <= 1) {
        dim3 grid((unsigned)((natoms + kEpgThreads - 1) / kEpgThreads), gen_blocks);
        roa_kernel<<<grid, kEpgThreads, 0, st>>>(a);
    } else {
        int G = 32, ipl = 0;
        roa_iso_layout(a.n_iso, &G, &ipl);
        const long long apc = kEpgThreads / G;
        dim3 grid((unsigned)((natoms + apc - 1) / apc), gen_blocks);
        switch (ipl) {
        case 1: roa_iso_kernel<1><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        case 2: roa_iso_kernel<2><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        case 4: roa_iso_kernel<4><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        case 7: roa_iso_kernel<7><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        case 8: roa_iso_kernel<8><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        default: roa_iso_kernel<13><<<grid, kEpgThreads, 0, st>>>(a, G); break;
        }
    }
    note_launches(1);
    return cudaGetLastError();
}

#endif  // SNAPMRF_EPG_DEVICE_HELPERS_ONLY

}  // namespace snapmrf
