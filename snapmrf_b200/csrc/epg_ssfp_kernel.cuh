// The bSSFP recursion (epg_ssfp, src/functions.cu:935-1019) in the frame of
// the RF phase.
//
// With z = e^{i phi_t}, G+ = conj(z) F+, G- = z F- and Y = -i Z, the RF pulse of
// any phase has real coefficients,
//   G+' = c G+ + s G- + S Y,  G-' = (G+ + G-) - G+',  Y' = -S/2 (G+ - G-) + C Y
// (C = cos a, S = sin a, c = (1 + C)/2, s = (1 - C)/2), so a pulse takes 8
// two-wide operations per state on (re, im) instead of 36 scalar ones.  What
// lies between two pulses multiplies F+ by one complex number and F- by its
// conjugate, whatever the order: relaxation over TE and TR - TE, precession
// over both, and the change of frame, w = E2(TR) e^{i theta(TR)} z_t
// conj(z_{t+1}); it commutes with the dephasing shift (F+[0] = conj F-[0] keeps
// the form), so the shift is only which register the product goes to.  Z's
// relaxation over TR is folded into the next pulse's Y column, its recovery
// enters through that column on state 0.  24 FP32 operations per state and
// step instead of 64.  The constants are the reference's (its sines of alpha
// and of the precession over TE and over TR - TE), so the atoms differ from
// the reference order's by rounding only.
// 111,008 atoms, T = 500, w = 50 (4 lanes x 13 states): 8.49 -> 2.99 ms, 1.87
// ms of it the 24 operations at the measured FP32 peak; the atoms within
// 2.1e-6 of their peak of the reference order's (4.9e-6 with quadratic RF
// phases), as far from 64 bits as those (3.1e-6; 2.7 against 3.3e-6).
#pragma once

#include "epg_kernels.cuh"

namespace snapmrf {

constexpr int kSsfpMaxStates = 16;  // states per lane
constexpr int kSsfpChunk = 16;      // steps staged per chunk

struct SsfpStep {
    float2 rf;   // cos, sin of the flip angle
    float2 z;    // frame of this step
    float2 zz;   // z_t conj(z_{t+1})
};

struct SsfpAtom {
    double rate;   // 2 pi B0 / 1000 (rad / ms)
    float T1, T2;
};

inline size_t epg_ssfp_smem_bytes(int L) {
    const int apc = 32 / L;
    return kSsfpChunk * sizeof(SsfpStep) +
           (size_t)apc * ((kSsfpChunk + 1) * (sizeof(float4) + 2 * sizeof(float2)) + sizeof(SsfpAtom));
}

// a + b i times c + d i, and the first's product with the conjugate.
__device__ __forceinline__ float2 c_mul_fma(float2 w, float2 v) {
    return make_float2(fmaf(w.x, v.x, -w.y * v.y), fmaf(w.x, v.y, w.y * v.x));
}
__device__ __forceinline__ float2 c_mul_conj(float2 w, float2 v) {
    return make_float2(fmaf(w.x, v.x, w.y * v.y), fmaf(w.x, v.y, -w.y * v.x));
}

// One warp per CTA, 32 / L atoms, S states per lane.  TAIL: the layout pads at
// most three states, so slot w (which the shift feeds from w - 1 and which has
// to stay zero) is one of the last lane's last three.
template <int S, bool TAIL>
__global__ void __launch_bounds__(32) epg_ssfp_kernel(EpgArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = a.L, apc = 32 / L;
    const int lane = threadIdx.x, g = lane / L, gl = lane % L;
    const bool lane0 = gl == 0, last = gl == L - 1;
    const long long blk = blockIdx.y, nreps = a.nreps;
    const long long atom0 = (long long)blockIdx.x * apc, ab = atom0 + g;
    const bool active = ab < a.natoms;
    const long long gatom = blk * a.natoms + ab;
    SsfpStep *sS = reinterpret_cast<SsfpStep *>(smem_raw);
    SsfpAtom *sP = reinterpret_cast<SsfpAtom *>(sS + kSsfpChunk);         // [apc]
    float4 *sW = reinterpret_cast<float4 *>(sP + apc);                    // [apc][chunk + 1]: w, E1, recovery before
    float2 *sD = reinterpret_cast<float2 *>(sW + apc * (kSsfpChunk + 1)); // readout factors
    float2 *sR = sD + apc * (kSsfpChunk + 1);                             // readouts
    if (lane < apc) {
        const long long at = atom0 + lane;
        SsfpAtom q = {0.0, 1.f, 1.f};
        if (at < a.natoms) {
            const float *p = a.params + (a.own_params ? blk * a.natoms + at : at) * a.nparams;
            q = {2 * M_PI * p[2] / 1000.0, p[0], p[1]};
        }
        sP[lane] = q;
    }
    __syncwarp();
    const float *alpha = a.alpha + blk * nreps, *phi = a.sched + nreps;
    const float *TR = a.sched + 2 * nreps, *TE = a.sched + 3 * nreps;
    const int w = a.nstates;

    // the inversion (st_init) in the frame of the first pulse
    float2 p[S], m[S], y[S];
    {
        LaneState<1> s0;
        st_init<1>(s0, lane0, sP[g].T1, sP[g].T2, a.init_alpha_deg, a.init_phi_deg, a.init_ti);
        float sp, cp;
        sincosf(phi[0], &sp, &cp);
        const float2 z0 = make_float2(cp, sp);
#pragma unroll
        for (int j = 0; j < S; j++) p[j] = m[j] = y[j] = make_float2(0.f, 0.f);
        p[0] = c_mul_conj(z0, s0.fp[0]);
        m[0] = c_mul_fma(z0, s0.fm[0]);
        y[0] = make_float2(s0.zz[0].y, -s0.zz[0].x);
    }
    // TAIL: 0 at slot w, for the last three slots of the lane
    float kt[3] = {1.f, 1.f, 1.f};
    if (TAIL) {
#pragma unroll
        for (int q = 0; q < 3; q++)
            if (gl * S + S - 1 - q == w) kt[q] = 0.f;
    }
    const float2 minus = make_float2(-1.f, -1.f);
    float nrm = 0.f;
    float2 *out = a.atoms + gatom * nreps;
    for (long long t0 = 0; t0 < nreps; t0 += kSsfpChunk) {
        const int nch = (int)min((long long)kSsfpChunk, nreps - t0);
        __syncwarp();
        if (lane < nch) {
            const long long t = t0 + lane;
            SsfpStep k;
            __sincosf(alpha[t], &k.rf.y, &k.rf.x);
            sincosf(phi[t], &k.z.y, &k.z.x);
            float2 zn = make_float2(1.f, 0.f);
            if (t + 1 < nreps) sincosf(phi[t + 1], &zn.y, &zn.x);
            k.zz = c_mul_conj(zn, k.z);
            sS[lane] = k;
        }
        __syncwarp();
        for (int idx = lane; idx < apc * nch; idx += 32) {
            const int ga = idx / nch, i = idx - ga * nch;
            const long long t = t0 + i;
            const SsfpAtom q = sP[ga];
            const float te = TE[t], tb = TR[t] - te;
            float2 ea, eb;
            __sincosf((float)(q.rate * te), &ea.y, &ea.x);
            __sincosf((float)(q.rate * tb), &eb.y, &eb.x);
            // (products of the two intervals' factors, as the reference's two
            // relaxations apply them: one exponential over TR from 1 / T
            // moved single atoms by 1.0e-5 of their peak against it, these
            // by 2.1e-6, for 0.14 ms of 3.0)
            const float E2a = expf(-te / q.T2), E2 = E2a * expf(-tb / q.T2);
            float E1 = 1.f, rec = 0.f;
            if (t > 0) {
                const float tep = TE[t - 1], tbp = TR[t - 1] - tep;
                const float e1a = expf(-tep / q.T1), e1b = expf(-tbp / q.T1);
                E1 = e1a * e1b;
                rec = fmaf(1 - e1a, e1b, 1 - e1b);
            }
            const float2 wv = c_scale(c_mul_fma(c_mul_fma(ea, eb), sS[i].zz), E2);
            sW[ga * (kSsfpChunk + 1) + i] = make_float4(wv.x, wv.y, E1, rec);
            sD[ga * (kSsfpChunk + 1) + i] = c_scale(c_mul_fma(ea, sS[i].z), E2a);
        }
        __syncwarp();
        for (int i = 0; i < nch; i++) {
            const float4 k = sW[g * (kSsfpChunk + 1) + i];
            const float2 cs = sS[i].rf;
            const float C = cs.x, Sn = cs.y;
            const float fc = (1 + C) / 2, fs = (1 - C) / 2, fS = Sn * k.z, fh = -0.5f * Sn, fC = C * k.z;
            const float2 c2 = make_float2(fc, fc), s2 = make_float2(fs, fs), S2 = make_float2(fS, fS),
                         h2 = make_float2(fh, fh), C2 = make_float2(fC, fC);
#pragma unroll
            for (int j = 0; j < S; j++) {
                const float2 u = p[j], v = m[j], q = y[j];
                const float2 np = __ffma2_rn(S2, q, __ffma2_rn(s2, v, __fmul2_rn(c2, u)));
                const float2 d = __ffma2_rn(v, minus, u);
                y[j] = __ffma2_rn(C2, q, __fmul2_rn(h2, d));
                m[j] = __ffma2_rn(np, minus, __fadd2_rn(u, v));
                p[j] = np;
            }
            if (lane0) {
                // the recovery -i (1 - E1) of Y0 through the pulse's Y column
                p[0].y = fmaf(-Sn, k.w, p[0].y);
                m[0].y = fmaf(Sn, k.w, m[0].y);
                y[0].y = fmaf(-C, k.w, y[0].y);
                const float2 v = c_mul_fma(sD[g * (kSsfpChunk + 1) + i], p[0]);
                sR[g * (kSsfpChunk + 1) + i] = v;
                nrm = fmaf(v.x, v.x, fmaf(v.y, v.y, nrm));
            }
            // the interval's factor and the shift
            const float2 wv = make_float2(k.x, k.y);
            float2 up, dn;
            up.x = __shfl_up_sync(0xffffffffu, p[S - 1].x, 1, L);
            up.y = __shfl_up_sync(0xffffffffu, p[S - 1].y, 1, L);
            dn.x = __shfl_down_sync(0xffffffffu, m[0].x, 1, L);
            dn.y = __shfl_down_sync(0xffffffffu, m[0].y, 1, L);
            const float2 m0 = m[0];
            if (last) dn = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = S - 1; j >= 1; j--) p[j] = c_mul_fma(wv, p[j - 1]);
            p[0] = c_mul_fma(wv, up);
#pragma unroll
            for (int j = 0; j < S - 1; j++) m[j] = c_mul_conj(wv, m[j + 1]);
            m[S - 1] = c_mul_conj(wv, dn);
            // (one state: nothing shifts, F+[0] takes the unshifted F-[0])
            if (lane0) p[0] = w == 1 ? c_conj(c_mul_conj(wv, m0)) : c_conj(m[0]);
            if (TAIL) {
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (q < S) {
                        p[S - 1 - q].x *= kt[q];
                        p[S - 1 - q].y *= kt[q];
                    }
            } else {
#pragma unroll
                for (int j = 0; j < S; j++)
                    if (gl * S + j == w) p[j] = make_float2(0.f, 0.f);
            }
        }
        __syncwarp();
        if (active)
            for (int q = gl; q < nch; q += L) out[t0 + q] = sR[g * (kSsfpChunk + 1) + q];
    }
    if (a.normalize || a.norms) {
        nrm = __shfl_sync(0xffffffffu, nrm, 0, L);
        if (a.norms && lane0 && active) a.norms[gatom] = sqrtf(nrm);
        if (a.normalize) {
            __syncwarp();
            const float inv = nrm > 0.f ? 1.f / sqrtf(nrm) : nrm;
            // the whole warp on each of its atoms
            for (int q = 0; q < apc && atom0 + q < a.natoms; q++) {
                const float iv = __shfl_sync(0xffffffffu, inv, q * L);
                float2 *row = a.atoms + (blk * a.natoms + atom0 + q) * nreps;
                for (long long t = lane; t < nreps; t += 32) row[t] = c_scale(row[t], iv);
            }
        }
    }
}

}  // namespace snapmrf
