// pssfp_real.cuh — pSSFP isochromat simulation of sequences with real RF samples.
//
// With a real RF train and waveform every rotation axis lies in the x-z plane, a = (ax, 0, az), and the
// rotation by |a| = θ needs one common factor: with b = az·mx - ax·mz, S = sin θ/θ, H = (1 - cos θ)/θ²,
//     u = S·my + H·b,   mx' = mx - az·u,   mz' = mz + ax·u,   my' = cos θ·my + S·b = K·u - my,
// K = S/H = θ·cot(θ/2), and u = H·(K·my + b). (src/operators/isochromat.cuh:14-73 for a_y = 0.) The sign of
// my' is absorbed by keeping s = ±my, the sign alternating from sample to sample together with that of
// the axis: s' = s + K·u. The relaxation between the samples of a pulse (src/simulate/pssfp_kernels.cuh:
// 46-55) is divided out: the kernel keeps mx/E2^i, s/E2^i and (mz - 1)/E1^i at sample i, whose
// relaxations are ratios of the coefficients of the coupling, -ax·E2^-i, -ax·(E1/E2)^i and
// -ax·(E2/E1)^i, common to the isochromats of a voxel; the pulse's whole decay multiplies the precession
// that follows it. That is 12 or 14 operations per isochromat and RF sample (K and H to second or third
// order in θ²), 24 before. Pairs of isochromats run as two-wide FP32 instructions.
//
// Which order, and whether the division is safe, is decided once per voxel: the order from the largest
// axis of the sequence (the table's second flag) and its isochromats, the division from its
// relaxation. Samples whose angles may pass half a radian take longer series (and sincos above 3π/2), and a
// voxel that a pulse outlasts by far relaxes explicitly after every sample. The warp's vote only picks the
// cheapest of three loops that does what all its voxels need; in each of them a voxel gets the same bits
// (what it does not need enters as a factor of 1 or a highest coefficient of 0), so its echoes
// do not depend on its neighbours. Loop 2, in us for 20000 voxels, 60 TRs of 15 samples, 9 / 35 z (with the
// 24-operation rotation in brackets): 30 % of the voxels with T2 = 0 293 / 588 (350 / 729; no such voxel, loop
// 0: 166 / 388), az of 1 rad at the outer z 488 / 1077 (1349 / 2810); pulses of one sample of 40° 53 / 115 (139 / 219).
//
// Bound by the FP32 pipe. 35 z, 15 RF samples: 50176 voxels, 320 TRs 4.85 ms (7.93 ms with the 24-operation
// rotation), tangents at 100 TRs 3.25 ms (6.3); 2500 voxels, 743 TRs 1.34 ms (3.37). The loop over the samples
// holds an even and an odd body and a third for the last sample of an odd count: with a branch in
// the loop instead, 10 % slower.
#pragma once

#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "job_args.cuh"

namespace compas {
namespace kernels {

// one operation on an isochromat (float) or on a pair (float2), the same rounding either way
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return mul2(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
template<class T>
__device__ __forceinline__ T vset(float s) {
    if constexpr (sizeof(T) == 4) return s;
    else return bcast2(s);
}

// RF sample i of a pulse on one voxel
struct RealSample {
    float nb0, nb1, nb2;  // -B·E2^-i, -B·(E1/E2)^i, -B·(E2/E1)^i, B = ±ax
    float nax2;           // -ax²
    bool small;           // θ² ≤ 1/4 for every isochromat of the voxel
};

// What a voxel needs of the loop it runs in (file header)
struct RealNeeds {
    float k6, h6;   // highest coefficients of K and -H: those of the third order, or 0
    float E1, E2;   // the relaxation after a sample where it is not divided out, else 1
};

// -sin θ/θ, -(1 - cos θ)/θ², -cos θ for y = -θ² of a large angle, or NaN
struct RealRotation {
    float ns, nh, nc;
};
static __device__ __noinline__ RealRotation real_sincos(float y) {  // rarely run: one copy of the sincos
    RealRotation q;
    const float th = sqrtf(-y);
    float sn, cs;
    sincosf(th, &sn, &cs);
    q.ns = -sn / th;
    q.nh = (1.0f - cs) / y;
    q.nc = -cs;
    return q;
}
__device__ __forceinline__ void real_rotation(float y, float& ns, float& nh, float& nc) {
    const RealRotation q = real_sincos(y);
    ns = q.ns, nh = q.nh, nc = q.nc;
}

// -sin θ/θ, -(1 - cos θ)/θ², -cos θ for y = -θ² ≥ kRealSeriesMin (θ ≤ 3π/2) on an isochromat or a pair, from
// q = sin(θ/2)/(θ/2) and the cosine of the half angle: Taylor series in y/4 (the next terms are below 3e-9
// and 1e-9), sin θ/θ = q·cos(θ/2), (1 - cos θ)/θ² = q²/2
constexpr float kRealSeriesMin = -22.2f;
template<class T>
__device__ __forceinline__ void real_series(T y, T& ns, T& nh, T& nc) {
    const T h = vmul(vset<T>(0.25f), y);
    T q = vfma(h, vset<T>(1.0f / 1307674368000.0f), vset<T>(1.0f / 6227020800.0f));
    q = vfma(h, q, vset<T>(1.0f / 39916800.0f));
    q = vfma(h, q, vset<T>(1.0f / 362880.0f));
    q = vfma(h, q, vset<T>(1.0f / 5040.0f));
    q = vfma(h, q, vset<T>(1.0f / 120.0f));
    q = vfma(h, q, vset<T>(1.0f / 6.0f));
    q = vfma(h, q, vset<T>(1.0f));
    T c = vfma(h, vset<T>(1.0f / 20922789888000.0f), vset<T>(1.0f / 87178291200.0f));
    c = vfma(h, c, vset<T>(1.0f / 479001600.0f));
    c = vfma(h, c, vset<T>(1.0f / 3628800.0f));
    c = vfma(h, c, vset<T>(1.0f / 40320.0f));
    c = vfma(h, c, vset<T>(1.0f / 720.0f));
    c = vfma(h, c, vset<T>(1.0f / 24.0f));
    c = vfma(h, c, vset<T>(0.5f));
    c = vfma(h, c, vset<T>(1.0f));
    const T nhq = vmul(vset<T>(-0.5f), q);
    ns = vmul(vmul(vset<T>(-1.0f), q), c);
    nh = vmul(nhq, q);
    nc = vfma(y, nh, vset<T>(-1.0f));
}

// One RF sample on one isochromat or pair: x, s, z the value, (x1, s1, z1) and (x2, s2, z2) its tangents
// ∂/∂T1, ∂/∂T2 (TAN), A = ±az, nA = -A. t1 = dt/T1², t2 = dt/T2².
// LOOP 0: θ² ≤ 0.02, 1: θ² ≤ 0.25 (the dropped terms of K and H are below 1e-8 and 1e-9), 2: any angle and
// relaxation.
template<int LOOP, bool TAN, class T>
__device__ __forceinline__ void real_step(T (&v)[TAN ? 9 : 3], T A, T nA, const RealSample& f, const RealNeeds& need,
                                          float t1, float t2) {
    const T y = vfma(nA, A, vset<T>(f.nax2));  // -θ²
    const T nb0 = vset<T>(f.nb0), nb1 = vset<T>(f.nb1), nb2 = vset<T>(f.nb2);
    if (LOOP < 2 || f.small) {
        T K, nH;
        if constexpr (LOOP == 0) {
            K = vfma(y, vfma(y, vset<T>(-1.0f / 360.0f), vset<T>(1.0f / 6.0f)), vset<T>(2.0f));
            nH = vfma(y, vfma(y, vset<T>(-1.0f / 720.0f), vset<T>(-1.0f / 24.0f)), vset<T>(-0.5f));
        } else {
            K = vfma(y, vfma(y, vfma(y, vset<T>(need.k6), vset<T>(-1.0f / 360.0f)), vset<T>(1.0f / 6.0f)), vset<T>(2.0f));
            nH = vfma(y, vfma(y, vfma(y, vset<T>(need.h6), vset<T>(-1.0f / 720.0f)), vset<T>(-1.0f / 24.0f)), vset<T>(-0.5f));
        }
#pragma unroll
        for (int q = 0; q < (TAN ? 3 : 1); q++) {
            T &x = v[3 * q], &s = v[3 * q + 1], &z = v[3 * q + 2];
            // (the tangents' regrowth is that of the value)
            const T b = vfma(A, x, q == 0 ? vfma(nb1, z, nb0) : vmul(nb1, z));
            const T u = vmul(nH, vfma(K, s, b));
            x = vfma(A, u, x);
            s = vfma(K, u, s);
            z = vfma(nb2, u, z);
        }
    } else {
        T nS, nH, c;
        real_series(y, nS, nH, c);
        if constexpr (sizeof(T) == 4) {
            if (!(y >= kRealSeriesMin)) real_rotation(y, nS, nH, c);
        } else if (!(y.x >= kRealSeriesMin && y.y >= kRealSeriesMin)) {
            if (!(y.x >= kRealSeriesMin)) real_rotation(y.x, nS.x, nH.x, c.x);
            if (!(y.y >= kRealSeriesMin)) real_rotation(y.y, nS.y, nH.y, c.y);
        }
#pragma unroll
        for (int q = 0; q < (TAN ? 3 : 1); q++) {
            T &x = v[3 * q], &s = v[3 * q + 1], &z = v[3 * q + 2];
            const T b = vfma(A, x, q == 0 ? vfma(nb1, z, nb0) : vmul(nb1, z));
            const T u = vfma(nS, s, vmul(nH, b));
            x = vfma(A, u, x);
            s = vfma(c, s, vmul(nS, b));
            z = vfma(nb2, u, z);
        }
    }
    if constexpr (LOOP == 2) {
        const T e1 = vset<T>(need.E1), e2 = vset<T>(need.E2);
#pragma unroll
        for (int q = 0; q < (TAN ? 3 : 1); q++) {
            v[3 * q] = vmul(e2, v[3 * q]);
            v[3 * q + 1] = vmul(e2, v[3 * q + 1]);
            v[3 * q + 2] = vmul(e1, v[3 * q + 2]);
        }
    }
    if constexpr (TAN) {  // the relaxation's own derivative, at the new state
        v[5] = vfma(vset<T>(t1), v[2], v[5]);
        v[6] = vfma(vset<T>(t2), v[0], v[6]);
        v[7] = vfma(vset<T>(t2), v[1], v[7]);
    }
}

// Precession by (c, sn) with relaxation (E1, E2) on one isochromat or pair (v as real_step, the sign of s
// settled: s = my, z = mz - 1); t1 = dt_pr/T1², t2 = dt_pr/T2²
template<bool TAN, class T>
__device__ __forceinline__ void real_precess(T (&v)[TAN ? 9 : 3], T c, T sn, T nsn, float E1, float E2, float t1, float t2) {
    const T e1 = vset<T>(E1), e2 = vset<T>(E2);
#pragma unroll
    for (int q = 0; q < (TAN ? 3 : 1); q++) {
        const T x = v[3 * q], y = v[3 * q + 1];
        v[3 * q] = vmul(e2, vfma(c, x, vmul(nsn, y)));
        v[3 * q + 1] = vmul(e2, vfma(c, y, vmul(sn, x)));
        v[3 * q + 2] = vmul(e1, v[3 * q + 2]);
    }
    if constexpr (TAN) {
        v[5] = vfma(vset<T>(t1), v[2], v[5]);
        v[6] = vfma(vset<T>(t2), v[0], v[6]);
        v[7] = vfma(vset<T>(t2), v[1], v[7]);
    }
}

// One tile (128/GZ voxels) of a simulation: GZ lanes per voxel, ZT isochromats per lane, slots p and
// p + ZT/2 in a pair, an odd last slot by itself. The isochromats evolve in the same bits in every layout (what a
// voxel needs follows from all of them); the echo sums a lane's slots in order and the lanes as a tree.
// QUEUE: the layout is the batch's, the sum that of `own`, the job's layout in a call of its own, where the two differ:
// through shared memory (`sums`, ZT entries per thread), own.zt isochromats in order and own.lanes of these as the
// same tree.
template<int ZT, int GZ, bool TAN, bool QUEUE = false>
__device__ __forceinline__ void pssfp_real_tile(const PssfpArgs& a, const int tile, const PssfpOrder own = {},
                                                float2* sums = nullptr) {
    constexpr int ZP = ZT / 2, ODD = ZT % 2, ZA = ZP > 0 ? ZP : 1, NV = TAN ? 9 : 3;
    const int lane = threadIdx.x & 31;
    const int sub = lane % GZ;
    const int first = sub * ZT, count = a.nz - first;  // the lane's first isochromat; its slots below count hold one
    const int vloc = (tile * blockDim.x + threadIdx.x) / GZ;
    const bool vok = vloc < a.nvoxels;
    const int64_t vcol = a.voxel_begin + (vok ? vloc : a.nvoxels - 1);
    const float T1 = a.params[0 * a.param_stride + vcol];
    const float T2 = a.params[1 * a.param_stride + vcol];
    const float B1 = a.params[2 * a.param_stride + vcol];
    const float B0 = a.params[3 * a.param_stride + vcol];
    const float R1 = 1.0f / T1, R2 = 1.0f / T2;
    const float E1_ex = expf(-a.dt_ex * R1), E2_ex = expf(-a.dt_ex * R2);
    const float E1_pr = expf(-a.dt_pr * R1), E2_pr = expf(-a.dt_pr * R2);
    const float E1_inv = expf(-a.dt_inv * R1);
    const float t1_ex = a.dt_ex * R1 * R1, t2_ex = a.dt_ex * R2 * R2;
    const float t1_pr = a.dt_pr * R1 * R1, t2_pr = a.dt_pr * R2 * R2;
    constexpr float kTwoPi = 6.28318530717958647692f;

    float2 P[ZA][NV], az[ZA], naz[ZA], cpr[ZA], spr[ZA], nspr[ZA];
    float O[NV], oaz = 0.f, ocpr = 1.f, ospr = 0.f;
    float azmax2 = 0.f;
    // inversion: mz = cos(πB1), then relaxation (isochromat.cuh:100-112); z - 1 and its T1 derivative
    const float z0 = __fmul_rn(E1_inv, __fadd_rn(cospif(B1), -1.0f));
    const float z0_1 = a.dt_inv * R1 * R1 * z0;
    auto position = [&](int k) { return k < count ? a.z[first + k] : 0.0f; };
    auto axis = [&](int k, float z) {
        const float v = __fmaf_rn(-a.gz_ex, z, -(a.dt_ex * kTwoPi * B0));
        if (k < count) azmax2 = fmaxf(azmax2, v * v);
        return v;
    };
    auto angle = [&](float g, float z) { return __fmaf_rn(-(g * a.gz_pr), z, -(a.dt_pr * kTwoPi * B0)); };
#pragma unroll
    for (int p = 0; p < ZP; p++) {
        const float zl = position(p), zh = position(p + ZP);
        az[p] = make_float2(axis(p, zl), axis(p + ZP, zh));
        naz[p] = make_float2(-az[p].x, -az[p].y);
        sincosf(angle(1.0f, zl), &spr[p].x, &cpr[p].x);
        sincosf(angle(1.0f, zh), &spr[p].y, &cpr[p].y);
        nspr[p] = make_float2(-spr[p].x, -spr[p].y);
#pragma unroll
        for (int q = 0; q < NV; q++) P[p][q] = bcast2(q == 2 ? z0 : q == 5 ? z0_1 : 0.f);
    }
    if constexpr (ODD) {
        const float z = position(2 * ZP);
        oaz = axis(2 * ZP, z);
        sincosf(angle(1.0f, z), &ospr, &ocpr);
#pragma unroll
        for (int q = 0; q < NV; q++) O[q] = q == 2 ? z0 : q == 5 ? z0_1 : 0.f;
    }

    // what the voxel needs: its largest angle of any sample, and whether its E1 and E2 to the power of
    // the pulse's samples stay far from the ends of the range (a NaN fails every comparison)
#pragma unroll
    for (int d = GZ / 2; d > 0; d /= 2) azmax2 = fmaxf(azmax2, __shfl_xor_sync(0xffffffffu, azmax2, d, GZ));
    const float zap_max = __ldg(&a.zap[int64_t(a.nTR + 1) * a.nRF].y);
    const float th2 = __fmaf_rn(zap_max * B1, zap_max * B1, azmax2);
    const float pulse = float(a.nRF) * a.dt_ex * fmaxf(fabsf(R1), fabsf(R2));
    const bool scaled = pulse <= 40.0f, second = th2 <= 0.02f, third = th2 <= 0.25f;
    RealNeeds need;
    need.k6 = second ? 0.0f : 1.0f / 15120.0f;
    need.h6 = second ? 0.0f : -1.0f / 40320.0f;
    need.E1 = scaled ? 1.0f : E1_ex;
    need.E2 = scaled ? 1.0f : E2_ex;
    const int loop = !__all_sync(0xffffffffu, scaled && third) ? 2 : __all_sync(0xffffffffu, second) ? 0 : 1;
    // the pulse's decay, and the steps of the running ratios less 1 (a relaxation per sample is so close to
    // 1 that its rounding, repeated every sample, would be the largest error: as products of the factors
    // the echoes were 2e-5 off, like this 3e-6)
    const float E1_all = scaled ? expf(-float(a.nRF) * a.dt_ex * R1) : 1.0f;
    const float E2_all = scaled ? expf(-float(a.nRF) * a.dt_ex * R2) : 1.0f;
    const float g0 = scaled ? expm1f(a.dt_ex * R2) : 0.0f;
    const float g1 = scaled ? expm1f(a.dt_ex * __fadd_rn(R2, -R1)) : 0.0f;
    const float g2 = scaled ? expm1f(a.dt_ex * __fadd_rn(R1, -R2)) : 0.0f;

    // (every lambda that touches the states is inlined by force: a call would move them to local memory)
    auto excite = [&](int row, auto loop_tag) __attribute__((always_inline)) {
        constexpr int LOOP = decltype(loop_tag)::value;
        const float2* zr = a.zap + int64_t(row) * a.nRF;
        float f0 = 1.f, f1 = 1.f, f2 = 1.f;
        auto sample = [&](int i, bool negative) __attribute__((always_inline)) {
            const float ax = __fmul_rn(__ldg(&zr[i].x), B1);
            const float nb = negative ? ax : -ax;
            RealSample f;
            f.nb0 = __fmul_rn(nb, f0);
            f.nb1 = __fmul_rn(nb, f1);
            f.nb2 = __fmul_rn(nb, f2);
            f.nax2 = -__fmul_rn(ax, ax);
            f.small = LOOP < 2 || __fmaf_rn(ax, ax, azmax2) <= 0.25f;
            f0 = __fmaf_rn(f0, g0, f0);
            f1 = __fmaf_rn(f1, g1, f1);
            f2 = __fmaf_rn(f2, g2, f2);
#pragma unroll
            for (int p = 0; p < ZP; p++) {
                if (negative) real_step<LOOP, TAN>(P[p], naz[p], az[p], f, need, t1_ex, t2_ex);
                else real_step<LOOP, TAN>(P[p], az[p], naz[p], f, need, t1_ex, t2_ex);
            }
            if constexpr (ODD) real_step<LOOP, TAN>(O, negative ? -oaz : oaz, negative ? oaz : -oaz, f, need, t1_ex, t2_ex);
        };
        int i = 0;
        for (; i + 1 < a.nRF; i += 2) {
            sample(i, false);
            sample(i + 1, true);
        }
        if (i < a.nRF) {  // an odd count ends on s = -my
            sample(i, false);
#pragma unroll
            for (int q = 1; q < NV; q += 3) {
#pragma unroll
                for (int p = 0; p < ZP; p++) P[p][q] = make_float2(-P[p][q].x, -P[p][q].y);
                if constexpr (ODD) O[q] = -O[q];
            }
        }
    };
    auto precess = [&](float E1, float E2) __attribute__((always_inline)) {
#pragma unroll
        for (int p = 0; p < ZP; p++) real_precess<TAN>(P[p], cpr[p], spr[p], nspr[p], E1, E2, t1_pr, t2_pr);
        if constexpr (ODD) real_precess<TAN>(O, ocpr, ospr, -ospr, E1, E2, t1_pr, t2_pr);
    };
    const float E1_first = E1_all * E1_pr, E2_first = E2_all * E2_pr;

    // the whole sequence, once for each loop: in a common one, what the others need takes registers from
    // loop 0 throughout (5 % of its time)
    auto simulate = [&](auto loop_tag) __attribute__((always_inline)) {
        auto pulse_of = [&](int row) __attribute__((always_inline)) { excite(row, loop_tag); };
        // α/2 pulse, then re- and prephaser with twice the prephasing gradient (pssfp_kernels.cuh:73-80)
        pulse_of(0);
#pragma unroll
        for (int p = 0; p < ZP; p++) {
            float2 c, s;
            sincosf(angle(2.0f, position(p)), &s.x, &c.x);
            sincosf(angle(2.0f, position(p + ZP)), &s.y, &c.y);
            real_precess<TAN>(P[p], c, s, make_float2(-s.x, -s.y), E1_first, E2_first, t1_pr, t2_pr);
        }
        if constexpr (ODD) {
            float c, s;
            sincosf(angle(2.0f, position(2 * ZP)), &s, &c);
            real_precess<TAN>(O, c, s, -s, E1_first, E2_first, t1_pr, t2_pr);
        }

        for (int t = 0; t < a.nTR; t++) {  // pssfp_kernels.cuh:83-107
            pulse_of(t + 1);
            precess(E1_first, E2_first);
            const int64_t at = int64_t(t) * a.echo_stride + a.voxel_begin + vloc;
#pragma unroll
            for (int q = 0; q < NV; q += 3) {
                float2* out = q == 0 ? a.echo : q == 3 ? a.dT1 : a.dT2;
                if (QUEUE && (own.zt != ZT || own.lanes != GZ)) {
                    float2* m = sums + (threadIdx.x / GZ) * (ZT * GZ);  // the voxel's isochromats
#pragma unroll
                    for (int p = 0; p < ZP; p++) {
                        if (p < count) m[first + p] = make_float2(P[p][q].x, P[p][q + 1].x);
                        if (p + ZP < count) m[first + p + ZP] = make_float2(P[p][q].y, P[p][q + 1].y);
                    }
                    if (ODD && 2 * ZP < count) m[first + 2 * ZP] = make_float2(O[q], O[q + 1]);
                    __syncwarp();
                    const int used = (a.nz + own.zt - 1) / own.zt;  // the other lanes' sums are zero
                    for (int v = sub; v < used; v += GZ) {
                        float2 s = make_float2(0.f, 0.f);
                        for (int z = v * own.zt; z < min((v + 1) * own.zt, a.nz); z++) s.x += m[z].x, s.y += m[z].y;
                        m[v * own.zt] = s;
                    }
                    for (int d = own.lanes / 2; d > 0; d /= 2) {
                        __syncwarp();
                        for (int v = sub; v < d && v + d < used; v += GZ) {
                            float2 &s = m[v * own.zt], t = m[(v + d) * own.zt];
                            s.x += t.x, s.y += t.y;
                        }
                    }
                    if (sub == 0 && vok) out[at] = m[0];
                    __syncwarp();
                    continue;
                }
                float sx = 0.0f, sy = 0.0f;  // over the slots in order
#pragma unroll
                for (int p = 0; p < ZP; p++)
                    if (p < count) {
                        sx += P[p][q].x;
                        sy += P[p][q + 1].x;
                    }
#pragma unroll
                for (int p = 0; p < ZP; p++)
                    if (p + ZP < count) {
                        sx += P[p][q].y;
                        sy += P[p][q + 1].y;
                    }
                if (ODD && 2 * ZP < count) {
                    sx += O[q];
                    sy += O[q + 1];
                }
#pragma unroll
                for (int d = GZ / 2; d > 0; d /= 2) {
                    sx += __shfl_xor_sync(0xffffffffu, sx, d, GZ);
                    sy += __shfl_xor_sync(0xffffffffu, sy, d, GZ);
                }
                if (sub == 0 && vok) out[at] = make_float2(sx, sy);
            }
            precess(E1_pr, E2_pr);
        }
    };
    if (loop == 0) simulate(std::integral_constant<int, 0> {});
    else if (loop == 1) simulate(std::integral_constant<int, 1> {});
    else simulate(std::integral_constant<int, 2> {});
}

// True when every RF sample of the sequence is real (Im zap = 0: a real RF train, as with 0-π phase
// cycling, and a real waveform).
__device__ __forceinline__ bool pssfp_real_rf(const PssfpArgs& a) {
    return __ldg(&a.zap[int64_t(a.nTR + 1) * a.nRF].x) == 0.0f;
}

// One simulation (TAN: with its T1 and T2 tangents into a.dT1, a.dT2). Returns at once when the RF is not
// real: the general kernel launched beside it runs then.
template<int ZT, int GZ, bool TAN>
__global__ void __launch_bounds__(128) pssfp_real_kernel(PssfpArgs a, HostAnswer ask) {
    if (!TAN && a.skip != nullptr && *a.skip != 0) return;  // uniform over the grid
    answer_host(ask, pssfp_real_rf(a));
    if (!pssfp_real_rf(a)) return;
    pssfp_real_tile<ZT, GZ, TAN>(a, blockIdx.x);
}

// Work-queue form for batches (see pssfp_queue_kernel): every job's RF is real; own: each job's own order of the sum.
template<int ZT, int GZ, bool TAN>
__global__ void __launch_bounds__(128) pssfp_real_queue_kernel(const PssfpArgs* __restrict__ jobs,
                                                               const int2* __restrict__ items, int nitems,
                                                               int* __restrict__ head, const PssfpOrder* __restrict__ own) {
    __shared__ float2 sums[128 * ZT];
    __shared__ PssfpArgs job;
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(head, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= nitems) break;
        const int2 w = items[it];
        if (threadIdx.x == 0) job = jobs[w.x];
        __syncthreads();
        pssfp_real_tile<ZT, GZ, TAN, true>(job, w.y, own[w.x], sums);
        __syncthreads();
    }
}

}  // namespace kernels

struct PssfpRealKernels {
    int ZT, GZ;
    void (*fn)(kernels::PssfpArgs, kernels::HostAnswer);
    void (*queue)(const kernels::PssfpArgs*, const int2*, int, int*, const kernels::PssfpOrder*);
};
// the real-RF value and tangent kernels of a layout (every layout of pssfp.cu has them)
const PssfpRealKernels& pssfp_real_kernels(int ZT, int GZ);
const PssfpRealKernels& pssfp_real_tangent_kernels(int ZT, int GZ);

}  // namespace compas
