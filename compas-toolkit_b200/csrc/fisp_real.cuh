// fisp_real.cuh — FISP extended-phase-graph simulation of sequences with real RF phases.
//
// Off-resonance leaves the magnitude of the echoes alone: within a TR the precession multiplies F+
// by e^{iθ} (F- by e^{-iθ}), θ = 2π·B0·TR, and the spoiler shifts F+ one state up and F- one state
// down, so the states of order k carry exactly the factor e^{iθk} at the start of every TR, whatever
// was played before, and excitation mixes only states of one order. In F±_k·e^{-iθk}, Z_k·e^{-iθk}
// the precession is gone; order 0, the echo, has no factor but the e^{2πi·B0·TE} of its echo time.
// With real RF phases (e^{iφ} = ±1) what is left is real: F+ = i·p, conj(F-) = i·n, Z = z, and with
// s = sin(α/2), c = cos(α/2) (α signed by the phase), E1, E2 the relaxation of the TR before:
//     d = p + n,   t = E2·s²·d + E1·sin α·z,
//     p' = E2·p - t,   n' = E2·n - t,   z' = E1·cos α·z + E2·s·c·d:
// 7 FP32 operations per state and TR instead of the 24 of the complex update (fisp.cu), on 3 reals per
// state instead of 6, so that 25 states leave room for twice the warps per SM. (src/operators/epg.cuh:
// 37-111,182-298 composed for e^{iφ} = ±1; the truncation at N states and the spoiling only zero whole
// states.) State 0 has p = n = q and takes the regrowth 1 - E1; it is kept by itself, the states 1..N-1
// as KP pairs for the two-wide FP32 instructions. At 25 states: 12 pairs, no padding.
//
// The form holds from one repetition to the next as long as no precession happens without a spoiler
// while F is not zero: that is the wait TW of a sequence with neither inversion prepulse nor wait
// spoiling, which stays on the general kernels (fisp_real_covers).
//
// Bound by the FP32 pipe (182 lane operations per voxel, position and TR at 25 states: 12 pairs of 14, state 0
// and the coefficients). MR-STAT slice (50176 voxels, 1120 TRs, 25 states, 35 positions): 12.6 ms,
// 41.7 ms as complex states; its tangents at 9216 voxels: 9.9 ms, 42.7 ms before; 4096 voxels, 400 TRs,
// 8 states, 1 position: 35 us, 113 us before. The two-wide instructions of the states run at 86 % of the
// pipe's rate (8 against 25 states; ncu: pipe 76 % busy overall); the scalar forms of the same operations,
// all or every second pair, ran 5-10 % slower.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "fisp_common.cuh"
#include "job_args.cuh"

namespace compas {
namespace kernels {

// Excitation coefficients of one TR with the relaxation before it (file header). Every operation has
// an explicit rounding, so all instantiations give the same bits.
struct RealCoefs {
    float2 nal, nbe, f, D, E2;  // -E2·s², -E1·sin α, E1·cos α, E2·s·c, E2, in both angles (the two-wide
                                // FMA has no operand negation: the negated coefficients make -t)
    float sa, ca, E1, regrow;   // sin α, cos α; state 0: E1, 1 - E1
};

// The sine and cosine are those of α itself, with s² = (1 - cos α)/2 and s·c = sin α/2: four operations
// fewer per TR than from α/2. Both functions are good to about 5e-7 absolute for |α| ≤ π, the range for
// which CUDA bounds them; beyond it the reduction of the argument adds its rounding, 6e-8·|α|. Against 64
// bits the echoes are as close as or closer than from α/2 over the whole range (25 states, 1000 TRs, B1 0.8-1.2, in 1e-6):
// constant flips of 1° 7.7 (from α/2 14.5), 5° 3.9 (8.8), 30° 4.9 (12.7), 90° 2.6 (10.9), 180° 5.8 (5.7), 360° 4.6
// (11.0), 720° 4.9 (11.5), random flips of 0-70° 1.6 (2.3) and 150-360° 2.0 (2.6).
__device__ __forceinline__ RealCoefs real_coefs(float alpha, float B1, float E1, float E2, float regrow) {
    RealCoefs k;
    __sincosf(__fmul_rn(alpha, B1), &k.sa, &k.ca);  // (epg.cuh:41-51)
    const float h = 0.5f * E2;
    k.nal = bcast2(__fmaf_rn(h, k.ca, -h));
    k.nbe = bcast2(-__fmul_rn(E1, k.sa));
    k.f = bcast2(__fmul_rn(E1, k.ca));
    k.D = bcast2(__fmul_rn(h, k.sa));
    k.E2 = bcast2(E2);
    k.E1 = E1;
    k.regrow = regrow;
    return k;
}

// The states of one (voxel, slice position) on G lanes (sub = 0 .. G-1 of the group): state 0 in q, z0
// of lane 0 (the other lanes run along on values that nothing reads), states 1 + sub·2KP + i,
// i = 0 .. 2KP-1, on lane sub: pair j holds i = j (.x) and i = j + KP (.y).
template<int KP, int G>
struct EPGReal {
    float q, z0;
    float2 p[KP], n[KP], z[KP];

    __device__ __forceinline__ void init(float z_start) {
        q = 0.f;
        z0 = z_start;
#pragma unroll
        for (int j = 0; j < KP; j++) p[j] = n[j] = z[j] = make_float2(0.f, 0.f);
    }

    // the spoiler (epg.cuh:229-298): n one state down, zero at the top, p one state up, q = n of state 0.
    // cut: a bit for the slot of state N when the layout holds it, on the lane that does: its p is kept
    // zero, so that it and the states above stay zero in all three components and state N-1 takes a
    // zero n. (A bit test per slot: an index compare could move the states to local memory.)
    __device__ __forceinline__ void shift(int sub, unsigned cut) {
        float np = q, nn = 0.f;  // what enters the lane's first p and last n
        if constexpr (G > 1) {
            const float up = __shfl_up_sync(0xffffffffu, p[KP - 1].y, 1, G);
            const float down = __shfl_down_sync(0xffffffffu, n[0].x, 1, G);
            if (sub > 0) np = up;
            if (sub < G - 1) nn = down;
        }
        const float cn = n[0].y, cp = p[KP - 1].x;
        q = n[0].x;
#pragma unroll
        for (int j = 0; j < KP - 1; j++) n[j] = n[j + 1];
        n[KP - 1] = make_float2(cn, nn);
#pragma unroll
        for (int j = KP - 1; j > 0; j--) p[j] = p[j - 1];
        p[0] = make_float2(np, cp);
        if constexpr (G == 1) {  // N = 2·KP or 2·KP + 1: state N is the last slot or beyond
            if (cut) p[KP - 1].y = 0.f;
        } else {
#pragma unroll
            for (int j = 0; j < KP; j++) {
                if (cut & (1u << j)) p[j].x = 0.f;
                if (cut & (1u << (j + KP))) p[j].y = 0.f;
            }
        }
    }

    // pair j, in place
    __device__ __forceinline__ static void excite_pair(const RealCoefs& k, float2& p, float2& n, float2& z) {
        const float2 d = add2(p, n);
        const float2 nt = fma2(k.nal, d, mul2(k.nbe, z));
        const float2 Dd = mul2(k.D, d);
        p = fma2(k.E2, p, nt);
        n = fma2(k.E2, n, nt);
        z = fma2(k.f, z, Dd);
    }

    // state 0 from its relaxed values x (F) and y (Z)
    __device__ __forceinline__ void excite_first(const RealCoefs& k, float x, float y) {
        q = __fmaf_rn(k.ca, x, -__fmul_rn(k.sa, y));
        z0 = __fmaf_rn(k.ca, y, __fmul_rn(k.sa, x));
    }

    __device__ __forceinline__ void excite(const RealCoefs& k) {
        excite_first(k, __fmul_rn(k.E2.x, q), __fmaf_rn(k.E1, z0, k.regrow));
#pragma unroll
        for (int j = 0; j < KP; j++) excite_pair(k, p[j], n[j], z[j]);
    }

    // F·E2, Z·E1, Z0 += regrow
    __device__ __forceinline__ void relax(float E1, float E2, float regrow) {
        const float2 e1 = bcast2(E1), e2 = bcast2(E2);
        q = __fmul_rn(E2, q);
        z0 = __fmaf_rn(E1, z0, regrow);
#pragma unroll
        for (int j = 0; j < KP; j++) {
            p[j] = mul2(e2, p[j]);
            n[j] = mul2(e2, n[j]);
            z[j] = mul2(e1, z[j]);
        }
    }

    __device__ __forceinline__ void spoil() {
        q = 0.f;
#pragma unroll
        for (int j = 0; j < KP; j++) p[j] = n[j] = make_float2(0.f, 0.f);
    }
};

// The relaxation of an interval t on one voxel
struct RealInterval {
    float E1, E2;  // e^{-t/T1}, e^{-t/T2}
    float s1, s2;  // t/T1², t/T2² (tangents)
};

// The value alone
template<int KP, int G>
struct RealValue {
    static constexpr int kPlanes = 1;
    EPGReal<KP, G> x;

    __device__ __forceinline__ void init() { x.init(1.f); }
    __device__ __forceinline__ void shift(int sub, unsigned cut) { x.shift(sub, cut); }
    __device__ __forceinline__ void excite(const RealCoefs& k, float, float) { x.excite(k); }
    __device__ __forceinline__ void relax(const RealInterval& r) { x.relax(r.E1, r.E2, 1.0f - r.E1); }
    __device__ __forceinline__ void spoil() { x.spoil(); }
    // inversion, spoiling, longitudinal relaxation over TI
    __device__ __forceinline__ void invert_decay(const RealInterval& r) {
        x.spoil();
        x.relax(-r.E1, 0.f, 1.0f - r.E1);
    }
    __device__ __forceinline__ float sample(int, float) const { return x.q; }
};

// The value and its tangents ∂/∂T1 and ∂/∂T2 (the phase factors depend on neither). Every step is
// affine in the state, and with the relaxation folded into the excitation the tangents are the same
// excitation of (p1, n1, z1 + s1·(z - δ_{n0})) and (p2 + s2·p, n2 + s2·n, z2), s1 = t/T1², s2 = t/T2²
// (EPGTangent in fisp.cu): 8 and 9 operations per state beside the value's 7.
template<int KP, int G>
struct RealTangents {
    static constexpr int kPlanes = 3;
    EPGReal<KP, G> x, d1, d2;

    __device__ __forceinline__ void init() {
        x.init(1.f);
        d1.init(0.f);
        d2.init(0.f);
    }
    __device__ __forceinline__ void shift(int sub, unsigned cut) {
        x.shift(sub, cut);
        d1.shift(sub, cut);
        d2.shift(sub, cut);
    }
    __device__ __forceinline__ void excite(const RealCoefs& k, float s1, float s2) {
        d1.excite_first(k, __fmul_rn(k.E2.x, d1.q),
                        __fmul_rn(k.E1, __fmaf_rn(s1, __fadd_rn(x.z0, -1.0f), d1.z0)));
        d2.excite_first(k, __fmul_rn(k.E2.x, __fmaf_rn(s2, x.q, d2.q)), __fmul_rn(k.E1, d2.z0));
        x.excite_first(k, __fmul_rn(k.E2.x, x.q), __fmaf_rn(k.E1, x.z0, k.regrow));
        const float2 S1 = bcast2(s1), S2 = bcast2(s2);
#pragma unroll
        for (int j = 0; j < KP; j++) {
            d1.z[j] = fma2(S1, x.z[j], d1.z[j]);
            d2.p[j] = fma2(S2, x.p[j], d2.p[j]);
            d2.n[j] = fma2(S2, x.n[j], d2.n[j]);
            EPGReal<KP, G>::excite_pair(k, x.p[j], x.n[j], x.z[j]);
            EPGReal<KP, G>::excite_pair(k, d1.p[j], d1.n[j], d1.z[j]);
            EPGReal<KP, G>::excite_pair(k, d2.p[j], d2.n[j], d2.z[j]);
        }
    }
    __device__ __forceinline__ void relax(const RealInterval& r) {
        const float2 S1 = bcast2(r.s1), S2 = bcast2(r.s2);
        d1.z0 = __fmaf_rn(r.s1, __fadd_rn(x.z0, -1.0f), d1.z0);
        d2.q = __fmaf_rn(r.s2, x.q, d2.q);
#pragma unroll
        for (int j = 0; j < KP; j++) {
            d1.z[j] = fma2(S1, x.z[j], d1.z[j]);
            d2.p[j] = fma2(S2, x.p[j], d2.p[j]);
            d2.n[j] = fma2(S2, x.n[j], d2.n[j]);
        }
        x.relax(r.E1, r.E2, 1.0f - r.E1);
        d1.relax(r.E1, r.E2, 0.f);
        d2.relax(r.E1, r.E2, 0.f);
    }
    __device__ __forceinline__ void spoil() {
        x.spoil();
        d1.spoil();
        d2.spoil();
    }
    __device__ __forceinline__ void invert_decay(const RealInterval& r) {
        spoil();
        x.relax(-1.f, 0.f, 0.f);
        d1.relax(-1.f, 0.f, 0.f);
        d2.relax(-1.f, 0.f, 0.f);
        relax(RealInterval {r.E1, 0.f, r.s1, 0.f});
    }
    // the sample's T2 tangent has the share of the decay over TE, s2 = TE/T2²
    __device__ __forceinline__ float sample(int plane, float s2) const {
        return plane == 0 ? x.q : plane == 1 ? d1.q : __fmaf_rn(s2, x.q, d2.q);
    }
};

// Rows of samples per chunk: the CTA's warps meet once per chunk of TRs to sum their positions. (Three
// planes of 32 voxels leave room for half the rows.)
template<int G, int PLANES>
constexpr int kRealRows = PLANES == 3 && G == 1 ? 32 : 64;
constexpr int kRealAngles = 68;  // angles per warp in shared memory

// shared memory of a CTA of W warps: float2 cte[W][VB], float angles[W][kRealAngles], float
// samples[W][kRealRows][VB] per plane, VB = 32 / G voxels per warp
template<int G, int PLANES>
constexpr size_t real_smem_bytes(int W) {
    return size_t(W) * ((32 / G) * sizeof(float2) + (kRealAngles + PLANES * kRealRows<G, PLANES> * (32 / G)) * sizeof(float));
}

// The items [item_begin, item_end) of a simulation (BAL: in the order `ord`), in rounds of one item
// per warp, as fisp_items (fisp.cu) runs them: an item is one (tile of VB voxels, slice position), a
// warp keeps one voxel per group of G lanes, and the positions of a voxel are summed one at a time in
// increasing order, so the echoes do not depend on the layout or on the split into rounds, CTAs or
// launches. The samples and the partial sums are the real q; the sum over the positions times i·c_TE is
// the echo. A partial sum lies in the first half of its tile's part of the echo row, 4 bytes per voxel.
// DIRECT: one slice position and G = 1, every warp writes its echoes itself.
template<class State, int KP, int G, bool BAL = false, bool DIRECT = false>
__device__ __forceinline__ void fisp_real_items(const FispArgs& a, const int item_begin, const int item_end,
                                                float2* smem, const FispOrder* ord = nullptr) {
    static_assert(!DIRECT || (G == 1 && State::kPlanes == 1), "one lane per voxel writes its echoes");
    constexpr int VB = 32 / G, NQ = State::kPlanes, CH = kRealRows<G, NQ>, RS = CH * VB;
    const int W = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane / G, sub = lane % G;
    const int P = a.P;
    // the slot of state N (index N-1 behind state 0), if the layout holds it
    const unsigned cut = a.N - 1 < 2 * KP * G && sub == (a.N - 1) / (2 * KP) ? 1u << ((a.N - 1) % (2 * KP)) : 0u;
    float2* cte = smem;
    float* angles = reinterpret_cast<float*>(smem + W * VB) + warp * kRealAngles;
    float* samples = reinterpret_cast<float*>(smem + W * VB) + W * kRealAngles;
    const int plane = W * RS;

    auto item_at = [&](int u) { return BAL ? ord->item[u] : u; };
    int nact;  // warps with an item this round
    for (int base = item_begin; base < item_end; base += nact) {
        nact = min(W, item_end - base);
        // a round that would reach from the tail into the head ends with the tail: what a CTA publishes then
        // never waits for another CTA (25 states, 35 positions, 400 TRs: 6560 voxels 664 us, 685 with waits
        // that chained; 8000 voxels, where they did not hold anything up, 799 and 758)
        if (BAL && base < ord->publish_u && ord->wait_u < base + nact) nact = ord->publish_u - base;
        if (BAL && base <= ord->wait_u && ord->wait_u < base + nact) {
            // this round reaches the head: its tile's first positions come from CTA cta - 1
            if (threadIdx.x == 0) handoff_wait(ord->handoff + ord->cta - 1, ord->status);
            __syncthreads();
        }
        const int item = item_at(base + min(warp, nact - 1));
        const bool pok = warp < nact;  // warp-uniform
        const int tile = item / P, p = item % P;
        const int vloc = tile * VB + grp;
        const bool vok = vloc < a.nvoxels;
        const int64_t vcol = a.voxel_begin + (vok ? vloc : a.nvoxels - 1);

        const float T1 = a.params[0 * a.param_stride + vcol];
        const float T2 = a.params[1 * a.param_stride + vcol];
        const float B1 = a.params[2 * a.param_stride + vcol];
        const float B0 = a.params[3 * a.param_stride + vcol];
        // per-voxel relaxation factors (fisp_kernels.cuh:110-144)
        const float R1 = 1.0f / T1, R2 = 1.0f / T2;
        auto interval = [&](float t) {
            return RealInterval {expf(-t * R1), expf(-t * R2), t * R1 * R1, t * R2 * R2};
        };
        const RealInterval tr = interval(a.TR);
        const float regrow = 1.0f - tr.E1;
        const float s2_TE = a.TE * R2 * R2;
        float2 c_TE = make_float2(1.f, 0.f);
        if (B0 != 0.0f) sincospif(2.0f * a.TE * B0, &c_TE.y, &c_TE.x);
        c_TE = cscale(expf(-a.TE * R2), c_TE);
        if (!DIRECT && sub == 0) cte[warp * VB + grp] = c_TE;  // read after the barrier of the first chunk

        // segments of this round: runs of consecutive warps on the same tile (bit w set where
        // warp w starts one); every thread derives the same mask
        unsigned starts = 0;
        if (!DIRECT)
            for (int w = 0; w < nact; w++)
                if (w == 0 || item_at(base + w) / P != item_at(base + w - 1) / P) starts |= 1u << w;

        const float4* tab = a.table + int64_t(p) * a.nTR;
        State st;
        st.init();
        for (int rep = a.reps; rep >= 1; rep--) {
            const bool sampled = (rep == 1);
            if (a.inversion) st.invert_decay(interval(a.TI));  // fisp_kernels.cuh:146-152
            for (int t0 = 0; t0 < a.nTR; t0 += CH) {
                const int nt = min(CH, a.nTR - t0);
                if (pok) {
                    // the chunk's signed angles (uniform over the lanes: read back as broadcasts)
                    __syncwarp();
                    for (int i = lane; i < nt; i += 32) angles[i] = __ldg(&tab[t0 + i].w);
                    __syncwarp();
                    float* mine = samples + warp * RS + grp;
                    float2* dst = a.echo + int64_t(t0) * a.uf * a.echo_stride + vcol;
                    auto sample = [&](int j) {
                        if (!sampled) return;
                        if (!DIRECT) {
                            if (sub == 0) {
#pragma unroll
                                for (int qn = 0; qn < NQ; qn++) mine[qn * plane + j * VB] = st.sample(qn, s2_TE);
                            }
                            return;
                        }
                        const float q = st.sample(0, s2_TE);
                        const float2 e = make_float2(-__fmul_rn(c_TE.y, q), __fmul_rn(c_TE.x, q));  // i·c_TE·q
                        for (int u = 0; u < a.uf; u++) {
                            if (vok) __stcs(dst, e);
                            dst += a.echo_stride;
                        }
                    };
                    int j = 0;
                    if (t0 == 0) {  // no relaxation before the first excitation
                        st.excite(real_coefs(angles[0], B1, 1.0f, 1.0f, 0.0f), 0.f, 0.f);
                        sample(0);
                        j = 1;
                    }
                    // four TRs per iteration let the compiler absorb most dephasing shifts in register
                    // renaming (25 states, MR-STAT slice: 12.6 ms; with KP TRs, where the renaming
                    // closes, 12.8 ms)
#pragma unroll 4
                    for (; j < nt; j++) {
                        const RealCoefs k = real_coefs(angles[j], B1, tr.E1, tr.E2, regrow);
                        st.shift(sub, cut);
                        st.excite(k, tr.s1, tr.s2);
                        sample(j);
                    }
                }
                if (sampled && !DIRECT) {
                    __syncthreads();
                    // per segment, add its positions in increasing order to the tile's partial sum
                    // (unless the segment starts at position 0); after the last position write the
                    // undersampling-expanded rows (fisp_kernels.cuh:246-259)
                    const uint64_t l2_keep = l2_policy_evict_last();
                    // two voxels per lane; no other warp touches a row
                    constexpr int kRows = 64 / VB;
                    const int jh = lane / (VB / 2), vp = 2 * (lane % (VB / 2));
                    for (int w0 = 0; w0 < nact;) {
                        int w1 = w0 + 1;
                        while (w1 < nact && !(starts & (1u << w1))) w1++;
                        const int seg_tile = item_at(base + w0) / P;
                        const bool first = item_at(base + w0) % P == 0;
                        const bool last = item_at(base + w1 - 1) % P == P - 1;
                        const int left = a.nvoxels - seg_tile * VB - vp;
                        const float2 c0 = cte[w0 * VB + vp], c1 = cte[w0 * VB + vp + 1];
#pragma unroll
                        for (int qn = 0; qn < NQ; qn++) {
                            float2* out = qn == 0 ? a.echo : qn == 1 ? a.dT1 : a.dT2;
                            for (int jb = kRows * warp; jb < nt; jb += kRows * W) {
                                const int j = jb + jh;
                                const bool in = j < nt && left > 0;
                                float2* row = out + int64_t(t0 + j) * a.uf * a.echo_stride + a.voxel_begin + seg_tile * VB;
                                float2* part = row + vp / 2;
                                const float2* col = reinterpret_cast<const float2*>(samples + qn * plane + j * VB + vp);
                                float2 acc = make_float2(0.f, 0.f);
                                if (in) {
                                    acc = col[w0 * (RS / 2)];
                                    if (!first) acc = add2(__ldcg(part), acc);
                                    for (int w = w0 + 1; w < w1; w++) acc = add2(acc, col[w * (RS / 2)]);
                                }
                                if (last) {
                                    __syncwarp();  // a lane's echoes cover other lanes' partial sums
                                    const float2 e0 = make_float2(-__fmul_rn(c0.y, acc.x), __fmul_rn(c0.x, acc.x));  // i·c_TE·acc
                                    const float2 e1 = make_float2(-__fmul_rn(c1.y, acc.y), __fmul_rn(c1.x, acc.y));
                                    if (in)
                                        for (int u = 0; u < a.uf; u++) {
                                            __stcs(row + int64_t(u) * a.echo_stride + vp, e0);
                                            if (left > 1) __stcs(row + int64_t(u) * a.echo_stride + vp + 1, e1);
                                        }
                                } else if (in) {
                                    // read again by a later round (or the next CTA): keep it in L2
                                    st_l2_hint(part, acc, l2_keep);
                                }
                            }
                        }
                        w0 = w1;
                    }
                    __syncthreads();
                }
            }
            if (rep > 1 && pok) {  // close the repetition: relax to TR, dephase, spoil, wait (fisp_kernels.cuh:195-200)
                st.relax(tr);
                st.shift(sub, cut);
                if (a.wait_spoil) st.spoil();
                st.relax(interval(a.TW));
            }
        }
        if (BAL && base < ord->publish_u && ord->publish_u <= base + nact) {
            // the tail's partial sums are written (the summation ends with a barrier): hand them over
            if (threadIdx.x == 0) handoff_publish(ord->handoff + ord->cta);
        }
    }
}

// Warps per CTA (one CTA per SM), by the registers: 6·KP for each state vector and about 60 besides. A
// multiple of 4, so that the four schedulers of an SM get the same number. Measured: 8 states, 35
// positions, 50176 voxels: 5.91 ms with 16 warps, 6.60 with 24 (spills); tangents of 25 states (6 pairs on
// 2 lanes), 9216 voxels: 9.86 ms with 8 warps, 11.1 with 12 (spills).
template<int KP, int PLANES>
constexpr int kRealWarps = KP * PLANES <= 8 ? 16 : KP * PLANES <= 12 ? 12 : 8;

// One FISP simulation with real phases on a persistent grid (returns at once when the sequence's
// phases are not real: the general kernel launched beside it runs then). State: RealValue, or
// RealTangents, which also writes a.dT1 and a.dT2. BAL: the balanced split of the (tile, position)
// items, see fisp_epg_kernel.
template<template<int, int> class State, int KP, int G, bool BAL>
__global__ void __launch_bounds__(32 * kRealWarps<KP, State<KP, G>::kPlanes>, 1)
    fisp_real_kernel(FispArgs a, HostAnswer ask, int ntiles, int* handoff, unsigned int* status) {
    extern __shared__ float2 smem[];
    if (a.skip != nullptr && *a.skip != 0) return;  // uniform over the grid
    answer_host(ask, fisp_real_phases(a));
    if (!fisp_real_phases(a)) return;
    if constexpr (BAL) {
        __shared__ FispOrder ord;
        const int n = fisp_balanced_order(ord, ntiles, a.P, handoff, status);
        fisp_real_items<State<KP, G>, KP, G, true>(a, 0, n, smem, &ord);
    } else {
        const int2 r = cta_tile_range(ntiles, blockIdx.x, gridDim.x);
        if constexpr (G == 1 && State<KP, G>::kPlanes == 1) {
            if (a.P == 1) {
                fisp_real_items<State<KP, G>, KP, G, false, true>(a, r.x, r.y, smem);
                return;
            }
        }
        fisp_real_items<State<KP, G>, KP, G>(a, r.x * a.P, r.y * a.P, smem);
    }
}

// Work-queue form for batches (see fisp_queue_kernel): every job's phases are real.
template<template<int, int> class State, int KP, int G>
__global__ void __launch_bounds__(32 * kRealWarps<KP, State<KP, G>::kPlanes>, 1)
    fisp_real_queue_kernel(const FispArgs* __restrict__ jobs, const int2* __restrict__ items, int nitems,
                           int* __restrict__ head) {
    extern __shared__ float2 smem[];
    __shared__ FispArgs job;
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(head, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= nitems) break;
        const int2 w = items[it];
        if (threadIdx.x == 0) job = jobs[w.x];
        __syncthreads();
        const int tiles = (job.nvoxels + 32 / G - 1) / (32 / G);
        const int t_end = min(w.y + fisp_queue_tiles_per_item(job.P, blockDim.x >> 5), tiles);
        fisp_real_items<State<KP, G>, KP, G>(job, w.y * job.P, t_end * job.P, smem);
        __syncthreads();  // job and s_item are rewritten by the next item
    }
}

}  // namespace kernels

// Up to this many (voxel, position) pairs the states of a pair go over 4 lanes: three warps for each
// scheduler of the GPU's 148 SMs on 4 lanes. 200 TRs, one lane (tangents: the layout for many pairs) against
// four, in us: values of 25 states 60.7 / 41.5 at 9470 pairs, 61.9 / 73.0 at 18940, of 5 states 31.0 / 28.7
// and 31.6 / 53.8; tangents of 25 states 109 / 95 and 173 / 162, of 8 states 93.5 / 56.6 and 93.6 / 104.
constexpr int64_t kRealSplitPairs = 148 * 3 * 32;

using RealKernel = void (*)(kernels::FispArgs, kernels::HostAnswer, int, int*, unsigned int*);
using RealQueueKernel = void (*)(const kernels::FispArgs*, const int2*, int, int*);
struct RealLayout {
    int KP, G;     // states 0 .. 2·KP·G
    int warps;     // at most, per CTA
    int smem;      // shared memory per warp
    RealKernel fn, balanced;  // balanced: null when the layout has no such form
    RealQueueKernel queue;
};

}  // namespace compas
