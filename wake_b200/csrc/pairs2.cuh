// TRT (+ Smagorinsky) for two nodes at once in packed FP32.
//
// sm_100 executes add / mul / fma on a pair of FP32 values as one instruction
// (PTX add/mul/fma .f32x2, CUDA __fadd2_rn / __fmul2_rn / __ffma2_rn), so a
// thread that carries two nodes in the two halves of float2 registers issues
// half the arithmetic of the one-node form. The algebra is the pair form:
// pair sums s = f_q + f_opp and differences
// d = f_q - f_opp, rho = f_0 + sum s, j = sum c d, LES stress from
// s - s_eq, and the update
//     f_q'   = f_q   - omega_s/2 (s - s_eq) - omega_a/2 (d - d_eq)
//     f_opp' = f_opp - omega_s/2 (s - s_eq) + omega_a/2 (d - d_eq)
// with s_eq = 2 w rho (1 - 1.5 u^2 + 4.5 (c.u)^2) and d_eq = 6 w rho (c.u).
//
// HS = true works on shifted populations h = f / w - 1 (the FP16 / BF16
// storage format) directly: with S = h_q + h_opp, D = h_q - h_opp,
//     rho = 1 + w_0 h_0 + sum w S,   j = sum c w D,
//     S_eq = 2 rho (1 - 1.5 u^2 + 4.5 (c.u)^2) - 2,   D_eq = 6 rho (c.u),
// and the same update in h, so stored values are used without decoding.
// gy (FP32 forms) is the y body force of the two nodes, P.g[1] twice,
// and `forced` whether any body force acts.
// Every rounding is explicit (packed ops are never contracted by the compiler).
#pragma once

#include "lattice.cuh"

namespace wk {

// (On the host the same roundings one by one.)
__host__ __device__ __forceinline__ float2 bc2(float s) { return make_float2(s, s); }
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
#else
__host__ __device__ inline float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ inline float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__host__ __device__ inline float2 fma2(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
#endif
__host__ __device__ __forceinline__ float2 sub2(float2 a, float2 b) { return add2(a, make_float2(-b.x, -b.y)); }

// acc + c v (f-space) or acc + c w v (h-space) for a lattice component c in {-1, 0, 1};
// the branches fold away once the pair loop is unrolled
__host__ __device__ __forceinline__ float2 acc_c(float2 acc, int c, float2 v) {
    return c > 0 ? add2(acc, v) : (c < 0 ? sub2(acc, v) : acc);
}
__device__ __forceinline__ float2 acc_cw(float2 acc, int c, float w, float2 v) {
    return c > 0 ? fma2(bc2(w), v, acc) : (c < 0 ? fma2(bc2(-w), v, acc) : acc);
}
__host__ __device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// Shifted populations. The body force is P.g for both nodes (as packed gy it cost the pipelined row kernel 4 more spilled
// values a thread: D3Q19 F16 256^3 box with Smagorinsky 267 us a step, 257 so).
template <int Q, bool LES>
__device__ __forceinline__ void trt_pairs2_h(float2* f, const Physics& P, const bool forced, float2& rho, float2 u[3]) {
    using L = Lat<Q>;
    constexpr int NP = (Q - 1) / 2;
    float2 s[NP], d[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p), o = L::opp(q);
        s[p] = add2(f[q], f[o]);
        d[p] = sub2(f[q], f[o]);
    }
    float2 r, jx = bc2(0.f), jy = bc2(0.f), jz = bc2(0.f);
    r = fma2(bc2(L::w(0)), f[0], bc2(1.0f));
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p);
        r = fma2(bc2(L::w(q)), s[p], r);
        jx = acc_cw(jx, L::cx(q), L::w(q), d[p]);
        jy = acc_cw(jy, L::cy(q), L::w(q), d[p]);
        jz = acc_cw(jz, L::cz(q), L::w(q), d[p]);
    }
    rho = r;
    const float2 inv = make_float2(__fdividef(1.0f, r.x), __fdividef(1.0f, r.y));
    const float* g = P.g;
    const float2 hr = mul2(bc2(0.5f), r);
    u[0] = mul2(forced ? fma2(hr, bc2(g[0]), jx) : jx, inv);
    u[1] = mul2(forced ? fma2(hr, bc2(g[1]), jy) : jy, inv);
    u[2] = mul2(forced ? fma2(hr, bc2(g[2]), jz) : jz, inv);
    const float2 u2 = fma2(u[2], u[2], fma2(u[1], u[1], mul2(u[0], u[0])));
    const float2 a0 = fma2(bc2(-1.5f), u2, bc2(1.0f));
    // per pair: c.u and the non-equilibrium parts nS = s - s_eq, nD = d - d_eq, with the even
    // equilibrium written s_eq = (9 rho (c.u)) (c.u) + 2 rho a0 - 2
    float2 nS[NP], nD[NP];
    const float2 rm6 = mul2(bc2(-6.0f), r);
    const float2 e0h = fma2(add2(r, r), a0, bc2(-2.0f)), r9 = mul2(bc2(9.0f), r);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p);
        // c.u from the nonzero components (no multiplications by +-1)
        const int cx = L::cx(q), cy = L::cy(q), cz = L::cz(q);
        float2 cu = cx ? (cx > 0 ? u[0] : neg2(u[0])) : bc2(0.f);
        if (cy) cu = cx ? acc_c(cu, cy, u[1]) : (cy > 0 ? u[1] : neg2(u[1]));
        if (cz) cu = (cx || cy) ? acc_c(cu, cz, u[2]) : (cz > 0 ? u[2] : neg2(u[2]));
        nS[p] = sub2(s[p], fma2(mul2(r9, cu), cu, e0h));
        nD[p] = fma2(rm6, cu, d[p]);
    }
    float2 hs, ha;  // omega_s / 2, omega_a / 2 per node
    if constexpr (LES) {
        float2 pxx = bc2(0.f), pyy = bc2(0.f), pzz = bc2(0.f), pxy = bc2(0.f), pyz = bc2(0.f), pxz = bc2(0.f);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int q = pair_q<Q>(p);
            const int x = L::cx(q), y = L::cy(q), z = L::cz(q);
            // stress contribution w (S - S_eq)
            const float wq = L::w(q);
            if (x) pxx = fma2(bc2(wq), nS[p], pxx);
            if (y) pyy = fma2(bc2(wq), nS[p], pyy);
            if (z) pzz = fma2(bc2(wq), nS[p], pzz);
            if (x && y) pxy = fma2(bc2(x * y > 0 ? wq : -wq), nS[p], pxy);
            if (y && z) pyz = fma2(bc2(y * z > 0 ? wq : -wq), nS[p], pyz);
            if (x && z) pxz = fma2(bc2(x * z > 0 ? wq : -wq), nS[p], pxz);
        }
        const float2 off = fma2(pxz, pxz, fma2(pyz, pyz, mul2(pxy, pxy)));
        const float2 sum = fma2(bc2(2.0f), off, fma2(pzz, pzz, fma2(pyy, pyy, mul2(pxx, pxx))));
        const float tx = smagorinsky_tau_eff(P.tau, P.cs_smag, r.x, sum.x);
        const float ty = smagorinsky_tau_eff(P.tau, P.cs_smag, r.y, sum.y);
        hs = make_float2(__fdividef(0.5f, tx), __fdividef(0.5f, ty));
        ha = make_float2(__fdividef(0.5f, trt_tau_a(P.lambda_trt, tx)), __fdividef(0.5f, trt_tau_a(P.lambda_trt, ty)));
    } else {
        const float tau_a = 0.5f + P.lambda_trt / fmaxf(1e-4f, P.tau - 0.5f);
        hs = bc2(0.5f / P.tau);
        ha = bc2(0.5f / tau_a);
    }
    // rest population: relaxes to rho a0 - 1
    const float2 e0 = fma2(r, a0, bc2(-1.0f));
    f[0] = fma2(mul2(bc2(-2.0f), hs), sub2(f[0], e0), f[0]);
    float2 ug;
    float2 ps, pa;
    if (forced) {
        ug = fma2(u[2], bc2(g[2]), fma2(u[1], bc2(g[1]), mul2(u[0], bc2(g[0]))));
        ps = fma2(bc2(-1.0f), hs, bc2(1.0f));  // 1 - omega_s / 2
        pa = fma2(bc2(-1.0f), ha, bc2(1.0f));
        // Guo term of the rest population: (1 - omega_s/2) w_0 rho (-3 u.g)
        const float2 fr = r;
        f[0] = fma2(mul2(ps, fr), mul2(bc2(-3.0f), ug), f[0]);
    }
    if (!forced) {
        // f_q' = f_q - hs nS - ha nD, f_opp' = f_opp - hs nS + ha nD, two fused steps each
        const float2 nhs = neg2(hs), nha = neg2(ha);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int q = pair_q<Q>(p), o = L::opp(q);
            f[q] = fma2(nhs, nS[p], fma2(nha, nD[p], f[q]));
            f[o] = fma2(nhs, nS[p], fma2(ha, nD[p], f[o]));
        }
        return;
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p), o = L::opp(q);
        float2 A = mul2(hs, nS[p]), B = mul2(ha, nD[p]);
        {
            // Guo forcing of the pair (collide_trt_t in lattice.cuh): even part
            // (1 - omega_s/2) w rho (-3 u.g + 9 (c.u)(c.g)), odd part (1 - omega_a/2) w rho 3 (c.g)
            float cg = L::cx(q) > 0 ? g[0] : (L::cx(q) < 0 ? -g[0] : 0.0f);
            if (L::cy(q)) cg = __fadd_rn(cg, L::cy(q) > 0 ? g[1] : -g[1]);
            if (L::cz(q)) cg = __fadd_rn(cg, L::cz(q) > 0 ? g[2] : -g[2]);
            float2 cu = fma2(bc2(float(L::cz(q))), u[2], fma2(bc2(float(L::cy(q))), u[1], mul2(bc2(float(L::cx(q))), u[0])));
            const float2 fr = r;
            const float2 ev = mul2(mul2(ps, fr), fma2(bc2(__fmul_rn(9.0f, cg)), cu, mul2(bc2(-3.0f), ug)));
            const float2 od = mul2(mul2(pa, fr), bc2(__fmul_rn(3.0f, cg)));
            A = sub2(A, ev);
            B = sub2(B, od);
        }
        const float2 fq = sub2(sub2(f[q], A), B);
        const float2 fo = add2(sub2(f[o], A), B);
        f[q] = fq;
        f[o] = fo;
    }
}

// FP32 populations. Pair sums, differences and non-equilibrium parts are formed anew in each of the three passes
// (moments, stress, update) from f instead of kept (36 to 72 registers of two nodes in D3Q19): at the 96 registers
// of before, 17 values per thread spilled, and every spilled value is a store to L2 (1.55 times the step's own
// writes there).
template <int Q, bool LES>
__device__ __forceinline__ void trt_pairs2_f(float2* f, const Physics& P, const float2 gy, const bool forced, float2& rho,
                                             float2 u[3]) {
    using L = Lat<Q>;
    constexpr int NP = (Q - 1) / 2;
    // hide from the compiler that f is unchanged since the last pass: it would keep what it computed
    auto forget = [&]() {
#pragma unroll
        for (int q = 1; q < Q; ++q) asm volatile("" : "+f"(f[q].x), "+f"(f[q].y));
    };
    float2 r = f[0], jx = bc2(0.f), jy = bc2(0.f), jz = bc2(0.f);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p);
        const float2 d = sub2(f[q], f[L::opp(q)]);
        r = add2(r, add2(f[q], f[L::opp(q)]));
        jx = acc_c(jx, L::cx(q), d);
        jy = acc_c(jy, L::cy(q), d);
        jz = acc_c(jz, L::cz(q), d);
    }
    forget();
    rho = r;
    const float2 inv = make_float2(__fdividef(1.0f, r.x), __fdividef(1.0f, r.y));
    const float* g = P.g;
    const float2 hr = mul2(bc2(0.5f), r);
    u[0] = mul2(forced ? fma2(hr, bc2(g[0]), jx) : jx, inv);
    u[1] = mul2(forced ? fma2(hr, gy, jy) : jy, inv);
    u[2] = mul2(forced ? fma2(hr, bc2(g[2]), jz) : jz, inv);
    const float2 u2 = fma2(u[2], u[2], fma2(u[1], u[1], mul2(u[0], u[0])));
    const float2 a0 = fma2(bc2(-1.5f), u2, bc2(1.0f));
    auto cdotu = [&](int q) {  // c.u from the nonzero components (no multiplications by +-1)
        const int cx = L::cx(q), cy = L::cy(q), cz = L::cz(q);
        float2 cu = cx ? (cx > 0 ? u[0] : neg2(u[0])) : bc2(0.f);
        if (cy) cu = cx ? acc_c(cu, cy, u[1]) : (cy > 0 ? u[1] : neg2(u[1]));
        if (cz) cu = (cx || cy) ? acc_c(cu, cz, u[2]) : (cz > 0 ? u[2] : neg2(u[2]));
        return cu;
    };
    // s - s_eq of a pair, s_eq = (9 w rho (c.u)) (c.u) + 2 w rho a0; the weight-class products are shared by its pairs
    auto even = [&](int q, float2 cu) {
        const float w = L::w(q);
        const float2 e0w = mul2(mul2(bc2(2.0f * w), r), a0);
        return sub2(add2(f[q], f[L::opp(q)]), fma2(mul2(mul2(bc2(9.0f * w), r), cu), cu, e0w));
    };
    float2 hs, ha;  // omega_s / 2, omega_a / 2 per node
    if constexpr (LES) {
        float2 pxx = bc2(0.f), pyy = bc2(0.f), pzz = bc2(0.f), pxy = bc2(0.f), pyz = bc2(0.f), pxz = bc2(0.f);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int q = pair_q<Q>(p), x = L::cx(q), y = L::cy(q), z = L::cz(q);
            const float2 n = even(q, cdotu(q));
            if (x) pxx = add2(pxx, n);
            if (y) pyy = add2(pyy, n);
            if (z) pzz = add2(pzz, n);
            pxy = acc_c(pxy, x * y, n);
            pyz = acc_c(pyz, y * z, n);
            pxz = acc_c(pxz, x * z, n);
        }
        forget();
        const float2 off = fma2(pxz, pxz, fma2(pyz, pyz, mul2(pxy, pxy)));
        const float2 sum = fma2(bc2(2.0f), off, fma2(pzz, pzz, fma2(pyy, pyy, mul2(pxx, pxx))));
        const float tx = smagorinsky_tau_eff(P.tau, P.cs_smag, r.x, sum.x);
        const float ty = smagorinsky_tau_eff(P.tau, P.cs_smag, r.y, sum.y);
        hs = make_float2(__fdividef(0.5f, tx), __fdividef(0.5f, ty));
        ha = make_float2(__fdividef(0.5f, trt_tau_a(P.lambda_trt, tx)), __fdividef(0.5f, trt_tau_a(P.lambda_trt, ty)));
    } else {
        hs = bc2(0.5f / P.tau);
        ha = bc2(0.5f / (0.5f + P.lambda_trt / fmaxf(1e-4f, P.tau - 0.5f)));
    }
    // rest population: relaxes to w_0 rho a0
    f[0] = fma2(mul2(bc2(-2.0f), hs), sub2(f[0], mul2(mul2(bc2(L::w(0)), r), a0)), f[0]);
    const float2 nhs = neg2(hs), nha = neg2(ha);
    float2 ug, ps, pa;
    if (forced) {
        ug = fma2(u[2], bc2(g[2]), fma2(u[1], gy, mul2(u[0], bc2(g[0]))));
        ps = fma2(bc2(-1.0f), hs, bc2(1.0f));  // 1 - omega_s / 2
        pa = fma2(bc2(-1.0f), ha, bc2(1.0f));
        // Guo term of the rest population: (1 - omega_s/2) w_0 rho (-3 u.g)
        f[0] = fma2(mul2(ps, mul2(bc2(L::w(0)), r)), mul2(bc2(-3.0f), ug), f[0]);
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = pair_q<Q>(p), o = L::opp(q);
        const int cx = L::cx(q), cy = L::cy(q), cz = L::cz(q);
        const float w = L::w(q);
        const float2 cu = cdotu(q), nS = even(q, cu);
        const float2 nD = fma2(mul2(bc2(-6.0f * w), r), cu, sub2(f[q], f[o]));
        if (!forced) {
            // f_q' = f_q - hs nS - ha nD, f_opp' = f_opp - hs nS + ha nD, two fused steps each
            f[q] = fma2(nhs, nS, fma2(nha, nD, f[q]));
            f[o] = fma2(nhs, nS, fma2(ha, nD, f[o]));
        } else {
            // Guo forcing of the pair (collide_trt_t in lattice.cuh): even part
            // (1 - omega_s/2) w rho (-3 u.g + 9 (c.u)(c.g)), odd part (1 - omega_a/2) w rho 3 (c.g)
            float2 cg = bc2(cx > 0 ? g[0] : (cx < 0 ? -g[0] : 0.0f));
            cg = acc_c(cg, cy, gy);
            cg = acc_c(cg, cz, bc2(g[2]));
            const float2 fr = mul2(bc2(w), r);
            const float2 ev = mul2(mul2(ps, fr), fma2(mul2(bc2(9.0f), cg), cu, mul2(bc2(-3.0f), ug)));
            const float2 od = mul2(mul2(pa, fr), mul2(bc2(3.0f), cg));
            const float2 A = sub2(mul2(hs, nS), ev), B = sub2(mul2(ha, nD), od);
            f[q] = sub2(sub2(f[q], A), B);
            f[o] = add2(sub2(f[o], A), B);
        }
    }
}

template <int Q, bool LES, bool HS>
__device__ __forceinline__ void trt_pairs2(float2* f, const Physics& P, const float2 gy, const bool forced, float2& rho,
                                           float2 u[3]) {
    if constexpr (HS) trt_pairs2_h<Q, LES>(f, P, forced, rho, u);
    else trt_pairs2_f<Q, LES>(f, P, gy, forced, rho, u);
}

// Smagorinsky tau of two nodes from the non-equilibrium stress.
__device__ __forceinline__ float2 smagorinsky_tau2(const Physics& P, float2 r, float2 xx, float2 yy, float2 zz, float2 xy,
                                                   float2 yz, float2 xz) {
    const float2 off = fma2(xz, xz, fma2(yz, yz, mul2(xy, xy)));
    const float2 sum = fma2(bc2(2.0f), off, fma2(zz, zz, fma2(yy, yy, mul2(xx, xx))));
    return make_float2(smagorinsky_tau_eff(P.tau, P.cs_smag, r.x, sum.x), smagorinsky_tau_eff(P.tau, P.cs_smag, r.y, sum.y));
}

// Density and momentum of two FP32 nodes and, for Smagorinsky's tau, the stress moments of f - w: `dev` = sum (f - w) and
// p = sum c c (f - w) (xx, yy, zz, xy, yz, xz). The moments of f themselves are near 1/3, and the small stress that is
// left of them would keep their roundings.
template <int Q, bool LES>
__host__ __device__ __forceinline__ void bgk_sums2(const float2* f, float2& r, float2 j[3], float2& dev, float2 p[6]) {
    using L = Lat<Q>;
    r = dev = bc2(0.f);
#pragma unroll
    for (int k = 0; k < 6; ++k) p[k] = bc2(0.f);
#pragma unroll
    for (int a = 0; a < 3; ++a) j[a] = bc2(0.f);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int x = L::cx(q), y = L::cy(q), z = L::cz(q);
        r = add2(r, f[q]);
        j[0] = acc_c(j[0], x, f[q]);
        j[1] = acc_c(j[1], y, f[q]);
        j[2] = acc_c(j[2], z, f[q]);
        if constexpr (LES) {
            const float2 d = sub2(f[q], bc2(L::w(q)));
            dev = add2(dev, d);
            p[0] = acc_c(p[0], x * x, d);
            p[1] = acc_c(p[1], y * y, d);
            p[2] = acc_c(p[2], z * z, d);
            p[3] = acc_c(p[3], x * y, d);
            p[4] = acc_c(p[4], y * z, d);
            p[5] = acc_c(p[5], x * z, d);
        }
    }
}

// The non-equilibrium stress sum c c (f - f_eq) = p - 1/3 dev - rho u u from those moments, in their place. Its error
// against FP64 (diagonal, rms of 200,000 nodes, density and velocity rounded): D3Q19 2.5e-9, D3Q27 7.5e-10;
// from the moments of f 3.4e-8 and 4.8e-8, from the non-equilibrium pair sums of smagorinsky_tau 2.6e-8 and 3.3e-8.
__host__ __device__ __forceinline__ void bgk_stress2(float2 r, const float2 u[3], float2 dev, float2 p[6]) {
    const float2 d3 = mul2(bc2(-1.0f / 3.0f), dev), rx = mul2(r, neg2(u[0])), ry = mul2(r, neg2(u[1])), rz = mul2(r, neg2(u[2]));
    p[0] = fma2(rx, u[0], add2(p[0], d3));
    p[1] = fma2(ry, u[1], add2(p[1], d3));
    p[2] = fma2(rz, u[2], add2(p[2], d3));
    p[3] = fma2(rx, u[1], p[3]);
    p[4] = fma2(ry, u[2], p[4]);
    p[5] = fma2(rx, u[2], p[5]);
}

// BGK (collide_bgk) of two FP32 nodes of a 3D lattice. Each population relaxes by itself: written over pair sums like the
// TRT update, a 20,000-step drag history drifted three times as far from FP64 (1.3e-4 against 4.6e-5). For the same
// reason BGK and MRT round the reciprocal of rho correctly.
template <int Q, bool LES>
__device__ __forceinline__ void bgk_pairs2(float2* f, const Physics& P, const float2 gy, const bool forced, float2& rho,
                                           float2 u[3]) {
    using L = Lat<Q>;
    float2 r, j[3], dev, p[6];
    bgk_sums2<Q, LES>(f, r, j, dev, p);
    rho = r;
    const float2 inv = make_float2(__frcp_rn(r.x), __frcp_rn(r.y)), hr = mul2(bc2(0.5f), r);
    const float2 g[3] = {bc2(P.g[0]), gy, bc2(P.g[2])};
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = mul2(forced ? fma2(hr, g[a], j[a]) : j[a], inv);
    float2 om;
    if constexpr (LES) {
        bgk_stress2(r, u, dev, p);
        const float2 t = smagorinsky_tau2(P, r, p[0], p[1], p[2], p[3], p[4], p[5]);
        om = make_float2(__frcp_rn(t.x), __frcp_rn(t.y));
    } else {
        om = bc2(1.0f / P.tau);
    }
    const float2 u2 = fma2(u[2], u[2], fma2(u[1], u[1], mul2(u[0], u[0]))), nom = neg2(om);
    const float2 pre = fma2(bc2(-0.5f), om, bc2(1.0f));
    float2 ug = bc2(0.f);
    if (forced) ug = fma2(u[2], g[2], fma2(u[1], g[1], mul2(u[0], g[0])));
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int cx = L::cx(q), cy = L::cy(q), cz = L::cz(q);
        float2 cu = cx ? (cx > 0 ? u[0] : neg2(u[0])) : bc2(0.f);
        if (cy) cu = cx ? acc_c(cu, cy, u[1]) : (cy > 0 ? u[1] : neg2(u[1]));
        if (cz) cu = (cx || cy) ? acc_c(cu, cz, u[2]) : (cz > 0 ? u[2] : neg2(u[2]));
        const float2 wr = mul2(bc2(L::w(q)), r);
        const float2 t = fma2(bc2(-1.5f), u2, fma2(mul2(bc2(4.5f), cu), cu, fma2(bc2(3.0f), cu, bc2(1.0f))));
        const float2 d = fma2(neg2(wr), t, f[q]);
        f[q] = fma2(nom, d, f[q]);
        if (forced) {
            float2 cg = bc2(cx > 0 ? P.g[0] : (cx < 0 ? -P.g[0] : 0.0f));
            cg = acc_c(cg, cy, g[1]);
            cg = acc_c(cg, cz, g[2]);
            f[q] = fma2(mul2(pre, wr), fma2(mul2(bc2(9.0f), cu), cg, mul2(bc2(3.0f), sub2(cg, ug))), f[q]);
        }
    }
}

// Inverse row of the D3Q19 MRT (D3Q19Minv) for direction q over moments 3 .. 18 of one parity: the odd moments change
// sign with the direction, so a pair needs one even and one odd row.
template <bool R, int q, bool ODD, int... k>
__device__ __forceinline__ float2 d3q19_inv_part(const float2* m, float2 a, std::integer_sequence<int, k...>) {
    (((((k + 3 <= 8 || k + 3 >= 16) == ODD) && D3Q19Minv<R, q, k + 3>::v != 0.0f)
          ? (void)(a = fma2(bc2(D3Q19Minv<R, q, k + 3>::v), m[k + 3], a))
          : (void)0),
     ...);
    return a;
}
template <bool R, int p>
__device__ __forceinline__ void d3q19_inv_pair(float2* f, const float2* m, float2 axis, float2 diagonal) {
    constexpr int q = pair_q<19>(p), o = Lat<19>::opp(q);
    using K = std::make_integer_sequence<int, 16>;
    const float2 e = d3q19_inv_part<R, q, false>(m, q < 7 ? axis : diagonal, K{});
    const float2 d = d3q19_inv_part<R, q, true>(m, bc2(0.f), K{});
    f[q] = add2(e, d);
    f[o] = sub2(e, d);
}
template <bool R, int... p>
__device__ __forceinline__ void d3q19_inverse2(float2* f, const float2* m, std::integer_sequence<int, p...>) {
    auto low = [&](auto w0, auto w1, auto w2) { return fma2(bc2(w2), m[2], fma2(bc2(w1), m[1], mul2(bc2(w0), m[0]))); };
    const float2 axis = low(D3Q19Minv<R, 1, 0>::v, D3Q19Minv<R, 1, 1>::v, D3Q19Minv<R, 1, 2>::v);
    const float2 diagonal = low(D3Q19Minv<R, 7, 0>::v, D3Q19Minv<R, 7, 1>::v, D3Q19Minv<R, 7, 2>::v);
    f[0] = low(D3Q19Minv<R, 0, 0>::v, D3Q19Minv<R, 0, 1>::v, D3Q19Minv<R, 0, 2>::v);
    (d3q19_inv_pair<R, p>(f, m, axis, diagonal), ...);
}

// D3Q19 MRT (collide_mrt_d3q19) of two nodes. The moments of the d'Humieres basis are sums and differences of a few
// pair sums (even moments) and pair differences (odd moments), and an inverse row is an even and an odd half that the
// two directions of a pair share: about 190 packed operations for two nodes where the dense 19 x 19 products and their
// scalar relaxation take about 600 per node.
template <bool LES>
__device__ __forceinline__ void mrt19_pairs2(float2* f, const Physics& P, const float2 gy, const bool forced, float2& rho,
                                             float2 u[3]) {
    auto S = [&](int q) { return add2(f[q], f[Lat<19>::opp(q)]); };
    auto D = [&](int q) { return sub2(f[q], f[Lat<19>::opp(q)]); };
    float2 m[19];
    const float2 sx = S(1), sy = S(3), sz = S(5);
    const float2 a1 = S(7), a2 = S(8), b1 = S(11), b2 = S(12), c1 = S(15), c2 = S(16);
    const float2 xy = add2(a1, a2), xz = add2(b1, b2), yz = add2(c1, c2);
    const float2 A = add2(add2(sx, sy), sz), G = add2(add2(xy, xz), yz);
    m[0] = add2(add2(f[0], A), G);
    m[1] = fma2(bc2(8.0f), G, fma2(bc2(-11.0f), A, mul2(bc2(-30.0f), f[0])));
    m[2] = add2(G, fma2(bc2(-4.0f), A, mul2(bc2(12.0f), f[0])));
    const float2 p9 = sub2(sub2(add2(sx, sx), sy), sz), r9 = fma2(bc2(-2.0f), yz, add2(xy, xz));
    m[9] = add2(p9, r9);
    m[10] = fma2(bc2(-2.0f), p9, r9);
    const float2 p11 = sub2(sy, sz), r11 = sub2(xy, xz);
    m[11] = add2(p11, r11);
    m[12] = fma2(bc2(-2.0f), p11, r11);
    m[13] = sub2(a1, a2);
    m[14] = sub2(c1, c2);
    m[15] = sub2(b1, b2);
    const float2 dx = D(1), dy = D(3), dz = D(5);
    const float2 e1 = D(7), e2 = D(8), g1 = D(11), g2 = D(12), h1 = D(15), h2 = D(16);
    const float2 em = sub2(e1, e2), gm = sub2(g1, g2), hm = sub2(h1, h2);
    const float2 ep = add2(e1, e2), gp = add2(g1, g2), hp = add2(h1, h2);
    const float2 jx = add2(em, gm), jy = add2(ep, hm), jz = add2(gp, hp);
    m[3] = add2(dx, jx);
    m[4] = fma2(bc2(-4.0f), dx, jx);
    m[5] = add2(dy, jy);
    m[6] = fma2(bc2(-4.0f), dy, jy);
    m[7] = add2(dz, jz);
    m[8] = fma2(bc2(-4.0f), dz, jz);
    m[16] = sub2(em, gm);
    m[17] = sub2(hm, ep);
    m[18] = sub2(hp, gp);
    const float2 r = m[0];
    rho = r;
    const float2 inv = make_float2(__frcp_rn(r.x), __frcp_rn(r.y)), hr = mul2(bc2(0.5f), r);
    const float* g = P.g;
    u[0] = mul2(forced ? fma2(hr, bc2(g[0]), m[3]) : m[3], inv);
    u[1] = mul2(forced ? fma2(hr, gy, m[5]) : m[5], inv);
    u[2] = mul2(forced ? fma2(hr, bc2(g[2]), m[7]) : m[7], inv);
    const float2 rx = mul2(r, u[0]), ry = mul2(r, u[1]), rz = mul2(r, u[2]);
    const float2 xx = mul2(rx, u[0]), yy = mul2(ry, u[1]), zz = mul2(rz, u[2]);
    const float2 qxy = mul2(rx, u[1]), qyz = mul2(ry, u[2]), qxz = mul2(rx, u[2]), ru2 = add2(add2(xx, yy), zz);
    float2 sn;  // minus the shear rate
    if constexpr (LES) {
        const float2 r3 = mul2(bc2(1.0f / 3.0f), r);
        const float2 t = smagorinsky_tau2(P, r, sub2(sub2(add2(add2(sx, xy), xz), r3), xx),
                                          sub2(sub2(add2(add2(sy, xy), yz), r3), yy),
                                          sub2(sub2(add2(add2(sz, xz), yz), r3), zz), sub2(m[13], qxy), sub2(m[14], qyz),
                                          sub2(m[15], qxz));
        sn = make_float2(-__frcp_rn(t.x), -__frcp_rn(t.y));
    } else {
        sn = bc2(-1.0f / P.tau);
    }
    // rates d3q19_collision_mrt.ispc:41-48; equilibria :119-138; forcing on j and q :141-148
    auto relax = [&](int k, float2 ms, float2 eq) { m[k] = fma2(ms, sub2(m[k], eq), m[k]); };
    relax(1, bc2(-1.0f / P.tau_bulk), fma2(bc2(19.0f), ru2, mul2(bc2(-11.0f), r)));
    relax(2, bc2(-1.4f), fma2(bc2(-5.5f), ru2, mul2(bc2(3.0f), r)));
    relax(4, bc2(-1.2f), mul2(bc2(-2.0f / 3.0f), rx));
    relax(6, bc2(-1.2f), mul2(bc2(-2.0f / 3.0f), ry));
    relax(8, bc2(-1.2f), mul2(bc2(-2.0f / 3.0f), rz));
    const float2 eq9 = sub2(sub2(add2(xx, xx), yy), zz), eq11 = sub2(yy, zz);
    relax(9, sn, eq9);
    relax(10, bc2(-1.4f), mul2(bc2(-0.5f), eq9));
    relax(11, sn, eq11);
    relax(12, bc2(-1.4f), mul2(bc2(-0.5f), eq11));
    relax(13, sn, qxy);
    relax(14, sn, qyz);
    relax(15, sn, qxz);
    for (int k = 16; k < 19; ++k) m[k] = mul2(bc2(1.0f - 1.98f), m[k]);
    if (forced) {
        const float2 F[3] = {mul2(r, bc2(g[0])), mul2(r, gy), mul2(r, bc2(g[2]))};
        for (int c = 0; c < 3; ++c) {
            m[3 + 2 * c] = add2(m[3 + 2 * c], F[c]);
            m[4 + 2 * c] = fma2(bc2(-2.0f / 3.0f), F[c], m[4 + 2 * c]);
        }
    }
    using Pairs = std::make_integer_sequence<int, 9>;
    if (P.mrt_exact) d3q19_inverse2<false>(f, m, Pairs{});
    else d3q19_inverse2<true>(f, m, Pairs{});
}

// D3Q27 raw-moment MRT (collide_mrt_d3q27) of two nodes without body force, in place: v = f - f_eq, its raw moments
// (three sweeps of nine 3-point transforms), the part that stays after relaxation, back, plus f_eq formed anew.
template <bool LES>
__device__ __forceinline__ void mrt27_pairs2(float2* f, const Physics& P, float2& rho, float2 u[3]) {
    using L = Lat<27>;
    float2 r = f[0], j[3] = {bc2(0.f), bc2(0.f), bc2(0.f)};
#pragma unroll
    for (int p = 0; p < 13; ++p) {
        const int q = pair_q<27>(p);
        const float2 d = sub2(f[q], f[L::opp(q)]);
        r = add2(r, add2(f[q], f[L::opp(q)]));
        j[0] = acc_c(j[0], L::cx(q), d);
        j[1] = acc_c(j[1], L::cy(q), d);
        j[2] = acc_c(j[2], L::cz(q), d);
    }
    rho = r;
    const float2 inv = make_float2(__frcp_rn(r.x), __frcp_rn(r.y));
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = mul2(j[a], inv);
    const float2 u2 = fma2(u[2], u[2], fma2(u[1], u[1], mul2(u[0], u[0])));
    const float2 ra0 = mul2(r, fma2(bc2(-1.5f), u2, bc2(1.0f)));
    float2 v[27];
    // even and odd part of a pair's equilibrium: w rho (1 - 1.5 u^2 + 4.5 (c.u)^2), 3 w rho (c.u)
    auto equilibrium = [&](int q, float2& even, float2& odd) {
        const int cx = L::cx(q), cy = L::cy(q), cz = L::cz(q);
        float2 cu = cx ? (cx > 0 ? u[0] : neg2(u[0])) : bc2(0.f);
        if (cy) cu = cx ? acc_c(cu, cy, u[1]) : (cy > 0 ? u[1] : neg2(u[1]));
        if (cz) cu = (cx || cy) ? acc_c(cu, cz, u[2]) : (cz > 0 ? u[2] : neg2(u[2]));
        even = fma2(mul2(mul2(bc2(4.5f * L::w(q)), r), cu), cu, mul2(bc2(L::w(q)), ra0));
        odd = mul2(mul2(bc2(3.0f * L::w(q)), r), cu);
    };
    v[d3q27_slot(0)] = sub2(f[0], mul2(bc2(L::w(0)), ra0));
#pragma unroll
    for (int p = 0; p < 13; ++p) {
        const int q = pair_q<27>(p), o = L::opp(q);
        float2 e, d;
        equilibrium(q, e, d);
        v[d3q27_slot(q)] = sub2(f[q], add2(e, d));
        v[d3q27_slot(o)] = sub2(f[o], sub2(e, d));
    }
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        const int st = axis == 0 ? 1 : (axis == 1 ? 3 : 9), o1 = axis == 0 ? 3 : 1, o2 = axis == 2 ? 3 : 9;
#pragma unroll
        for (int l = 0; l < 9; ++l) {
            const int b = (l % 3) * o1 + (l / 3) * o2;
            const float2 lo = v[b], mid = v[b + st], hi = v[b + 2 * st], sum = add2(hi, lo);
            v[b] = add2(sum, mid);
            v[b + st] = sub2(hi, lo);
            v[b + 2 * st] = sum;
        }
    }
    // what relaxation leaves: conserved moments, shear (1 - 1/tau), trace (1 - 1/tau_bulk), third order (1 - s3),
    // higher (1 - s4)
    float2 ks;
    if constexpr (LES) {
        const float2 t = smagorinsky_tau2(P, r, v[2], v[6], v[18], v[4], v[12], v[10]);
        ks = make_float2(1.0f - __frcp_rn(t.x), 1.0f - __frcp_rn(t.y));
    } else {
        ks = bc2(1.0f - 1.0f / P.tau);
    }
    const float2 kb = bc2(1.0f - 1.0f / P.tau_bulk), k3 = bc2(1.0f - P.s3), k4 = bc2(1.0f - P.s4);
#pragma unroll
    for (int k = 0; k < 27; ++k) {
        const int a = k % 3, b = (k / 3) % 3, c = k / 9, o = a + b + c;
        if (o == 2 && a < 2 && b < 2 && c < 2) v[k] = mul2(ks, v[k]);
        else if (o == 3) v[k] = mul2(k3, v[k]);
        else if (o > 3) v[k] = mul2(k4, v[k]);
    }
    const float2 T = mul2(kb, add2(add2(v[2], v[6]), v[18])), B = mul2(ks, sub2(v[2], v[6])), C = mul2(ks, sub2(v[2], v[18]));
    const float2 third = bc2(1.0f / 3.0f);
    v[2] = mul2(third, add2(add2(T, B), C));
    v[6] = mul2(third, fma2(bc2(-2.0f), B, add2(T, C)));
    v[18] = mul2(third, fma2(bc2(-2.0f), C, add2(T, B)));
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        const int st = axis == 0 ? 1 : (axis == 1 ? 3 : 9), o1 = axis == 0 ? 3 : 1, o2 = axis == 2 ? 3 : 9;
#pragma unroll
        for (int l = 0; l < 9; ++l) {
            const int b = (l % 3) * o1 + (l / 3) * o2;
            const float2 m0 = v[b], m1 = mul2(bc2(0.5f), v[b + st]), m2 = v[b + 2 * st];
            v[b] = fma2(bc2(0.5f), m2, neg2(m1));
            v[b + st] = sub2(m0, m2);
            v[b + 2 * st] = fma2(bc2(0.5f), m2, m1);
        }
    }
    f[0] = fma2(bc2(L::w(0)), ra0, v[d3q27_slot(0)]);
#pragma unroll
    for (int p = 0; p < 13; ++p) {
        const int q = pair_q<27>(p), o = L::opp(q);
        float2 e, d;
        equilibrium(q, e, d);
        f[q] = add2(v[d3q27_slot(q)], add2(e, d));
        f[o] = add2(v[d3q27_slot(o)], sub2(e, d));
    }
}

// How a model's nodes are computed. TRT: two per thread (trt_pairs2) where the node's row segment is all pure
// gathers, one per thread (collide) elsewhere. BGK and MRT on FP32 3D lattices: two per thread everywhere. The rest,
// and a coupled temperature: one per thread (16-bit populations would have to be decoded and encoded around the
// packed form, D2Q9 is bound by memory either way). Each rule gives one result for a node, whatever kernel steps it.
template <int Q, int COLL, int S>
__host__ __device__ constexpr bool all_pairs() {
    return COLL != COLL_TRT && S == STORE_F32 && Q != 9;
}
template <int Q, int COLL, int S>
__host__ __device__ constexpr bool pure_pairs() {
    return COLL == COLL_TRT || all_pairs<Q, COLL, S>();
}

template <int Q, int COLL, int S, bool LES>
__device__ __forceinline__ void collide_pairs2(float2* f, const Physics& P, const float2 gy, const bool forced, float2& rho,
                                               float2 u[3]) {
    if constexpr (COLL == COLL_TRT) {
        trt_pairs2<Q, LES, S != STORE_F32>(f, P, gy, forced, rho, u);
    } else if constexpr (COLL == COLL_BGK) {
        bgk_pairs2<Q, LES>(f, P, gy, forced, rho, u);
    } else if constexpr (Q == 19) {
        mrt19_pairs2<LES>(f, P, gy, forced, rho, u);
    } else {
        if (!forced) {
            mrt27_pairs2<LES>(f, P, rho, u);
            return;
        }
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {  // with a body force, one node after the other
            float t[27], rh, uh[3];
#pragma unroll
            for (int q = 0; q < 27; ++q) t[q] = h ? f[q].y : f[q].x;
            node_moments<27>(t, P.g, rh, uh);
            collide<27, COLL_MRT, LES>(t, rh, uh, P);
#pragma unroll
            for (int q = 0; q < 27; ++q) (h ? f[q].y : f[q].x) = t[q];
            (h ? rho.y : rho.x) = rh;
            for (int a = 0; a < 3; ++a) (h ? u[a].y : u[a].x) = uh[a];
        }
    }
}

// The same with the uniform body force P.g.
template <int Q, bool LES, bool HS>
__device__ __forceinline__ void trt_pairs2(float2* f, const Physics& P, float2& rho, float2 u[3]) {
    trt_pairs2<Q, LES, HS>(f, P, bc2(P.g[1]), P.g[0] != 0.0f || P.g[1] != 0.0f || P.g[2] != 0.0f, rho, u);
}

}  // namespace wk
