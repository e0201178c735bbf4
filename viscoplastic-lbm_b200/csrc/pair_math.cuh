// pair_math.cuh -- the arithmetic of the half-precision step, for one node
// (float) or for two at once (float2).  (FP32 storage: step_math_f32.cuh.)
//
// The z-paired kernel (k_step2) holds the nodes (x, y, z) and (x, y, z + NZ/2)
// in the two lanes of float2 values and evaluates moments, stress magnitude
// and collision with sm_100's packed FP32x2 instructions (FFMA2 / FADD2 /
// FMUL2: two FP32 operations per issued instruction); the one-node kernel uses
// the same functions on floats.  All work on deviations g_i = f_i - w_i rho0.
//
// The half-precision step is limited by instruction issue, not by HBM, so the
// sums are shared: opposite populations enter as e = g_i + g_opp and o = g_i -
// g_opp; the two diagonals of a coordinate plane (7/8 and 13/14 for xy) share
// their sum, which goes to rho and two second moments, and the collision
// writes each population as (E + O) or (E - O) with
//     E = K + sum_ab c_a c_b T_ab,     O = sum_a c_a V_a,
// the tensor T and the vector V being formed once per node instead of c.u, c.F
// and c_a c_b Pi_ab once per population pair.  D3Q19 regularized: about 160
// packed operations per node pair instead of 230, D3Q27 210 instead of 350.
// FP16 Bingham, steps and one read-out: 256^3 D3Q19 (20 steps) 5.89 -> 5.42 ms,
// 256x128x64 (50) 1.86 -> 1.72 ms, D3Q27 144x56x56 duct (100) 1.43 -> 1.27 ms.
#pragma once
#include <cuda_runtime.h>
#include "internal.h"
#include "lattice.cuh"

namespace vlbm {

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(__frcp_rn(a.x), __frcp_rn(a.y)); }
// One node: the same roundings as a lane of the packed operations (no
// contraction).
__device__ __forceinline__ float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub2(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul2(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float rcp2(float a) { return __frcp_rn(a); }
template <class F> __device__ __forceinline__ F vs(float a);   // a in every lane
template <> __device__ __forceinline__ float vs<float>(float a) { return a; }
template <> __device__ __forceinline__ float2 vs<float2>(float a) { return f2(a); }
__device__ __forceinline__ float lane_of(const float2& v, int lane) { return lane ? v.y : v.x; }
__device__ __forceinline__ void set_lane(float2& v, int lane, float a) {
    if (lane) v.y = a; else v.x = a;
}

// Moments of a node: rho, u (with half force, lbm.cu:79-111), non-equilibrium
// second moments (lbm.cu:149-190).
template <class F>
struct MomT {
    F rho, drho, ux, uy, uz;
    F jx, jy, jz;               // sum c g
    F hx, hy, hz;               // rho u = j + F / 2
    F pxx, pyy, pzz, pxy, pxz, pyz;
};
using Mom = MomT<float>;
using Mom2 = MomT<float2>;

// Moments of the deviations g_i = f_i - w_i rho0: rho = rho0 + sum g,
// rho u = sum c g + F/2, and the non-equilibrium second moments
// Pi_ab = sum c_a c_b f - rho (u_a u_b + delta_ab / 3)
//       = sum c_a c_b g - rho u_a u_b - delta_ab (rho - rho0) / 3.
//
// SCALED: g holds the stored half-precision values, deviations times a power
// of two (1 / inv_scale); the ten sums are scaled back instead of the Q
// populations, which gives the same bits (a power-of-two scale is exact).
//
// The reciprocal is correctly rounded: u = j/rho enters every equilibrium, and
// a biased approximate reciprocal (the hardware result is within 2 ulp but not
// unbiased) acts like a spurious force proportional to the momentum, which
// shifts a slow channel flow by ~1e-3 over 1e4 steps.
template <int Q, bool NEED_PI, bool SCALED, class F>
__device__ __forceinline__ MomT<F> moments_of(const F (&g)[Q], F fx, F fy, F fz, float rho0, float inv_scale) {
    MomT<F> m;
    // axis pairs 1/2, 3/4, 5/6
    const F ex = add2(g[1], g[2]), ey = add2(g[3], g[4]), ez = add2(g[5], g[6]);
    F jx = sub2(g[1], g[2]), jy = sub2(g[3], g[4]), jz = sub2(g[5], g[6]);
    F sxy, sxz, syz, exy, exz, eyz;   // per coordinate plane: c_a c_b sum and plain sum of its diagonals
    {
        const F ep = add2(g[7], g[8]), em = add2(g[13], g[14]);      // (1,1,0), (1,-1,0)
        const F op = sub2(g[7], g[8]), om = sub2(g[13], g[14]);
        sxy = sub2(ep, em); exy = add2(ep, em);
        jx = add2(jx, add2(op, om)); jy = add2(jy, sub2(op, om));
    }
    {
        const F ep = add2(g[9], g[10]), em = add2(g[15], g[16]);     // (1,0,1), (1,0,-1)
        const F op = sub2(g[9], g[10]), om = sub2(g[15], g[16]);
        sxz = sub2(ep, em); exz = add2(ep, em);
        jx = add2(jx, add2(op, om)); jz = add2(jz, sub2(op, om));
    }
    {
        const F ep = add2(g[11], g[12]), em = add2(g[17], g[18]);    // (0,1,1), (0,1,-1)
        const F op = sub2(g[11], g[12]), om = sub2(g[17], g[18]);
        syz = sub2(ep, em); eyz = add2(ep, em);
        jy = add2(jy, add2(op, om)); jz = add2(jz, sub2(op, om));
    }
    F rho = add2(add2(add2(ex, ey), ez), add2(add2(exy, exz), eyz));
    F sxx = add2(ex, add2(exy, exz)), syy = add2(ey, add2(exy, eyz)), szz = add2(ez, add2(exz, eyz));
    if constexpr (Q == 27) {   // (1,1,1), (1,1,-1), (1,-1,1), (-1,1,1)
        const F e0 = add2(g[19], g[20]), e1 = add2(g[21], g[22]), e2 = add2(g[23], g[24]), e3 = add2(g[25], g[26]);
        const F o0 = sub2(g[19], g[20]), o1 = sub2(g[21], g[22]), o2 = sub2(g[23], g[24]), o3 = sub2(g[25], g[26]);
        const F a = add2(e0, e1), b = add2(e2, e3), c = sub2(e0, e1), d = sub2(e2, e3), all = add2(a, b);
        rho = add2(rho, all);
        sxx = add2(sxx, all); syy = add2(syy, all); szz = add2(szz, all);
        sxy = add2(sxy, sub2(a, b)); sxz = add2(sxz, add2(c, d)); syz = add2(syz, sub2(c, d));
        const F p = add2(o0, o1), q = sub2(o2, o3);
        jx = add2(jx, add2(p, q)); jy = add2(jy, sub2(p, q));
        jz = add2(jz, add2(sub2(o0, o1), add2(o2, o3)));
    }
    rho = add2(rho, g[0]);
    if (SCALED) {
        const F k = vs<F>(inv_scale);
        rho = mul2(rho, k);
        jx = mul2(jx, k); jy = mul2(jy, k); jz = mul2(jz, k);
        if (NEED_PI) {
            sxx = mul2(sxx, k); syy = mul2(syy, k); szz = mul2(szz, k);
            sxy = mul2(sxy, k); sxz = mul2(sxz, k); syz = mul2(syz, k);
        }
    }
    m.drho = rho;
    rho = add2(rho, vs<F>(rho0));
    m.rho = rho;
    const F inv = rcp2(rho), h = vs<F>(0.5f);
    m.jx = jx; m.jy = jy; m.jz = jz;
    m.hx = fma2(fx, h, jx);
    m.hy = fma2(fy, h, jy);
    m.hz = fma2(fz, h, jz);
    m.ux = mul2(m.hx, inv);
    m.uy = mul2(m.hy, inv);
    m.uz = mul2(m.hz, inv);
    if (NEED_PI) {
        const F rux = mul2(m.hx, vs<F>(-1.f)), ruy = mul2(m.hy, vs<F>(-1.f)), ruz = mul2(m.hz, vs<F>(-1.f));
        const F dr3 = mul2(m.drho, vs<F>(1.f / 3.f));
        m.pxx = fma2(rux, m.ux, sub2(sxx, dr3));
        m.pyy = fma2(ruy, m.uy, sub2(syy, dr3));
        m.pzz = fma2(ruz, m.uz, sub2(szz, dr3));
        m.pxy = fma2(rux, m.uy, sxy);
        m.pxz = fma2(rux, m.uz, sxz);
        m.pyz = fma2(ruy, m.uz, syz);
    } else {
        m.pxx = m.pyy = m.pzz = m.pxy = m.pxz = m.pyz = vs<F>(0.f);
    }
    return m;
}
template <int Q, bool NEED_PI>
__device__ __forceinline__ Mom moments(const float (&f)[Q], float fx, float fy, float fz, float rho0) {
    return moments_of<Q, NEED_PI, false, float>(f, fx, fy, fz, rho0, 1.f);
}
template <int Q, bool NEED_PI, bool SCALED = false>
__device__ __forceinline__ Mom2 moments2(const float2 (&g)[Q], float2 fx, float2 fy, float2 fz, float rho0,
                                         float inv_scale = 1.f) {
    return moments_of<Q, NEED_PI, SCALED, float2>(g, fx, fy, fz, rho0, inv_scale);
}

// The squared stress magnitude |S|^2 = S_ab S_ab / 2 of the rheology models, with
// the force correction (lbm.cu:192-208), and its square root: the hardware
// reciprocal square root (<= 2 ulp).
template <class F>
__device__ __forceinline__ F stress_square(const MomT<F>& m, F fx, F fy, F fz) {
    const F a = fma2(m.ux, fx, m.pxx), b = fma2(m.uy, fy, m.pyy), c = fma2(m.uz, fz, m.pzz);
    const F h = vs<F>(0.5f);
    const F d = fma2(h, fma2(m.ux, fy, mul2(m.uy, fx)), m.pxy);
    const F e = fma2(h, fma2(m.ux, fz, mul2(m.uz, fx)), m.pxz);
    const F k = fma2(h, fma2(m.uy, fz, mul2(m.uz, fy)), m.pyz);
    const F off = fma2(d, d, fma2(e, e, mul2(k, k)));
    return mul2(h, fma2(a, a, fma2(b, b, fma2(c, c, add2(off, off)))));
}
__device__ __forceinline__ float root_of(float q) { return q > 0.f ? q * rsqrtf(q) : 0.f; }
__device__ __forceinline__ float stress_aux(const Mom& m, float fx, float fy, float fz) {
    return root_of(stress_square<float>(m, fx, fy, fz));
}
__device__ __forceinline__ float2 stress_aux2(const Mom2& m, float2 fx, float2 fy, float2 fz) {
    const float2 q = stress_square<float2>(m, fx, fy, fz);
    return make_float2(root_of(q.x), root_of(q.y));
}

// Collision in place on deviations:
//  regularized (lbm.cu:263-461):
//    f*_i = w_i [ A (Q_i:Pi - c_i.F/3) + rho(1 - 1.5u^2 + 3cu + 4.5cu^2) + B(3(c_i-u).F + 9 cu cF) ]
//    A = 4.5(1-omega), B = 1-omega/2
//  BGK (collisionForceNoReg.txt): f*_i = (1-omega) f_i + omega f_eq_i + B F_i
// The rest part w_i rho0 is not formed (for BGK (1 - omega) w rho0 + omega w
// rho0 cancels against it).
//
// Odd part: V = 3 w (rho u + F/2), since 3B - A/3 = 3/2 for every omega; BGK:
// 3 w (omega rho u + B F).  Even part: with q = 3/2 V + (6.75 - 4.5 omega) w F
// (BGK: 4.5 w B F), which is 4.5 w rho u + 9 w B F,
//    T_aa = w A Pi_aa + u_a q_a,  T_ab + T_ba = 2 w A Pi_ab + u_a q_b + u_b q_a,
//    K = w (rho - rho0) - tr(T) / 3   (the -1.5 rho u^2, -3 B u.F and -A tr(Pi)/3
// of the formula; taken from T itself, so that they cancel in the sum over the
// populations).  w is the weight of the face diagonals; axis, body and rest
// weights differ from it by a power of two (and D3Q19's rest by 12).
//
// A slow body-force flow (u / F ~ 1e4) shows every rounding that has the same
// sign at all nodes and steps: it acts as a force along the momentum.  So the
// constants 3 w and 1/3 are products with their exact value (a second term
// carries what rounding the constant leaves).  The half force enters the
// regularized V as F minus what rounding j + F/2 has added already, and drops
// out of BGK's: omega rho u + B F = omega j + F.  FP16 storage, 256x128x64
// Bingham channel after 50,000 steps, velocity against 64 bits at yield stresses
// of 1.1e-6, 5.3e-6 and 4.7e-5: regularized D3Q19 1.7e-4, 1.7e-4, 1.7e-4 (7.2e-4,
// 7.0e-4, 3.5e-4 with the formula evaluated per population), D3Q27 1.5e-4, 1.5e-4,
// 1.6e-4 (7.2e-4, 6.9e-4, 3.5e-4); BGK D3Q19 1.3e-4, 2.3e-4 (7.6e-4, 6.9e-4) and
// 5.9e-3 (5.7e-3) at the largest, where the plug hardly relaxes and keeps the
// noise of the stores.  The D3Q19 one-node BGK step takes 21.4 us for Bingham and
// 24.5 for Power-Law on 96x90x91 nodes, 21.5 and 25.3 with the half force in omega
// h + omega (F - (h - j)) + (1 - omega) F.
//
// `gscale` is what the incoming g must be multiplied by to be deviations
// (inv_scale for stored half values, 1 otherwise); the result is deviations
// times `oscale` (the storage scale for half storage, 1 otherwise).  Both are
// powers of two, folded into the weights and BGK's (1 - omega) factor, which
// gives the same bits as scaling before and after.
template <int Q, int OP, class F>
__device__ __forceinline__ void collide_of(F (&g)[Q], const MomT<F>& m, F omega, F fx, F fy, F fz, float gscale,
                                           float oscale) {
    constexpr bool REG = OP == VLBM_OP_REGULARIZED;
    constexpr float AXIS = Q == 27 ? 4.f : 2.f, REST = Q == 27 ? 16.f : 12.f, BODY = 0.25f;
    const float w = Lattice<Q>::w(7) * oscale;
    constexpr float W3 = (float)(3.0 * Lattice<Q>::wd(7)), W3LO = (float)(3.0 * Lattice<Q>::wd(7) - (double)W3);
    const F w3 = vs<F>(W3 * oscale), w3lo = vs<F>(W3LO * oscale);
    F Vx, Vy, Vz, cq, A, A2, om1 = vs<F>(0.f);
    if constexpr (REG) {
        // F minus the half force as it was rounded into h
        const F ex = sub2(fx, sub2(m.hx, m.jx)), ey = sub2(fy, sub2(m.hy, m.jy)), ez = sub2(fz, sub2(m.hz, m.jz));
        Vx = fma2(m.hx, w3, fma2(ex, w3, mul2(m.hx, w3lo)));
        Vy = fma2(m.hy, w3, fma2(ey, w3, mul2(m.hy, w3lo)));
        Vz = fma2(m.hz, w3, fma2(ez, w3, mul2(m.hz, w3lo)));
        cq = fma2(omega, vs<F>(-4.5f * w), vs<F>(6.75f * w));
        A = fma2(omega, vs<F>(-4.5f * w), vs<F>(4.5f * w));
        A2 = add2(A, A);
    } else {   // the half force drops out: omega rho u + B F = omega j + F
        const F ow = mul2(omega, w3);
        const F owlo = fma2(omega, w3lo, fma2(omega, w3, mul2(ow, vs<F>(-1.f))));   // what rounding 3 w omega leaves
        Vx = fma2(m.jx, ow, fma2(fx, w3, mul2(m.jx, owlo)));
        Vy = fma2(m.jy, ow, fma2(fy, w3, mul2(m.jy, owlo)));
        Vz = fma2(m.jz, ow, fma2(fz, w3, mul2(m.jz, owlo)));
        cq = fma2(omega, vs<F>(-2.25f * w), vs<F>(4.5f * w));
        om1 = mul2(sub2(vs<F>(1.f), omega), vs<F>(gscale * oscale));
    }
    const F c15 = vs<F>(1.5f);
    const F qx = fma2(Vx, c15, mul2(cq, fx)), qy = fma2(Vy, c15, mul2(cq, fy)), qz = fma2(Vz, c15, mul2(cq, fz));
    F Txy = mul2(m.uy, qx), Txz = mul2(m.uz, qx), Tyz = mul2(m.uz, qy);
    F Txx, Tyy, Tzz;
    if constexpr (REG) {
        Txx = fma2(A, m.pxx, mul2(m.ux, qx)); Tyy = fma2(A, m.pyy, mul2(m.uy, qy));
        Tzz = fma2(A, m.pzz, mul2(m.uz, qz));
        Txy = fma2(A2, m.pxy, Txy); Txz = fma2(A2, m.pxz, Txz); Tyz = fma2(A2, m.pyz, Tyz);
    }
    // v + T_aa.  BGK's T_aa is a bare product: the sum is written as a fused
    // operation, because the compiler may fuse a packed product and sum by itself
    auto plus_t = [&](F v, int a) {
        if constexpr (REG) return add2(v, a == 0 ? Txx : (a == 1 ? Tyy : Tzz));
        else return a == 0 ? fma2(m.ux, qx, v) : (a == 1 ? fma2(m.uy, qy, v) : fma2(m.uz, qz, v));
    };
    Txy = fma2(m.ux, qy, Txy); Txz = fma2(m.ux, qz, Txz); Tyz = fma2(m.uy, qz, Tyz);
    constexpr float T3 = -1.f / 3.f, T3LO = (float)(-1.0 / 3.0 - (double)T3);
    if constexpr (!REG) Txx = mul2(m.ux, qx);
    const F tr = plus_t(plus_t(Txx, 1), 2);
    const F K = fma2(tr, vs<F>(T3), fma2(tr, vs<F>(T3LO), mul2(REG ? m.drho : mul2(omega, m.drho), vs<F>(w))));
    if constexpr (REG) g[0] = mul2(K, vs<F>(REST));
    else g[0] = fma2(om1, g[0], mul2(K, vs<F>(REST)));
    // populations i and i + 1 = opp(i) from the even part E and the odd part O
    auto put = [&](int i, F E, F O) {
        if constexpr (REG) {
            g[i] = add2(E, O);
            g[i + 1] = sub2(E, O);
        } else {
            g[i] = fma2(om1, g[i], add2(E, O));
            g[i + 1] = fma2(om1, g[i + 1], sub2(E, O));
        }
    };
    const F Kx = plus_t(K, 0), Ky = plus_t(K, 1), Kz = plus_t(K, 2);
    const F ax = vs<F>(AXIS);
    put(1, mul2(Kx, ax), mul2(Vx, ax));
    put(3, mul2(Ky, ax), mul2(Vy, ax));
    put(5, mul2(Kz, ax), mul2(Vz, ax));
    const F Exy = plus_t(Kx, 1), Exz = plus_t(Kx, 2), Eyz = plus_t(Ky, 2);
    const F Vp = add2(Vx, Vy), Vm = sub2(Vx, Vy);
    put(7, add2(Exy, Txy), Vp);
    put(13, sub2(Exy, Txy), Vm);
    put(9, add2(Exz, Txz), add2(Vx, Vz));
    put(15, sub2(Exz, Txz), sub2(Vx, Vz));
    put(11, add2(Eyz, Tyz), add2(Vy, Vz));
    put(17, sub2(Eyz, Tyz), sub2(Vy, Vz));
    if constexpr (Q == 27) {
        const F bd = vs<F>(BODY);
        const F E = mul2(plus_t(Exy, 2), bd), Sxy = mul2(Txy, bd);
        const F p = mul2(add2(Txz, Tyz), bd), q = mul2(sub2(Txz, Tyz), bd);
        const F b1 = add2(E, Sxy), b2 = sub2(E, Sxy);
        const F vp = mul2(Vp, bd), vm = mul2(Vm, bd), vz = mul2(Vz, bd);
        put(19, add2(b1, p), add2(vp, vz));      // (1,1,1)
        put(21, sub2(b1, p), sub2(vp, vz));      // (1,1,-1)
        put(23, add2(b2, q), add2(vm, vz));      // (1,-1,1)
        put(25, sub2(b2, q), sub2(vz, vm));      // (-1,1,1)
    }
}
template <int Q, int OP>
__device__ __forceinline__ void collide(float (&f)[Q], const Mom& m, float omega, float fx, float fy, float fz) {
    collide_of<Q, OP, float>(f, m, omega, fx, fy, fz, 1.f, 1.f);
}
template <int Q, int OP>
__device__ __forceinline__ void collide2(float2 (&g)[Q], const Mom2& m, float2 omega, float2 fx, float2 fy,
                                         float2 fz, float gscale = 1.f, float oscale = 1.f) {
    collide_of<Q, OP, float2>(g, m, omega, fx, fy, fz, gscale, oscale);
}

}  // namespace vlbm
