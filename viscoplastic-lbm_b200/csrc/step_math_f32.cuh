// step_math_f32.cuh -- the step's arithmetic for FP32 storage, evaluated per
// population pair: one node (scalars) and two nodes (packed FP32x2).
//
// The shared sums of pair_math.cuh would make the FP32 step 3 to 5 % faster (with
// the layouts as they are, 50 steps of the 256x128x64 D3Q19 Bingham channel 2.80 ->
// 2.66 ms, 20 steps of the 256^3 D3Q27 Power-Law cavity 15.6 -> 15.0 ms) and bring
// it closer to 64 bits.  It keeps these so that FP32 results stay those it has
// always had, to the bit: a quantity that nearly cancels, such as the mean of a
// wave over a plane, differs between the two by 1e-4 of itself after 150 steps.
#pragma once
#include <cuda_runtime.h>
#include "internal.h"
#include "lattice.cuh"
#include "pair_math.cuh"

namespace vlbm {
namespace f32 {

template <int Q, bool NEED_PI>
__device__ __forceinline__ Mom moments(const float (&f)[Q], float fx, float fy, float fz, float rho0) {
    // Sums over opposite pairs: e = g_i + g_opp feeds the even moments (rho,
    // second moments), o = g_i - g_opp the odd ones (momentum).
    Mom m;
    float rho = f[0], jx = 0.f, jy = 0.f, jz = 0.f;
    float sxx = 0.f, syy = 0.f, szz = 0.f, sxy = 0.f, sxz = 0.f, syz = 0.f;
#pragma unroll
    for (int i = 1; i < Q; i += 2) {
        const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
        const float e = f[i] + f[i + 1], o = f[i] - f[i + 1];
        rho += e;
        if (cx) jx += cx * o;
        if (cy) jy += cy * o;
        if (cz) jz += cz * o;
        if (NEED_PI) {
            if (cx) sxx += e;
            if (cy) syy += e;
            if (cz) szz += e;
            if (cx && cy) sxy += cx * cy * e;
            if (cx && cz) sxz += cx * cz * e;
            if (cy && cz) syz += cy * cz * e;
        }
    }
    // correctly rounded reciprocal: u = j/rho enters every equilibrium, and a
    // biased approximate reciprocal (the hardware MUFU result is within 2 ulp
    // but not unbiased) acts like a spurious force proportional to the
    // momentum, which shifts a slow channel flow by ~1e-3 over 1e4 steps
    const float drho = rho;
    rho += rho0;
    const float inv = __frcp_rn(rho);
    m.rho = rho;
    m.drho = drho;
    m.ux = (jx + 0.5f * fx) * inv;
    m.uy = (jy + 0.5f * fy) * inv;
    m.uz = (jz + 0.5f * fz) * inv;
    if (NEED_PI) {
        const float dr3 = drho * (1.f / 3.f);
        m.pxx = sxx - rho * m.ux * m.ux - dr3;
        m.pyy = syy - rho * m.uy * m.uy - dr3;
        m.pzz = szz - rho * m.uz * m.uz - dr3;
        m.pxy = sxy - rho * m.ux * m.uy;
        m.pxz = sxz - rho * m.ux * m.uz;
        m.pyz = syz - rho * m.uy * m.uz;
    } else {
        m.pxx = m.pyy = m.pzz = m.pxy = m.pxz = m.pyz = 0.f;
    }
    return m;
}

__device__ __forceinline__ float stress_aux(const Mom& m, float fx, float fy, float fz) {
    const float a = m.pxx + m.ux * fx, b = m.pyy + m.uy * fy, c = m.pzz + m.uz * fz;
    const float d = m.pxy + 0.5f * (m.ux * fy + m.uy * fx);
    const float e = m.pxz + 0.5f * (m.ux * fz + m.uz * fx);
    const float g = m.pyz + 0.5f * (m.uy * fz + m.uz * fy);
    const float q = 0.5f * (a * a + b * b + c * c + 2.f * (d * d + e * e + g * g));
    return q > 0.f ? q * rsqrtf(q) : 0.f;  // hardware reciprocal square root (<= 2 ulp)
}

template <int Q, int OP>
__device__ __forceinline__ void collide(float (&f)[Q], const Mom& m, float omega, float fx, float fy, float fz) {
    // Populations i (odd index) and opp(i) = i+1 have opposite velocities: they
    // share Q_i:Pi, while c.u and c.F change sign.  Each pair is evaluated as an
    // even part E and an odd part O with f*_i = w (E + O), f*_opp = w (E - O).
    const float B = 1.f - 0.5f * omega;
    const float uu = m.ux * m.ux + m.uy * m.uy + m.uz * m.uz;
    const float uF = m.ux * fx + m.uy * fy + m.uz * fz;
    if (OP == VLBM_OP_REGULARIZED) {
        const float A = 4.5f * (1.f - omega);
        const float tr = (m.pxx + m.pyy + m.pzz) * (1.f / 3.f);
        // the rest part w_i rho0 is not formed: K0 is the deviation of rho(1 - 1.5 u^2)
        const float K0 = m.drho - 1.5f * m.rho * uu - 3.f * B * uF - A * tr;
        const float alpha = 3.f * B - A * (1.f / 3.f);
        const float r3 = 3.f * m.rho, r45 = 4.5f * m.rho, b9 = 9.f * B;
        f[0] = Lattice<Q>::w(0) * K0;
        // coefficients with the weight of each velocity class folded in
        float cK[3], cA[3], cr45[3], cb9[3], cal[3], cr3[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // representative population of the class: 1 (axis), 7 (face), 19 (body, D3Q27 only)
            const float w = Lattice<Q>::w(k == 0 ? 1 : (k == 1 ? 7 : (Q == 27 ? 19 : 1)));
            cK[k] = w * K0; cA[k] = w * A; cr45[k] = w * r45; cb9[k] = w * b9; cal[k] = w * alpha; cr3[k] = w * r3;
        }
        const float pxy2 = 2.f * m.pxy, pxz2 = 2.f * m.pxz, pyz2 = 2.f * m.pyz;
#pragma unroll
        for (int i = 1; i < Q; i += 2) {
            const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
            const int k = lat_norm1(i) - 1;   // 0 axis, 1 face diagonal, 2 body diagonal
            float S = 0.f, cu = 0.f, cF = 0.f;
            if (cx) { S += m.pxx; cu += cx * m.ux; cF += cx * fx; }
            if (cy) { S += m.pyy; cu += cy * m.uy; cF += cy * fy; }
            if (cz) { S += m.pzz; cu += cz * m.uz; cF += cz * fz; }
            if (cx && cy) S += cx * cy * pxy2;
            if (cx && cz) S += cx * cz * pxz2;
            if (cy && cz) S += cy * cz * pyz2;
            const float E = cK[k] + cA[k] * S + cu * (cr45[k] * cu + cb9[k] * cF);
            const float O = cal[k] * cF + cr3[k] * cu;
            f[i] = E + O;
            f[i + 1] = E - O;
        }
    } else {
        const float om1 = 1.f - omega;
        // on deviations: (1 - omega) w rho0 + omega w rho0 cancels against w rho0
        const float base = omega * (m.drho - 1.5f * m.rho * uu) - 3.f * B * uF;
        const float r45 = 4.5f * omega * m.rho, r3 = 3.f * omega * m.rho, b9 = 9.f * B, b3 = 3.f * B;
        f[0] = om1 * f[0] + Lattice<Q>::w(0) * base;
#pragma unroll
        for (int i = 1; i < Q; i += 2) {
            const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
            float cu = 0.f, cF = 0.f;
            if (cx) { cu += cx * m.ux; cF += cx * fx; }
            if (cy) { cu += cy * m.uy; cF += cy * fy; }
            if (cz) { cu += cz * m.uz; cF += cz * fz; }
            const float w = Lattice<Q>::w(i);
            const float E = w * (base + cu * (r45 * cu + b9 * cF));
            const float O = w * (r3 * cu + b3 * cF);
            f[i] = om1 * f[i] + (E + O);
            f[i + 1] = om1 * f[i + 1] + (E - O);
        }
    }
}

template <int Q, bool NEED_PI>
__device__ __forceinline__ Mom2 moments2(const float2 (&g)[Q], float2 fx, float2 fy, float2 fz, float rho0) {
    Mom2 m;
    float2 rho = g[0], jx = f2(0.f), jy = f2(0.f), jz = f2(0.f);
    float2 sxx = f2(0.f), syy = f2(0.f), szz = f2(0.f), sxy = f2(0.f), sxz = f2(0.f), syz = f2(0.f);
#pragma unroll
    for (int i = 1; i < Q; i += 2) {
        const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
        const float2 e = add2(g[i], g[i + 1]), o = sub2(g[i], g[i + 1]);
        rho = add2(rho, e);
        if (cx > 0) jx = add2(jx, o); else if (cx < 0) jx = sub2(jx, o);
        if (cy > 0) jy = add2(jy, o); else if (cy < 0) jy = sub2(jy, o);
        if (cz > 0) jz = add2(jz, o); else if (cz < 0) jz = sub2(jz, o);
        if (NEED_PI) {
            if (cx) sxx = add2(sxx, e);
            if (cy) syy = add2(syy, e);
            if (cz) szz = add2(szz, e);
            if (cx && cy) sxy = (cx * cy > 0) ? add2(sxy, e) : sub2(sxy, e);
            if (cx && cz) sxz = (cx * cz > 0) ? add2(sxz, e) : sub2(sxz, e);
            if (cy && cz) syz = (cy * cz > 0) ? add2(syz, e) : sub2(syz, e);
        }
    }
    m.drho = rho;
    rho = add2(rho, f2(rho0));
    m.rho = rho;
    const float2 inv = make_float2(__frcp_rn(rho.x), __frcp_rn(rho.y));
    m.ux = mul2(fma2(fx, f2(0.5f), jx), inv);
    m.uy = mul2(fma2(fy, f2(0.5f), jy), inv);
    m.uz = mul2(fma2(fz, f2(0.5f), jz), inv);
    if (NEED_PI) {
        const float2 rn = mul2(rho, f2(-1.f));
        const float2 rux = mul2(rn, m.ux), ruy = mul2(rn, m.uy), ruz = mul2(rn, m.uz);
        const float2 dr3 = mul2(m.drho, f2(1.f / 3.f));
        m.pxx = fma2(rux, m.ux, sub2(sxx, dr3));
        m.pyy = fma2(ruy, m.uy, sub2(syy, dr3));
        m.pzz = fma2(ruz, m.uz, sub2(szz, dr3));
        m.pxy = fma2(rux, m.uy, sxy);
        m.pxz = fma2(rux, m.uz, sxz);
        m.pyz = fma2(ruy, m.uz, syz);
    } else {
        m.pxx = m.pyy = m.pzz = m.pxy = m.pxz = m.pyz = f2(0.f);
    }
    return m;
}

__device__ __forceinline__ float2 stress_aux2(const Mom2& m, float2 fx, float2 fy, float2 fz) {
    const float2 a = fma2(m.ux, fx, m.pxx), b = fma2(m.uy, fy, m.pyy), c = fma2(m.uz, fz, m.pzz);
    const float2 h = f2(0.5f);
    const float2 d = fma2(h, fma2(m.ux, fy, mul2(m.uy, fx)), m.pxy);
    const float2 e = fma2(h, fma2(m.ux, fz, mul2(m.uz, fx)), m.pxz);
    const float2 k = fma2(h, fma2(m.uy, fz, mul2(m.uz, fy)), m.pyz);
    const float2 off = fma2(d, d, fma2(e, e, mul2(k, k)));
    const float2 q = mul2(h, fma2(a, a, fma2(b, b, fma2(c, c, add2(off, off)))));
    return make_float2(q.x > 0.f ? q.x * rsqrtf(q.x) : 0.f, q.y > 0.f ? q.y * rsqrtf(q.y) : 0.f);
}

template <int Q, int OP>
__device__ __forceinline__ void collide2(float2 (&g)[Q], const Mom2& m, float2 omega, float2 fx, float2 fy,
                                         float2 fz) {
    const float2 B = fma2(omega, f2(-0.5f), f2(1.f));
    const float2 uu = fma2(m.ux, m.ux, fma2(m.uy, m.uy, mul2(m.uz, m.uz)));
    const float2 uF = fma2(m.ux, fx, fma2(m.uy, fy, mul2(m.uz, fz)));
    const float2 BuF = mul2(B, uF);
    if (OP == VLBM_OP_REGULARIZED) {
        const float2 A = fma2(omega, f2(-4.5f), f2(4.5f));
        const float2 tr = mul2(add2(add2(m.pxx, m.pyy), m.pzz), f2(1.f / 3.f));
        float2 K0 = fma2(mul2(m.rho, uu), f2(-1.5f), m.drho);
        K0 = fma2(BuF, f2(-3.f), K0);
        K0 = sub2(K0, mul2(A, tr));
        const float2 alpha = fma2(B, f2(3.f), mul2(A, f2(-1.f / 3.f)));
        const float2 r3 = mul2(m.rho, f2(3.f)), r45 = mul2(m.rho, f2(4.5f)), b9 = mul2(B, f2(9.f));
        const float2 pxy2 = add2(m.pxy, m.pxy), pxz2 = add2(m.pxz, m.pxz), pyz2 = add2(m.pyz, m.pyz);
        g[0] = mul2(f2(Lattice<Q>::w(0)), K0);
#pragma unroll
        for (int i = 1; i < Q; i += 2) {
            const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
            float2 S = f2(0.f), cu = f2(0.f), cF = f2(0.f);
            bool first = true;
            if (cx) { S = m.pxx; first = false; cu = cx > 0 ? m.ux : mul2(m.ux, f2(-1.f)); cF = cx > 0 ? fx : mul2(fx, f2(-1.f)); }
            if (cy) {
                S = first ? m.pyy : add2(S, m.pyy);
                cu = first ? (cy > 0 ? m.uy : mul2(m.uy, f2(-1.f))) : (cy > 0 ? add2(cu, m.uy) : sub2(cu, m.uy));
                cF = first ? (cy > 0 ? fy : mul2(fy, f2(-1.f))) : (cy > 0 ? add2(cF, fy) : sub2(cF, fy));
                first = false;
            }
            if (cz) {
                S = first ? m.pzz : add2(S, m.pzz);
                cu = first ? (cz > 0 ? m.uz : mul2(m.uz, f2(-1.f))) : (cz > 0 ? add2(cu, m.uz) : sub2(cu, m.uz));
                cF = first ? (cz > 0 ? fz : mul2(fz, f2(-1.f))) : (cz > 0 ? add2(cF, fz) : sub2(cF, fz));
            }
            if (cx && cy) S = (cx * cy > 0) ? add2(S, pxy2) : sub2(S, pxy2);
            if (cx && cz) S = (cx * cz > 0) ? add2(S, pxz2) : sub2(S, pxz2);
            if (cy && cz) S = (cy * cz > 0) ? add2(S, pyz2) : sub2(S, pyz2);
            const float2 E = fma2(cu, fma2(r45, cu, mul2(b9, cF)), fma2(A, S, K0));
            const float2 O = fma2(alpha, cF, mul2(r3, cu));
            const float2 w = f2(Lattice<Q>::w(i));
            g[i] = mul2(w, add2(E, O));
            g[i + 1] = mul2(w, sub2(E, O));
        }
    } else {
        const float2 om1 = sub2(f2(1.f), omega);
        const float2 base = fma2(omega, fma2(mul2(m.rho, uu), f2(-1.5f), m.drho), mul2(BuF, f2(-3.f)));
        const float2 orho = mul2(omega, m.rho);
        const float2 r45 = mul2(orho, f2(4.5f)), r3 = mul2(orho, f2(3.f)), b9 = mul2(B, f2(9.f)),
                     b3 = mul2(B, f2(3.f));
        g[0] = fma2(om1, g[0], mul2(f2(Lattice<Q>::w(0)), base));
#pragma unroll
        for (int i = 1; i < Q; i += 2) {
            const int cx = lat_cx(i), cy = lat_cy(i), cz = lat_cz(i);
            float2 cu = f2(0.f), cF = f2(0.f);
            bool first = true;
            if (cx) { cu = cx > 0 ? m.ux : mul2(m.ux, f2(-1.f)); cF = cx > 0 ? fx : mul2(fx, f2(-1.f)); first = false; }
            if (cy) {
                cu = first ? (cy > 0 ? m.uy : mul2(m.uy, f2(-1.f))) : (cy > 0 ? add2(cu, m.uy) : sub2(cu, m.uy));
                cF = first ? (cy > 0 ? fy : mul2(fy, f2(-1.f))) : (cy > 0 ? add2(cF, fy) : sub2(cF, fy));
                first = false;
            }
            if (cz) {
                cu = first ? (cz > 0 ? m.uz : mul2(m.uz, f2(-1.f))) : (cz > 0 ? add2(cu, m.uz) : sub2(cu, m.uz));
                cF = first ? (cz > 0 ? fz : mul2(fz, f2(-1.f))) : (cz > 0 ? add2(cF, fz) : sub2(cF, fz));
            }
            const float2 w = f2(Lattice<Q>::w(i));
            const float2 E = mul2(w, fma2(cu, fma2(r45, cu, mul2(b9, cF)), base));
            const float2 O = mul2(w, fma2(r3, cu, mul2(b3, cF)));
            g[i] = fma2(om1, g[i], add2(E, O));
            g[i + 1] = fma2(om1, g[i + 1], sub2(E, O));
        }
    }
}

}  // namespace f32

// The functions of a storage type.
template <int ST, int Q, bool NEED_PI>
__device__ __forceinline__ Mom moments_st(const float (&f)[Q], float fx, float fy, float fz, float rho0) {
    if constexpr (ST == VLBM_STORE_F32) return f32::moments<Q, NEED_PI>(f, fx, fy, fz, rho0);
    else return moments<Q, NEED_PI>(f, fx, fy, fz, rho0);
}
template <int ST>
__device__ __forceinline__ float stress_aux_st(const Mom& m, float fx, float fy, float fz) {
    if constexpr (ST == VLBM_STORE_F32) return f32::stress_aux(m, fx, fy, fz);
    else return stress_aux(m, fx, fy, fz);
}
template <int ST, int Q, int OP>
__device__ __forceinline__ void collide_st(float (&f)[Q], const Mom& m, float omega, float fx, float fy, float fz) {
    if constexpr (ST == VLBM_STORE_F32) f32::collide<Q, OP>(f, m, omega, fx, fy, fz);
    else collide<Q, OP>(f, m, omega, fx, fy, fz);
}
template <int ST, int Q, bool NEED_PI, bool SCALED>
__device__ __forceinline__ Mom2 moments2_st(const float2 (&g)[Q], float2 fx, float2 fy, float2 fz, float rho0,
                                            float inv_scale) {
    if constexpr (ST == VLBM_STORE_F32) return f32::moments2<Q, NEED_PI>(g, fx, fy, fz, rho0);
    else return moments2<Q, NEED_PI, SCALED>(g, fx, fy, fz, rho0, inv_scale);
}
template <int ST>
__device__ __forceinline__ float2 stress_aux2_st(const Mom2& m, float2 fx, float2 fy, float2 fz) {
    if constexpr (ST == VLBM_STORE_F32) return f32::stress_aux2(m, fx, fy, fz);
    else return stress_aux2(m, fx, fy, fz);
}
template <int ST, int Q, int OP>
__device__ __forceinline__ void collide2_st(float2 (&g)[Q], const Mom2& m, float2 omega, float2 fx, float2 fy,
                                            float2 fz, float gscale, float oscale) {
    if constexpr (ST == VLBM_STORE_F32) f32::collide2<Q, OP>(g, m, omega, fx, fy, fz);
    else collide2<Q, OP>(g, m, omega, fx, fy, fz, gscale, oscale);
}

}  // namespace vlbm
