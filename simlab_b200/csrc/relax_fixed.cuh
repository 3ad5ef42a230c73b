// The regularized D3Q19 collision (relax_m without forcing and without the
// u_inf absorbing target) with every rounding written out: which products a
// sum is fused with does not depend on where the compiler inlines it, so a
// kernel can change its loads, its stores or the number of cells a thread
// carries and give the same bits.  The choices below are the ones the
// compiler makes for relax_m; they differ between its run-time-switched form
// (the direct kernel) and its compile-time form (the staged kernel), and
// flags in V select them.
#pragma once
#include "f32x2.cuh"
#include "lbm_device.cuh"

namespace lbm {

__device__ __forceinline__ float xfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xmul_apart(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float xrcp(float a) { return 1.0f / a; }
__device__ __forceinline__ float xsqrt(float a) { return sqrtf(a); }
template <class T> __device__ __forceinline__ T xval(float s) { return T(s); }

// V: the odd part O cu fused into the sum; the absorbing shift fused into the
// coefficient it joins; the product beside tau0^2 fused, not tau0^2; 1 - 1.5
// u.u fused; the axis pairs' sum in the edges' order
constexpr int RF_ODD = 1, RF_SHIFT = 2, RF_TAU = 4, RF_USQ = 8, RF_AXIS = 16;
// the direct kernel's choices, and the staged kernel's
template <class S, int P> constexpr int rf_direct() { return P == 0 ? 0 : (sizeof(S) == 2 ? RF_AXIS : RF_USQ); }
template <int P> constexpr int rf_staged() { return RF_ODD | RF_SHIFT | (P == 0 ? RF_TAU : 0); }

// tau of a cell's sponge factor (shader.rs:832-833)
__device__ __forceinline__ float sponge_tau(const Consts<float> &k, float sp, float tau) {
    return (sp > 0.0f && k.sponge_tau > tau) ? xfma(xmul(sp, sp), xadd(k.sponge_tau, -tau), tau) : tau;
}

__device__ __forceinline__ F2 sponge_tau(const Consts<float> &k, F2 sp, F2 tau) {
    return F2(sponge_tau(k, sp.v.x, tau.v.x), sponge_tau(k, sp.v.y, tau.v.y));
}

// m: the moments of f in storage units (scale SC); sp: the sponge factor (0
// without sponges); f receives the post-collision populations, scaled.
template <class T, int SC, bool LES, int V>
__device__ __forceinline__ void relax_fixed(const Consts<float> &k, const Moments<T> &m, T sp, T *f) {
    const T one = xval<T>(1.0f), t3 = xval<T>((float)(1.0 / 3.0));
    const T rho1 = SC != 1 ? xmul(m.rho1, xval<T>(1.0f / SC)) : m.rho1;
    const T rho = xadd(one, rho1);
    const T ir = xrcp(rho);
    const T irs = SC != 1 ? xmul(ir, xval<T>(1.0f / SC)) : ir;
    const T ux = xmul(m.jx, irs), uy = xmul(m.jy, irs), uz = xmul(m.jz, irs);
    const T rs = SC != 1 ? xmul(rho, xval<T>((float)SC)) : rho;
    const T rx = xmul(rs, ux), ry = xmul(rs, uy), rz = xmul(rs, uz);
    const T pxx = xfma(-m.rho1, t3, xfma(-rx, ux, m.sxx)), pyy = xfma(-m.rho1, t3, xfma(-ry, uy, m.syy)),
            pzz = xfma(-m.rho1, t3, xfma(-rz, uz, m.szz));
    const T pxy = xfma(-rx, uy, m.sxy), pxz = xfma(-rx, uz, m.sxz), pyz = xfma(-ry, uz, m.syz);
    T tau = xval<T>(k.tau0);
    if (LES) {
        const T d = xfma(pzz, pzz, xfma(pxx, pxx, xmul(pyy, pyy)));
        const T e = xfma(pyz, pyz, xfma(pxy, pxy, xmul(pxz, pxz)));
        const T qn = xsqrt(xmul(xval<T>(2.0f), xfma(xval<T>(2.0f), e, d)));
        const T x = xmul(xval<T>(xmul(18.0f, k.smag2)), qn), t0 = xval<T>(k.tau0);
        const T t2 = (V & RF_TAU) ? xfma(x, irs, xmul(t0, t0)) : xfma(t0, t0, xmul(x, irs));
        tau = xmul(xval<T>(0.5f), xadd(t0, xsqrt(t2)));
    }
    tau = sponge_tau(k, sp, tau);
    const T om1 = xadd(one, -xrcp(tau));
    const T uu = xfma(uz, uz, xfma(ux, ux, xmul(uy, uy)));
    const T usq = xmul(xval<T>(1.5f), uu);
    const T sg = xmul(xmul(xval<T>(k.sigma), sp), sp);
    const T s3 = xadd(xadd(pxx, pyy), pzz), tr = xmul(s3, t3);
    const T bq = xfma(-rho, usq, rho1), sr = xmul(sg, rho1);
    const T left = (V & RF_USQ) ? xfma(xval<T>(-1.5f), uu, one) : xadd(one, -usq);
    const T cb = (V & RF_SHIFT) ? xfma(-sr, left, bq) : xadd(bq, xmul_apart(-sr, left));
    const T c0 = xadd(rho, -sr);
    const T cA = xmul(xval<T>(4.5f), c0), cO = xmul(xval<T>(3.0f), c0);
    const T wa = xval<T>((float)(SC / 18.0)), we = xval<T>((float)(SC / 36.0)), w0 = xval<T>((float)(SC / 3.0));
    const T Aa = xmul(wa, cA), Ae = xmul(we, cA), Ba = xmul(wa, cb), Be = xmul(we, cb), Oa = xmul(wa, cO), Oe = xmul(we, cO);
    // 4.5 w (1 - omega), the weights of the stress (in storage units already)
    const T Ca = xmul(xval<T>(0.25f), om1), Ce = xmul(xval<T>(0.125f), om1), Cr = xmul(xval<T>(1.5f), om1);
    const T ht = xmul(xval<T>(0.5f), tr);
    const T qx = xadd(pxx, -ht), qy = xadd(pyy, -ht), qz = xadd(pzz, -ht);
    f[0] = xfma(w0, cb, -xmul(Cr, tr));
#pragma unroll
    for (int kk = 0; kk < 9; kk++) {
        const int i = 2 * kk + 1;
        T cu, en;
        if (kk < 3) {
            cu = kk == 0 ? ux : (kk == 1 ? uy : uz);
            const T ccp = xadd(kk == 0 ? pxx : (kk == 1 ? pyy : pzz), -tr);
            en = xfma(Ca, ccp, (V & RF_AXIS) ? xfma(Aa, xmul(cu, cu), Ba) : xfma(wa, cb, xmul(Aa, xmul(cu, cu))));
        } else {
            const T ua = CX(i) ? ux : uy, ub = CZ(i) ? uz : uy;  // the two axes of the edge, the first positive
            const int sgn = CX(i) * CY(i) + CX(i) * CZ(i) + CY(i) * CZ(i);
            cu = sgn > 0 ? xadd(ua, ub) : xadd(ua, -ub);
            const T pab = (CX(i) && CY(i)) ? pxy : ((CX(i) && CZ(i)) ? pxz : pyz);
            const T ccp = xfma(xval<T>((float)(2 * sgn)), pab, xadd(CX(i) ? qx : qy, CZ(i) ? qz : qy));
            en = xfma(Ce, ccp, xfma(Ae, xmul(cu, cu), Be));
        }
        const T O = kk < 3 ? Oa : Oe;
        if (V & RF_ODD) {
            f[i] = xfma(O, cu, en);
            f[i + 1] = xfma(-O, cu, en);
        } else {
            const T odd = xmul(O, cu);
            f[i] = xadd(en, odd);
            f[i + 1] = xadd(en, -odd);
        }
    }
}

}  // namespace lbm
