// The force pass's pair terms, shared by its two kernels (sphx_force.cu, sphx_team_force.cu).
#pragma once
#include "sphx_passes.cuh"

namespace sphx {

// The pair term of particle t against candidate j: the pressure-force contribution
// m_j * (P_t + P_j)/(2 rho_j) * gradW (the caller adds its negation, which equals
// subtracting it; +0 when |r| < 1e-6, where the reference skips it, and adding -0 leaves
// every float unchanged) and the viscosity contribution ((m_j/rho_j) mu (v_j - v_t))
// laplacianW (added), each with the reference's operations; aj.w holds (m_j/rho_j) mu.
template <int K>
__device__ __forceinline__ void force_term(const StepConst& c, const float4& xt,
                                           const float4& vt, float Pt, const float4& xj,
                                           const float4& vj, const float4& aj, float* p3,
                                           float* v3) {
    const Diff d = diff(xt, xj);
    const float r_len = xsqrt(d.d2);
    const bool skip = r_len < 1e-6f;
    p3[0] = p3[1] = p3[2] = 0.0f;
    float lap;
    if (K == SPHX_KERNEL_GAUSSIAN) {
        // GaussianKernel::gradW / laplacianW (kernels.cpp:215-225): both use
        // exp(-r_sq * sigma_sq_inv_) of the same r_sq -- one evaluation serves both
        const float e = expf(xmul(-d.d2, c.gs));
        if (!skip) {
            const float pt = xdiv(xadd(Pt, aj.y), aj.z);
            const float k = xmul(c.gg, e);
            const float sp = xmul(xj.w, pt);
            p3[0] = xmul(sp, xmul(k, d.x));
            p3[1] = xmul(sp, xmul(k, d.y));
            p3[2] = xmul(sp, xmul(k, d.z));
        }
        lap = xmul(xmul(c.gl, e), xsub(xmul(c.g2s, d.d2), 3.0f));
    } else {
        const float q = xdiv_fixed(r_len, c.h, c.rcp_h, c.fast_div_h);
        if (!skip) {
            const float pt = xdiv(xadd(Pt, aj.y), aj.z);
            const float sp = xmul(xj.w, pt);
            if (K == SPHX_KERNEL_WENDLAND_C2) {
                // WendlandC2Kernel::gradW (kernels.cpp:180-192):
                // norm * dW/dq * (r / (r_len h)), dW/dq = -5 tmp^3 q; 0 for q >= 2
                if (!(q >= 2.0f)) {
                    const float tmp = xsub(1.0f, xmul(0.5f, q));
                    const float dw = xmul(xmul(xmul(xmul(-5.0f, tmp), tmp), tmp), q);
                    const float gsc = xmul(c.wnorm, dw);
                    const float den = xmul(r_len, c.h);
                    p3[0] = xmul(sp, xmul(gsc, xdiv(d.x, den)));
                    p3[1] = xmul(sp, xmul(gsc, xdiv(d.y, den)));
                    p3[2] = xmul(sp, xmul(gsc, xdiv(d.z, den)));
                } else {
                    p3[0] = xmul(sp, 0.0f);
                    p3[1] = xmul(sp, 0.0f);
                    p3[2] = xmul(sp, 0.0f);
                }
            } else {
                float gx = 0.0f, gy = 0.0f, gz = 0.0f;
                if ((q >= 0.0f && q <= 1.0f) || (q > 1.0f && q <= 2.0f)) {
                    const float gf = cubic_grad_factor(c, q);
                    gx = xmul(gf, xdiv(d.x, r_len));
                    gy = xmul(gf, xdiv(d.y, r_len));
                    gz = xmul(gf, xdiv(d.z, r_len));
                }
                p3[0] = xmul(sp, xdiv_fixed(gx, c.h, c.rcp_h, c.fast_div_h));
                p3[1] = xmul(sp, xdiv_fixed(gy, c.h, c.rcp_h, c.fast_div_h));
                p3[2] = xmul(sp, xdiv_fixed(gz, c.h, c.rcp_h, c.fast_div_h));
            }
        }
        lap = K == SPHX_KERNEL_WENDLAND_C2 ? wendland_lap(c, q) : cubic_lap(c, q);
    }
    const float sv = aj.w;  // (m_j / rho_j) * mu, formed by the density pass
    v3[0] = xmul(xmul(sv, xsub(vj.x, vt.x)), lap);
    v3[1] = xmul(xmul(sv, xsub(vj.y, vt.y)), lap);
    v3[2] = xmul(xmul(sv, xsub(vj.z, vt.z)), lap);
}

// The terms of two neighbours, one in each half of packed FP32 pairs: px, py, pz the negated
// pressure-force contributions (every sum then only adds), wx, wy, wz the viscosity ones.  The
// three divisions by |r| (cubic spline) or |r| h (Wendland)
// share one reciprocal, the division by 2 rho_j has its reciprocal with the candidate, and
// those by h and h^2 need no range tests.  Valid where StepConst::force_nz is 2 and
// DevState::general is 0: a component of x_t - x_j is then 0 or in [2^-68, r], P_t + P_j 0 or
// in [2^-74, 2^61] and rho in [2^-60, 2^40], and every dividend below stays in the range its
// division needs.  Where force_nz is 1 or a particle left those ranges (kCheck), the terms come
// with the answer whether this pair is in range: its components, the dividends of the division
// by h, and the candidate, whose factor 1 / (2 rho_j) is 0 if its density or pressure is out of
// range.  The signs of zero terms are not kept: the sums start at +0 and so never
// become -0, and adding a zero of either sign leaves any other value unchanged.  A pair with
// |r| < 1e-6, whose pressure term the reference skips, gets m_j pt = 0 and with it zero terms
// (what it multiplies is finite there).
//
// The work on a pair of neighbours is split in two (PairStart::start, pair_terms): a lane starts
// its next pair in the same straight-line code that finishes the one before, so that the two
// chains of dependent operations overlap.
struct PairStart {
    F2 dx, dy, dz;  // x_t - x_j
    F2 m;           // m_j
    F2 s, ns, hr;   // |r|, -|r|, 1/(2 |r|) scaled (sqrt2_exact)
    int qa, qb;     // ring slots
    bool ha = false, hb = false;
    __device__ __forceinline__ void start(const PairLits& k, const float4& xt, const float4& xa,
                                          const float4& xb) {
        dx = f2(xt.x) - f2(xa.x, xb.x);
        dy = f2(xt.y) - f2(xa.y, xb.y);
        dz = f2(xt.z) - f2(xa.z, xb.z);
        m = f2(xa.w, xb.w);
        s = sqrt2_exact(k, pair_d2(dx, dy, dz, F2{k.neg0}), hr, ns);
    }
};
struct PairTerms {
    F2 px, py, pz, wx, wy, wz;
    bool oka, okb;  // (kCheck)
};
// three numbers 0 or at least `least` in magnitude
__device__ __forceinline__ bool zero_or_above(float x, float y, float z, float least) {
    auto order = [](float v) { return 2u * __float_as_uint(v) - 1u; };  // (0 becomes the largest)
    return min(min(order(x), order(y)), order(z)) >= order(least);
}
template <int K, bool kCheck = false>
__device__ __forceinline__ PairTerms pair_terms(const PairLits& k, const PairConst& c,
                                                const float4& vt, float Pt, const PairStart& p,
                                                const float4& va, const float4& vb,
                                                const float2& fa, const float2& fb) {
    const F2 zero = f2(0.0f), neg0{k.neg0};
    const F2 dx = p.dx, dy = p.dy, dz = p.dz, ns = p.ns;
    const F2 q = div_fixed2(p.s, F2{c.neg_h}, F2{c.rcp_h});
    const float2 su = upk2(p.s.v), qu = upk2(q.v);
    const bool la = !(su.x < 1e-6f), lb = !(su.y < 1e-6f);
    const F2 rho = f2(va.w, vb.w);
    const F2 nPj = pmul(F2{c.gas}, F2{c.rest} - rho, neg0);
    const F2 npt = div_rcp2(f2(-Pt) + nPj, F2{k.neg2} * rho, f2(fa.y, fb.y));
    const F2 sp = select2(la, lb, p.m * npt, zero);  // -m_j pt
    const F2 y1 = p.hr * F2{k.p2p21};               // ~ 1/|r|
    F2 px, py, pz, lap;
    bool oka = true, okb = true;
    if (kCheck) {
        const float2 x = upk2(dx.v), y = upk2(dy.v), z = upk2(dz.v);
        oka = fa.y != 0.0f && zero_or_above(x.x, y.x, z.x, kLeastStep);
        okb = fb.y != 0.0f && zero_or_above(x.y, y.y, z.y, kLeastStep);
    }
    // beyond the support q = 2 the clamped 2 - q (1 - q/2) makes the terms the zeros that the
    // reference returns there
    if (K == SPHX_KERNEL_WENDLAND_C2) {
        // norm dW/dq (r / (|r| h)), dW/dq = -5 t^3 q (kernels.cpp:180-192)
        const F2 t = max0(F2{k.one} - F2{k.half} * q);
        const F2 gsc = F2{c.wnorm} * (F2{k.neg5} * t * t * t * q);
        const F2 nden = ns * F2{c.h};
        const F2 y = rcp2_exact(k, nden, y1 * F2{c.rcp_h});
        px = sp * (gsc * div_rcp2(dx, nden, y));
        py = sp * (gsc * div_rcp2(dy, nden, y));
        pz = sp * (gsc * div_rcp2(dz, nden, y));
        lap = F2{c.wl} * t * t * (pmul(F2{k.five}, q, neg0) - F2{k.three});
    } else {
        // gradient factor (kernels.cpp:96-108): sigma (-2 q + 1.5 q q) or -sigma (0.5 t) t
        const bool ia = qu.x <= 1.0f, ib = qu.y <= 1.0f;
        const F2 t = max0(F2{k.two} - q);
        const F2 g1 = F2{c.sigma} * (F2{k.neg2} * q + pmul(F2{k.onehalf} * q, q, neg0));
        const F2 g2 = F2{c.neg_sigma} * (F2{k.half} * t * t);
        const F2 gf = select2(ia, ib, g1, g2);
        const F2 y = rcp2_exact(k, ns, y1);
        const F2 ux = gf * div_rcp2(dx, ns, y), uy = gf * div_rcp2(dy, ns, y),
                 uz = gf * div_rcp2(dz, ns, y);
        if (kCheck) {
            const float2 a = upk2(ux.v), e = upk2(uy.v), f = upk2(uz.v);
            oka = oka && zero_or_above(a.x, e.x, f.x, 0x1p-100f);
            okb = okb && zero_or_above(a.y, e.y, f.y, 0x1p-100f);
        }
        px = sp * div_fixed2(ux, F2{c.neg_h}, F2{c.rcp_h});
        py = sp * div_fixed2(uy, F2{c.neg_h}, F2{c.rcp_h});
        pz = sp * div_fixed2(uz, F2{c.neg_h}, F2{c.rcp_h});
        // Laplacian (kernels.cpp:130-138)
        const F2 l = select2(ia, ib, F2{k.neg2} + pmul(F2{k.three}, q, neg0), t);
        lap = div_fixed2(F2{c.sigma} * l, F2{c.neg_hsq}, F2{c.rcp_hsq});
    }
    const F2 mv = f2(fa.x, fb.x);  // (m_j / rho_j) mu, formed by the density pass
    return {px, py, pz, mv * (f2(va.x, vb.x) - f2(vt.x)) * lap,
            mv * (f2(va.y, vb.y) - f2(vt.y)) * lap, mv * (f2(va.z, vb.z) - f2(vt.z)) * lap,
            oka, okb};
}

}  // namespace sphx
