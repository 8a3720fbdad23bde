// Force + acceleration + leapfrog + wall-clamp pass of the step (compute_forces,
// sph_engine.cpp:226-244, 390-443; integrate_leapfrog, cpp:290-310; apply_boundary_conditions,
// particle.cpp:122-153).
#include "sphx_passes.cuh"

namespace sphx {

// ---------------------------------------------------------------------------------------
// force + acceleration (+ leapfrog + wall clamp when kIntegrate)
// (compute_pressure_force / compute_viscosity_force / compute_acceleration,
//  sph_engine.cpp:390-443; integrate_leapfrog, cpp:290-310;
//  ParticleSystem::apply_boundary_conditions, particle.cpp:122-153)
// ---------------------------------------------------------------------------------------
// Per warp: the candidate ring -- positions and mass, velocities and density, the two
// per-candidate factors -- the lanes' masks and the tile's row segments.  40 bytes a candidate:
// 12 chunks leave room for 12 warps per SM; 8 chunks (16 warps) took 9% longer on the 1M dam
// break, 10 (14 warps) 8%, 16 (8 warps) 17%.
//
// Bound: instruction issue (64% of the slots with 3 warps per scheduler) and the FP32 pipe
// (58%; a packed instruction holds it two cycles): about 1,200 warp instructions per particle
// in 5.7 turns, each finishing one pair of neighbours per lane and starting the next.  1M dam
// break, force + leapfrog: 1.52 ms; walking and culling the candidates again instead of
// reading the density pass's list 1.71 ms; with hit lists, terms passed through shared memory and
// in-order folds by their lanes (2,479 instructions) 2.60 ms; one neighbour per turn with the
// compiler's division and square root 2.72 ms, pairs 2.08, staged by asynchronous copies 1.83,
// the two halves of a turn overlapped 1.73.
constexpr int kForceRing = 12;
struct ForceSmem {
    float4 pos[kForceRing * 32];  // x, y, z, m
    float4 vel[kForceRing * 32];  // vx, vy, vz, rho
    float2 fac[kForceRing * 32];  // (m / rho) mu, 1 / (2 rho)
    uint32_t mask[kForceRing * 32];
    int2 seg[kMaxSegments + 1];
};
static_assert(sizeof(ForceSmem) % 16 == 0, "per-warp regions stay 16-byte aligned");

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


// A lane's running force sums: pressure and viscosity, each in the walk's order.
struct ForceSums {
    float px = 0.0f, py = 0.0f, pz = 0.0f, vx = 0.0f, vy = 0.0f, vz = 0.0f;
};

// force_term added to the sums (the general form; a call of its own, so that the forms below
// keep their registers)
template <int K>
__device__ __noinline__ ForceSums add_term_general(const StepConst& c, float4 xt, float4 vt,
                                                   float Pt, float4 xj, float4 vj, float4 aj,
                                                   ForceSums F) {
    float p3[3], v3[3];
    force_term<K>(c, xt, vt, Pt, xj, vj, aj, p3, v3);
    F.px = xsub(F.px, p3[0]);
    F.py = xsub(F.py, p3[1]);
    F.pz = xsub(F.pz, p3[2]);
    F.vx = xadd(F.vx, v3[0]);
    F.vy = xadd(F.vy, v3[1]);
    F.vz = xadd(F.vz, v3[2]);
    return F;
}

// The terms of two neighbours, one in each half of packed FP32 pairs, added to the sums in
// order (a if ha, b if hb).  The three divisions by |r| (cubic spline) or |r| h (Wendland)
// share one reciprocal, the division by 2 rho_j has its reciprocal with the candidate, and
// those by h and h^2 need no range tests.  Valid where StepConst::force_nz holds and
// DevState::general is 0: a component of x_t - x_j is then 0 or in [2^-68, r], P_t + P_j 0 or
// in [2^-64, 2^61] and rho in [2^-30, 2^40], and every dividend below stays in the range its
// division needs.  The signs of zero terms are not kept: the sums start at +0 and so never
// become -0, and adding a zero of either sign leaves any other value unchanged.  A pair with
// |r| < 1e-6, whose pressure term the reference skips, gets m_j pt = 0 and with it zero terms
// (what it multiplies is finite there).
//
// The work on a pair of neighbours is split in two (PairStart::start, add_pair): a lane starts
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
template <int K>
__device__ __forceinline__ void add_pair(const PairLits& k, const PairConst& c, const float4& vt, float Pt,
                                         const PairStart& p, const float4& va, const float4& vb,
                                         const float2& fa, const float2& fb, ForceSums& F) {
    const F2 zero = f2(0.0f), neg0{k.neg0};
    const F2 dx = p.dx, dy = p.dy, dz = p.dz, ns = p.ns;
    const bool ha = p.ha, hb = p.hb;
    const F2 q = div_fixed2(p.s, F2{c.neg_h}, F2{c.rcp_h});
    const float2 su = upk2(p.s.v), qu = upk2(q.v);
    const bool la = !(su.x < 1e-6f), lb = !(su.y < 1e-6f);
    const F2 rho = f2(va.w, vb.w);
    const F2 Pj = pmul(F2{c.gas}, rho - F2{c.rest}, neg0);
    const F2 pt = div_rcp2(f2(Pt) + Pj, F2{k.neg2} * rho, f2(fa.y, fb.y));
    const F2 sp = select2(la, lb, p.m * pt, zero);  // m_j pt
    const F2 y1 = p.hr * F2{k.p2p21};               // ~ 1/|r|
    F2 px, py, pz, lap;
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
        px = sp * div_fixed2(gf * div_rcp2(dx, ns, y), F2{c.neg_h}, F2{c.rcp_h});
        py = sp * div_fixed2(gf * div_rcp2(dy, ns, y), F2{c.neg_h}, F2{c.rcp_h});
        pz = sp * div_fixed2(gf * div_rcp2(dz, ns, y), F2{c.neg_h}, F2{c.rcp_h});
        // Laplacian (kernels.cpp:130-138)
        const F2 l = select2(ia, ib, F2{k.neg2} + pmul(F2{k.three}, q, neg0), t);
        lap = div_fixed2(F2{c.sigma} * l, F2{c.neg_hsq}, F2{c.rcp_hsq});
    }
    const F2 mv = f2(fa.x, fb.x);  // (m_j / rho_j) mu, formed by the density pass
    const F2 wx = mv * (f2(va.x, vb.x) - f2(vt.x)) * lap, wy = mv * (f2(va.y, vb.y) - f2(vt.y)) * lap,
             wz = mv * (f2(va.z, vb.z) - f2(vt.z)) * lap;
    const float2 ax = upk2(px.v), ay = upk2(py.v), az = upk2(pz.v);
    const float2 bx = upk2(wx.v), by = upk2(wy.v), bz = upk2(wz.v);
    if (ha) {
        F.px = xsub(F.px, ax.x);
        F.py = xsub(F.py, ay.x);
        F.pz = xsub(F.pz, az.x);
        F.vx = xadd(F.vx, bx.x);
        F.vy = xadd(F.vy, by.x);
        F.vz = xadd(F.vz, bz.x);
    }
    if (hb) {
        F.px = xsub(F.px, ax.y);
        F.py = xsub(F.py, ay.y);
        F.pz = xsub(F.pz, az.y);
        F.vx = xadd(F.vx, bx.y);
        F.vy = xadd(F.vy, by.y);
        F.vz = xadd(F.vz, bz.y);
    }
}

// Candidates go from global to shared memory by asynchronous copies (cp.async), a round of the
// ring ahead of their use.
template <bool kIntegrate, bool kBatch, int kKern, bool kNZ>
__global__ void __launch_bounds__(128, 3) k_force(const StepConst cp, const Buffers b,
                                                  DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_raw_f[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ForceSmem* S = reinterpret_cast<ForceSmem*>(smem_raw_f) + warp;
    const uint32_t ntiles = ds->n_tiles;
    const uint32_t lt = (1u << lane) - 1u;
    const PairLits& lit = cp.lit;
    const bool nz = kNZ && !ds->general;
    const TileQueue queue(&ds->work[1], b.num_sms);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        const uint2 tile = b.tiles[t];
        const int scene = kBatch ? (int)b.scene_s[tile.x] : 0;
        const StepConst& c = kBatch ? b.scenes[scene].c : cp;
        const Geom g = kBatch ? scene_geom(b.scenes[scene], ds) : grid_geom(ds);
        Tile T;
        float4 xi;
        bool valid;
        int i;
        tile_setup(c, b, g, tile, lane, T, i, xi, valid);
        const float4 vi0 = valid ? b.vel4_s[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float Pi = valid ? b.aux4_s[i].y : 0.0f;
        // the density pass's records of this tile: its kept candidates and the lanes' masks
        const uint2 list = b.records ? b.tile_list[t] : make_uint2(kNoSlot, 0u);
        const bool listed = list.x != kNoSlot;
        const uint32_t* rec = b.records + (size_t)list.x * 32 + lane;
        const int nlist = listed ? (int)list.y : 0;  // candidates
        uint32_t ahead = lane < nlist ? __ldcs(rec) : 0u;  // the next chunk's, read ahead
        TileBox B;
        int nseg = 0;
        if (!listed) {
            B = tile_box(xi, valid);
            __syncwarp();  // the previous tile's segments are read
            nseg = build_segments(b, g, T, lane, S->seg);
            __syncwarp();
        }
        RawStream st(S->seg, nseg);
        ForceSums F;
        int kept = 0, ready = 0, staged = 0, head = 0, self = -1;
        RingLane<kForceRing> at;
        PairStart pair;  // started, not yet added
        pair.qa = pair.qb = 0;
        pair.start(lit, xi, xi, xi);
        int need = 0;  // first chunk the lane still needs
        for (;;) {
            cp_async_wait_all();
            __syncwarp();  // staged chunks are in place, every lane is done with those before head
            ready = staged;
            auto copy = [&](int q, uint32_t j) {  // candidate j to ring slot q
                cp_async16(&S->pos[q], &b.pos4_s[j]);
                cp_async16(&S->vel[q], &b.vel4_s[j]);
                cp_async8(&S->fac[q], &b.aux4_s[j].z);
            };
            for (; staged * 32 < nlist && staged < head + kForceRing; ++staged) {
                const int f = (staged % kForceRing) * 32;
                if (staged * 32 + lane < nlist) copy(f + 31 - lane, ahead);
                cp_async4(&S->mask[f + lane], rec + 32);
                rec += 64;
                if ((staged + 1) * 32 + lane < nlist) ahead = __ldcs(rec);
            }
            // without records: the walk, culled and tested again
            while (st.more() && kept + 32 <= (head + kForceRing) * 32) {
                const int m = st.count(), s = st.s;
                bool near = false;
                if (lane < m) near = box_near(B, b.pos4_s[s + lane], c.r2 * 1.0001f);
                const uint32_t surv = __ballot_sync(kFull, near);
                if ((unsigned)(i - s) < (unsigned)m)
                    self = kept + __popc(surv & ((1u << (i - s)) - 1u));
                if ((surv >> lane) & 1u)
                    copy(ring_slot<kForceRing>(kept + __popc(surv & lt)), (uint32_t)(s + lane));
                st.next();
                kept += __popc(surv);
                while ((kept >> 5) > staged || (!st.more() && kept > staged * 32)) {
                    const int f = (staged % kForceRing) * 32;
                    cp_async_wait_all();
                    __syncwarp();
                    uint32_t mask = 0;
                    for (int q = 0; q < 32; ++q)
                        if (diff_d2(xi, S->pos[f + q]) <= c.r2) mask |= 1u << q;
                    mask = valid ? mask & chunk_valid(kept - staged * 32) : 0u;
                    if (self >> 5 == staged) mask &= ~(0x80000000u >> (self & 31));
                    S->mask[f + lane] = mask;
                    ++staged;
                }
            }
            const bool all = !st.more() && staged * 32 >= nlist && ready == staged;
            const int until = all ? ready : min(head + 1, ready);
            if (nz) {
                // starts `next` and adds `done`; false when no lane needs a chunk before `until`
                auto turn = [&](PairStart& next, const PairStart& done) -> bool {
                    at.advance(S->mask, ready, lane);
                    at.take2(next.qa, next.qb, next.ha, next.hb);
                    next.start(lit, xi, S->pos[next.qa], S->pos[next.qb]);
                    add_pair<kKern>(lit, c.pair, vi0, Pi, done, S->vel[done.qa], S->vel[done.qb],
                                    S->fac[done.qa], S->fac[done.qb], F);
                    need = at.next - (next.ha ? 1 : 0);
                    return __any_sync(kFull, need < until);
                };
                for (;;) {
                    PairStart other;
                    if (!turn(other, pair)) {
                        pair = other;
                        break;
                    }
                    if (!turn(pair, other)) break;
                }
            } else {
                for (;;) {
                    at.advance(S->mask, ready, lane);
                    need = at.need();
                    if (!__any_sync(kFull, need < until)) break;
                    int q[2];
                    bool h[2];
                    at.take2(q[0], q[1], h[0], h[1]);
                    for (int k = 0; k < 2; ++k) {
                        if (!h[k]) continue;
                        const float4 vj = S->vel[q[k]];
                        const float Pj = xmul(c.gas, xsub(vj.w, c.rest));
                        F = add_term_general<kKern>(
                            c, xi, vi0, Pi, S->pos[q[k]], vj,
                            make_float4(vj.w, Pj, xmul(2.0f, vj.w), S->fac[q[k]].x), F);
                    }
                }
            }
            if (all) break;
            head = __reduce_min_sync(kFull, need);
        }
        if (!valid) continue;
        const float mi = xi.w;
        const float ax = xdiv(xadd(xadd(F.px, F.vx), xmul(0.0f, mi)), mi);
        const float ay = xdiv(xadd(xadd(F.py, F.vy), xmul(c.grav, mi)), mi);
        const float az = xdiv(xadd(xadd(F.pz, F.vz), xmul(0.0f, mi)), mi);
        b.acc4_s[i] = make_float4(ax, ay, az, 0.0f);
        if (!kIntegrate) continue;
        const float dt = kBatch ? b.scenes[scene].dt : ds->dt;
        const float4 vi = vi0;
        const uint32_t id = b.id_s[i];
        float x[3] = {xi.x, xi.y, xi.z}, v[3] = {vi.x, vi.y, vi.z};
        const float acc[3] = {ax, ay, az};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float half = xmul(xmul(0.5f, acc[a]), dt);
            float vv = xadd(v[a], half);
            x[a] = xadd(x[a], xmul(vv, dt));
            vv = xadd(vv, half);
            v[a] = xmul(vv, c.damping);
            if (x[a] < c.lo[a]) {
                x[a] = c.lo[a];
                v[a] = xmul(v[a], -0.8f);
            } else if (x[a] > c.hi[a]) {
                x[a] = c.hi[a];
                v[a] = xmul(v[a], -0.8f);
            }
        }
        b.pos4[id] = make_float4(x[0], x[1], x[2], mi);
        b.vel4[id] = make_float4(v[0], v[1], v[2], 0.0f);
        if (kBatch) {
            if (id == b.scenes[scene].start) {  // accelerations_[0] of the scene
                b.scenes[scene].a0[0] = ax;
                b.scenes[scene].a0[1] = ay;
                b.scenes[scene].a0[2] = az;
            }
        } else if (id == 0) {
            ds->a0[0] = ax;
            ds->a0[1] = ay;
            ds->a0[2] = az;
        }
    }
}

template <bool kIntegrate, bool kBatch, int kKern, bool kNZ>
static void launch_force_t(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                           DevState* ds) {
    const int threads = 32 * L.warps_per_block;
    const size_t sm = (size_t)L.warps_per_block * sizeof(ForceSmem);
    static LaunchShapeCache cache;
    const int nb = cached_resident_blocks(
        cache, L, k_force<kIntegrate, kBatch, kKern, kNZ>, threads, sm);
    k_force<kIntegrate, kBatch, kKern, kNZ><<<nb, threads, sm, L.stream>>>(c, b, ds);
}

template <int kKern, bool kNZ>
static void launch_force_n(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                           DevState* ds, int integrate) {
    const bool batch = b.nscenes > 0;
    if (integrate) {
        if (batch) launch_force_t<true, true, kKern, kNZ>(L, c, b, ds);
        else launch_force_t<true, false, kKern, kNZ>(L, c, b, ds);
    } else {
        if (batch) launch_force_t<false, true, kKern, kNZ>(L, c, b, ds);
        else launch_force_t<false, false, kKern, kNZ>(L, c, b, ds);
    }
}

// Precision mode (single scene) runs the tile sweep (sphx_sweep.cu); exact mode k_force.
int launch_force(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                 int integrate) {
    if (c.precise && b.nscenes == 0) return launch_force_sweep(L, c, b, ds, integrate);
    if (c.kern == SPHX_KERNEL_WENDLAND_C2) {
        if (c.force_nz) launch_force_n<SPHX_KERNEL_WENDLAND_C2, true>(L, c, b, ds, integrate);
        else launch_force_n<SPHX_KERNEL_WENDLAND_C2, false>(L, c, b, ds, integrate);
    } else if (c.kern == SPHX_KERNEL_GAUSSIAN) {
        launch_force_n<SPHX_KERNEL_GAUSSIAN, false>(L, c, b, ds, integrate);
    } else if (c.force_nz) {
        launch_force_n<SPHX_KERNEL_CUBIC_SPLINE, true>(L, c, b, ds, integrate);
    } else {
        launch_force_n<SPHX_KERNEL_CUBIC_SPLINE, false>(L, c, b, ds, integrate);
    }
    return 1;
}

}  // namespace sphx
