// Force + acceleration + leapfrog + wall-clamp pass of the step (compute_forces,
// sph_engine.cpp:226-244, 390-443; integrate_leapfrog, cpp:290-310; apply_boundary_conditions,
// particle.cpp:122-153).
#include "sphx_pairs.cuh"

namespace sphx {

// ---------------------------------------------------------------------------------------
// force + acceleration (+ leapfrog + wall clamp when kIntegrate)
// (compute_pressure_force / compute_viscosity_force / compute_acceleration,
//  sph_engine.cpp:390-443; integrate_leapfrog, cpp:290-310;
//  ParticleSystem::apply_boundary_conditions, particle.cpp:122-153)
// ---------------------------------------------------------------------------------------
// Per warp: the candidate ring -- positions and mass, velocities and density, the two
// per-candidate factors -- the lanes' masks and the tile's row segments.  40 bytes a candidate:
// 13 chunks are what 12 warps per SM leave room for; on the 1M dam break 12 chunks took 4%
// longer, 8 (16 warps) 13%, 10 (14 warps) 12%, 16 (8 warps) 21%.
//
// Bound: instruction issue (64% of the slots with 3 warps per scheduler) and the FP32 pipe
// (58%; a packed instruction holds it two cycles): about 1,130 warp instructions per particle
// in 5.7 turns, each finishing one pair of neighbours per lane and starting the next.  1M dam
// break, force + leapfrog: 1.41 ms (1.53 with 12 chunks and a branch at each new mask); walking
// and culling the candidates again instead of reading the density pass's list 1.71 ms; with hit lists, terms passed through shared memory and
// in-order folds by their lanes (2,479 instructions) 2.60 ms; one neighbour per turn with the
// compiler's division and square root 2.72 ms, pairs 2.08, staged by asynchronous copies 1.83,
// the two halves of a turn overlapped 1.73.
constexpr int kForceRing = 13;
struct ForceSmem {
    float4 pos[kForceRing * 32];  // x, y, z, m
    float4 vel[kForceRing * 32];  // vx, vy, vz, rho
    float2 fac[kForceRing * 32];  // (m / rho) mu, 1 / (2 rho)
    uint32_t mask[kForceRing * 32];
    int2 seg[kMaxSegments + 1];
};
static_assert(sizeof(ForceSmem) % 16 == 0, "per-warp regions stay 16-byte aligned");

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

// add_term_general of the candidate in ring slot q
template <int K>
__device__ __forceinline__ void add_slot_general(const StepConst& c, const ForceSmem* S, int q,
                                                 const float4& xt, const float4& vt, float Pt,
                                                 ForceSums& F) {
    const float4 vj = S->vel[q];
    const float Pj = xmul(c.gas, xsub(vj.w, c.rest));
    F = add_term_general<K>(c, xt, vt, Pt, S->pos[q], vj,
                            make_float4(vj.w, Pj, xmul(2.0f, vj.w), S->fac[q].x), F);
}

// the terms added to the sums in order (a if ha, b if hb)
__device__ __forceinline__ void add_terms(const PairTerms& t, bool ha, bool hb, ForceSums& F) {
    const float2 ax = upk2(t.px.v), ay = upk2(t.py.v), az = upk2(t.pz.v);
    const float2 bx = upk2(t.wx.v), by = upk2(t.wy.v), bz = upk2(t.wz.v);
    if (ha) {
        F.px = xadd(F.px, ax.x);
        F.py = xadd(F.py, ay.x);
        F.pz = xadd(F.pz, az.x);
        F.vx = xadd(F.vx, bx.x);
        F.vy = xadd(F.vy, by.x);
        F.vz = xadd(F.vz, bz.x);
    }
    if (hb) {
        F.px = xadd(F.px, ax.y);
        F.py = xadd(F.py, ay.y);
        F.pz = xadd(F.pz, az.y);
        F.vx = xadd(F.vx, bx.y);
        F.vy = xadd(F.vy, by.y);
        F.vz = xadd(F.vz, bz.y);
    }
}

// pair_terms of `p`, added to the sums
template <int K>
__device__ __forceinline__ void add_pair(const PairLits& k, const PairConst& c, const float4& vt,
                                         float Pt, const PairStart& p, const float4& va,
                                         const float4& vb, const float2& fa, const float2& fb,
                                         ForceSums& F) {
    add_terms(pair_terms<K>(k, c, vt, Pt, p, va, vb, fa, fb), p.ha, p.hb, F);
}

// pair_terms of two neighbours with the answer whether they are in range, added to the sums: in
// the general form where one of the two, or the lane's own particle (`out`), is not.
template <int K>
__device__ __forceinline__ void add_pair_checked(const PairLits& k, const StepConst& c,
                                                 const ForceSmem* S, const float4& xt,
                                                 const float4& vt, float Pt, bool out,
                                                 const PairStart& p, ForceSums& F) {
    const PairTerms t = pair_terms<K, true>(k, c.pair, vt, Pt, p, S->vel[p.qa], S->vel[p.qb],
                                            S->fac[p.qa], S->fac[p.qb]);
    if (((out || !t.oka) && p.ha) || ((out || !t.okb) && p.hb)) {
        if (p.ha) add_slot_general<K>(c, S, p.qa, xt, vt, Pt, F);
        if (p.hb) add_slot_general<K>(c, S, p.qb, xt, vt, Pt, F);
    } else {
        add_terms(t, p.ha, p.hb, F);
    }
}
// the same as a call
template <int K>
__device__ __noinline__ ForceSums add_slots_checked(const PairLits& k, const StepConst& c,
                                                    const ForceSmem* S, float4 xt, float4 vt,
                                                    float Pt, bool out, int qa, int qb, bool hb,
                                                    ForceSums F) {
    PairStart p;
    p.qa = qa;
    p.qb = qb;
    p.ha = true;
    p.hb = hb;
    p.start(k, xt, S->pos[qa], S->pos[qb]);
    add_pair_checked<K>(k, c, S, xt, vt, Pt, out, p, F);
    return F;
}

// The forms of the pair terms that a kernel takes, by StepConst::force_nz: 0 the general one; 1
// the packed one with a range check for every pair (the cubic spline's, for h above 0.045); 2 the
// packed one as it is, and where a particle is out of range (DevState::general) the checked one
// as a call, so that it takes no registers from the first.  1M dam break, ms, with the general
// form and now: at h = 0.05 4.32 and 1.53, with one coordinate of 1e-20 4.40 and 2.06.  The
// Wendland kernel keeps the general one there (2.90, with the checked one 1.94, but then the
// first loop takes 1.304 instead of 1.287); both loops in one kernel cost it 8%.
//
// Candidates go from global to shared memory by asynchronous copies (cp.async), a round of the
// ring ahead of their use.
template <bool kIntegrate, bool kBatch, int kKern, int kForm>
__global__ void __launch_bounds__(128, 3) k_force(const StepConst cp, const Buffers b,
                                                  DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_raw_f[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ForceSmem* S = reinterpret_cast<ForceSmem*>(smem_raw_f) + warp;
    const uint32_t ntiles = ds->n_tiles;
    const uint32_t lt = (1u << lane) - 1u;
    const PairLits& lit = cp.lit;
    const bool nz = kForm == 2 && !ds->general;
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
        // (see pair_range)
        const bool out = (kForm == 1 || (kForm == 2 && !nz)) && valid && b.aux4_s[i].w == 0.0f;
        // the density pass's records of this tile: its kept candidates and the lanes' masks
        const uint2 list = b.records ? b.tile_list[t] : make_uint2(kNoSlot, 0u);
        const bool listed = list.x != kNoSlot;
        const uint32_t* rec = b.records + (size_t)list.x * 32 + lane;
        // candidates; a single one is a lone particle's own
        const int nlist = listed && list.y > 1 ? (int)list.y : 0;
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
        // A lone particle takes no turns (1M lone particles 1.56 ms, with a round of turns over its
        // own candidate 2.15).  The Wendland kernel takes one even so (1.82 ms): with the test its
        // loop is 1.5% slower wherever there are neighbours.
        while (kKern == SPHX_KERNEL_WENDLAND_C2 || !listed || nlist > 0) {
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
            if (kForm == 1 || nz) {
                // starts `next` and adds `done`; false when no lane needs a chunk before `until`
                auto turn = [&](PairStart& next, const PairStart& done) -> bool {
                    at.advance_flat(S->mask, ready, lane);
                    at.take2(next.qa, next.qb, next.ha, next.hb);
                    next.start(lit, xi, S->pos[next.qa], S->pos[next.qb]);
                    if (kForm == 1) add_pair_checked<kKern>(lit, c, S, xi, vi0, Pi, out, done, F);
                    else add_pair<kKern>(lit, c.pair, vi0, Pi, done, S->vel[done.qa], S->vel[done.qb],
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
                    if constexpr (kForm == 2 && kKern == SPHX_KERNEL_CUBIC_SPLINE) {
                        if (h[0])
                            F = add_slots_checked<kKern>(lit, c, S, xi, vi0, Pi, out, q[0], q[1],
                                                         h[1], F);
                    } else {
                        for (int k = 0; k < 2; ++k)
                            if (h[k]) add_slot_general<kKern>(c, S, q[k], xi, vi0, Pi, F);
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
        leapfrog_exact(c, dt, acc, x, v);
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

template <bool kIntegrate, bool kBatch, int kKern, int kForm>
static void launch_force_t(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                           DevState* ds) {
    const int threads = 32 * L.warps_per_block;
    const size_t sm = (size_t)L.warps_per_block * sizeof(ForceSmem);
    static LaunchShapeCache cache;
    const int nb = cached_resident_blocks(
        cache, L, k_force<kIntegrate, kBatch, kKern, kForm>, threads, sm);
    k_force<kIntegrate, kBatch, kKern, kForm><<<nb, threads, sm, L.stream>>>(c, b, ds);
}

template <int kKern, int kForm>
static void launch_force_n(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                           DevState* ds, int integrate) {
    const bool batch = b.nscenes > 0;
    if (integrate) {
        if (batch) launch_force_t<true, true, kKern, kForm>(L, c, b, ds);
        else launch_force_t<true, false, kKern, kForm>(L, c, b, ds);
    } else {
        if (batch) launch_force_t<false, true, kKern, kForm>(L, c, b, ds);
        else launch_force_t<false, false, kKern, kForm>(L, c, b, ds);
    }
}

// Precision mode (single scene) runs the tile sweep (sphx_sweep.cu); exact mode k_force, or on
// tiles of at most 8 particles (small sets: pass_tile) k_force_team.
int launch_force(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                 int integrate) {
    if (c.precise && b.nscenes == 0) return launch_force_sweep(L, c, b, ds, integrate);
    if (b.tile_n <= kTeamTile) return launch_force_team(L, c, b, ds, integrate);
    constexpr int kCubic = SPHX_KERNEL_CUBIC_SPLINE, kWendland = SPHX_KERNEL_WENDLAND_C2,
                  kGaussian = SPHX_KERNEL_GAUSSIAN;
    if (c.kern == kWendland) {
        if (c.force_nz == 2) launch_force_n<kWendland, 2>(L, c, b, ds, integrate);
        else launch_force_n<kWendland, 0>(L, c, b, ds, integrate);
    } else if (c.kern == kGaussian) {
        launch_force_n<kGaussian, 0>(L, c, b, ds, integrate);
    } else if (c.force_nz == 2) {
        launch_force_n<kCubic, 2>(L, c, b, ds, integrate);
    } else if (c.force_nz == 1) {
        launch_force_n<kCubic, 1>(L, c, b, ds, integrate);
    } else {
        launch_force_n<kCubic, 0>(L, c, b, ds, integrate);
    }
    return 1;
}

}  // namespace sphx
