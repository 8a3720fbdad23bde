// Force + acceleration (+ leapfrog + wall clamp) pass with four lanes per particle (see
// sphx_team.cuh).
#include "sphx_team.cuh"

namespace sphx {

constexpr int kForceQueue = 64, kForceWarps = 12;
struct ForceQueue {
    uint32_t j[kForceQueue];  // sorted positions
};
// A particle's terms of one turn: per component (px, py, pz, vx, vy, vz) those of its 16
// neighbours in order, 20 floats apart; with 144 floats a particle the lanes' 128-bit stores
// and loads fall into different banks.
constexpr int kFoldComp = kTeamTurn + 4, kFoldStride = 144;
struct ForceTeamSmem {
    float fold[kTeamTile * kFoldStride];
    TeamSmem<ForceQueue> walk;  // for tiles without a list
};
static_assert(sizeof(ForceTeamSmem) % 16 == 0, "per-warp regions stay 16-byte aligned");

// Two neighbours of the lane's particle.
struct Gathered {
    float4 xa, xb, va, vb;
    float2 fa, fb;
    bool ha, hb;  // a missing one holds the values of the lane's own particle
    __device__ __forceinline__ void load(const Buffers& b, uint32_t ja, uint32_t jb, int own) {
        ha = ja != kNoSlot;
        hb = jb != kNoSlot;
        const uint32_t a = ha ? ja : (uint32_t)own, q = hb ? jb : (uint32_t)own;
        xa = b.pos4_s[a];
        xb = b.pos4_s[q];
        va = b.vel4_s[a];
        vb = b.vel4_s[q];
        fa = *reinterpret_cast<const float2*>(&b.aux4_s[a].z);
        fb = *reinterpret_cast<const float2*>(&b.aux4_s[q].z);
    }
};

// force_term with the pressure part negated (the general form; a call of its own, so that the
// other keeps its registers)
struct Terms6 {
    float v[6];
};
template <int K>
__device__ __noinline__ Terms6 general_terms(const StepConst& c, float4 xt, float4 vt, float Pt,
                                             float4 xj, float4 vj, float2 fj) {
    float p3[3], v3[3];
    const float Pj = xmul(c.gas, xsub(vj.w, c.rest));
    force_term<K>(c, xt, vt, Pt, xj, vj, make_float4(vj.w, Pj, xmul(2.0f, vj.w), fj.x), p3, v3);
    return {{-p3[0], -p3[1], -p3[2], v3[0], v3[1], v3[2]}};
}

// Reads the density pass's rows and gathers the neighbours' data straight into registers, a
// pair ahead; the 26 KB that a tile touches stay in L1.  Bound: the L1 wavefronts of the gathers
// (62% of the peak while it runs, on the SMs with three warps per scheduler 77%).  10k dam break
// 25 us, 4k 17 us (a lane per particle, candidates staged in shared memory: 67 and 60).
template <bool kBatch, int kKern, bool kNZ>
__global__ void __launch_bounds__(32 * kForceWarps, 1) k_force_team(const StepConst cp, const Buffers b,
                                                       DevState* ds, int integrate) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_raw_tf[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane & (kTeam - 1), team = lane / kTeam;
    ForceTeamSmem* S = reinterpret_cast<ForceTeamSmem*>(smem_raw_tf) + warp;
    uint32_t* const queue = S->walk.queue[team].j;
    const uint32_t qa = smem_u32(queue);
    const uint32_t ntiles = ds->n_tiles;
    const PairLits& lit = cp.lit;
    const bool nz = kNZ && !ds->general;
    // the components that the lane sums: sub, and 4 + sub in the team's first two lanes
    float* const fold = S->fold + team * kFoldStride;
    const float4* const fold0 = reinterpret_cast<const float4*>(fold + sub * kFoldComp);
    const float4* const fold1 = reinterpret_cast<const float4*>(fold + min(4 + sub, 5) * kFoldComp);
    const TileQueue tiles(&ds->work[1], b.num_sms);
    for (uint32_t t = tiles.start(); t < ntiles; t = tiles.next(lane)) {
        const uint2 tile = b.tiles[t];
        const int scene = kBatch ? (int)b.scene_s[tile.x] : 0;
        const StepConst& c = kBatch ? b.scenes[scene].c : cp;
        const uint2 list = b.records ? b.tile_list[t] : make_uint2(kNoSlot, 0u);
        const bool valid = team < (int)tile.y;
        const int i = valid ? (b.tgt ? (int)b.tgt[tile.x + team] : (int)tile.x + team) : (int)tile.x;
        const float4 xi = b.pos4_s[i];
        const float4 vi = b.vel4_s[i];
        const float Pi = b.aux4_s[i].y;
        float s0 = 0.0f, s1 = 0.0f;
        float2 w[2][6];  // the terms of a turn's two pairs
        auto terms = [&](const Gathered& G, float2* w) {
            if (nz) {
                PairStart p;
                p.start(lit, xi, G.xa, G.xb);
                const PairTerms q = pair_terms<kKern>(lit, c.pair, vi, Pi, p, G.va, G.vb, G.fa, G.fb);
                w[0] = upk2(q.px.v);
                w[1] = upk2(q.py.v);
                w[2] = upk2(q.pz.v);
                w[3] = upk2(q.wx.v);
                w[4] = upk2(q.wy.v);
                w[5] = upk2(q.wz.v);
            } else {
                const Terms6 ta = general_terms<kKern>(c, xi, vi, Pi, G.xa, G.va, G.fa);
                const Terms6 tb = general_terms<kKern>(c, xi, vi, Pi, G.xb, G.vb, G.fb);
#pragma unroll
                for (int k = 0; k < 6; ++k) w[k] = make_float2(ta.v[k], tb.v[k]);
            }
            if (!__all_sync(kFull, G.hb)) {  // adding -0 leaves every float as it is
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    if (!G.ha) w[k].x = -0.0f;
                    if (!G.hb) w[k].y = -0.0f;
                }
            }
        };
        auto add = [&]() {  // the turn's terms, in order
#pragma unroll
            for (int k = 0; k < 6; ++k)
                *reinterpret_cast<float4*>(fold + k * kFoldComp + 4 * sub) =
                    make_float4(w[0][k].x, w[0][k].y, w[1][k].x, w[1][k].y);
            __syncwarp();
#pragma unroll
            for (int o = 0; o < kTeam; ++o) {
                const float4 a = fold0[o], e = fold1[o];
                s0 = xadd(xadd(xadd(xadd(s0, a.x), a.y), a.z), a.w);
                s1 = xadd(xadd(xadd(xadd(s1, e.x), e.y), e.z), e.w);
            }
            __syncwarp();
        };
        if (list.x != kNoSlot) {
            // the density pass's rows: 16 neighbours of each particle, 4 per lane; read a row
            // ahead, their neighbours' data a pair ahead
            const int rows = (int)list.y;
            const uint32_t* rec = b.records + (size_t)list.x * 32 + lane * 4;
            const uint4 none = make_uint4(kNoSlot, kNoSlot, kNoSlot, kNoSlot);
            uint4 j = rows > 0 ? __ldcs(reinterpret_cast<const uint4*>(rec)) : none;
            Gathered even, odd;
            even.load(b, j.x, j.y, i);
            for (int r = 1; r <= rows; ++r) {
                rec += 128;
                const uint4 jn = r < rows ? __ldcs(reinterpret_cast<const uint4*>(rec)) : none;
                odd.load(b, j.z, j.w, i);
                terms(even, w[0]);
                even.load(b, jn.x, jn.y, i);
                terms(odd, w[1]);
                add();
                j = jn;
            }
        } else {  // the walk, culled and tested again
            const Geom g = kBatch ? scene_geom(b.scenes[scene], ds) : grid_geom(ds);
            Tile T;
            float4 xt;
            bool vt;
            int it;
            tile_setup(c, b, g, tile, team, T, it, xt, vt);
            const TileBox B = tile_box(xt, vt);
            TeamQueue Q;
            uint32_t nn = 0, rows = 0;
            const uint32_t turn0 = (uint32_t)team * kTeamTurn;
            auto turn = [&](bool last) {
                const bool act =
                    last ? Q.done < rows * kTeamTurn : Q.have - Q.done >= (uint32_t)kTeamTurn;
                const uint32_t k = Q.done + 4 * sub;
                const uint4 e = *reinterpret_cast<const uint4*>(
                    queue + ((turn0 + k) & (kForceQueue - 1)));
                const int n = act ? (int)(Q.have - k) : 0;  // neighbours the lane may take
                Gathered G;
                G.load(b, n > 0 ? e.x : kNoSlot, n > 1 ? e.y : kNoSlot, i);
                terms(G, w[0]);
                G.load(b, n > 2 ? e.z : kNoSlot, n > 3 ? e.w : kNoSlot, i);
                terms(G, w[1]);
                add();
                if (act) Q.done += kTeamTurn;
            };
            team_walk<kForceQueue>(
                b, g, T, B, it, xt, vt, c.r2, lane, &S->walk, F2{lit.neg0}, Q, nn,
                [&](uint32_t hit, uint32_t& n4, float, float, uint32_t j) {
                    append_if(hit, n4, qa + ((n4 + 4 * turn0) & (4 * kForceQueue - 1)), j);
                },
                turn);
            rows = __reduce_max_sync(kFull, (Q.have + kTeamTurn - 1) / kTeamTurn);
            while (__any_sync(kFull, Q.done < rows * kTeamTurn)) turn(true);
        }
        const float px = __shfl_sync(kFull, s0, 0, kTeam), py = __shfl_sync(kFull, s0, 1, kTeam),
                    pz = __shfl_sync(kFull, s0, 2, kTeam), fx = __shfl_sync(kFull, s0, 3, kTeam),
                    fy = __shfl_sync(kFull, s1, 0, kTeam), fz = __shfl_sync(kFull, s1, 1, kTeam);
        if (!valid || sub != 0) continue;
        const float mi = xi.w;
        const float acc[3] = {xdiv(xadd(xadd(px, fx), xmul(0.0f, mi)), mi),
                              xdiv(xadd(xadd(py, fy), xmul(c.grav, mi)), mi),
                              xdiv(xadd(xadd(pz, fz), xmul(0.0f, mi)), mi)};
        b.acc4_s[i] = make_float4(acc[0], acc[1], acc[2], 0.0f);
        if (!integrate) continue;
        const float dt = kBatch ? b.scenes[scene].dt : ds->dt;
        const uint32_t id = b.id_s[i];
        float x[3] = {xi.x, xi.y, xi.z}, v[3] = {vi.x, vi.y, vi.z};
        leapfrog_exact(c, dt, acc, x, v);
        b.pos4[id] = make_float4(x[0], x[1], x[2], mi);
        b.vel4[id] = make_float4(v[0], v[1], v[2], 0.0f);
        if (kBatch) {
            if (id == b.scenes[scene].start) {  // accelerations_[0] of the scene
                for (int a = 0; a < 3; ++a) b.scenes[scene].a0[a] = acc[a];
            }
        } else if (id == 0) {
            for (int a = 0; a < 3; ++a) ds->a0[a] = acc[a];
        }
    }
}

template <bool kBatch, int kKern, bool kNZ>
static void launch_team_t(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                          int integrate) {
    constexpr int threads = 32 * kForceWarps;
    constexpr size_t sm = kForceWarps * sizeof(ForceTeamSmem);
    static LaunchShapeCache cache;
    const int nb = cached_resident_blocks(cache, L, k_force_team<kBatch, kKern, kNZ>, threads, sm);
    k_force_team<kBatch, kKern, kNZ><<<nb, threads, sm, L.stream>>>(c, b, ds, integrate);
}

template <int kKern>
static void launch_team_k(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                          int integrate) {
    constexpr bool kPairs = kKern != SPHX_KERNEL_GAUSSIAN;
    const bool nz = kPairs && c.force_nz == 2;
    if (b.nscenes > 0) {
        if (nz) launch_team_t<true, kKern, kPairs>(L, c, b, ds, integrate);
        else launch_team_t<true, kKern, false>(L, c, b, ds, integrate);
    } else if (nz) launch_team_t<false, kKern, kPairs>(L, c, b, ds, integrate);
    else launch_team_t<false, kKern, false>(L, c, b, ds, integrate);
}

int launch_force_team(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                      int integrate) {
    if (c.kern == SPHX_KERNEL_WENDLAND_C2) launch_team_k<SPHX_KERNEL_WENDLAND_C2>(L, c, b, ds, integrate);
    else if (c.kern == SPHX_KERNEL_GAUSSIAN) launch_team_k<SPHX_KERNEL_GAUSSIAN>(L, c, b, ds, integrate);
    else launch_team_k<SPHX_KERNEL_CUBIC_SPLINE>(L, c, b, ds, integrate);
    return 1;
}

}  // namespace sphx
