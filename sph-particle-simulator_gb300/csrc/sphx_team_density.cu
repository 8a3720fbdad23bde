// Density + pressure pass with four lanes per particle (see sphx_team.cuh).
#include "sphx_team.cuh"

namespace sphx {

constexpr int kDensityQueue = 128, kDensityWarps = 12;
struct DensityQueue {  // squared distances, masses and sorted positions
    float d2[kDensityQueue], m[kDensityQueue];
    uint32_t j[kDensityQueue];
};
struct DensityTeamSmem {
    TeamSmem<DensityQueue> walk;
    float fold[kTeamTile * kTeamTurn];  // a turn's terms, in order
};
static_assert(sizeof(DensityTeamSmem) % 16 == 0, "per-warp regions stay 16-byte aligned");

// Bound: dependent latency (0.4 instructions per cycle with the 2 warps per scheduler of a 10k
// set) and the number of instructions: 8,700 per tile in 22 steps of the walk, 17 chunks tested
// and 15 turns.  10k dam break 32 us, 4k 28 us (a lane per particle: 67 and 64).  Queues of 64
// entries take 38 turns of 8 where 128 take 27; turns of 16 share the loop between two pairs.
template <bool kBatch, int kKern, bool kNZ>
__global__ void __launch_bounds__(32 * kDensityWarps, 1) k_density_team(const StepConst cp, const Buffers b,
                                                         DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_raw_td[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane & (kTeam - 1), team = lane / kTeam;
    DensityTeamSmem* S = reinterpret_cast<DensityTeamSmem*>(smem_raw_td) + warp;
    DensityQueue& queue = S->walk.queue[team];
    const uint32_t qa = smem_u32(queue.d2);
    float4* const fold = reinterpret_cast<float4*>(S->fold + team * kTeamTurn);
    const uint32_t ntiles = ds->n_tiles;
    const F2 neg0{cp.lit.neg0};
    const bool nz = kNZ && !ds->general;
    uint32_t my_max = 0;
    const TileQueue tiles(&ds->work[0], b.num_sms);
    RecordRegion region(b, tiles, ntiles);
    for (uint32_t t = tiles.start(); t < ntiles; t = tiles.next(lane)) {
        const uint2 tile = b.tiles[t];
        const int scene = kBatch ? (int)b.scene_s[tile.x] : 0;
        const StepConst& c = kBatch ? b.scenes[scene].c : cp;
        const Geom g = kBatch ? scene_geom(b.scenes[scene], ds) : grid_geom(ds);
        Tile T;
        float4 xi;
        bool valid;
        int i;
        tile_setup(c, b, g, tile, team, T, i, xi, valid);
        const TileBox B = tile_box(xi, valid);
        const int room = (int)((region.end - region.cur) >> 2);  // rows
        uint32_t* const rec = b.records + (size_t)region.cur * 32 + lane * 4;
        float rho = xmul(xi.w, c.w0);
        uint32_t nn = 0, rows = 0;
        // the teams' queues start 16 entries apart, in different banks
        TeamQueue Q;
        const uint32_t turn0 = (uint32_t)team * kTeamTurn;
        auto turn = [&](bool last) {
            const bool act = last ? Q.done < rows * kTeamTurn : Q.have - Q.done >= (uint32_t)kTeamTurn;
            const uint32_t k = Q.done + 4 * sub, at = (turn0 + k) & (kDensityQueue - 1);
            const float4 d2 = *reinterpret_cast<const float4*>(&queue.d2[at]);
            const float4 m = *reinterpret_cast<const float4*>(&queue.m[at]);
            const int n = act ? (int)(Q.have - k) : 0;  // neighbours the lane may take
            const int row = (int)(Q.done / kTeamTurn);
            if (act && row < room) {
                const uint4 j = *reinterpret_cast<const uint4*>(&queue.j[at]);
                __stcs(reinterpret_cast<uint4*>(rec + row * 128),
                       make_uint4(n > 0 ? j.x : kNoSlot, n > 1 ? j.y : kNoSlot,
                                  n > 2 ? j.z : kNoSlot, n > 3 ? j.w : kNoSlot));
            }
            float2 w, z;
            if (nz) {
                w = upk2((f2(m.x, m.y) * pair_w_exact2<kKern>(cp.lit, c.pair, f2(d2.x, d2.y))).v);
                z = upk2((f2(m.z, m.w) * pair_w_exact2<kKern>(cp.lit, c.pair, f2(d2.z, d2.w))).v);
            } else {
                w.x = xmul(m.x, pair_w_exact<kKern>(c, d2.x));
                w.y = xmul(m.y, pair_w_exact<kKern>(c, d2.y));
                z.x = xmul(m.z, pair_w_exact<kKern>(c, d2.z));
                z.y = xmul(m.w, pair_w_exact<kKern>(c, d2.w));
            }
            // adding -0 leaves every float as it is
            fold[sub] = make_float4(n > 0 ? w.x : -0.0f, n > 1 ? w.y : -0.0f, n > 2 ? z.x : -0.0f,
                                    n > 3 ? z.y : -0.0f);
            __syncwarp();
#pragma unroll
            for (int o = 0; o < kTeam; ++o) {
                const float4 a = fold[o];
                rho = xadd(xadd(xadd(xadd(rho, a.x), a.y), a.z), a.w);
            }
            __syncwarp();
            if (act) Q.done += kTeamTurn;
        };
        team_walk<kDensityQueue>(
            b, g, T, B, i, xi, valid, c.r2, lane, &S->walk, neg0, Q, nn,
            [&](uint32_t hit, uint32_t& n4, float d2, float m, uint32_t j) {
                append3_if<kDensityQueue>(hit, n4, qa + ((n4 + 4 * turn0) & (4 * kDensityQueue - 1)),
                                          d2, m, j);
            },
            turn);
        // the rest: every team as many rows as the longest one's, the missing entries marked
        rows = __reduce_max_sync(kFull, (Q.have + kTeamTurn - 1) / kTeamTurn);
        while (__any_sync(kFull, Q.done < rows * kTeamTurn)) turn(true);
        if (b.records) {
            const bool fits = (int)rows <= room;
            if (lane == 0) b.tile_list[t] = make_uint2(fits ? region.cur : kNoSlot, rows);
            if (fits) region.cur += 4u * rows;
        }
        if (valid) {
            my_max = max(my_max, nn);
            if (sub == 0) {
                const float P = xmul(c.gas, xsub(rho, c.rest));
                // see k_density
                const float mr = xdiv(xi.w, rho);
                const bool in = pair_range(rho, P);
                b.aux4_s[i] = make_float4(rho, P, xmul(mr, c.visc),
                                          in ? __frcp_rn(xmul(2.0f, rho)) : 0.0f);
                if (!in) ds->general = 1;
                b.vel4_s[i].w = rho;
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) my_max = max(my_max, __shfl_xor_sync(kFull, my_max, o));
    if (lane == 0 && my_max) atomicMax(&ds->max_nn, (unsigned long long)my_max);
}

template <bool kBatch, int kKern, bool kNZ>
static void launch_team_t(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds) {
    constexpr int threads = 32 * kDensityWarps;
    constexpr size_t sm = kDensityWarps * sizeof(DensityTeamSmem);
    static LaunchShapeCache cache;
    const int nb = cached_resident_blocks(cache, L, k_density_team<kBatch, kKern, kNZ>, threads, sm);
    k_density_team<kBatch, kKern, kNZ><<<nb, threads, sm, L.stream>>>(c, b, ds);
}

template <int kKern>
static void launch_team_k(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds) {
    constexpr bool kDiv = kKern != SPHX_KERNEL_GAUSSIAN;
    const bool nz = kDiv && c.div_nz;
    if (b.nscenes > 0) {
        if (nz) launch_team_t<true, kKern, kDiv>(L, c, b, ds);
        else launch_team_t<true, kKern, false>(L, c, b, ds);
    } else if (nz) launch_team_t<false, kKern, kDiv>(L, c, b, ds);
    else launch_team_t<false, kKern, false>(L, c, b, ds);
}

int launch_density_team(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds) {
    if (c.kern == SPHX_KERNEL_WENDLAND_C2) launch_team_k<SPHX_KERNEL_WENDLAND_C2>(L, c, b, ds);
    else if (c.kern == SPHX_KERNEL_GAUSSIAN) launch_team_k<SPHX_KERNEL_GAUSSIAN>(L, c, b, ds);
    else launch_team_k<SPHX_KERNEL_CUBIC_SPLINE>(L, c, b, ds);
    return 1;
}

}  // namespace sphx
