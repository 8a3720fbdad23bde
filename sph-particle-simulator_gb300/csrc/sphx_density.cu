// Density + pressure pass of the step (compute_densities / compute_pressures,
// sph_engine.cpp:203-224, 370-388).
#include "sphx_passes.cuh"

namespace sphx {

// ---------------------------------------------------------------------------------------
// density + pressure:  rho_i = m_i W(0) + sum_{j in N(i), j != i} m_j W(r_ij)
//                      P_i = k (rho_i - rho0)
// (compute_density / compute_pressure, sph_engine.cpp:370-388)
// ---------------------------------------------------------------------------------------
// Per warp: the candidate ring as coordinate arrays (the distance test reads four candidates'
// x, y or z in one 128-bit load), their masses, the lanes' masks, the tile's row segments.
// 16 chunks (10.9 KB a warp, 20 warps per SM) let the lanes run as far apart as they want to
// on the lattice; 8 and 12 chunks (24 warps) took 1.08 and 1.03 ms on the 1M dam break where
// 16 take 0.97, 20 (16 warps) 1.05.
//
// Bound: instruction issue (72% of the slots) and the FP32 pipe (56%; a packed instruction
// holds it two cycles).  Of 882 warp instructions per particle about 220 are distance tests
// (900 kept candidates per tile, 29 chunks), 110 the walk, box cull and lists, 500 the pair terms
// (5 turns of two neighbours per lane and particle).  1M dam break: 0.96 ms; with hit lists
// worked through by the whole warp and folded back lane by lane (1,502 instructions, of which
// the lists and folds were half) 1.45 ms.  Five CTAs per SM leave 96 registers, at which 8 bytes
// spill; four without spill 1.00 ms.
constexpr int kDensityRing = 16;
struct DensitySmem {
    float cx[kDensityRing * 32], cy[kDensityRing * 32], cz[kDensityRing * 32];
    float cm[kDensityRing * 32];
    uint32_t mask[kDensityRing * 32];
    int2 seg[kMaxSegments + 1];
};
static_assert(sizeof(DensitySmem) % 16 == 0, "per-warp regions stay 16-byte aligned");

// If `on`: a candidate's coordinates and mass into the ring arrays and, if there is `room`, its
// position j into the tile's records (a streaming store: the records must not evict the
// candidates from L2).  Predicated stores; the compiler branches around them.
__device__ __forceinline__ void keep_candidate(uint32_t on, uint32_t slot, const float4& p,
                                               bool room, uint32_t* rec, uint32_t j) {
    constexpr int kArray = kDensityRing * 32 * 4;  // bytes
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %0, 0;\n\tsetp.ne.and.u32 q, %6, 0, p;\n\t"
        "@p st.shared.f32 [%1], %2;\n\t@p st.shared.f32 [%1+%9], %3;\n\t"
        "@p st.shared.f32 [%1+%10], %4;\n\t@p st.shared.f32 [%1+%11], %5;\n\t"
        "@q st.global.cs.u32 [%7], %8;\n\t}"
        ::"r"(on), "r"(slot), "f"(p.x), "f"(p.y), "f"(p.z), "f"(p.w), "r"((uint32_t)room), "l"(rec),
        "r"(j), "n"(kArray), "n"(2 * kArray), "n"(3 * kArray) : "memory");
}

// kNZ: the pair forms' divisions are in range (StepConst::div_nz)
template <bool kBatch, int kKern, bool kNZ>
__global__ void __launch_bounds__(128, 5) k_density(const StepConst cp, const Buffers b,
                                                    DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_raw_d[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    DensitySmem* S = reinterpret_cast<DensitySmem*>(smem_raw_d) + warp;
    const uint32_t ntiles = ds->n_tiles;
    const uint32_t lt = (1u << lane) - 1u;
    const F2 neg0{cp.lit.neg0};
    const bool nz = kNZ && !ds->general;
    uint32_t my_max = 0;
    const TileQueue queue(&ds->work[0], b.num_sms);
    RecordRegion region(b, queue, ntiles);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        const uint2 tile = b.tiles[t];
        const int scene = kBatch ? (int)b.scene_s[tile.x] : 0;
        const StepConst& c = kBatch ? b.scenes[scene].c : cp;
        const Geom g = kBatch ? scene_geom(b.scenes[scene], ds) : grid_geom(ds);
        const float r2m = c.r2 * 1.0001f;
        Tile T;
        float4 xi;
        bool valid;
        int i;
        tile_setup(c, b, g, tile, lane, T, i, xi, valid);
        const TileBox B = tile_box(xi, valid);
        __syncwarp();  // the previous tile's segments are read
        const int nseg = build_segments(b, g, T, lane, S->seg);
        __syncwarp();
        // records of this tile: per chunk of 32 kept candidates their sorted positions, then
        // the lanes' masks
        const int room = (int)((region.end - region.cur) >> 1);  // chunks
        uint32_t* const rec = b.records + (size_t)region.cur * 32;
        RawStream st(S->seg, nseg);
        float4 pl = make_float4(0.f, 0.f, 0.f, 0.f);  // the next chunk's candidate, read ahead
        if (st.more() && lane < st.count()) pl = b.pos4_s[st.s + lane];
        float rho = xmul(xi.w, c.w0);
        uint32_t nn = 0;
        int kept = 0, tested = 0, head = 0, self = -1;
        RingLane<kDensityRing> at;
        for (;;) {
            __syncwarp();  // every lane is done with the chunks before head
            while (st.more() && kept + 32 <= (head + kDensityRing) * 32) {
                const int m = st.count(), s = st.s;
                const uint32_t surv =
                    __ballot_sync(kFull, lane < m && box_near(B, pl, r2m));
                const int a = kept + __popc(surv & lt);
                keep_candidate((surv >> lane) & 1u, smem_u32(&S->cx[ring_slot<kDensityRing>(a)]), pl,
                               (a >> 5) < room, rec + (a >> 5) * 64 + (a & 31), (uint32_t)(s + lane));
                if ((unsigned)(i - s) < (unsigned)m) self = kept + __popc(surv & ((1u << (i - s)) - 1u));
                st.next();
                if (st.more() && lane < st.count()) pl = b.pos4_s[st.s + lane];
                kept += __popc(surv);
                while ((kept >> 5) > tested || (!st.more() && kept > tested * 32)) {
                    __syncwarp();
                    const int f = (tested % kDensityRing) * 32;
                    uint32_t mask = ring_hits(S->cx + f, S->cy + f, S->cz + f, xi, c.r2, neg0);
                    mask = valid ? mask & chunk_valid(kept - tested * 32) : 0u;
                    nn += __popc(mask);
                    if (self >> 5 == tested) mask &= ~(0x80000000u >> (self & 31));
                    if (tested < room) __stcs(rec + tested * 64 + 32 + lane, mask);
                    S->mask[f + lane] = mask;
                    ++tested;
                }
            }
            // the lanes' neighbours in the ring; while candidates are left, until no lane
            // needs the oldest chunk any more
            const int until = st.more() ? head + 1 : tested;
            for (;;) {
                at.advance(S->mask, tested, lane);
                if (!__any_sync(kFull, at.need() < until)) break;
                int qa, qb;
                bool ha, hb;
                at.take2(qa, qb, ha, hb);
                if (nz) {
                    const F2 d2 = pair_d2(f2(xi.x) - f2(S->cx[qa], S->cx[qb]),
                                          f2(xi.y) - f2(S->cy[qa], S->cy[qb]),
                                          f2(xi.z) - f2(S->cz[qa], S->cz[qb]), neg0);
                    const float2 w = upk2((f2(S->cm[qa], S->cm[qb]) *
                                           pair_w_exact2<kKern>(cp.lit, c.pair, d2)).v);
                    if (ha) rho = xadd(rho, w.x);
                    if (hb) rho = xadd(rho, w.y);
                } else {
                    auto add = [&](int q) {
                        const float4 xj = make_float4(S->cx[q], S->cy[q], S->cz[q], S->cm[q]);
                        rho = xadd(rho,
                                   xmul(xj.w, pair_w_exact<kKern>(c, diff_d2(xi, xj))));
                    };
                    if (ha) add(qa);
                    if (hb) add(qb);
                }
            }
            if (!st.more()) break;
            head = __reduce_min_sync(kFull, at.need());
        }
        if (b.records) {
            const bool fits = tested <= room;
            if (lane == 0) b.tile_list[t] = make_uint2(fits ? region.cur : kNoSlot, (uint32_t)kept);
            if (fits) region.cur += 2u * (uint32_t)tested;
        }
        if (valid) {
            const float P = xmul(c.gas, xsub(rho, c.rest));
            // the per-candidate factors of the force pass's pair terms, each formed once here
            // with the rounding the reference applies per pair: (rho, P, (m / rho) mu, 1 / 2 rho)
            const float mr = xdiv(xi.w, rho);
            // (0: the force pass takes the particle's pairs in the general form)
            const bool in = pair_range(rho, P);
            b.aux4_s[i] = make_float4(rho, P, xmul(mr, c.visc),
                                      in ? __frcp_rn(xmul(2.0f, rho)) : 0.0f);
            if (!in) ds->general = 1;
            b.vel4_s[i].w = rho;  // read with the candidate's velocity by the force pass
            my_max = max(my_max, nn);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) my_max = max(my_max, __shfl_xor_sync(kFull, my_max, o));
    if (lane == 0 && my_max) atomicMax(&ds->max_nn, (unsigned long long)my_max);
}

template <bool kBatch, int kKern, bool kNZ>
static void launch_density_t(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                             DevState* ds) {
    const int threads = 32 * L.warps_per_block;
    const size_t sm = (size_t)L.warps_per_block * sizeof(DensitySmem);
    static LaunchShapeCache cache;
    const int nb = cached_resident_blocks(cache, L, k_density<kBatch, kKern, kNZ>, threads, sm);
    k_density<kBatch, kKern, kNZ><<<nb, threads, sm, L.stream>>>(c, b, ds);
}

template <int kKern>
static void launch_density_k(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                             DevState* ds) {
    // the Gaussian divides by neither h nor h^2
    constexpr bool kDiv = kKern != SPHX_KERNEL_GAUSSIAN;
    const bool nz = kDiv && c.div_nz;
    if (b.nscenes > 0) {
        if (nz) launch_density_t<true, kKern, kDiv>(L, c, b, ds);
        else launch_density_t<true, kKern, false>(L, c, b, ds);
    } else if (nz) launch_density_t<false, kKern, kDiv>(L, c, b, ds);
    else launch_density_t<false, kKern, false>(L, c, b, ds);
}

// Precision mode (single scene) runs the tile sweep (sphx_sweep.cu); exact mode k_density, or on
// tiles of at most 8 particles (small sets: pass_tile) k_density_team.
int launch_density(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds) {
    if (c.precise && b.nscenes == 0) return launch_density_sweep(L, c, b, ds);
    if (b.tile_n <= kTeamTile) return launch_density_team(L, c, b, ds);
    if (c.kern == SPHX_KERNEL_WENDLAND_C2) launch_density_k<SPHX_KERNEL_WENDLAND_C2>(L, c, b, ds);
    else if (c.kern == SPHX_KERNEL_GAUSSIAN) launch_density_k<SPHX_KERNEL_GAUSSIAN>(L, c, b, ds);
    else launch_density_k<SPHX_KERNEL_CUBIC_SPLINE>(L, c, b, ds);
    return 1;
}

}  // namespace sphx
