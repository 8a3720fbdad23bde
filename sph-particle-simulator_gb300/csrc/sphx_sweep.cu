// Precision-mode neighbour passes: density + pressure, and force + acceleration + leapfrog +
// wall clamp, of the cell + offset step (compute_densities / compute_pressures /
// compute_forces, sph_engine.cpp:203-244, 370-443; integrate_leapfrog, cpp:290-310;
// apply_boundary_conditions, particle.cpp:122-153).
//
// The precision mode is judged against an FP64 evaluation, not against the reference's
// summation order, so its passes sweep: one warp owns one tile (up to 32 particles of one cell
// column, one per lane), appends the candidates its box can reach to a small buffer in shared
// memory in the tile's frame, and whenever 32 have come together every lane evaluates all of
// them against its own particle, two per packed FP32 instruction and without branches: the
// pair's term is formed whatever the distance and is zero (or zeroed) when the candidate is
// not a neighbour.  Every lane is busy on every instruction and the terms are independent of
// one another; the price is the terms of the non-neighbours (about two of three), which costs
// less here than taking each lane's neighbours one by one (the exact passes' way, whose terms
// are four times as long: 0.90 and 1.49 ms for density and force on the 1M dam break).  The
// density pass also lists the kept candidates that are a neighbour of some lane at all (750 of
// 920 per tile); the force pass sweeps only those.
//
// The particle itself is swept like any other: its W is W(0) (the reference's m_i W(0)
// term) and its force terms are zero (r = 0 gives a zero gradient; v_i - v_i = 0).
//
// Smoothing kernels in the "max form" (a = max(2 - q, 0), b = max(1 - q, 0) for the cubic
// spline), which is zero beyond the support without a test:
//   cubic spline  dW/dq = sigma/2 (4 b^2 - a^2), d2W/dq2 = sigma (a - 4 b) (kernels.cpp:23-60,
//                 piecewise there); W itself keeps the piecewise form (sweep_w)
//   Wendland C2   t = max(1 - q/2, 0):  W = norm t^4 (1 + 2 q), dW/dq = -5 norm t^3 q,
//                 laplacian = norm (5/h^2) t^2 (5 q - 3)      (kernels.cpp:172-200)
//   Gaussian      no compact support: every term is masked by the neighbour test
//                                                             (kernels.cpp:210-225)
// A pair is a neighbour when |r|^2 <= r_search^2 (spatial_hash.cpp:46-50); when the search
// radius is at least the support 2h, the max form already zeroes every non-neighbour and
// the terms need no selection (kCut = false).
//
// Positions are in units of h (the tile's frame scaled by 1/h): |r|/h = q comes without a
// multiplication, and every force term that needs the direction uses r_vec / |r|, which is
// the same in any unit.  The pressure term of a pair closer than 1e-6 m, which the reference
// skips, is formed here (it is at most |grad W| 1e-6 m, far below the stated bound; a
// coincident pair, |r| = 0, gives exactly 0 as in the reference).
#include "sphx_passes.cuh"

namespace sphx {

namespace {

__device__ __forceinline__ F2 keep(bool ka, bool kb, F2 a) {
    const float2 u = upk2(a.v);
    return f2(ka ? u.x : 0.0f, kb ? u.y : 0.0f);
}

// hardware square root (a few ulp)
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float exp_approx(float x) { return __expf(x); }

// position of an empty slot: far enough to be no particle's neighbour, near
// enough that every term formed from it stays finite (|r|^2 of 3e30)
constexpr float kFar = 1.0e15f;

// The sweeps' lengths in units of h.
struct SweepUnits {
    float inv;   // 1/h: metres -> sweep units
    float cs;    // the cell size in sweep units
    float r2;    // r_search^2 / h^2: the neighbour test
    float r2m;   // the same with the box cull's margin
    float skip2; // (1e-6 m / h)^2: the Gaussian's pressure-term skip
};
__device__ __forceinline__ SweepUnits sweep_units(const StepConst& c) {
    return SweepUnits{c.rcp_h, c.sw_cs, c.sw_r2, c.sw_r2m, c.sw_skip2};
}
// A particle (cell, offset o, mass in o.w) in the tile's frame, in sweep units: the cell
// difference times the cell size plus the offset scaled, one rounding each (as frame_pos
// does in metres).
__device__ __forceinline__ float4 frame_pos_h(const int4& cell, const int4& frame,
                                              const float4& o, const SweepUnits& U) {
    return make_float4(fmaf((float)(cell.x - frame.x), U.cs, o.x * U.inv),
                       fmaf((float)(cell.y - frame.y), U.cs, o.y * U.inv),
                       fmaf((float)(cell.z - frame.z), U.cs, o.z * U.inv), o.w);
}

// W of two pairs (d2 = (|r|/h)^2 of each) up to the kernel's constant factor
// (sweep_w_scale); the Gaussian's exp(-|r|^2 / h^2) is exp(-d2).  The cubic spline is the
// reference's piecewise polynomial (2/3 - q^2 + q^3/2 on [0, 1], (2 - q)^3 / 6 beyond, with
// 2 - q clamped at 0), selected per pair: no cancellation at small q.
template <int K>
__device__ __forceinline__ F2 sweep_w(const StepConst& c, F2 d2) {
    const float2 e = upk2(d2.v);
    if (K == SPHX_KERNEL_GAUSSIAN) return f2(exp_approx(-e.x), exp_approx(-e.y));
    const F2 q = f2(sqrt_approx(e.x), sqrt_approx(e.y));
    if (K == SPHX_KERNEL_WENDLAND_C2) {
        const F2 t = max0(fma2(q, F2{c.lit.neg_half}, F2{c.lit.one}));
        const F2 t2 = t * t;
        return (t2 * t2) * fma2(q, F2{c.lit.two}, F2{c.lit.one});
    }
    const F2 w1 = fma2(q * q, fma2(q, F2{c.lit.half}, F2{c.lit.neg1}), F2{c.lit.two_thirds});
    const F2 t = max0(F2{c.lit.two} - q);
    const F2 w2 = (t * t) * (t * F2{c.lit.one_sixth});
    const float2 qv = upk2(q.v), a = upk2(w1.v), bb = upk2(w2.v);
    return f2(qv.x <= 1.0f ? a.x : bb.x, qv.y <= 1.0f ? a.y : bb.y);
}
__host__ __device__ __forceinline__ float sweep_w_scale(const StepConst& c) {
    return c.kern == SPHX_KERNEL_CUBIC_SPLINE ? c.sigma : c.wnorm;
}

// ---------------------------------------------------------------------------------------
// density + pressure
// ---------------------------------------------------------------------------------------
// Candidates kept by the tile wait in a buffer of two chunks of 32; a chunk is swept once
// complete (the last one padded with empty slots: far, without mass).
struct SweepDensitySmem {
    float cx[64], cy[64], cz[64], cm[64];  // tile frame; mass
    uint32_t idx[64];                      // sorted position
    int2 seg[kMaxSegments + 1];
};
static_assert(sizeof(SweepDensitySmem) % 16 == 0, "per-warp regions stay 16-byte aligned");
// The spread tiles' launch (sweep_density_spread) stages whole candidates.
struct SweepDensitySpreadSmem {
    int2 seg[kMaxSegments];
    int4 scell[32];   // candidate j of the chunk: its cell
    float4 soff[32];  // its offset in sweep units, mass
};

// A tile is spread when one of its particles lies more than kSpreadCells cells from the
// frame (a folded grid puts far cells together; on an unfolded grid the column runs keep
// every tile within kRunCells cells of its first particle's cell): frame
// coordinates that large would carry rounding of the size of their magnitude, so such a
// tile sweeps with each lane's own cell as its frame (the separation of a pair is
// (cell_j - cell_t) cs + (o_j - o_t), the cell difference exact), unculled, one candidate
// pair at a time.  Rare and slow; exact to the same few ulps as a compact tile.
constexpr int kSpreadCells = 4;
static_assert(kRunCells <= kSpreadCells, "a run's tiles would be spread");
// cell difference a - b as a float (wrapping: cells are clamped to +-2^30, so only a pair
// that far apart can wrap, and it stays far)
__device__ __forceinline__ float cdiff(int a, int b) {
    return (float)(int)((unsigned)a - (unsigned)b);
}
__device__ __forceinline__ bool far_cell(const int4& c, const int4& f) {
    return fabsf(cdiff(c.x, f.x)) > kSpreadCells || fabsf(cdiff(c.y, f.y)) > kSpreadCells ||
           fabsf(cdiff(c.z, f.z)) > kSpreadCells;
}
// A spread tile's offset o / h (sweep units) and mass.  The products are rounded on their
// own (__fmul_rn): the lane's particle and its own staged copy then give a separation of
// exactly 0, where a product contracted into the difference (fma(o, 1/h, -o')) would leave
// its rounding error, a separation of ~1e-8 h whose gradient term does not vanish.
__device__ __forceinline__ float4 spread_off(const float4& o, const SweepUnits& U) {
    return make_float4(__fmul_rn(o.x, U.inv), __fmul_rn(o.y, U.inv), __fmul_rn(o.z, U.inv),
                       o.w);
}
// separations (sweep units) of candidates a, b from the lane's particle (cell ct, offset ot)
__device__ __forceinline__ void spread_sep(const SweepUnits& U, const int4& ct, const float4& ot,
                                           const int4& ca, const float4& oa, const int4& cb,
                                           const float4& ob, F2& dx, F2& dy, F2& dz) {
    dx = f2(fmaf(cdiff(ct.x, ca.x), U.cs, ot.x - oa.x), fmaf(cdiff(ct.x, cb.x), U.cs, ot.x - ob.x));
    dy = f2(fmaf(cdiff(ct.y, ca.y), U.cs, ot.y - oa.y), fmaf(cdiff(ct.y, cb.y), U.cs, ot.y - ob.y));
    dz = f2(fmaf(cdiff(ct.z, ca.z), U.cs, ot.z - oa.z), fmaf(cdiff(ct.z, cb.z), U.cs, ot.z - ob.z));
}

// The density sweep of a spread tile: every candidate of every chunk against the lane's
// particle in the lane's own frame (ct, ot: its cell and offset in sweep units).
template <int kKern>
__device__ __forceinline__ void sweep_density_spread(const StepConst& c, const Buffers& b,
                                                  const SweepUnits& U,
                                                  SweepDensitySpreadSmem* S,
                                                  int nseg, int lane, bool valid, int4 ct,
                                                  float4 ot, KSum& rk, uint32_t& nn) {
    for (int sg = 0; sg < nseg; ++sg) {
        const int2 se = S->seg[sg];
        for (int s = se.x; s < se.y; s += 32) {
            const int m = min(32, se.y - s);
            __syncwarp();
            if (lane < m) {
                const float4 o = b.pos4_s[s + lane];
                S->scell[lane] = b.cell4_s[s + lane];
                S->soff[lane] = spread_off(o, U);
            } else {  // empty slot: far, no mass
                S->scell[lane] = ct;
                S->soff[lane] = make_float4(kFar, kFar, kFar, 0.0f);
            }
            __syncwarp();
            F2 acc = f2(0.0f);
            for (int j = 0; j < m; j += 2) {
                F2 dx, dy, dz;
                spread_sep(U, ct, ot, S->scell[j], S->soff[j], S->scell[j + 1], S->soff[j + 1],
                           dx, dy, dz);
                const F2 d2 = fma2(dx, dx, fma2(dy, dy, dz * dz));
                const float2 e = upk2(d2.v);
                const bool ha = valid && e.x <= U.r2, hb = valid && e.y <= U.r2;
                nn += (uint32_t)ha + (uint32_t)hb;
                acc = fma2(f2(S->soff[j].w, S->soff[j + 1].w), keep(ha, hb, sweep_w<kKern>(c, d2)),
                           acc);
            }
            const float2 a2 = upk2(acc.v);
            rk.add(a2.x + a2.y);
        }
    }
}

// The density epilogue of the lane's particle: rho, P and the force sweep's per-candidate
// factor m / (2 rho) (the viscosity's is a multiple of it: StepConst::sw_kappa).
__device__ __forceinline__ void density_out(const StepConst& c, const Buffers& b, int i,
                                            bool cells, float mi, const KSum& rk) {
    const float rho = cells ? rk.value() * sweep_w_scale(c) : xmul(mi, c.w0);
    const float P = xmul(c.gas, xsub(rho, c.rest));
    const float mr = xdiv(mi, rho);
    b.aux4_s[i] = make_float4(rho, P, 0.5f * mr, 0.0f);
}

// A tile with a particle more than kSpreadCells cells from its frame (listed for the
// spread launch by the density pass, skipped by both passes).
__device__ __forceinline__ bool spread_tile(const Tile& T, const int4& cell, bool valid,
                                            const int4& frame) {
    return T.cells && __any_sync(kFull, valid && far_cell(cell, frame));
}

// A chunk's terms added to acc; returns the mask of the lane's neighbours in it (bit 31 - j:
// slot j; quads past nq unset).
template <int kKern, bool kCut>
__device__ __forceinline__ uint32_t sweep_density_chunk(const StepConst& c, const float* cx,
                                                        const float* cy, const float* cz,
                                                        const float* cm, int nq, F2 X, F2 Y, F2 Z,
                                                        float r2, F2& acc) {
    const F2 R2 = f2(r2);
    uint32_t miss = 0;
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
        const ulonglong2 x = reinterpret_cast<const ulonglong2*>(cx)[q];
        const ulonglong2 y = reinterpret_cast<const ulonglong2*>(cy)[q];
        const ulonglong2 z = reinterpret_cast<const ulonglong2*>(cz)[q];
        const ulonglong2 m = reinterpret_cast<const ulonglong2*>(cm)[q];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const F2 dx = X - F2{h ? x.y : x.x}, dy = Y - F2{h ? y.y : y.x},
                     dz = Z - F2{h ? z.y : z.x};
            const F2 d2 = fma2(dx, dx, fma2(dy, dy, dz * dz));
            const float2 t = upk2((R2 - d2).v);  // negative: not a neighbour
            miss = __funnelshift_l(__float_as_uint(t.x), miss, 1);
            miss = __funnelshift_l(__float_as_uint(t.y), miss, 1);
            F2 w = sweep_w<kKern>(c, d2);
            if (kCut) w = keep(!(t.x < 0.0f), !(t.y < 0.0f), w);
            acc = fma2(F2{h ? m.y : m.x}, w, acc);
        }
    }
    return ~miss << (32 - 4 * nq);
}

// kCut: the search radius is below the support 2h (or the kernel is the Gaussian): W is
// selected by the neighbour test; otherwise W is already 0 beyond 2h and the test only
// counts the neighbours and finds the candidates some lane needs.
//
// Bound: instruction issue (73% of the slots) and the FP32 pipe: 653 warp instructions per
// particle, of which 415 are the chunks (27.7 per pair of candidates, 29 chunks a tile) and
// most of the rest the walk of 55 chunks of 32, its conversion to the tile's frame and its box
// cull.  1M dam break: 0.74 ms (0.76 with a sweep of each culled chunk on its own, without the
// list for the force pass).  Six CTAs per SM leave 80 registers, at which up to 12 bytes spill;
// five without spill take as long.
template <int kKern, bool kCut>
__global__ void __launch_bounds__(128, 6) k_density_sweep(const StepConst c, const Buffers b,
                                                          DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_sweep_d[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepDensitySmem* S = reinterpret_cast<SweepDensitySmem*>(smem_sweep_d) + warp;
    const uint32_t ntiles = ds->n_tiles;
    const uint32_t lt = (1u << lane) - 1u;
    const Geom g = grid_geom(ds);
    const SweepUnits U = sweep_units(c);
    uint32_t my_max = 0;
    const TileQueue queue(&ds->work[0], b.num_sms);
    RecordRegion region(b, queue, ntiles);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        Tile T;
        int i;
        int4 cell, frame;
        float4 o;
        bool valid;
        tile_setup_cells(c, b, g, b.tiles[t], lane, T, i, cell, o, valid, frame);
        if (spread_tile(T, cell, valid, frame)) {
            if (lane == 0) b.spread_tiles[atomicAdd(&ds->n_spread, 1u)] = t;
            continue;  // swept by the spread launch
        }
        const float4 xi = frame_pos_h(cell, frame, o, U);
        const TileBox B = tile_box(xi, valid);
        __syncwarp();  // the previous tile's segments are read
        const int nseg = build_segments(b, g, T, lane, S->seg);
        __syncwarp();
        // the tile's list of needed candidates, one after another in its records
        uint32_t* const list = b.records + (size_t)region.cur * 32;
        const uint32_t room = (region.end - region.cur) * 32;
        const F2 X = f2(xi.x), Y = f2(xi.y), Z = f2(xi.z);
        KSum rk;  // sum of m_j W_ij / scale over the stencil, the particle itself included
        uint32_t nn = 0, needed = 0;
        int kept = 0, swept = 0;
        auto put = [&](int q, float x, float y, float z, float m) {
            S->cx[q] = x;
            S->cy[q] = y;
            S->cz[q] = z;
            S->cm[q] = m;
        };
        auto sweep = [&](int left) {  // chunk `swept`, `left` candidates
            const int f = (swept & 1) * 32;
            __syncwarp();
            F2 acc = f2(0.0f);
            uint32_t mask = sweep_density_chunk<kKern, kCut>(c, S->cx + f, S->cy + f, S->cz + f,
                                                             S->cm + f, (left + 3) >> 2, X, Y, Z,
                                                             U.r2, acc);
            const float2 a2 = upk2(acc.v);
            rk.add(a2.x + a2.y);  // compensated across chunks
            mask = valid ? mask & chunk_valid(left) : 0u;
            nn += __popc(mask);
            const uint32_t used = __brev(__reduce_or_sync(kFull, mask));
            const uint32_t at = needed + __popc(used & lt);
            // (streaming stores: the lists must not evict the candidates from L2)
            if (((used >> lane) & 1u) && at < room) __stcs(list + at, S->idx[f + lane]);
            needed += __popc(used);
            ++swept;
            __syncwarp();  // the chunk's slots may be written again
        };
        for (int sg = 0; sg < nseg; ++sg) {
            const int2 se = S->seg[sg];
            for (int s = se.x; s < se.y; s += 32) {
                const bool in = lane < se.y - s;
                float4 pl = make_float4(kFar, kFar, kFar, 0.0f);
                if (in) pl = frame_pos_h(b.cell4_s[s + lane], frame, b.pos4_s[s + lane], U);
                const uint32_t surv = __ballot_sync(kFull, in && box_near(B, pl, U.r2m));
                if ((surv >> lane) & 1u) {
                    const int q = (kept + __popc(surv & lt)) & 63;
                    put(q, pl.x, pl.y, pl.z, pl.w);
                    S->idx[q] = (uint32_t)(s + lane);
                }
                kept += __popc(surv);
                if ((kept >> 5) > swept) sweep(32);
            }
        }
        if (kept > swept * 32) {
            const int left = kept - swept * 32;
            if (lane >= left) put((swept & 1) * 32 + lane, kFar, kFar, kFar, 0.0f);
            sweep(left);
        }
        if (b.records) {
            const bool fits = needed <= room;
            if (lane == 0) b.tile_list[t] = make_uint2(fits ? region.cur : kNoSlot, needed);
            if (fits) region.cur += (needed + 31) >> 5;
        }
        if (valid) {
            density_out(c, b, i, T.cells, o.w, rk);
            my_max = max(my_max, nn);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) my_max = max(my_max, __shfl_xor_sync(kFull, my_max, o));
    if (lane == 0 && my_max) atomicMax(&ds->max_nn, (unsigned long long)my_max);
}

// The spread tiles the density launch listed, each lane in its own frame (its own launch,
// so that this code and its shared memory stay out of the main one).
template <int kKern>
__global__ void __launch_bounds__(128, 4) k_density_sweep_spread(const StepConst c,
                                                                 const Buffers b,
                                                                 DevState* ds) {
    if (ds->status || ds->n_spread == 0) return;  // (an empty list: no atomics)
    extern __shared__ __align__(16) unsigned char smem_sweep_ds[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepDensitySpreadSmem* S = reinterpret_cast<SweepDensitySpreadSmem*>(smem_sweep_ds) + warp;
    const uint32_t ntiles = ds->n_spread;
    const Geom g = grid_geom(ds);
    const SweepUnits U = sweep_units(c);
    uint32_t my_max = 0;
    const TileQueue queue(&ds->spread_work[0], b.num_sms);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        Tile T;
        int i;
        int4 ct, frame;
        float4 o;
        bool valid;
        tile_setup_cells(c, b, g, b.tiles[b.spread_tiles[t]], lane, T, i, ct, o, valid, frame);
        KSum rk;
        uint32_t nn = 0;
        const int nseg = build_segments(b, g, T, lane, S->seg);
        __syncwarp();
        sweep_density_spread<kKern>(c, b, U, S, nseg, lane, valid, ct, spread_off(o, U), rk, nn);
        if (valid) {
            density_out(c, b, i, T.cells, o.w, rk);
            my_max = max(my_max, nn);
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) my_max = max(my_max, __shfl_xor_sync(kFull, my_max, o));
    if (lane == 0 && my_max) atomicMax(&ds->max_nn, (unsigned long long)my_max);
}

// ---------------------------------------------------------------------------------------
// force + acceleration (+ leapfrog + wall clamp when kIntegrate)
// ---------------------------------------------------------------------------------------
struct SweepForceSmem {  // one chunk of candidates
    float cx[32], cy[32], cz[32];  // tile frame
    float vx[32], vy[32], vz[32];
    float pf[32], cf[32];          // kg m / (2 rho), the same times P
    int2 seg[kMaxSegments + 1];
};
static_assert(sizeof(SweepForceSmem) % 16 == 0, "per-warp regions stay 16-byte aligned");
// The spread tiles' launch (sweep_force_spread) stages whole candidates.
struct SweepForceSpreadSmem {
    int2 seg[kMaxSegments + 1];
    int4 scell[32];   // candidate j of the chunk: its cell
    float4 soff[32];  // its offset in sweep units, P
    float4 svel[32];  // its velocity, kg m / (2 rho)
};

// Pressure and viscosity factors of the kernel: the force on particle t from candidate j is
//   kg (m_j / (2 rho_j)) (P_t + P_j) G' r_vec  +  kl (m_j / rho_j) mu L' (v_j - v_t)
// with G' and L' the kernel's gradient and Laplacian shapes below: grad W_tj = -kg G' r_vec
// and laplacian W_tj = kl L' (r_vec = x_t - x_j, in units of h).  The host forms kg and the
// constant kappa = 2 kl / kg mu between the two factors (StepConst::sw_kg, sw_kappa).

// (|r|/h)^2 of a pair is formed with kCoincident added: far below the rounding of any other pair
__device__ __forceinline__ F2 sweep_d2(const PairLits& k, F2 dx, F2 dy, F2 dz) {
    return fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, F2{k.coincident})));
}

// The gradient shape over |r| and the Laplacian shape of two pairs, from their (|r|/h)^2.
template <int K>
__device__ __forceinline__ void sweep_shapes(const PairLits& k, const SweepUnits& U, F2 d2, F2& G, F2& L) {
    const float2 e = upk2(d2.v);
    if (K == SPHX_KERNEL_GAUSSIAN) {
        const F2 ex = f2(exp_approx(-e.x), exp_approx(-e.y));
        G = keep(e.x >= U.skip2, e.y >= U.skip2, ex);
        L = ex * fma2(d2, F2{k.two}, F2{k.neg3});  // 2 |r|^2 / h^2 - 3
        return;
    }
    // 1/|r| (h units); a coincident pair (d2 = kCoincident) gets a finite value and q = 1e-15,
    // where the gradient shapes below are 0
    const F2 R = f2(rsqrt_approx(e.x), rsqrt_approx(e.y));
    const F2 q = d2 * R;
    if (K == SPHX_KERNEL_WENDLAND_C2) {
        const F2 t = max0(fma2(q, F2{k.neg_half}, F2{k.one}));
        const F2 t2 = t * t;
        G = ((t2 * t) * q) * R;
        L = t2 * fma2(q, F2{k.five}, F2{k.neg3});
    } else {
        const F2 a = max0(F2{k.two} - q), b2 = max0(fma2(q, F2{k.neg2}, F2{k.two}));  // b2 = 2b
        G = ((b2 - a) * (b2 + a)) * R;  // 4 b^2 - a^2
        L = fma2(b2, F2{k.neg2}, a);     // a - 4 b
    }
}

// The terms of two candidates from the separations x_t - x_j (dx, dy, dz, sweep units) and the
// candidates' velocities and factors (pf = kg m / (2 rho), cf = pf P), added to the packed
// sums.  kMask: zero the terms of non-neighbours by selection (needed when the search radius
// is below the support, for the Gaussian, and when a candidate carries a non-finite velocity
// or factor, which a zero factor would not cancel).
template <int K, bool kMask>
__device__ __forceinline__ void sweep_force_terms(const PairLits& k, const SweepUnits& U, F2 kappa, F2 dx, F2 dy,
                                                  F2 dz, const float4& vt, float Pt, F2 vx, F2 vy,
                                                  F2 vz, F2 pf, F2 cf, F2& Fx, F2& Fy, F2& Fz) {
    const F2 d2 = sweep_d2(k, dx, dy, dz);
    F2 G, L;
    sweep_shapes<K>(k, U, d2, G, L);
    F2 cp = fma2(f2(Pt), pf, cf) * G, cv = (pf * kappa) * L;
    F2 ux = vx - f2(vt.x), uy = vy - f2(vt.y), uz = vz - f2(vt.z);
    if (kMask) {
        const float2 e = upk2(d2.v);
        const bool ha = e.x <= U.r2, hb = e.y <= U.r2;
        cp = keep(ha, hb, cp);
        cv = keep(ha, hb, cv);
        ux = keep(ha, hb, ux);
        uy = keep(ha, hb, uy);
        uz = keep(ha, hb, uz);
    }
    Fx = fma2(cv, ux, fma2(cp, dx, Fx));
    Fy = fma2(cv, uy, fma2(cp, dy, Fy));
    Fz = fma2(cv, uz, fma2(cp, dz, Fz));
}

// The staged chunk (nq quads) against the lane's particle.
template <int K, bool kMask>
__device__ __forceinline__ void sweep_force_chunk(const PairLits& k, const SweepUnits& U, F2 kappa,
                                                  const SweepForceSmem* S, int nq, F2 X,
                                                  F2 Y, F2 Z, const float4& vt, float Pt, F2& Fx,
                                                  F2& Fy, F2& Fz) {
    auto quad = [&](const float* a, int q) {
        return reinterpret_cast<const ulonglong2*>(a)[q];
    };
#pragma unroll 4
    for (int q = 0; q < nq; ++q) {
        const ulonglong2 x = quad(S->cx, q), y = quad(S->cy, q), z = quad(S->cz, q),
                         vx = quad(S->vx, q), vy = quad(S->vy, q), vz = quad(S->vz, q),
                         pf = quad(S->pf, q), cf = quad(S->cf, q);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            sweep_force_terms<K, kMask>(k, U, kappa, X - F2{h ? x.y : x.x}, Y - F2{h ? y.y : y.x},
                                        Z - F2{h ? z.y : z.x}, vt, Pt, F2{h ? vx.y : vx.x},
                                        F2{h ? vy.y : vy.x}, F2{h ? vz.y : vz.x},
                                        F2{h ? pf.y : pf.x}, F2{h ? cf.y : cf.x}, Fx, Fy, Fz);
    }
}

// The force sweep of a spread tile: every candidate of every chunk against the lane's
// particle in the lane's own frame (ct, ot), masked by the neighbour test.
template <int kKern>
__device__ __forceinline__ void sweep_force_spread(const PairLits& k, const Buffers& b, const SweepUnits& U, float kg,
                                                   F2 kappa, SweepForceSpreadSmem* S, int nseg,
                                                   int lane, int4 ct, float4 ot, const float4& vt,
                                                   float Pt, KSum& Sx, KSum& Sy, KSum& Sz) {
    for (int sg = 0; sg < nseg; ++sg) {
        const int2 se = S->seg[sg];
        for (int s = se.x; s < se.y; s += 32) {
            const int m = min(32, se.y - s);
            __syncwarp();
            if (lane < m) {
                const float4 o = spread_off(b.pos4_s[s + lane], U), v = b.vel4_s[s + lane],
                             a = b.aux4_s[s + lane];
                S->scell[lane] = b.cell4_s[s + lane];
                S->soff[lane] = make_float4(o.x, o.y, o.z, a.y);
                S->svel[lane] = make_float4(v.x, v.y, v.z, kg * a.z);
            } else {  // empty slot: far
                S->scell[lane] = ct;
                S->soff[lane] = make_float4(kFar, kFar, kFar, 0.0f);
                S->svel[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            __syncwarp();
            F2 Fx = f2(0.0f), Fy = Fx, Fz = Fx;
            for (int j = 0; j < m; j += 2) {
                const float4 oa = S->soff[j], ob = S->soff[j + 1];
                F2 dx, dy, dz;
                spread_sep(U, ct, ot, S->scell[j], oa, S->scell[j + 1], ob, dx, dy, dz);
                const float4 va = S->svel[j], vb = S->svel[j + 1];
                const F2 pf = f2(va.w, vb.w);
                sweep_force_terms<kKern, true>(k, U, kappa, dx, dy, dz, vt, Pt, f2(va.x, vb.x),
                                               f2(va.y, vb.y), f2(va.z, vb.z), pf,
                                               pf * f2(oa.w, ob.w), Fx, Fy, Fz);
            }
            const float2 fx = upk2(Fx.v), fy = upk2(Fy.v), fz = upk2(Fz.v);
            Sx.add(fx.x + fx.y);
            Sy.add(fy.x + fy.y);
            Sz.add(fz.x + fz.y);
        }
    }
}

// The force epilogue of the lane's particle: the acceleration, and (kIntegrate) the
// leapfrog step with the wall clamp, scattered back to insertion order.
template <bool kIntegrate>
__device__ __forceinline__ void force_out(const StepConst& c, const Buffers& b, DevState* ds,
                                          int i, float mi, const KSum& Sx, const KSum& Sy,
                                          const KSum& Sz) {
    const float ax = Sx.value() / mi;
    const float ay = (Sy.value() + c.grav * mi) / mi;
    const float az = Sz.value() / mi;
    b.acc4_s[i] = make_float4(ax, ay, az, 0.0f);
    if (!kIntegrate) return;
    const uint32_t id = b.id_s[i];
    int4 cell = b.cell4_s[i];
    const float4 own = b.pos4_s[i];
    const float4 vi = b.vel4_s[i];  // loaded again: not held across the sweep
    float o[3] = {own.x, own.y, own.z}, v[3] = {vi.x, vi.y, vi.z};
    const float acc[3] = {ax, ay, az};
    if (!cell.w) integrate_cells(c, ds->dt, acc, o, v, cell);
    b.cell4[id] = cell;
    b.pos4[id] = make_float4(o[0], o[1], o[2], mi);
    b.vel4[id] = make_float4(v[0], v[1], v[2], 0.0f);
    if (id == 0) {
        ds->a0[0] = ax;
        ds->a0[1] = ay;
        ds->a0[2] = az;
    }
}

// Bound: the FP32 pipe (27 packed instructions of two cycles per pair of candidates, 374 pairs
// a tile and lane).  1M dam break: 0.81 ms; walking and culling the candidates again instead
// of reading the density pass's list (1.8 times the instructions) 1.14 ms, sweeping all kept
// candidates 1.20 ms.  Four CTAs per SM leave 128 registers, at which up to 28 bytes spill in
// some forms; three without spill 0.84 ms.
template <bool kIntegrate, int kKern, bool kCut>
__global__ void __launch_bounds__(128, 4) k_force_sweep(const StepConst c, const Buffers b,
                                                        DevState* ds) {
    if (ds->status) return;
    extern __shared__ __align__(16) unsigned char smem_sweep_f[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepForceSmem* S = reinterpret_cast<SweepForceSmem*>(smem_sweep_f) + warp;
    const uint32_t ntiles = ds->n_tiles;
    const Geom g = grid_geom(ds);
    const SweepUnits U = sweep_units(c);
    const float kg = c.sw_kg;
    const F2 kappa{c.sw_kappa2};
    const TileQueue queue(&ds->work[1], b.num_sms);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        Tile T;
        int i;
        int4 cell, frame;
        float4 o;
        bool valid;
        tile_setup_cells(c, b, g, b.tiles[t], lane, T, i, cell, o, valid, frame);
        if (spread_tile(T, cell, valid, frame))
            continue;  // listed by the density launch, swept by the spread launch
        const float4 xi = frame_pos_h(cell, frame, o, U);
        const float4 vi = b.vel4_s[i];
        const float Pi = b.aux4_s[i].y;
        const F2 X = f2(xi.x), Y = f2(xi.y), Z = f2(xi.z);
        KSum Sx, Sy, Sz;  // force sums, compensated
        // a candidate as loaded, and how a chunk of them is staged and swept (`left` of them in
        // lane order; an empty lane's has no factor and lies far away)
        struct Cand {
            int4 cell;
            float4 o, v, a;
        };
        const Cand empty{frame, make_float4(kFar, kFar, kFar, 0.0f),
                         make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        auto load = [&](bool has, uint32_t j) {
            Cand d = empty;
            if (has) {
                d.cell = b.cell4_s[j];
                d.o = b.pos4_s[j];
                d.v = b.vel4_s[j];
                d.a = b.aux4_s[j];
            }
            return d;
        };
        auto stage = [&](const Cand& d) {  // returns whether the chunk needs the masked sweep
            const float4 x = frame_pos_h(d.cell, frame, d.o, U);
            const float pf = kg * d.a.z;
            __syncwarp();  // the previous chunk's reads are done
            S->cx[lane] = x.x;
            S->cy[lane] = x.y;
            S->cz[lane] = x.z;
            S->vx[lane] = d.v.x;
            S->vy[lane] = d.v.y;
            S->vz[lane] = d.v.z;
            S->pf[lane] = pf;
            S->cf[lane] = pf * d.a.y;
            __syncwarp();
            // a non-finite velocity or factor (the pressure's, the viscosity's) is not cancelled
            // by a zero shape
            return kCut || __any_sync(kFull, !isfinite(d.v.x + d.v.y + d.v.z + d.a.y +
                                                       pf * d.a.y + pf * c.sw_kappa));
        };
        auto sweep = [&](bool masked, int left) {
            F2 Fx = f2(0.0f), Fy = Fx, Fz = Fx;
            const int nq = (left + 3) >> 2;
            if (masked) sweep_force_chunk<kKern, true>(c.lit, U, kappa, S, nq, X, Y, Z, vi, Pi, Fx, Fy, Fz);
            else sweep_force_chunk<kKern, false>(c.lit, U, kappa, S, nq, X, Y, Z, vi, Pi, Fx, Fy, Fz);
            const float2 fx = upk2(Fx.v), fy = upk2(Fy.v), fz = upk2(Fz.v);
            Sx.add(fx.x + fx.y);  // compensated across chunks
            Sy.add(fy.x + fy.y);
            Sz.add(fz.x + fz.y);
        };
        // the candidates that some lane needs, listed by the density pass: positions read two
        // chunks ahead, their data one
        const uint2 list = b.records ? b.tile_list[t] : make_uint2(kNoSlot, 0u);
        if (list.x != kNoSlot) {
            const uint32_t* p = b.records + (size_t)list.x * 32;
            const uint32_t n = list.y;
            auto at = [&](uint32_t q) { return q < n ? __ldcs(p + q) : 0u; };
            Cand d = load((uint32_t)lane < n, at(lane));
            uint32_t j = at(32 + lane);
            for (uint32_t q = 0; q < n; q += 32) {
                const bool masked = stage(d);
                d = load(q + 32 + lane < n, j);
                j = at(q + 64 + lane);
                sweep(masked, (int)min(32u, n - q));
            }
        } else {  // no list: every chunk of the walk that the tile's box reaches
            const TileBox B = tile_box(xi, valid);
            __syncwarp();  // the previous tile's segments are read
            const int nseg = build_segments(b, g, T, lane, S->seg);
            __syncwarp();
            for (int sg = 0; sg < nseg; ++sg) {
                const int2 se = S->seg[sg];
                for (int s = se.x; s < se.y; s += 32) {
                    const bool in = lane < se.y - s;
                    const Cand d = load(in, (uint32_t)(s + lane));
                    const bool near = in && box_near(B, frame_pos_h(d.cell, frame, d.o, U), U.r2m);
                    if (__any_sync(kFull, near)) sweep(stage(d), min(32, se.y - s));
                }
            }
        }
        if (!valid) continue;
        force_out<kIntegrate>(c, b, ds, i, o.w, Sx, Sy, Sz);
    }
}

// The spread tiles the density launch listed, each lane in its own frame (its own launch).
template <bool kIntegrate, int kKern>
__global__ void __launch_bounds__(128, 4) k_force_sweep_spread(const StepConst c,
                                                               const Buffers b, DevState* ds) {
    if (ds->status || ds->n_spread == 0) return;
    extern __shared__ __align__(16) unsigned char smem_sweep_fs[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SweepForceSpreadSmem* S = reinterpret_cast<SweepForceSpreadSmem*>(smem_sweep_fs) + warp;
    const uint32_t ntiles = ds->n_spread;
    const Geom g = grid_geom(ds);
    const SweepUnits U = sweep_units(c);
    const float kg = c.sw_kg;
    const F2 kappa{c.sw_kappa2};
    const TileQueue queue(&ds->spread_work[1], b.num_sms);
    for (uint32_t t = queue.start(); t < ntiles; t = queue.next(lane)) {
        Tile T;
        int i;
        int4 ct, frame;
        float4 o;
        bool valid;
        tile_setup_cells(c, b, g, b.tiles[b.spread_tiles[t]], lane, T, i, ct, o, valid, frame);
        KSum Sx, Sy, Sz;
        const int nseg = build_segments(b, g, T, lane, S->seg);
        __syncwarp();
        sweep_force_spread<kKern>(c.lit, b, U, kg, kappa, S, nseg, lane, ct, spread_off(o, U),
                                  b.vel4_s[i], b.aux4_s[i].y, Sx, Sy, Sz);
        __syncwarp();
        if (!valid) continue;
        force_out<kIntegrate>(c, b, ds, i, o.w, Sx, Sy, Sz);
    }
}

template <class K>
void launch_sweep(const LaunchCtx& L, LaunchShapeCache& cache, K kernel, size_t smem_per_warp,
                  const StepConst& c, const Buffers& b, DevState* ds) {
    const int threads = 32 * L.warps_per_block;
    const size_t sm = (size_t)L.warps_per_block * smem_per_warp;
    const int nb = cached_resident_blocks(cache, L, kernel, threads, sm);
    kernel<<<nb, threads, sm, L.stream>>>(c, b, ds);
}

// the max form zeroes every pair beyond the support 2h; a search radius below it needs the
// neighbour test (the Gaussian has no compact support)
template <int kKern>
bool cut(const StepConst& c) {
    return kKern == SPHX_KERNEL_GAUSSIAN || c.r2 < 4.0f * c.h_sq;
}

template <int kKern, bool kCut>
void launch_density_sweep_v(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                            DevState* ds) {
    static LaunchShapeCache cache, cache_spread;
    launch_sweep(L, cache, k_density_sweep<kKern, kCut>, sizeof(SweepDensitySmem), c, b, ds);
    launch_sweep(L, cache_spread, k_density_sweep_spread<kKern>, sizeof(SweepDensitySpreadSmem),
                 c, b, ds);
}

template <int kKern>
void launch_density_sweep_k(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                            DevState* ds) {
    if (cut<kKern>(c)) launch_density_sweep_v<kKern, true>(L, c, b, ds);
    else launch_density_sweep_v<kKern, false>(L, c, b, ds);
}

template <bool kIntegrate, int kKern, bool kCut>
void launch_force_sweep_v(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                          DevState* ds) {
    static LaunchShapeCache cache, cache_spread;
    launch_sweep(L, cache, k_force_sweep<kIntegrate, kKern, kCut>, sizeof(SweepForceSmem), c, b,
                 ds);
    launch_sweep(L, cache_spread, k_force_sweep_spread<kIntegrate, kKern>,
                 sizeof(SweepForceSpreadSmem), c, b, ds);
}

template <int kKern>
void launch_force_sweep_k(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                          DevState* ds, int integrate) {
    const bool k = cut<kKern>(c);
    if (integrate) {
        if (k) launch_force_sweep_v<true, kKern, true>(L, c, b, ds);
        else launch_force_sweep_v<true, kKern, false>(L, c, b, ds);
    } else {
        if (k) launch_force_sweep_v<false, kKern, true>(L, c, b, ds);
        else launch_force_sweep_v<false, kKern, false>(L, c, b, ds);
    }
}

}  // namespace

int launch_density_sweep(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                         DevState* ds) {
    if (c.kern == SPHX_KERNEL_WENDLAND_C2) launch_density_sweep_k<SPHX_KERNEL_WENDLAND_C2>(L, c, b, ds);
    else if (c.kern == SPHX_KERNEL_GAUSSIAN) launch_density_sweep_k<SPHX_KERNEL_GAUSSIAN>(L, c, b, ds);
    else launch_density_sweep_k<SPHX_KERNEL_CUBIC_SPLINE>(L, c, b, ds);
    return 2;  // the main and the spread-tile launch
}

int launch_force_sweep(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                       int integrate) {
    if (c.kern == SPHX_KERNEL_WENDLAND_C2)
        launch_force_sweep_k<SPHX_KERNEL_WENDLAND_C2>(L, c, b, ds, integrate);
    else if (c.kern == SPHX_KERNEL_GAUSSIAN)
        launch_force_sweep_k<SPHX_KERNEL_GAUSSIAN>(L, c, b, ds, integrate);
    else launch_force_sweep_k<SPHX_KERNEL_CUBIC_SPLINE>(L, c, b, ds, integrate);
    return 2;  // the main and the spread-tile launch
}

}  // namespace sphx
