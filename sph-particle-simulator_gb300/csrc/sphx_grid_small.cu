// The grid build of a small set in one launch: bounding box, layout, dt, keys, stable sort,
// gather, cell offsets, in-cell order and tile list (what k_prepare, k_keys, the radix passes,
// k_reorder and k_order_tiles do for larger sets).
//
// One cluster of 16 CTAs: the CTAs meet at the hardware's cluster barrier, and the sort's items
// never leave shared memory (a CTA stores an item straight into the CTA that owns its place).
// Bound: latency.  Of the 13 us that 4k particles take (clock counts, one sort pass) the sort
// pass is 3.4, the gather and the tile flags 2 and 1.5, the bounding box 1.7, the barriers
// between them 0.3 each; at 64k a CTA moves 4k particles through one SM's load path and the
// gather (6 us) and the in-cell order (8 us) show.  As nine launches the build took 36 us at
// 4k, 42 at 10k, 54 at 64k; in one 19, 23 and 42 (with the launch).
#include <cooperative_groups.h>

#include "sphx_grid.cuh"

namespace sphx {

namespace cg = cooperative_groups;

constexpr int kSmallCtas = 16, kSmallThreads = 1024, kSmallWarps = kSmallThreads / 32;
constexpr int kSmallPer = kSmallMax / kSmallCtas;  // particles of a CTA at most
static_assert(kSmallPer % kSmallThreads == 0, "whole rounds");
// Runs of empty cells (their offsets are all the same): up to kShortRun are written by the thread
// of the particle behind them, longer ones by its warp, and those above 1/kMaxRuns of the grid
// (and kLongRun) by the whole cluster.  16 million cells, us for the density and force passes and
// the build with a thread for each run, whatever its length, and now: 4k particles spread evenly
// 2,190 and 319, 33k 961 and 254, 64k 818 and 322; two clumps far apart 69,000 and 120 to 410.
constexpr uint32_t kShortRun = 8, kLongRun = 1 << 16, kMaxRuns = 256;

struct SmallSmem {
    uint2 item[2][kSmallPer];  // (key, insertion index): the sort's two buffers
    uint32_t cnt[kSmallWarps][kRadixBuckets];
    uint32_t total[kRadixBuckets];  // of this CTA, read by the others
    uint32_t first[kRadixBuckets];  // where the CTA's keys of a digit go
    uint32_t scan[kSmallWarps];
    uint32_t flags[kSmallPer / 32 + 1], flags_before[kSmallPer / 32];
    uint32_t occ, max_occ, base;
    uint32_t runs;  // for the cluster: first cell, last cell + 1, offset (the same in every CTA)
    uint3 run[kMaxRuns];
    PrepPart part;
    DevState ds;                               // the step's grid
    alignas(4) uint8_t lev[kSmallPer + 2 * kZOrderMax];  // z levels, with those of the neighbours' ends
};

// sum of x over the block's threads before this one, in a block of kSmallThreads
__device__ __forceinline__ uint32_t scan_block(uint32_t x, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
    const uint32_t mine = warp_sums[lane];  // kSmallWarps == 32
    all = __reduce_add_sync(0xffffffffu, mine);
    before = __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0u);
    *total = all;
    __syncthreads();
    return before + inc - x;
}

// off[from .. to) = value, by `workers` (at least 4) threads; off is 16-byte aligned
__device__ __forceinline__ void fill_cells(uint32_t* off, uint32_t from, uint32_t to, uint32_t value,
                                           uint32_t worker, uint32_t workers) {
    const uint32_t a = min((from + 3u) & ~3u, to), e = max(a, to & ~3u);
    if (worker < a - from) off[from + worker] = value;
    if (worker < to - e) off[e + worker] = value;
    for (uint32_t q = a + 4u * worker; q < e; q += 4u * workers)
        *reinterpret_cast<uint4*>(off + q) = make_uint4(value, value, value, value);
}

template <bool kCells, bool kVmax>
__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallThreads, 1)
    k_grid_small(const StepConst c, const Buffers b, DevState* ds, int how, float host_dt, int per) {
    extern __shared__ __align__(16) unsigned char smem_raw_s[];
    SmallSmem& S = *reinterpret_cast<SmallSmem*>(smem_raw_s);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const int n = c.n, lo = rank * per, mine = max(0, min(per, n - lo));
    auto remote = [&](int r) { return cluster.map_shared_rank(&S, r); };

    // bounding box and max |v|, joined by every CTA for itself
    PrepPart p = prep_empty();
    for (int i = tid; i < mine; i += kSmallThreads) prep_add<kCells, kVmax>(p, c, b, lo + i);
    p = merge_block<kSmallThreads>(p);
    if (tid == 0) {
        S.part = p;
        S.runs = 0;
    }
    cluster.sync();
    if (warp == 0) {
        p = prep_empty();
        if (lane < kSmallCtas) p = remote(lane)->part;
        p = merge_warp(p);
        if (lane == 0) {
            for (int a = 0; a < 3; ++a) {
                S.ds.cmin[a] = p.mn[a];
                S.ds.cmax[a] = p.mx[a];
            }
            S.ds.nonfinite = p.bad;
            grid_setup(n, c.max_cells, &S.ds);
            S.occ = S.max_occ = 0;
            if (rank == 0) {
                for (int a = 0; a < 3; ++a) {
                    ds->cmin[a] = S.ds.cmin[a];
                    ds->cmax[a] = S.ds.cmax[a];
                    ds->dim[a] = S.ds.dim[a];
                    ds->wrap[a] = S.ds.wrap[a];
                }
                ds->ncells = S.ds.ncells;
                ds->passes = S.ds.passes;
                ds->nonfinite = p.bad;
                ds->general = p.general;
                reset_counters(ds);
                if (how != kNoStep) set_dt(c, ds, how, host_dt, p.vmax);
            }
        }
    }
    __syncthreads();

    // keys, then a stable radix sort through the cluster's shared memory; a warp owns a
    // contiguous part of the CTA's items and walks it in rounds of 32
    const int wper = per / kSmallWarps, w0 = warp * wper;
    const uint32_t nc = S.ds.ncells;
    {
        const KeyGrid g(&S.ds);
        for (int r = lane; r < wper; r += 32) {
            const int k = w0 + r;
            if (k < mine) S.item[0][k] = make_uint2(cell_key<kCells>(b, lo + k, c.inv_cell, g), lo + k);
        }
    }
    __syncwarp();
    const int passes = (int)S.ds.passes;
    for (int pass = 0; pass < passes; ++pass) {
        const uint2* in = S.item[pass & 1];
        const int shift = pass * kRadixBits;
        uint32_t* cnt = S.cnt[warp];
        for (int d = lane; d < kRadixBuckets; d += 32) cnt[d] = 0;
        __syncwarp();
        // a round's digit, its equals in the round and whether the lane holds an item
        auto round = [&](int r, uint2& it, uint32_t& d, uint32_t& peers) {
            const int k = w0 + r + lane;
            const bool ok = k < mine;
            it = ok ? in[k] : make_uint2(0, 0);
            d = ok ? (it.x >> shift) & (kRadixBuckets - 1) : 0xffffffffu;
            peers = __match_any_sync(0xffffffffu, d);
            return ok;
        };
        uint2 it;
        uint32_t d, peers;
        for (int r = 0; r < wper; r += 32) {
            if (round(r, it, d, peers) && (peers & lt) == 0) cnt[d] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < kRadixBuckets) {  // the warps' counts become places within the CTA's digit
            uint32_t run = 0;
#pragma unroll 8
            for (int w = 0; w < kSmallWarps; ++w) {
                const uint32_t x = S.cnt[w][tid];
                S.cnt[w][tid] = run;
                run += x;
            }
            S.total[tid] = run;
        }
        cluster.sync();
        uint32_t all = 0, before = 0, unused;
        if (tid < kRadixBuckets) {
            uint32_t t[kSmallCtas];
#pragma unroll
            for (int q = 0; q < kSmallCtas; ++q) t[q] = remote(q)->total[tid];
#pragma unroll
            for (int q = 0; q < kSmallCtas; ++q) {
                all += t[q];
                before += q < rank ? t[q] : 0u;
            }
        }
        const uint32_t start = scan_block(all, S.scan, &unused);
        if (tid < kRadixBuckets) S.first[tid] = start + before;
        __syncthreads();
        for (int r = 0; r < wper; r += 32) {
            const bool ok = round(r, it, d, peers);
            uint32_t to = 0;
            if (ok) to = S.first[d] + cnt[d] + __popc(peers & lt);
            __syncwarp();
            if (ok) {
                if ((peers & lt) == 0) cnt[d] += __popc(peers);
                const uint32_t q = to / (uint32_t)per;
                remote((int)q)->item[(pass & 1) ^ 1][to - q * (uint32_t)per] = it;
            }
            __syncwarp();
        }
        cluster.sync();
    }

    // gather, sorted keys and permutation, cell offsets (see k_reorder), z levels
    const uint2* sorted = S.item[passes & 1];
    const float levels = 16.0f / c.cs;
    const uint32_t long_run = max(kLongRun, nc / kMaxRuns);  // at most kMaxRuns are longer
    // the lanes' runs: off[from .. to) = value
    auto put_runs = [&](uint32_t from, uint32_t to, uint32_t value) {
        const bool by_warp = to - from > kShortRun;
        if (!by_warp)
            for (uint32_t q = from; q < to; ++q) b.off[q] = value;
        for (uint32_t todo = __ballot_sync(0xffffffffu, by_warp); todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const uint32_t f = __shfl_sync(0xffffffffu, from, src),
                           t = __shfl_sync(0xffffffffu, to, src),
                           v = __shfl_sync(0xffffffffu, value, src);
            if (t - f <= long_run) {
                fill_cells(b.off, f, t, v, (uint32_t)lane, 32u);
            } else if (lane < kSmallCtas) {
                SmallSmem* R = remote(lane);
                const uint32_t slot = atomicAdd(&R->runs, 1u);
                if (slot < kMaxRuns) R->run[slot] = make_uint3(f, t, v);  // always
            }
        }
    };
    for (int k0 = warp * 32; k0 < mine; k0 += kSmallThreads) {
        const int k = k0 + lane, at = lo + k;
        uint32_t from = 0, to = 0;
        if (k < mine) {
            const uint2 it = sorted[k];
            const float4 pos = b.pos4[it.y];
            to = it.x + 1u;
            if (k > 0) from = sorted[k - 1].x + 1u;
            else if (rank > 0) from = remote(rank - 1)->item[passes & 1][per - 1].x + 1u;
            b.key_s[at] = it.x;
            b.id_s[at] = it.y;
            if (b.rank) b.rank[it.y] = (uint32_t)at;
            b.pos4_s[at] = pos;
            b.vel4_s[at] = b.vel4[it.y];
            if (kCells) b.cell4_s[at] = b.cell4[it.y];
            S.lev[kZOrderMax + k] = z_level_of(pos.z, kCells, c.inv_cell, levels);
        }
        put_runs(from, to, (uint32_t)at);
        if (lo + k0 + 32 >= n)  // the cells after the last particle's
            put_runs(at == n - 1 ? to : 0u, at == n - 1 ? nc + 2u : 0u, (uint32_t)n);
    }
    cluster.sync();
    if (S.runs) {
        for (uint32_t r = 0; r < min(S.runs, kMaxRuns); ++r)
            fill_cells(b.off, S.run[r].x, S.run[r].y, S.run[r].z, (uint32_t)(rank * kSmallThreads + tid),
                       (uint32_t)(kSmallCtas * kSmallThreads));
        cluster.sync();
    }

    // in-cell order and tiles (see k_order_tiles)
    const bool folded_cells = !kCells && S.ds.wrap[2];
    const ColumnInfo col{0u, (uint32_t)S.ds.dim[2], !b.columns || folded_cells};
    if (b.columns && tid < 2 * kZOrderMax) {  // levels at the neighbours' ends
        const bool right = tid >= kZOrderMax;
        const int q = right ? rank + 1 : rank - 1;
        if (q >= 0 && q < kSmallCtas)
            S.lev[right ? per + tid : tid] = remote(q)->lev[right ? tid : per + tid];
    }
    if (mine > 0 && warp == 0) {  // the first 32 positions past the CTA's end its last tiles
        const int q = lo + per + lane;
        bool f = false;
        if (q < n) {
            const uint32_t kq = b.key_s[q], pq = b.key_s[q - 1];
            f = tile_starts(b, col, nc, q, kq, pq, pq != kq);
        }
        const uint32_t word = __ballot_sync(0xffffffffu, f);
        if (lane == 0) S.flags[per / 32] = word;
    }
    uint2* const cells_of = S.item[(passes & 1) ^ 1];  // first position and particles of k's cell
    for (int k = tid; k < per; k += kSmallThreads) {
        const int at = lo + k;
        uint32_t key = 0, cells = 0;
        bool start = false, new_cell = false;
        if (k < mine) {
            key = sorted[k].x;
            uint2 cell = make_uint2(0, 0);
            if (key < nc) {
                cell.x = b.off[key];
                cell.y = b.off[key + 1] - cell.x;
            }
            cells_of[k] = cell;
            const uint32_t prev = at ? (k ? sorted[k - 1].x : b.key_s[at - 1]) : 0u;
            new_cell = at == 0 || prev != key;
            start = tile_starts(b, col, nc, at, key, prev, new_cell);
            if (new_cell) cells = cell.y;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, start);
        const uint32_t occ = __ballot_sync(0xffffffffu, cells != 0);
        const uint32_t fullest = __reduce_max_sync(0xffffffffu, cells);
        if (lane == 0) {
            S.flags[k >> 5] = word;
            if (occ) {
                atomicAdd(&S.occ, (uint32_t)__popc(occ));
                atomicMax(&S.max_occ, fullest);
            }
        }
    }
    __syncthreads();
    {
        const int words = per / 32;
        uint32_t total;
        const uint32_t x = tid < words ? (uint32_t)__popc(S.flags[tid]) : 0u;
        const uint32_t before = scan_block(x, S.scan, &total);
        if (tid < words) S.flags_before[tid] = before;
        if (tid == 0) {
            S.base = total ? atomicAdd(&ds->n_tiles, total) : 0u;
            if (S.occ) {
                atomicAdd(&ds->occupied, S.occ);
                atomicMax(&ds->max_occ, S.max_occ);
            }
        }
    }
    __syncthreads();
    for (int k = tid; k < mine; k += kSmallThreads) {
        const int at = lo + k;
        if (b.columns) {
            const uint2 cell = cells_of[k];
            uint32_t to = (uint32_t)at;
            if (cell.y >= 2 && cell.y <= (uint32_t)kZOrderMax)
                to = ordered_place(S.lev, lo - kZOrderMax, (uint32_t)at, cell.x, cell.y);
            b.tgt[to] = (uint32_t)at;
        }
        const int w = k >> 5;
        if (S.flags[w] >> (k & 31) & 1u) {
            const unsigned long long rest =
                (S.flags[w] | (unsigned long long)S.flags[w + 1] << 32) >> (k & 31) >> 1;
            uint32_t m = min((uint32_t)b.tile_n, (uint32_t)(n - at));
            if (rest) m = min(m, (uint32_t)__ffsll((long long)rest));
            b.tiles[S.base + S.flags_before[w] + __popc(S.flags[w] & ((1u << (k & 31)) - 1u))] =
                make_uint2((uint32_t)at, m);
        }
    }
    cluster.sync();  // no CTA leaves while another reads its memory
}

template <bool kCells, bool kVmax>
static bool small_t(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds, int how,
                    float host_dt) {
    static LaunchShapeFlag ready;  // per device: 1 usable, 2 not
    auto kernel = k_grid_small<kCells, kVmax>;
    std::atomic<int>& slot = ready.at(L.device);
    int state = slot.load(std::memory_order_relaxed);
    if (!state) {
        state = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(SmallSmem)) == cudaSuccess &&
                        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                             1) == cudaSuccess
                    ? 1 : 2;
        if (state == 1) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(kSmallCtas);
            cfg.blockDim = dim3(kSmallThreads);
            cfg.dynamicSmemBytes = sizeof(SmallSmem);
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = kSmallCtas;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1)
                state = 2;
        }
        if (state == 2) cudaGetLastError();
        slot.store(state, std::memory_order_relaxed);
    }
    if (state != 1) return false;
    const int round = kSmallCtas * kSmallThreads;
    const int per = (c.n + round - 1) / round * kSmallThreads;
    kernel<<<kSmallCtas, kSmallThreads, sizeof(SmallSmem), L.stream>>>(c, b, ds, how, host_dt, per);
    return true;
}

bool launch_grid_small(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                       int how, float host_dt) {
    const bool cfl = how == kCflDt;
    if (c.precise) return cfl ? small_t<true, true>(L, c, b, ds, how, host_dt)
                              : small_t<true, false>(L, c, b, ds, how, host_dt);
    return cfl ? small_t<false, true>(L, c, b, ds, how, host_dt)
               : small_t<false, false>(L, c, b, ds, how, host_dt);
}

}  // namespace sphx
