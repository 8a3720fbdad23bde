// Grid build of one step (the GPU form of SpatialHash::build, spatial_hash.cpp:15-25),
// the CFL timestep (SPHEngine::compute_cfl_timestep, sph_engine.cpp:312-333), the FP64
// diagnostics and the host<->device packing kernels.
//
// Cells are the reference's own: floor(x * inv_cell) per axis with
// inv_cell = 1.0f / neighbor_search_radius (spatial_hash.h:30-36, 63-66).  Instead of a
// hash map of index vectors the occupied-cell box is laid out as a dense grid (folded
// per axis when the box is huge, see grid_setup) with a linear key
// ((cx * dy + cy) * dz + cz), the keys are radix-sorted stably from insertion order, and
// off[c] holds the first sorted position of cell c.  z is the fastest axis, so
// the three cells (cx+dx, cy+dy, cz-1..cz+1) of one stencil row are one contiguous range
// of the sorted arrays.  Particles with a NaN/inf coordinate get key == ncells: they sort
// last and are never anyone's neighbour (every distance test with them fails in the
// reference too).
#include "sphx_grid.cuh"

namespace sphx {

static inline int grid_blocks(const LaunchCtx& L, int n, int threads, int per_sm = 4) {
    const int need = (n + threads - 1) / threads;
    const int cap = L.num_sms * per_sm;
    return need < 1 ? 1 : (need < cap ? need : cap);
}

// ---- the step's first kernel --------------------------------------------------------------

// Box of occupied cells, non-finite count and max |v| over the particles: per-block partials,
// joined by the block that finishes last, which then lays out the grid and sets dt (one
// launch where a reset, two reductions by atomics and two one-thread kernels were five: 1M
// particles 0.036 -> 0.011 ms, 10k 0.012 -> 0.007).
template <bool kCells, bool kVmax>
__global__ void __launch_bounds__(kPrepThreads) k_prepare(const StepConst c, const Buffers b,
                                                          DevState* ds, int how, float host_dt) {
    PrepPart p = prep_empty();
    const int n = c.n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        prep_add<kCells, kVmax>(p, c, b, i);
    p = merge_block<kPrepThreads>(p);
    if (threadIdx.x == 0) b.prep[blockIdx.x] = p;
    if (!last_block(b.sync)) return;
    reset_step(ds, b);
    p = prep_empty();
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) merge(p, b.prep[k]);
    p = merge_block<kPrepThreads>(p);
    if (threadIdx.x != 0) return;
    for (int a = 0; a < 3; ++a) {
        ds->cmin[a] = p.mn[a];
        ds->cmax[a] = p.mx[a];
    }
    ds->nonfinite = p.bad;
    ds->general = p.general;
    grid_setup(n, c.max_cells, ds);
    if (how != kNoStep) set_dt(c, ds, how, host_dt, p.vmax);
}

static int launch_prepare(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                   int how, float host_dt) {
    // at least 4 particles a thread, so that the partials of small sets are few
    int nb = (c.n + 4 * kPrepThreads - 1) / (4 * kPrepThreads);
    nb = nb < 1 ? 1 : (nb > kMaxPrepBlocks ? kMaxPrepBlocks : nb);
    const bool cfl = how == kCflDt;
    if (c.precise && cfl) k_prepare<true, true><<<nb, kPrepThreads, 0, L.stream>>>(c, b, ds, how, host_dt);
    else if (c.precise) k_prepare<true, false><<<nb, kPrepThreads, 0, L.stream>>>(c, b, ds, how, host_dt);
    else if (cfl) k_prepare<false, true><<<nb, kPrepThreads, 0, L.stream>>>(c, b, ds, how, host_dt);
    else k_prepare<false, false><<<nb, kPrepThreads, 0, L.stream>>>(c, b, ds, how, host_dt);
    return 1;
}

// ---- grid -----------------------------------------------------------------------------

// Cell keys and their digit histograms.
template <bool kCells>
__global__ void __launch_bounds__(256) k_keys(const Buffers b, int n, float inv_cell,
                                              const DevState* ds) {
    if (ds->status) return;
    __shared__ uint32_t h[kMaxPasses][kRadixBuckets];
    for (int i = threadIdx.x; i < kMaxPasses * kRadixBuckets; i += 256) (&h[0][0])[i] = 0;
    __syncthreads();
    const KeyGrid g(ds);
    const uint32_t passes = ds->passes;
    for (int i0 = blockIdx.x * 256; i0 < n; i0 += gridDim.x * 256) {
        const int i = i0 + (int)threadIdx.x;
        uint32_t key = 0;
        if (i < n) {
            key = cell_key<kCells>(b, i, inv_cell, g);
            b.key[0][i] = key;
        }
        count_digits(h, key, i < n, passes);
    }
    __syncthreads();
    add_digits(h, b.hist, passes);
}

// Gathers the state into cell-sorted order, keeps the sorted keys and permutation, and writes
// the cell offsets: off[c] = first sorted position whose key is >= c, for c in
// [0, ncells + 1]; off[ncells] is the number of finite particles and off[ncells + 1] == n.
__global__ void k_reorder(const Buffers b, int n, DevState* ds) {
    if (ds->status) return;
    const int sel = ds->passes & 1;
    const uint32_t nc = ds->ncells;
    const uint32_t* __restrict__ ks = b.key[sel];
    const uint32_t* __restrict__ vs = b.val[sel];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k <= n; k += gridDim.x * blockDim.x) {
        const uint32_t hi = k == n ? nc + 1u : ks[k];
        for (uint32_t c = k == 0 ? 0u : ks[k - 1] + 1u; c <= hi; ++c) b.off[c] = (uint32_t)k;
        if (k == n) break;
        uint32_t id = vs[k];
        if (id >= (uint32_t)n) {  // never for a valid permutation: record, do not fault
            atomicExch(&ds->status, SPHX_ERR_CUDA);
            id = 0;
        }
        b.key_s[k] = hi;
        b.id_s[k] = id;
        if (b.rank) b.rank[id] = (uint32_t)k;
        b.pos4_s[k] = b.pos4[id];
        b.vel4_s[k] = b.vel4[id];
        if (b.cell4) b.cell4_s[k] = b.cell4[id];
        if (b.scene_s) b.scene_s[k] = b.scene_of[id];
    }
}

// ---- in-cell order and tile list --------------------------------------------------------
// One block per 256 positions: the tile list, and the order in which each cell's particles are
// taken as targets: z order (the in-cell offset quantised to 16 levels, stable within a
// level), so that a tile is a compact slab across the cells of its column.  The particles
// themselves keep the reference's insertion order, in which they are met as neighbours.  A
// particle's place is the number of its cell's particles before it in that order, counted by
// one thread per particle from the levels in shared memory, four at a time (a counting sort per
// cell by one warp took 0.038 ms at 1M for this kernel, 0.014 at 10k).  Cells of more than kZOrderMax particles (collapsed
// states, whose tiles are dense anyway) keep their order.
__global__ void __launch_bounds__(256) k_order_tiles(const Buffers b, int n, DevState* ds,
                                                     float inv_cell, float levels) {
    if (ds->status) return;
    __shared__ uint32_t flags[9];
    __shared__ uint32_t s_occ, s_max, s_base;
    __shared__ __align__(4) uint8_t lev[256 + 2 * kZOrderMax];  // positions k0 - kZOrderMax ...
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_occ = s_max = 0;
    const uint32_t nc = ds->ncells;
    // an exact step on a grid folded along z keeps one-cell tiles: a row that wraps is met in
    // each cell's own dz order
    const bool folded_cells = !b.cell4_s && ds->wrap[2];
    const int k0 = blockIdx.x * 256, k = k0 + tid;
    uint32_t key = 0, cnt = 0, first = 0;
    bool new_cell = false, flag = false;
    if (k < n) {
        key = b.key_s[k];
        const uint32_t prev = k ? b.key_s[k - 1] : 0u;
        new_cell = k == 0 || prev != key;
        flag = tile_starts(b, column_info(b, ds, k, folded_cells), nc, k, key, prev, new_cell);
        if (key < nc) {
            first = b.off[key];
            cnt = b.off[key + 1] - first;
        }
    }
    if (b.columns) {
        if (k < n) lev[kZOrderMax + tid] = z_level(b, k, inv_cell, levels);
        const int h = tid < kZOrderMax ? tid : 256 + tid;  // the halo on both sides
        const int q = k0 - kZOrderMax + h;
        if (q >= 0 && q < n) lev[h] = z_level(b, q, inv_cell, levels);
    }
    {
        const uint32_t f = __ballot_sync(0xffffffffu, flag);
        if (lane == 0) flags[warp] = f;
    }
    if (warp == 0) {  // the first 32 positions past the block end its last tiles
        const int q = k0 + 256 + lane;
        bool fq = false;
        if (q < n) {
            const uint32_t kq = b.key_s[q], pq = b.key_s[q - 1];
            fq = tile_starts(b, column_info(b, ds, q, folded_cells), nc, q, kq, pq, pq != kq);
        }
        const uint32_t f = __ballot_sync(0xffffffffu, fq);
        if (lane == 0) flags[8] = f;
    }
    __syncthreads();
    {   // occupied cells, fullest cell
        const uint32_t starts = __ballot_sync(0xffffffffu, new_cell && key < nc);
        const uint32_t occ = __reduce_max_sync(0xffffffffu, new_cell ? cnt : 0u);
        if (lane == 0 && starts) {
            atomicAdd(&s_occ, (uint32_t)__popc(starts));
            atomicMax(&s_max, occ);
        }
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t nt = 0;
        for (int w = 0; w < 8; ++w) nt += __popc(flags[w]);
        s_base = atomicAdd(&ds->n_tiles, nt);
        if (s_occ) {
            atomicAdd(&ds->occupied, s_occ);
            atomicMax(&ds->max_occ, s_max);
        }
    }
    if (b.columns && k < n) {
        uint32_t to = (uint32_t)k;
        if (cnt >= 2 && cnt <= (uint32_t)kZOrderMax)
            to = ordered_place(lev, k0 - kZOrderMax, (uint32_t)k, first, cnt);
        b.tgt[to] = (uint32_t)k;
    }
    __syncthreads();
    if (flag) {
        uint32_t t = s_base + __popc(flags[warp] & ((1u << lane) - 1u));
        for (int w = 0; w < warp; ++w) t += __popc(flags[w]);
        const unsigned long long rest =
            (flags[warp] | (unsigned long long)flags[warp + 1] << 32) >> lane >> 1;
        uint32_t m = min((uint32_t)b.tile_n, (uint32_t)(n - k));
        if (rest) m = min(m, (uint32_t)__ffsll((long long)rest));
        b.tiles[t] = make_uint2((uint32_t)k, m);
    }
}

static int launch_build_grid(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                             DevState* ds) {
    const int n = c.n;
    const int gb = grid_blocks(L, n, 256, 2);
    if (c.precise) k_keys<true><<<gb, 256, 0, L.stream>>>(b, n, c.inv_cell, ds);
    else k_keys<false><<<gb, 256, 0, L.stream>>>(b, n, c.inv_cell, ds);
    return 1 + launch_grid_sort(L, b, ds, n, c);
}

int launch_grid(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds, int how,
                float host_dt) {
    // up to kSmallMax one cluster's shared memory holds the sort, and one launch is faster than
    // eight over the whole GPU (k_grid_small: 0.019 against 0.036 ms at 4k, 0.035 against 0.052
    // at 33k, 0.042 against 0.054 at 64k)
    if (c.n >= 1 && c.n <= kSmallMax && launch_grid_small(L, c, b, ds, how, host_dt)) return 1;
    const int k = launch_prepare(L, c, b, ds, how, host_dt);
    return k + launch_build_grid(L, c, b, ds);
}

// Shared tail of the grid build: stable sort of the keys, gather into cell-sorted order with
// the cell offsets, in-cell order and tile list.
int launch_grid_sort(const LaunchCtx& L, const Buffers& b, DevState* ds, int n,
                     const StepConst& c) {
    const int r = launch_radix_sort(L, b, ds, n);
    k_reorder<<<grid_blocks(L, n + 1, 256, 8), 256, 0, L.stream>>>(b, n, ds);
    k_order_tiles<<<(n + 255) / 256, 256, 0, L.stream>>>(b, n, ds, c.inv_cell, 16.0f / c.cs);
    return 2 + r;
}

// ---- FP64 diagnostics of the state after a step -----------------------------------------
// sums: mass, momentum x/y/z, kinetic energy, potential energy (-m g y), density.
// Fixed partition and fixed-order final sum: bit-reproducible run to run.
__global__ void __launch_bounds__(kDiagThreads) k_diag_partial(
    const float4* __restrict__ pos4, const float4* __restrict__ vel4,
    const float4* __restrict__ aux4_s, const int4* __restrict__ cell4, double cs, int n,
    float grav, double* __restrict__ part) {
    double s[7] = {0, 0, 0, 0, 0, 0, 0};
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int i0 = blockIdx.x * per, i1 = min(n, i0 + per);
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const float4 p = pos4[i];
        const float4 v = vel4[i];
        const double m = p.w;
        s[0] += m;
        s[1] += m * v.x;
        s[2] += m * v.y;
        s[3] += m * v.z;
        s[4] += 0.5 * m * ((double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z);
        const double y = cell4 ? (double)cell4[i].y * cs + (double)p.y : (double)p.y;
        s[5] += -m * (double)grav * y;
        if (aux4_s) s[6] += (double)aux4_s[i].x;  // null: no density pass on this set yet
    }
    __shared__ double red[kDiagThreads / 32][7];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        double v = s[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double v = 0;
        for (int w = 0; w < kDiagThreads / 32; ++w) v += red[w][threadIdx.x];
        part[blockIdx.x * kDiagSums + threadIdx.x] = v;
    }
}

// One warp per sum: lane l adds partials l, l + 32, ... in order, then a fixed shuffle tree
// (the order never changes, so the sums are reproducible bit for bit).
__global__ void k_diag_final(const double* __restrict__ part, int nb, DevState* ds) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= 7) return;
    double v = 0;
    for (int b = lane; b < nb; b += 32) v += part[b * kDiagSums + k];
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) ds->sums[k] = v;
}

int launch_diag(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds) {
    k_diag_partial<<<b.diag_blocks, kDiagThreads, 0, L.stream>>>(
        b.pos4, b.vel4, b.aux4_s, c.precise ? b.cell4 : nullptr, c.cs_d, c.n, c.grav, b.diag_part);
    k_diag_final<<<1, 7 * 32, 0, L.stream>>>(b.diag_part, b.diag_blocks, ds);
    return 2;
}

// ---- packing ----------------------------------------------------------------------------

__global__ void k_pack(int n, const float* __restrict__ pos3, const float* __restrict__ vel3,
                       const float* __restrict__ mass, float4* __restrict__ pos4,
                       float4* __restrict__ vel4) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        pos4[i] = make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], mass[i]);
        vel4[i] = vel3 ? make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], 0.0f)
                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

void launch_pack(const LaunchCtx& L, int n, const float* pos3, const float* vel3,
                 const float* mass, float4* pos4, float4* vel4) {
    k_pack<<<grid_blocks(L, n, 256, 8), 256, 0, L.stream>>>(n, pos3, vel3, mass, pos4, vel4);
}

__global__ void k_unpack_state(int n, const float4* __restrict__ pos4,
                               const float4* __restrict__ vel4, float* __restrict__ pos3,
                               float* __restrict__ vel3) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (pos3) {
            const float4 p = pos4[i];
            pos3[3 * i] = p.x;
            pos3[3 * i + 1] = p.y;
            pos3[3 * i + 2] = p.z;
        }
        if (vel3) {
            const float4 v = vel4[i];
            vel3[3 * i] = v.x;
            vel3[3 * i + 1] = v.y;
            vel3[3 * i + 2] = v.z;
        }
    }
}

void launch_unpack_state(const LaunchCtx& L, int n, const float4* pos4, const float4* vel4,
                         float* pos3, float* vel3) {
    k_unpack_state<<<grid_blocks(L, n, 256, 8), 256, 0, L.stream>>>(n, pos4, vel4, pos3, vel3);
}

__global__ void k_unpack_sorted(int n, const uint32_t* __restrict__ id_s,
                                const float4* __restrict__ aux4_s,
                                const float4* __restrict__ acc4_s, float* __restrict__ rho,
                                float* __restrict__ pressure, float* __restrict__ acc3) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t id = id_s[k];
        const float4 a = aux4_s[k];
        if (rho) rho[id] = a.x;
        if (pressure) pressure[id] = a.y;
        if (acc3) {
            const float4 g = acc4_s[k];
            acc3[3 * id] = g.x;
            acc3[3 * id + 1] = g.y;
            acc3[3 * id + 2] = g.z;
        }
    }
}

void launch_unpack_sorted(const LaunchCtx& L, int n, const uint32_t* id_s, const float4* aux4_s,
                          const float4* acc4_s, float* rho, float* pressure, float* acc3) {
    k_unpack_sorted<<<grid_blocks(L, n, 256, 8), 256, 0, L.stream>>>(n, id_s, aux4_s, acc4_s,
                                                                     rho, pressure, acc3);
}

// Any of the download's fields straight to pinned host memory, in insertion order, and the
// status word with them.  Bound: the link to the host (44 bytes a particle): 1M particles 0.21 ms
// where staging, two unpack kernels and the copy engines take 0.25.  Only whole lines go out: the
// fields are gathered by rank, and triples pass through shared memory.  Scattered by insertion
// index instead, a collapsed set of 24k particles took 42 us for what takes 10 here.
constexpr int kDirectThreads = 128;

// The words of `count` particles' triples, in order, to `out`: 128-bit stores where the caller's
// array allows them.
__device__ __forceinline__ void store_triples(float* out, const float* words, int count) {
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        const int quads = 3 * count / 4;
        for (int w = threadIdx.x; w < quads; w += kDirectThreads)
            reinterpret_cast<float4*>(out)[w] = reinterpret_cast<const float4*>(words)[w];
        for (int w = 4 * quads + threadIdx.x; w < 3 * count; w += kDirectThreads) out[w] = words[w];
    } else {
        for (int w = threadIdx.x; w < 3 * count; w += kDirectThreads) out[w] = words[w];
    }
}
// kCells: positions are cell + offset (cell size cs)
template <bool kCells>
__global__ void __launch_bounds__(kDirectThreads)
    k_unpack_direct(int n, const Buffers b, const DevState* ds, double cs, float* pos3, float* vel3,
                    float* rho, float* pressure, float* acc3, int* status) {
    __shared__ __align__(16) float s[3][3 * kDirectThreads];
    const int k0 = blockIdx.x * kDirectThreads, k = k0 + threadIdx.x;
    if (k == 0) *status = ds->status;
    auto put = [&](float* to, float x, float y, float z) {
        to[3 * threadIdx.x] = x;
        to[3 * threadIdx.x + 1] = y;
        to[3 * threadIdx.x + 2] = z;
    };
    if (k < n) {
        if (rho || pressure || acc3) {
            // (a failed step may have left no order)
            const uint32_t at = min(b.rank[k], (uint32_t)n - 1u);
            if (acc3) {
                const float4 g = b.acc4_s[at];
                put(s[2], g.x, g.y, g.z);
            }
            if (rho || pressure) {
                const float4 a = b.aux4_s[at];
                if (rho) rho[k] = a.x;
                if (pressure) pressure[k] = a.y;
            }
        }
        if (pos3) {
            const float4 p = b.pos4[k];
            const int4 c = kCells ? b.cell4[k] : make_int4(0, 0, 0, 1);
            if (c.w) {
                put(s[0], p.x, p.y, p.z);
            } else {
                put(s[0], (float)((double)c.x * cs + (double)p.x), (float)((double)c.y * cs + (double)p.y),
                    (float)((double)c.z * cs + (double)p.z));
            }
        }
        if (vel3) {
            const float4 v = b.vel4[k];
            put(s[1], v.x, v.y, v.z);
        }
    }
    __syncthreads();
    const int count = min(kDirectThreads, n - k0);
    const size_t at = 3 * (size_t)k0;
    if (pos3) store_triples(pos3 + at, s[0], count);
    if (vel3) store_triples(vel3 + at, s[1], count);
    if (acc3) store_triples(acc3 + at, s[2], count);
}

void launch_unpack_direct(const LaunchCtx& L, int n, const Buffers& b, const DevState* ds,
                          double cs, float* pos3, float* vel3, float* rho, float* pressure,
                          float* acc3, int* status) {
    const auto kernel = b.cell4 ? k_unpack_direct<true> : k_unpack_direct<false>;
    kernel<<<n / kDirectThreads + (n % kDirectThreads != 0), kDirectThreads, 0, L.stream>>>(
        n, b, ds, cs, pos3, vel3, rho, pressure, acc3, status);
}

// Absolute position (double) -> integer cell + offset in [0, cs); non-finite -> w = 1.
__device__ __forceinline__ void to_cell(double X, double cs, int fp16, int& c, float& o) {
    double f = floor(X / cs);
    f = fmin(fmax(f, -(double)kCellClamp), (double)(kCellClamp - 1));
    c = (int)f;
    o = (float)(X - (double)c * cs);
    if (fp16) o = round_half(o);
    const float csf = (float)cs;
    if (o >= csf) {  // rounding reached the next cell
        o = 0.0f;
        c += 1;
    } else if (o < 0.0f) {
        o = 0.0f;
    }
}

__global__ void k_pack_cells(StepConst c, int n, const float* __restrict__ pos3f,
                             const double* __restrict__ pos3d, const float* __restrict__ vel3,
                             const float* __restrict__ mass, int4* __restrict__ cell4,
                             float4* __restrict__ pos4, float4* __restrict__ vel4) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double X[3];
        for (int a = 0; a < 3; ++a) X[a] = pos3d ? pos3d[3 * i + a] : (double)pos3f[3 * i + a];
        int4 cc = make_int4(0, 0, 0, 0);
        float o[3] = {0.0f, 0.0f, 0.0f};
        if (isfinite(X[0]) && isfinite(X[1]) && isfinite(X[2])) {
            to_cell(X[0], c.cs_d, c.fp16, cc.x, o[0]);
            to_cell(X[1], c.cs_d, c.fp16, cc.y, o[1]);
            to_cell(X[2], c.cs_d, c.fp16, cc.z, o[2]);
        } else {
            cc.w = 1;
            for (int a = 0; a < 3; ++a) o[a] = (float)X[a];
        }
        cell4[i] = cc;
        pos4[i] = make_float4(o[0], o[1], o[2], mass[i]);
        vel4[i] = vel3 ? make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], 0.0f)
                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

void launch_pack_cells(const LaunchCtx& L, const StepConst& c, int n, const float* pos3f,
                       const double* pos3d, const float* vel3, const float* mass, int4* cell4,
                       float4* pos4, float4* vel4) {
    k_pack_cells<<<grid_blocks(L, n, 256, 8), 256, 0, L.stream>>>(c, n, pos3f, pos3d, vel3, mass,
                                                                  cell4, pos4, vel4);
}

__global__ void k_unpack_cells(StepConst c, int n, const int4* __restrict__ cell4,
                               const float4* __restrict__ pos4, float* __restrict__ pos3f,
                               double* __restrict__ pos3d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 cc = cell4[i];
        const float4 p = pos4[i];
        double X[3];
        if (cc.w) {
            X[0] = p.x; X[1] = p.y; X[2] = p.z;
        } else {
            X[0] = (double)cc.x * c.cs_d + (double)p.x;
            X[1] = (double)cc.y * c.cs_d + (double)p.y;
            X[2] = (double)cc.z * c.cs_d + (double)p.z;
        }
        for (int a = 0; a < 3; ++a) {
            if (pos3d) pos3d[3 * i + a] = X[a];
            if (pos3f) pos3f[3 * i + a] = (float)X[a];
        }
    }
}

void launch_unpack_cells(const LaunchCtx& L, const StepConst& c, int n, const int4* cell4,
                         const float4* pos4, float* pos3f, double* pos3d) {
    k_unpack_cells<<<grid_blocks(L, n, 256, 8), 256, 0, L.stream>>>(c, n, cell4, pos4, pos3f, pos3d);
}

}  // namespace sphx
