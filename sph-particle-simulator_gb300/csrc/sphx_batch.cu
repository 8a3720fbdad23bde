// Batched scenes: many independent SPH scenes advanced by one step's launches.
//
// Every scene keeps the reference's semantics on its own (its own parameters, walls,
// CFL timestep from its own particles and its own first particle's acceleration, its own
// current time).  The scenes share one cell grid in which each scene owns a dense block
// of cells starting at `base` (a scan over the scenes' cell counts); the key of a particle
// is base + its linear cell index inside the scene's block, so one stable radix sort
// orders all scenes by (scene, cell, insertion index), and the density / force passes take
// tiles of every scene from one work counter.  No particle of one scene ever meets a
// particle of another: the rows of a tile never leave its scene's block.  Each scene's
// results are therefore bit-identical to stepping that scene alone.
#include "sphx_internal.cuh"

namespace sphx {

static inline int blocks_for(const LaunchCtx& L, int n, int threads, int per_sm = 4) {
    const int need = (n + threads - 1) / threads;
    const int cap = L.num_sms * per_sm;
    return need < 1 ? 1 : (need < cap ? need : cap);
}

// ---- the step's first kernel --------------------------------------------------------------

// What a warp has gathered of one scene.
struct SceneAcc {
    uint32_t scene;
    int mn[3], mx[3];
    uint32_t bad, vmax;
};
__device__ __forceinline__ void clear(SceneAcc& s, uint32_t scene) {
    s.scene = scene;
    for (int a = 0; a < 3; ++a) {
        s.mn[a] = 0x7fffffff;
        s.mx[a] = -0x7fffffff - 1;
    }
    s.bad = s.vmax = 0;
}
__device__ __forceinline__ void flush(const SceneAcc& s, SceneInfo* scenes, int lane) {
    SceneInfo& sc = scenes[s.scene];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int mn = __reduce_min_sync(0xffffffffu, s.mn[a]);
        const int mx = __reduce_max_sync(0xffffffffu, s.mx[a]);
        if (lane == 0 && mn != 0x7fffffff) atomicMin(&sc.acc_min[a], mn);
        if (lane == 0 && mx != -0x7fffffff - 1) atomicMax(&sc.acc_max[a], mx);
    }
    const uint32_t bad = __reduce_add_sync(0xffffffffu, s.bad);
    const uint32_t vm = __reduce_max_sync(0xffffffffu, s.vmax);
    if (lane == 0 && bad) atomicAdd(&sc.acc_bad, bad);
    if (lane == 0 && vm) atomicMax(&sc.acc_vmax, vm);
}
__device__ __forceinline__ void gather(SceneAcc& s, const float4& p, const float4* vel, int i,
                                       float inv_cell, bool& tiny) {
    if (vel) {
        const float4 v = vel[i];
        const float len = xsqrt(xdot3(v.x, v.y, v.z));
        if (!isnan(len)) s.vmax = max(s.vmax, __float_as_uint(len));  // NaN ignored like std::max
    }
    tiny = tiny || tiny_coord(p.x) || tiny_coord(p.y) || tiny_coord(p.z);
    if (!finite3(p.x, p.y, p.z)) {
        ++s.bad;
        return;
    }
    const int c[3] = {cell_coord(p.x, inv_cell), cell_coord(p.y, inv_cell),
                      cell_coord(p.z, inv_cell)};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        s.mn[a] = min(s.mn[a], c[a]);
        s.mx[a] = max(s.mx[a], c[a]);
    }
}

// Per scene: box of occupied cells, non-finite count, max |v| (a warp takes consecutive
// particles, so it meets few scenes and adds each to the scene's record once); the block that
// finishes last sets every scene's dt and time and lays the scenes' cell blocks end to end.
__global__ void __launch_bounds__(kPrepThreads) k_batch_prepare(const Buffers b, DevState* ds,
                                                                int n, int how, float host_dt,
                                                                uint32_t max_cells) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (kPrepThreads / 32);
    const int w = blockIdx.x * (kPrepThreads / 32) + (threadIdx.x >> 5);
    const long long rows = (n + 31) / 32;  // of 32 particles
    const int r0 = (int)(rows * w / warps), r1 = (int)(rows * (w + 1) / warps);
    SceneInfo* scenes = b.scenes;
    const float4* vel = how == kCflDt ? b.vel4 : nullptr;
    bool tiny = false;
    if (r0 < r1) {
        SceneAcc acc;
        clear(acc, b.scene_of[r0 * 32]);
        for (int r = r0; r < r1; ++r) {
            const int i = r * 32 + lane;
            const bool in = i < n;
            const uint32_t s = in ? b.scene_of[i] : b.scene_of[n - 1];
            const float4 p = in ? b.pos4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t todo = __ballot_sync(0xffffffffu, in);
            while (todo) {  // scenes are contiguous: usually one round
                const uint32_t cur = __shfl_sync(0xffffffffu, s, __ffs(todo) - 1);
                if (cur != acc.scene) {
                    flush(acc, scenes, lane);
                    clear(acc, cur);
                }
                if (in && s == cur) gather(acc, p, vel, i, scenes[cur].c.inv_cell, tiny);
                todo &= ~__ballot_sync(0xffffffffu, s == cur);
            }
        }
        flush(acc, scenes, lane);
    }
    if (tiny) b.sync->general = 1;
    if (!last_block(b.sync)) return;
    reset_step(ds, b);
    __shared__ unsigned long long warp_cells[kPrepThreads / 32];
    unsigned long long total = 0;  // cells of the scenes before this round's
    for (int s0 = 0; s0 < b.nscenes; s0 += kPrepThreads) {
        const int s = s0 + (int)threadIdx.x;
        unsigned long long cells = 0;
        if (s < b.nscenes) {
            SceneInfo& sc = scenes[s];
            const bool none = sc.acc_bad >= sc.count;  // no finite particle: one cell
            cells = 1;
            for (int a = 0; a < 3; ++a) {
                sc.cmin[a] = none ? 0 : sc.acc_min[a];
                sc.cmax[a] = none ? 0 : sc.acc_max[a];
                sc.acc_min[a] = 0x7fffffff;
                sc.acc_max[a] = -0x7fffffff - 1;
                const long long d = (long long)sc.cmax[a] - (long long)sc.cmin[a] + 1;
                sc.dim[a] = (int)(d < 0x7fffffff ? d : 0x7fffffff);
                cells *= (unsigned long long)(d < (long long)max_cells ? d : (long long)max_cells + 1);
                if (cells > (unsigned long long)max_cells) cells = (unsigned long long)max_cells + 1;
            }
            sc.ncells = (uint32_t)cells;
            // SPHEngine::step is a no-op on an empty scene
            if (how != kNoStep && sc.count) {
                const float dt = how == kCflDt ? cfl_dt(sc.c, __uint_as_float(sc.acc_vmax), sc.a0)
                                               : host_dt;
                sc.dt = dt;
                sc.time = xadd(sc.time, dt);
            }
            sc.acc_bad = sc.acc_vmax = 0;
        }
        unsigned long long x = cells;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_cells[threadIdx.x >> 5] = x;
        __syncthreads();
        unsigned long long before = total, all = 0;
        for (int v = 0; v < kPrepThreads / 32; ++v) {
            if (v < (int)(threadIdx.x >> 5)) before += warp_cells[v];
            all += warp_cells[v];
        }
        const unsigned long long base = before + x - cells;
        if (s < b.nscenes) scenes[s].base = (uint32_t)(base < 0xffffffffull ? base : 0xffffffffull);
        total += all;
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    ds->general = b.sync->general;
    b.sync->general = 0;
    ds->nonfinite = 0;
    if (total > (unsigned long long)max_cells) {  // each scene's box must fit unfolded
        ds->status = SPHX_ERR_DOMAIN;
        ds->ncells = 0;
        ds->passes = 0;
        return;
    }
    ds->ncells = (uint32_t)total;
    for (int a = 0; a < 3; ++a) {
        ds->dim[a] = 1;
        ds->wrap[a] = 0;
    }
    const int bits = 32 - __clz(ds->ncells);
    ds->passes = (uint32_t)((bits + kRadixBits - 1) / kRadixBits);
}

int launch_batch_prepare(const LaunchCtx& L, const Buffers& b, DevState* ds, int n, int how,
                         float host_dt, uint32_t max_cells) {
    int nb = (n + 4 * kPrepThreads - 1) / (4 * kPrepThreads);
    nb = nb < 1 ? 1 : (nb > kMaxPrepBlocks ? kMaxPrepBlocks : nb);
    k_batch_prepare<<<nb, kPrepThreads, 0, L.stream>>>(b, ds, n, how, host_dt, max_cells);
    return 1;
}

// ---- grid ------------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_batch_keys(const Buffers b, int n, const DevState* ds) {
    if (ds->status) return;
    __shared__ uint32_t h[kMaxPasses][kRadixBuckets];
    for (int i = threadIdx.x; i < kMaxPasses * kRadixBuckets; i += 256) (&h[0][0])[i] = 0;
    __syncthreads();
    const uint32_t sentinel = ds->ncells, passes = ds->passes;
    for (int i0 = blockIdx.x * 256; i0 < n; i0 += gridDim.x * 256) {
        const int i = i0 + (int)threadIdx.x;
        uint32_t key = sentinel;
        if (i < n) {
            const SceneInfo& sc = b.scenes[b.scene_of[i]];
            const float4 p = b.pos4[i];
            if (finite3(p.x, p.y, p.z)) {
                const float ic = sc.c.inv_cell;
                const uint32_t x = (uint32_t)(cell_coord(p.x, ic) - sc.cmin[0]);
                const uint32_t y = (uint32_t)(cell_coord(p.y, ic) - sc.cmin[1]);
                const uint32_t z = (uint32_t)(cell_coord(p.z, ic) - sc.cmin[2]);
                key = sc.base + (x * (uint32_t)sc.dim[1] + y) * (uint32_t)sc.dim[2] + z;
            }
            b.key[0][i] = key;
        }
        count_digits(h, key, i < n, passes);
    }
    __syncthreads();
    add_digits(h, b.hist, passes);
}

int launch_batch_grid(const LaunchCtx& L, const Buffers& b, DevState* ds, int n) {
    k_batch_keys<<<blocks_for(L, n, 256, 2), 256, 0, L.stream>>>(b, n, ds);
    return 1 + launch_grid_sort(L, b, ds, n, StepConst{});  // (scenes carry their own)
}

// ---- FP64 diagnostics per scene (one block per scene, fixed order) ----------------------
__global__ void __launch_bounds__(kDiagThreads) k_batch_diag(
    const float4* __restrict__ pos4, const float4* __restrict__ vel4,
    const float4* __restrict__ aux4_s, SceneInfo* scenes, const DevState* ds) {
    SceneInfo& sc = scenes[blockIdx.x];
    double s[6] = {0, 0, 0, 0, 0, 0};
    const double g = sc.c.grav;
    for (uint32_t i = sc.start + threadIdx.x; i < sc.start + sc.count; i += blockDim.x) {
        const float4 p = pos4[i];
        const float4 v = vel4[i];
        const double m = p.w;
        s[0] += m;
        s[1] += m * v.x;
        s[2] += m * v.y;
        s[3] += m * v.z;
        s[4] += 0.5 * m * ((double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z);
        s[5] += -m * g * (double)p.y;
    }
    __shared__ double red[kDiagThreads / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        double v = s[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0;
        for (int w = 0; w < kDiagThreads / 32; ++w) v += red[w][threadIdx.x];
        sc.sums[threadIdx.x] = v;
    }
}

int launch_batch_diag(const LaunchCtx& L, const Buffers& b, DevState* ds) {
    k_batch_diag<<<b.nscenes, kDiagThreads, 0, L.stream>>>(b.pos4, b.vel4, b.aux4_s, b.scenes, ds);
    return 1;
}

}  // namespace sphx
