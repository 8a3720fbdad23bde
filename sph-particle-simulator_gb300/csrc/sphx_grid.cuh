// Device code of the grid build that its two forms share (sphx_grid.cu, sphx_grid_small.cu).
#pragma once
#include "sphx_internal.cuh"

namespace sphx {

// Grid extent.  The occupied-cell box is laid out densely when it has at most max_cells
// cells.  Otherwise (particles spread over a huge box) every axis longer than F =
// floor(cbrt(max_cells)) >= 5 cells is folded: its cell index is taken modulo F.  Cells
// that fold onto each other are at least F - 2 cells apart, so a candidate from a folded
// neighbour fails the distance test; sets and visiting order are unchanged, only the
// number of candidates grows.
__device__ inline void grid_setup(int n, uint32_t max_cells, DevState* ds) {
    if ((int)ds->nonfinite >= n) {  // no finite particle: a one-cell grid, all keys sentinel
        for (int a = 0; a < 3; ++a) {
            ds->cmin[a] = 0;
            ds->cmax[a] = 0;
        }
    }
    long long d[3];
    unsigned long long cells = 1;
    bool fits = true;
    for (int a = 0; a < 3; ++a) {
        d[a] = (long long)ds->cmax[a] - (long long)ds->cmin[a] + 1;
        if (d[a] > (long long)max_cells) fits = false;
        else if ((cells *= (unsigned long long)d[a]) > (unsigned long long)max_cells) fits = false;
    }
    long long fold = 1;
    if (!fits) {
        while ((fold + 1) * (fold + 1) * (fold + 1) <= (long long)max_cells) ++fold;
    }
    cells = 1;
    for (int a = 0; a < 3; ++a) {
        const bool w = !fits && d[a] > fold;
        ds->wrap[a] = w ? 1 : 0;
        ds->dim[a] = (int)(w ? fold : d[a]);
        cells *= (unsigned long long)ds->dim[a];
    }
    ds->ncells = (uint32_t)cells;
    const int bits = 32 - __clz(ds->ncells);  // key range is [0, ncells]
    ds->passes = (uint32_t)((bits + kRadixBits - 1) / kRadixBits);
}

// dt of the step, then current_time_ += dt; precision mode: the same rule and the time in FP64.
__device__ inline void set_dt(const StepConst& c, DevState* ds, int how, float host_dt,
                       unsigned long long vmax) {
    if (!c.precise) {
        // (a NaN dt is used as given, like SPHEngine::step, cpp:99-101)
        const float dt = how == kCflDt ? cfl_dt(c, __uint_as_float((uint32_t)vmax), ds->a0)
                                       : host_dt;
        ds->dt = dt;
        ds->time = xadd(ds->time, dt);
        return;
    }
    double dt = host_dt;
    if (how == kCflDt) {
        const double vm = __longlong_as_double((long long)vmax);
        const double cfl = c.cfl, h = c.h;
        const double dt_cfl = cfl * h / (vm + 1e-6);
        const double a0 = sqrt((double)ds->a0[0] * ds->a0[0] + (double)ds->a0[1] * ds->a0[1] +
                               (double)ds->a0[2] * ds->a0[2]);
        const double dt_force = cfl * sqrt(h / (a0 + 1e-6));
        dt = dt_cfl;
        if (dt_force < dt) dt = dt_force;
        if ((double)c.timestep < dt) dt = c.timestep;
    }
    ds->dt64 = dt;
    ds->time64 += dt;
    ds->dt = (float)dt;
    ds->time = (float)ds->time64;
}

__device__ __forceinline__ PrepPart prep_empty() {
    PrepPart p;
    for (int a = 0; a < 3; ++a) {
        p.mn[a] = 0x7fffffff;
        p.mx[a] = -0x7fffffff - 1;
    }
    p.bad = p.general = 0;
    p.vmax = 0;
    return p;
}
__device__ __forceinline__ void merge(PrepPart& p, const PrepPart& q) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p.mn[a] = min(p.mn[a], q.mn[a]);
        p.mx[a] = max(p.mx[a], q.mx[a]);
    }
    p.bad += q.bad;
    p.general |= q.general;
    p.vmax = max(p.vmax, q.vmax);
}
__device__ __forceinline__ PrepPart merge_warp(PrepPart p) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        PrepPart q;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            q.mn[a] = __shfl_xor_sync(0xffffffffu, p.mn[a], o);
            q.mx[a] = __shfl_xor_sync(0xffffffffu, p.mx[a], o);
        }
        q.bad = __shfl_xor_sync(0xffffffffu, p.bad, o);
        q.general = __shfl_xor_sync(0xffffffffu, p.general, o);
        q.vmax = __shfl_xor_sync(0xffffffffu, p.vmax, o);
        merge(p, q);
    }
    return p;
}
// (the result: in the first warp)
template <int kThreads>
__device__ __forceinline__ PrepPart merge_block(PrepPart p) {
    __shared__ PrepPart part[kThreads / 32];
    p = merge_warp(p);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = p;
    __syncthreads();
    if (threadIdx.x < 32) {
        p = threadIdx.x < kThreads / 32 ? part[threadIdx.x] : prep_empty();
        p = merge_warp(p);
    }
    return p;
}
// particle i of the insertion order added to a partial; kCells (precision mode): the stored
// cells.  kVmax: NaN lengths are ignored, as std::max(m, v) keeps m when v is NaN
// (sph_engine.cpp:316-322); non-negative floats order like their bit patterns.
template <bool kCells, bool kVmax>
__device__ __forceinline__ void prep_add(PrepPart& p, const StepConst& c, const Buffers& b, int i) {
            if (kVmax) {
                const float4 v = b.vel4[i];
                if (kCells) {
                    const double len = sqrt((double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z);
                    if (!isnan(len)) p.vmax = max(p.vmax, (unsigned long long)__double_as_longlong(len));
                } else {
                    const float len = xsqrt(xdot3(v.x, v.y, v.z));
                    if (!isnan(len)) p.vmax = max(p.vmax, (unsigned long long)__float_as_uint(len));
                }
            }
            int cell[3];
            if (kCells) {
                const int4 q = b.cell4[i];
                if (q.w) {
                    ++p.bad;
                    return;
                }
                cell[0] = q.x, cell[1] = q.y, cell[2] = q.z;
            } else {
                const float4 q = b.pos4[i];
                p.general |= tiny_coord(q.x) || tiny_coord(q.y) || tiny_coord(q.z);
                if (!finite3(q.x, q.y, q.z)) {
                    ++p.bad;
                    return;
                }
                cell[0] = cell_coord(q.x, c.inv_cell);
                cell[1] = cell_coord(q.y, c.inv_cell);
                cell[2] = cell_coord(q.z, c.inv_cell);
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                p.mn[a] = min(p.mn[a], cell[a]);
                p.mx[a] = max(p.mx[a], cell[a]);
            }
}

// ---- cell keys ----------------------------------------------------------------------------
struct KeyGrid {
    int cmin[3];
    uint32_t dim[3], ncells;
    bool wrap[3];
    __device__ __forceinline__ explicit KeyGrid(const DevState* ds) {
        for (int a = 0; a < 3; ++a) {
            cmin[a] = ds->cmin[a];
            dim[a] = (uint32_t)ds->dim[a];
            wrap[a] = ds->wrap[a];
        }
        ncells = ds->ncells;
    }
};
// Key of particle i of the insertion order; kCells (precision mode): from the stored cells
// (w != 0 marks a particle with no finite position).
template <bool kCells>
__device__ __forceinline__ uint32_t cell_key(const Buffers& b, int i, float inv_cell,
                                             const KeyGrid& g) {
    int cx = 0, cy = 0, cz = 0;
    bool fin;
    if (kCells) {
        const int4 q = b.cell4[i];
        cx = q.x, cy = q.y, cz = q.z;
        fin = !q.w;
    } else {
        const float4 p = b.pos4[i];
        fin = finite3(p.x, p.y, p.z);
        if (fin) {
            cx = cell_coord(p.x, inv_cell);
            cy = cell_coord(p.y, inv_cell);
            cz = cell_coord(p.z, inv_cell);
        }
    }
    if (fin) {  // relative cell index (< 2^31), folded on the axes that wrap
        uint32_t x = (uint32_t)(cx - g.cmin[0]), y = (uint32_t)(cy - g.cmin[1]),
                 z = (uint32_t)(cz - g.cmin[2]);
        if (g.wrap[0]) x %= g.dim[0];
        if (g.wrap[1]) y %= g.dim[1];
        if (g.wrap[2]) z %= g.dim[2];
        return (x * g.dim[1] + y) * g.dim[2] + z;
    }
    return g.ncells;
}

// ---- tiles --------------------------------------------------------------------------------
// A tile is a run of at most tile_n consecutive positions of a cell (b.columns == 0) or of a
// cell column (x, y, *).  Whether a tile starts at position k is decided from the keys and
// cell offsets alone (no scan over the particles): at every tile_n-th position of the column
// and, so that no tile reaches far from its first cell, where a sparse stretch of the column
// is cut (kRunWindow / kRunAlign).  A tile whose first particle lies in cell z_a ends by cell
// z_a + kRunCells: the first multiple z_m of kRunAlign at or above z_a + kRunWindow + 1 is at
// most that plus kRunAlign - 1, and were the tile to reach cell z_m, the kRunWindow cells
// below z_m would lie wholly in it, fewer than tile_n particles, so a tile starts at z_m.
struct ColumnInfo {
    uint32_t base, d2;  // first cell of the scene's block, cells along z
    bool each_cell;     // tiles within one cell
};
__device__ __forceinline__ ColumnInfo column_info(const Buffers& b, const DevState* ds, int k,
                                                  bool folded_cells) {
    if (b.nscenes) {
        const SceneInfo& sc = b.scenes[b.scene_s[k]];
        return ColumnInfo{sc.base, (uint32_t)sc.dim[2], !b.columns};
    }
    return ColumnInfo{0u, (uint32_t)ds->dim[2], !b.columns || folded_cells};
}
__device__ __forceinline__ bool tile_starts(const Buffers& b, const ColumnInfo& g, uint32_t nc,
                                            int k, uint32_t key, uint32_t prev, bool new_cell) {
    const uint32_t tn = (uint32_t)b.tile_n;
    // (the group of particles without a cell is all scenes'; a tile has the constants of one)
    if (key >= nc && b.nscenes && k > 0 && b.scene_s[k] != b.scene_s[k - 1]) return true;
    if (key >= nc || g.each_cell) return ((uint32_t)k - b.off[key]) % tn == 0;
    const uint32_t z = (key - g.base) % g.d2, cb = key - z;
    if (((uint32_t)k - b.off[cb]) % tn == 0) return true;
    if (!new_cell) return false;
    // the cells between the last particle's and this one are empty: only the last multiple of
    // kRunAlign among them can be undecided (an earlier one implies an empty window there)
    const uint32_t zm = z - z % kRunAlign;
    return zm > (uint32_t)kRunWindow && cb + zm > prev &&
           b.off[cb + zm] - b.off[cb + zm - kRunWindow] < tn;
}

// The order in which a cell's particles are taken as targets: by the level of their z inside the
// cell (16 levels; k_order_tiles).  Cells with more particles than this keep their order.
constexpr int kZOrderMax = 128;
__device__ __forceinline__ uint8_t z_level_of(float z, bool offsets, float inv_cell, float levels) {
    const float u = z * inv_cell;
    const float l = offsets ? z * levels : (u - floorf(u)) * 16.0f;
    return (uint8_t)min(15, max(0, (int)l));
}
__device__ __forceinline__ uint8_t z_level(const Buffers& b, int k, float inv_cell, float levels) {
    if (b.nscenes) inv_cell = b.scenes[b.scene_s[k]].c.inv_cell;
    return z_level_of(b.pos4_s[k].z, b.cell4_s, inv_cell, levels);
}

// How many of lev[a .. b) are below `bound` (levels are at most 15, bound at most 16): four at a
// time, each byte's bit 7 telling whether it is not.  lev is 4-byte aligned.
__device__ __forceinline__ uint32_t count_below(const uint8_t* lev, int a, int b, uint32_t bound) {
    if (a >= b) return 0;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(lev);
    const uint32_t sub = bound * 0x01010101u;
    const int last = (b - 1) >> 2;
    uint32_t count = 0;
    for (int q = a >> 2; q <= last; ++q) {
        uint32_t below = ~((w[q] | 0x80808080u) - sub) & 0x80808080u;
        if (q == a >> 2) below &= 0xffffffffu << (8 * (a & 3));
        if (q == last) below &= 0xffffffffu >> (8 * (3 - ((b - 1) & 3)));
        count += __popc(below);
    }
    return count;
}
// Place of position k among its cell's particles first .. first + cells, by level, then by
// position; lev[q] is the level of position base + q.
__device__ __forceinline__ uint32_t ordered_place(const uint8_t* lev, int base, uint32_t k,
                                                  uint32_t first, uint32_t cells) {
    const int f = (int)first - base, o = (int)k - base;
    const uint32_t level = lev[o];
    return first + count_below(lev, f, o, level + 1) + count_below(lev, o, f + (int)cells, level);
}

}  // namespace sphx
