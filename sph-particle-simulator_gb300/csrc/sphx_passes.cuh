// Shared device code of the neighbour passes (density + pressure in sphx_density.cu, force +
// leapfrog + wall clamp in sphx_force.cu, the precision mode's in sphx_sweep.cu, the
// neighbour-list dump in sphx_passes.cu): tiles, the stencil walk, the candidate rings, the
// pair arithmetic helpers and the launch-shape cache.
//
// Work decomposition: one warp owns one tile (up to 32 particles of one cell column
// (x, y, *), one particle per lane; a tile may span several cells of its column).  All lanes
// of a tile share the tile's stencil: for each row (dx, dy) the cells cz+lo..cz+hi (covering
// every lane's cell +-1, +-2 near a face) are one contiguous range of the sorted arrays; the
// warp reads that range 32 candidates at a time, drops those the tile's box cannot reach and
// keeps the rest in a shared-memory ring from which every lane takes its own neighbours.
//
// Exactness.  The reference walks, for particle i, the cells (dx, dy, dz) of its stencil
// in lexicographic order and each cell's particles in insertion order
// (spatial_hash.cpp:31-57), and accumulates every sum sequentially in that order
// (sph_engine.cpp:370-432).  The sorted arrays hold each cell's particles in insertion
// order (stable sort from insertion order), the rows are walked in (dx, dy) order and
// each row in increasing z, so a lane meets its neighbours in exactly the reference's
// order, whichever particles share its tile.  The reference scans a 5x5x5 block
// (cell_radius = 2); a neighbour at distance
// <= r can only sit two cells away when the particle lies within rounding distance of a
// cell face, so the tile's stencil is the 3x3x3 block of each of its cells, widened on an
// axis to the second layer when some lane is that close to a face (guard band eps below).
// Cells of the tile's rows outside a lane's own 5x5x5 block hold no neighbour of it (they
// are more than two cells away), so they add only misses to that lane's walk, and the
// cells of its block keep their relative order.  Every distance test and
// every term uses the reference's float operations in the reference's order with
// IEEE round-to-nearest and no contraction, so each lane's sums are bit-identical.
#pragma once
#include "sphx_internal.cuh"

namespace sphx {

struct Tile {
    int k0;       // first sorted position of the tile
    int cnt;      // particles in the tile (<= 32)
    bool cells;   // false for the group of non-finite particles (no neighbours)
    int cx, cy, cz;
    int lo[3], hi[3];
};

// Geometry of the whole grid (single scene).
__device__ __forceinline__ Geom grid_geom(const DevState* ds) {
    Geom g;
    for (int a = 0; a < 3; ++a) {
        g.dim[a] = ds->dim[a];
        g.wrap[a] = ds->wrap[a];
    }
    g.base = 0;
    g.sentinel = ds->ncells;
    return g;
}

// Geometry of one scene's block of cells (batched mode; scene grids are never folded).
__device__ __forceinline__ Geom scene_geom(const SceneInfo& sc, const DevState* ds) {
    Geom g;
    for (int a = 0; a < 3; ++a) {
        g.dim[a] = sc.dim[a];
        g.wrap[a] = 0;
    }
    g.base = sc.base;
    g.sentinel = ds->ncells;
    return g;
}

// The tile's z range relative to its first particle's cell: every lane's cell +-1, or +-2
// on the side where the lane lies within the guard band of a cell face.
__device__ __forceinline__ void tile_z_range(const Buffers& b, const Geom& g, uint32_t k0,
                                             int lane, bool valid, bool near_lo, bool near_hi,
                                             Tile& T) {
    const uint32_t kl = valid ? b.key_s[k0 + lane] : b.key_s[k0];
    const int rz = (int)((kl - g.base) % (uint32_t)g.dim[2]) - T.cz;  // >= 0 (sorted)
    T.lo[2] = __reduce_min_sync(0xffffffffu, rz + (near_lo ? -2 : -1));
    T.hi[2] = __reduce_max_sync(0xffffffffu, rz + (near_hi ? 2 : 1));
}

// Sets up a tile; returns the sorted position i of the lane's particle and the particle
// (valid lanes only).
__device__ __forceinline__ void tile_setup(const StepConst& c, const Buffers& b, const Geom& g,
                                           uint2 tile, int lane, Tile& T, int& i, float4& xi,
                                           bool& valid) {
    const uint32_t k0 = tile.x;
    const uint32_t key = b.key_s[k0];
    T.k0 = (int)k0;
    T.cnt = (int)tile.y;
    valid = lane < T.cnt;
    i = (int)k0 + lane;
    if (b.tgt && valid) i = (int)b.tgt[k0 + lane];
    xi = valid ? b.pos4_s[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    T.cells = key < g.sentinel;
    if (!T.cells) return;
    const uint32_t local = key - g.base;
    const uint32_t dz = g.dim[2], dy = g.dim[1];
    T.cz = (int)(local % dz);
    T.cy = (int)((local / dz) % dy);
    T.cx = (int)(local / (dz * dy));
    const float x[3] = {xi.x, xi.y, xi.z};
    bool lo_z = false, hi_z = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // position inside the cell in cell units; the guard band covers the rounding of
        // x*inv_cell and of the distance test (a few ulps of |u|) with a wide margin
        const float u = xmul(x[a], c.inv_cell);
        const float frac = u - floorf(u);
        const float eps = 1.52587890625e-5f + fabsf(u) * 9.5367431640625e-7f;
        const bool near_lo = valid && frac < eps;
        const bool near_hi = valid && (1.0f - frac) < eps;
        if (a == 2) {
            lo_z = near_lo;
            hi_z = near_hi;
        } else {
            T.lo[a] = __any_sync(0xffffffffu, near_lo) ? -2 : -1;
            T.hi[a] = __any_sync(0xffffffffu, near_hi) ? 2 : 1;
        }
    }
    tile_z_range(b, g, k0, lane, valid, lo_z, hi_z, T);
}

// Precision mode: the tile's frame is the cell of its first particle; the lane's particle is
// (cell, offset o), for lanes past the tile's end its first one.  A position inside the frame
// is (cell - frame) * cs + offset, exact to a few ulps of the cell size however
// far the frame lies from the origin.
__device__ __forceinline__ float4 frame_pos(const int4& cell, const int4& frame, const float4& o,
                                            float cs) {
    return make_float4((float)(cell.x - frame.x) * cs + o.x, (float)(cell.y - frame.y) * cs + o.y,
                       (float)(cell.z - frame.z) * cs + o.z, o.w);
}

__device__ __forceinline__ void tile_setup_cells(const StepConst& c, const Buffers& b,
                                                 const Geom& g, uint2 tile, int lane, Tile& T,
                                                 int& i, int4& cell, float4& o, bool& valid,
                                                 int4& frame) {
    const uint32_t k0 = tile.x;
    const uint32_t key = b.key_s[k0];
    T.k0 = (int)k0;
    T.cnt = (int)tile.y;
    valid = lane < T.cnt;
    i = (int)k0 + (valid ? lane : 0);
    if (b.tgt) i = (int)b.tgt[i];
    cell = b.cell4_s[i];
    o = b.pos4_s[i];
    frame.x = __shfl_sync(0xffffffffu, cell.x, 0);
    frame.y = __shfl_sync(0xffffffffu, cell.y, 0);
    frame.z = __shfl_sync(0xffffffffu, cell.z, 0);
    frame.w = 0;
    T.cells = key < g.sentinel;
    if (!T.cells) return;
    const uint32_t local = key - g.base;
    const uint32_t dz = g.dim[2], dy = g.dim[1];
    T.cz = (int)(local % dz);
    T.cy = (int)((local / dz) % dy);
    T.cx = (int)(local / (dz * dy));
    const float off[3] = {o.x, o.y, o.z};
    const float eps = c.cs * 2.44140625e-4f;  // 2^-12 cells
    bool lo_z = false, hi_z = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool near_lo = valid && off[a] < eps;
        const bool near_hi = valid && (c.cs - off[a]) < eps;
        if (a == 2) {
            lo_z = near_lo;
            hi_z = near_hi;
        } else {
            T.lo[a] = __any_sync(0xffffffffu, near_lo) ? -2 : -1;
            T.hi[a] = __any_sync(0xffffffffu, near_hi) ? 2 : 1;
        }
    }
    tile_z_range(b, g, k0, lane, valid, lo_z, hi_z, T);
}

// Calls f(begin, end) for every stencil row of the tile, in the reference's order.  On a
// folded axis the neighbour index wraps; a row that wraps on z is two segments, visited
// in dz order.
template <class F>
__device__ __forceinline__ void for_each_row(const Buffers& b, const Geom& g, const Tile& T,
                                             F&& f) {
    if (!T.cells) return;
    const int d0 = g.dim[0], d1 = g.dim[1], d2 = g.dim[2];
    const bool w0 = g.wrap[0], w1 = g.wrap[1], w2 = g.wrap[2];
    // z range of every row: [z0, z1] plus, when z wraps past the end, [0, z2]
    int z0 = T.cz + T.lo[2], z1 = T.cz + T.hi[2], z2 = -1;
    int zp = -1, zq = -2;  // a wrapped piece at the front (dz < 0 past 0)
    if (w2 && z1 - z0 + 1 >= d2) {  // it covers the folded axis: each cell once
        zp = z0 < 0 ? z0 + d2 : z0;
        zq = d2 - 1;
        z0 = 0;
        z1 = zp - 1;
    } else if (w2) {
        if (z0 < 0) {
            zp = z0 + d2;
            zq = d2 - 1;
            z0 = 0;
        }
        if (z1 >= d2) {
            z2 = z1 - d2;
            z1 = d2 - 1;
        }
    } else {
        z0 = max(z0, 0);
        z1 = min(z1, d2 - 1);
    }
    for (int dx = T.lo[0]; dx <= T.hi[0]; ++dx) {
        int X = T.cx + dx;
        if (w0) X = (X + d0) % d0;
        else if (X < 0 || X >= d0) continue;
        for (int dy = T.lo[1]; dy <= T.hi[1]; ++dy) {
            int Y = T.cy + dy;
            if (w1) Y = (Y + d1) % d1;
            else if (Y < 0 || Y >= d1) continue;
            const uint32_t rb = g.base + ((uint32_t)X * (uint32_t)d1 + (uint32_t)Y) * (uint32_t)d2;
            if (zp <= zq) {
                const uint32_t a = b.off[rb + zp], e = b.off[rb + zq + 1];
                if (a < e) f((int)a, (int)e);
            }
            if (z0 <= z1) {
                const uint32_t a = b.off[rb + z0], e = b.off[rb + z1 + 1];
                if (a < e) f((int)a, (int)e);
            }
            if (z2 >= 0) {
                const uint32_t a = b.off[rb], e = b.off[rb + z2 + 1];
                if (a < e) f((int)a, (int)e);
            }
        }
    }
}

// The same walk as for_each_row, listed up front: writes the tile's non-empty row
// segments [a, e) to seg in visiting order and returns their number (<= 75: 5 x 5 rows of
// up to 3 pieces).  One lane per row (dx, dy) -- lane order is the rows' visiting order --
// and a warp scan places each row's pieces.
constexpr int kMaxSegments = 75;
__device__ __forceinline__ int build_segments(const Buffers& b, const Geom& g, const Tile& T,
                                              int lane, int2* seg) {
    if (!T.cells) return 0;
    const int d0 = g.dim[0], d1 = g.dim[1], d2 = g.dim[2];
    int z0 = T.cz + T.lo[2], z1 = T.cz + T.hi[2], z2 = -1;
    int zp = -1, zq = -2;
    if (g.wrap[2] && z1 - z0 + 1 >= d2) {  // it covers the folded axis: each cell once
        zp = z0 < 0 ? z0 + d2 : z0;
        zq = d2 - 1;
        z0 = 0;
        z1 = zp - 1;
    } else if (g.wrap[2]) {
        if (z0 < 0) {
            zp = z0 + d2;
            zq = d2 - 1;
            z0 = 0;
        }
        if (z1 >= d2) {
            z2 = z1 - d2;
            z1 = d2 - 1;
        }
    } else {
        z0 = max(z0, 0);
        z1 = min(z1, d2 - 1);
    }
    const int ny = T.hi[1] - T.lo[1] + 1;
    const int nrows = (T.hi[0] - T.lo[0] + 1) * ny;
    int2 p0 = make_int2(0, 0), p1 = p0, p2 = p0;  // the row's pieces, in dz order
    bool v0 = false, v1 = false, v2 = false;
    if (lane < nrows) {
        int X = T.cx + T.lo[0] + lane / ny;
        int Y = T.cy + T.lo[1] + lane % ny;
        bool ok = true;
        if (g.wrap[0]) X = (X + d0) % d0;
        else ok = X >= 0 && X < d0;
        if (g.wrap[1]) Y = (Y + d1) % d1;
        else ok = ok && Y >= 0 && Y < d1;
        if (ok) {
            const uint32_t rb = g.base + ((uint32_t)X * (uint32_t)d1 + (uint32_t)Y) * (uint32_t)d2;
            if (zp <= zq) {
                p0 = make_int2((int)b.off[rb + zp], (int)b.off[rb + zq + 1]);
                v0 = p0.x < p0.y;
            }
            if (z0 <= z1) {
                p1 = make_int2((int)b.off[rb + z0], (int)b.off[rb + z1 + 1]);
                v1 = p1.x < p1.y;
            }
            if (z2 >= 0) {
                p2 = make_int2((int)b.off[rb], (int)b.off[rb + z2 + 1]);
                v2 = p2.x < p2.y;
            }
        }
    }
    const uint32_t np = (uint32_t)v0 + (uint32_t)v1 + (uint32_t)v2;
    uint32_t x = np;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    uint32_t at = x - np;
    if (v0) seg[at++] = p0;
    if (v1) seg[at++] = p1;
    if (v2) seg[at] = p2;
    return (int)__shfl_sync(0xffffffffu, x, 31);
}

// d = x_i - x_j; d2 = dot(d, d)  (spatial_hash.h:70-73, sph_engine.cpp:378, 400, 424)
struct Diff {
    float x, y, z, d2;
};
__device__ __forceinline__ Diff diff(const float4& xi, const float4& xj) {
    Diff d;
    d.x = xsub(xi.x, xj.x);
    d.y = xsub(xi.y, xj.y);
    d.z = xsub(xi.z, xj.z);
    d.d2 = xdot3(d.x, d.y, d.z);
    return d;
}
// diff(xi, xj).d2 with the x and y steps as packed FP32 pairs (same rounding)
__device__ __forceinline__ float diff_d2(const float4& xi, const float4& xj) {
    const f32x2 dxy = xsub2(pk2(xi.x, xi.y), pk2(xj.x, xj.y));
    const float dz = xsub(xi.z, xj.z);
    const float2 sq = upk2(xmul2(dxy, dxy));
    return xadd(xadd(sq.x, sq.y), xmul(dz, dz));
}

constexpr uint32_t kFull = 0xffffffffu;

// Axis-aligned box of the tile's particles (valid lanes).
struct TileBox {
    float lo[3], hi[3];
};
__device__ __forceinline__ TileBox tile_box(const float4& xi, bool valid) {
    TileBox B;
    const float inf = __int_as_float(0x7f800000);
    B.lo[0] = valid ? xi.x : inf;
    B.lo[1] = valid ? xi.y : inf;
    B.lo[2] = valid ? xi.z : inf;
    B.hi[0] = valid ? xi.x : -inf;
    B.hi[1] = valid ? xi.y : -inf;
    B.hi[2] = valid ? xi.z : -inf;
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            B.lo[a] = fminf(B.lo[a], __shfl_xor_sync(kFull, B.lo[a], o));
            B.hi[a] = fmaxf(B.hi[a], __shfl_xor_sync(kFull, B.hi[a], o));
        }
    return B;
}

// Conservative: false only if no point of the box is within r of p (margin 1e-4 on r^2
// covers every rounding of this test and of the exact distance test).
__device__ __forceinline__ bool box_near(const TileBox& B, const float4& p, float r2_margin) {
    const float ex = fmaxf(fmaxf(B.lo[0] - p.x, p.x - B.hi[0]), 0.0f);
    const float ey = fmaxf(fmaxf(B.lo[1] - p.y, p.y - B.hi[1]), 0.0f);
    const float ez = fmaxf(fmaxf(B.lo[2] - p.z, p.z - B.hi[2]), 0.0f);
    return ex * ex + ey * ey + ez * ez <= r2_margin;
}

// ---------------------------------------------------------------------------------------
// Candidate rings (density and force passes).
//
// The candidates of the tile's walk that its box keeps are appended, in order, to a ring of
// kRing chunks of 32 in shared memory, and each complete chunk gets one 32-bit mask per lane:
// bit p is set when the candidate in slot p of the chunk is a neighbour of the lane's
// particle.  The j-th candidate of a chunk sits in slot 31 - j, so that the highest set bit is
// the next neighbour in order.  Every lane then takes its own neighbours one after another,
// each at its own place in the ring, forms the term and adds it to its sums in registers: no
// hit list, no staging of terms, and the additions happen in the walk's order by construction.
//
// What bounds the split: all lanes of a warp issue together, so a pass costs the largest
// number of terms any lane has between two points where the lanes must meet.  The lanes of a
// tile have about the same number of neighbours in all (270 on the lattice, within 7%) but
// meet them at different times: a particle on the low-x side of the tile meets its first
// third of the stream before one on the high side meets any.  The ring is what lets a lane
// run ahead; its length trades resident warps (shared memory) for that freedom.  Iterations
// per particle on the lattice (ideal 7.5): 21 with one chunk, 13 with 4, 11 with 8, 9.1 with
// 12, 8.0 with 16.
// ---------------------------------------------------------------------------------------

// The walk's row segments, 32 candidates at a time (warp-uniform).
struct RawStream {
    const int2* seg;
    int nseg, sg, s, e;
    __device__ __forceinline__ RawStream(const int2* segs, int n) : seg(segs), nseg(n), sg(0) {
        s = n ? segs[0].x : 0;
        e = n ? segs[0].y : 0;
    }
    __device__ __forceinline__ bool more() const { return sg < nseg; }
    __device__ __forceinline__ int count() const { return min(32, e - s); }
    __device__ __forceinline__ void next() {
        s += 32;
        if (s < e) return;
        if (++sg < nseg) {
            s = seg[sg].x;
            e = seg[sg].y;
        }
    }
};

// Ring slot of the a-th candidate kept (a counts from the tile's start).
template <int kRing>
__device__ __forceinline__ int ring_slot(int a) {
    return ((a >> 5) % kRing) * 32 + (31 - (a & 31));
}

// glm::dot(d, d) of two separations
__device__ __forceinline__ F2 pair_d2(F2 dx, F2 dy, F2 dz, F2 neg0) {
    return (pmul(dx, dx, neg0) + pmul(dy, dy, neg0)) + pmul(dz, dz, neg0);
}

// Neighbour mask of the lane's particle against a complete chunk (32 slots of cx, cy, cz): the
// reference's rounded test (x_i - x_j per axis, (dx*dx + dy*dy) + dz*dz, <= r^2), two
// candidates per packed FP32 instruction, element by element.  d2 <= r2 is read from the sign
// of r2 - d2 (exact: a rounded difference keeps its sign), shifted into the mask.
__device__ __forceinline__ uint32_t ring_hits(const float* cx, const float* cy, const float* cz,
                                              const float4& xi, float r2, F2 neg0) {
    const F2 X = f2(xi.x), Y = f2(xi.y), Z = f2(xi.z), R2 = f2(r2);
    uint32_t miss = 0;
#pragma unroll
    for (int q = 28; q >= 0; q -= 4) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(cx + q);
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(cy + q);
        const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(cz + q);
#pragma unroll
        for (int h = 1; h >= 0; --h) {
            const F2 dx = X - F2{h ? x.y : x.x}, dy = Y - F2{h ? y.y : y.x},
                     dz = Z - F2{h ? z.y : z.x};
            const float2 t = upk2((R2 - pair_d2(dx, dy, dz, neg0)).v);
            miss = __funnelshift_l(__float_as_uint(t.y), miss, 1);
            miss = __funnelshift_l(__float_as_uint(t.x), miss, 1);
        }
    }
    return ~miss;
}

// slots of a chunk that hold candidates when `left` of the stream remain from its start
__device__ __forceinline__ uint32_t chunk_valid(int left) {
    return left >= 32 ? kFull : ~(kFull >> left);
}

// position of the highest set bit
__device__ __forceinline__ uint32_t top_bit(uint32_t m) {
    uint32_t p;
    asm("bfind.u32 %0, %1;" : "=r"(p) : "r"(m));
    return p;
}

// A lane's place in the ring: the next chunk to load and what is left of the mask of the one
// before it.
template <int kRing>
struct RingLane {
    int next = 0;  // chunks from the tile's start
    int at = 0;    // first slot of the chunk being worked through
    int at_next = 0;
    uint32_t m = 0;
    // first chunk still needed
    __device__ __forceinline__ int need() const { return next - (m != 0); }
    // loads the next of the first n chunks when the last one is used up
    __device__ __forceinline__ void advance(const uint32_t* mask, int n, int lane) {
        if (m == 0 && next < n) {
            m = mask[at_next + lane];
            at = at_next;
            at_next = at == (kRing - 1) * 32 ? 0 : at + 32;
            ++next;
        }
    }
    // the same without a branch (force pass, 1M: 1.53 -> 1.50 ms; the density pass is faster with
    // the branch, 0.96 against 1.00)
    __device__ __forceinline__ void advance_flat(const uint32_t* mask, int n, int lane) {
        const bool take = m == 0 && next < n;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.u32 %0, [%1];\n\t}"
                     : "+r"(m) : "r"(smem_u32(mask + at_next + lane)), "r"((uint32_t)take) : "memory");
        at = take ? at_next : at;
        const int after = at_next == (kRing - 1) * 32 ? 0 : at_next + 32;
        at_next = take ? after : at_next;
        next += take;
    }
    // Slots of the next two neighbours of the chunk, removed from the mask; a: there is one,
    // b: there are two (otherwise the slot is some slot of the ring).
    __device__ __forceinline__ void take2(int& qa, int& qb, bool& a, bool& b) {
        a = m != 0;
        const uint32_t pa = top_bit(m) & 31u;
        m &= ~(1u << pa);
        b = m != 0;
        const uint32_t pb = top_bit(m) & 31u;
        m &= ~(1u << pb);
        qa = at + (int)pa;
        qb = at + (int)pb;
    }
};

// W of the pair with |x_i - x_j|^2 = d2 for smoothing kernel K, with the reference's float
// operations (Kernel::W, kernels.cpp:140-143, 172-178, 210-213).
template <int K>
__device__ __forceinline__ float pair_w_exact(const StepConst& c, float d2) {
    if (K == SPHX_KERNEL_GAUSSIAN) return xmul(c.wnorm, expf(xmul(-d2, c.gs)));
    const float q = xdiv_fixed(xsqrt(d2), c.h, c.rcp_h, c.fast_div_h);
    return K == SPHX_KERNEL_WENDLAND_C2 ? wendland_w(c, q) : cubic_w(c, q);
}

// pair_w_exact of two neighbours of the cubic spline or Wendland kernel (StepConst::div_nz and
// no tiny coordinate: d2 is 0 or at least 2^-136)
template <int K>
__device__ __forceinline__ F2 pair_w_exact2(const PairLits& k, const PairConst& c, F2 d2) {
    const F2 neg0{k.neg0};
    F2 hr, ns;
    const F2 q = div_fixed2(sqrt2_exact(k, d2, hr, ns), F2{c.neg_h}, F2{c.rcp_h});
    const float2 u = upk2(q.v);
    // beyond the support q = 2 the clamped 2 - q (1 - q/2) makes the outer branch the 0 that
    // the reference returns there; 0.5 q and 2 q are exact: contraction changes nothing
    if (K == SPHX_KERNEL_WENDLAND_C2) {
        const F2 t = max0(F2{k.one} - F2{k.half} * q);
        return F2{c.wnorm} * t * t * t * t * (F2{k.two} * q + F2{k.one});
    }
    const F2 t = max0(F2{k.two} - q);
    const F2 w1 = (F2{k.two_thirds} - pmul(q, q, neg0)) + pmul(F2{k.half} * q * q, q, neg0);
    const F2 w2 = F2{k.one_sixth} * t * t * t;
    return F2{c.sigma} * select2(u.x <= 1.0f, u.y <= 1.0f, w1, w2);
}

// integrate_leapfrog and the wall clamp (sph_engine.cpp:290-310, particle.cpp:122-153)
__device__ __forceinline__ void leapfrog_exact(const StepConst& c, float dt, const float* acc,
                                               float* x, float* v) {
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
}

// Precision-mode leapfrog + wall clamp on cell + offset positions (FP64 clamp).
__device__ __forceinline__ void integrate_cells(const StepConst& c, float dt, const float* acc,
                                                float* o, float* v, int4& cell) {
    int* cc[3] = {&cell.x, &cell.y, &cell.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float half = 0.5f * acc[a] * dt;
        float vv = v[a] + half;
        float on = o[a] + vv * dt;
        vv = vv + half;
        v[a] = vv * c.damping;
        if (!isfinite(on)) {  // the position is lost: park the particle as non-finite
            cell.w = 1;
            o[a] = on;
            continue;
        }
        double X = (double)(*cc[a]) * c.cs_d + (double)on;
        if (X < (double)c.lo[a]) {
            X = c.lo[a];
            v[a] = v[a] * -0.8f;
        } else if (X > (double)c.hi[a]) {
            X = c.hi[a];
            v[a] = v[a] * -0.8f;
        }
        double f = floor(X / c.cs_d);
        f = fmin(fmax(f, -(double)kCellClamp), (double)(kCellClamp - 1));
        int ci = (int)f;
        float oo = (float)(X - (double)ci * c.cs_d);
        if (c.fp16) oo = round_half(oo);
        if (oo >= c.cs) {
            oo = 0.0f;
            ci += 1;
        } else if (oo < 0.0f) {
            oo = 0.0f;
        }
        *cc[a] = ci;
        o[a] = oo;
    }
}

// Work distribution of a persistent pass: the first tile of every warp is fixed, later ones come
// from the pass's counter (dynamic, so crowded cells in degenerate states do not serialise the
// tail).  The first ones go round the SMs, then round each SM's sub-partitions (block k runs on
// SM k mod num_sms, warp w of a block on sub-partition w mod 4), so that a set of few tiles
// spreads over the whole GPU; handed out by the counter alone, the blocks that start first
// took up to a dozen each (10k particles, 352 tiles: force 0.133 -> 0.099 ms).
struct TileQueue {
    uint32_t* ctr;
    uint32_t first, warps;
    __device__ __forceinline__ TileQueue(uint32_t* counter, int num_sms) : ctr(counter) {
        const uint32_t per = blockDim.x >> 5, s = (uint32_t)num_sms;
        const uint32_t row = blockIdx.x / s, col = blockIdx.x % s;
        const uint32_t width = min(s, gridDim.x - row * s);  // blocks in this row
        first = row * s * per + (threadIdx.x >> 5) * width + col;
        warps = gridDim.x * per;
    }
    __device__ __forceinline__ uint32_t start() const { return first; }
    __device__ __forceinline__ uint32_t next(int lane) const {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(ctr, 1u) + warps;
        return __shfl_sync(kFull, t, 0);
    }
};

// A warp's share of the record pool (Buffers::records), filled tile after tile: an equal region
// for every warp that gets a tile at all (record indices fit 32 bits: the pool holds at most
// 0xffff0000 records).  Regions for all resident warps would be too small for one tile on
// small sets, whose force pass then walked and tested again (10k: 0.099 ms against 0.068).
struct RecordRegion {
    uint32_t cur, end;
    __device__ __forceinline__ RecordRegion(const Buffers& b, const TileQueue& q, uint32_t ntiles) {
        const uint32_t w = min(q.warps, ntiles);
        const uint32_t region = b.records && q.first < w ? (uint32_t)(b.record_cap / w) : 0u;
        cur = q.first * region;
        end = cur + region;
    }
};

// Persistent grid: as many CTAs as fit on the GPU (queried once per kernel).
template <class K>
inline int resident_blocks(const LaunchCtx& L, K kernel, int threads, size_t smem) {
    int per_sm = 0;
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
            cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    if (L.blocks_per_sm > 0 && L.blocks_per_sm < per_sm) per_sm = L.blocks_per_sm;
    return L.num_sms * per_sm;
}

// Grid sizes of the persistent passes, found once per (device, kernel instantiation, warps
// per block, requested CTAs per SM) and kept: one cache object per instantiation, indexed
// by device; any host thread may fill an entry (a racing fill stores the same value).
struct LaunchShapeCache {
    std::atomic<int> nb[kMaxCacheDevices][5][33];
    std::atomic<int>& at(const LaunchCtx& L) {
        const int d = L.device >= 0 && L.device < kMaxCacheDevices ? L.device : 0;
        const int w = L.warps_per_block >= 0 && L.warps_per_block <= 4 ? L.warps_per_block : 4;
        const int b = L.blocks_per_sm >= 0 && L.blocks_per_sm < 32 ? L.blocks_per_sm : 32;
        return nb[d][w][b];
    }
};

template <class K>
inline int cached_resident_blocks(LaunchShapeCache& cache, const LaunchCtx& L, K kernel,
                                  int threads, size_t smem) {
    std::atomic<int>& slot = cache.at(L);
    int nb = slot.load(std::memory_order_relaxed);
    if (!nb) {
        nb = resident_blocks(L, kernel, threads, smem);
        slot.store(nb, std::memory_order_relaxed);
    }
    return nb;
}

inline int pass_blocks(const LaunchCtx& L) {
    const int bps = L.blocks_per_sm > 0 ? L.blocks_per_sm : 8;
    return L.num_sms * bps;
}

}  // namespace sphx
