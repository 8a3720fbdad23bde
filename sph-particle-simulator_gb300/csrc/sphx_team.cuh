// Exact passes with a team of four lanes per particle, for sets too small to fill the GPU with
// a lane per particle (sphx_team_density.cu, sphx_team_force.cu).
//
// A tile is at most 8 particles of a cell column.  The four lanes of a team split the tile's
// candidates among themselves (8 of a chunk of 32 each), append the neighbours that they find
// to the particle's queue in shared memory, at the places that the order of the walk gives
// them, and take the queue's neighbours 16 at a time, four per lane.  The terms are then added
// to the particle's sums one after another in the queue's order, so that every sum is formed
// as by one lane walking the stencil, bit for bit.
//
// Why: with a lane per particle a warp works through its 32 particles' neighbours in some 130
// dependent turns whatever the size of the set, 65 us for each pass, while 10k particles give
// the 608 schedulers 313 warps.  A team's turns are a quarter of that, and there are four times
// as many warps.  The chunks' appends are predicated stores written out in PTX: as branches
// around each store they cost a third of the density pass (10k: 39.8 us, now 32.2).  One CTA
// per SM with as many warps as fit, so that the first tiles, dealt out a row of SMs at a time,
// spread evenly.
#pragma once
#include "sphx_pairs.cuh"

namespace sphx {

constexpr int kTeamTurn = 4 * kTeam;        // neighbours of a particle taken together

template <class Queue>
struct TeamSmem {
    // candidates that the tile's box keeps, their sorted positions: a ring of chunks
    float cx[128], cy[128], cz[128], cm[128];
    uint32_t cj[128];
    Queue queue[kTeamTile];  // neighbours per particle, a ring each
    int2 seg[kMaxSegments + 1];
};

// A particle's queue: entries appended and taken so far (the same in the team's lanes).
struct TeamQueue {
    uint32_t have = 0, done = 0;
};

// Predicated appends (the compiler would branch around each): if `on`, words to shared memory
// at a + 512 k, or at a + 4 kStride k with `at` advanced by a word.
__device__ __forceinline__ void store5_if(uint32_t on, uint32_t a, const float4& p, int j) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.f32 [%1], %2;\n\t"
        "@p st.shared.f32 [%1+512], %3;\n\t@p st.shared.f32 [%1+1024], %4;\n\t"
        "@p st.shared.f32 [%1+1536], %5;\n\t@p st.shared.u32 [%1+2048], %6;\n\t}"
        ::"r"(on), "r"(a), "f"(p.x), "f"(p.y), "f"(p.z), "f"(p.w), "r"(j) : "memory");
}
template <int kStride>
__device__ __forceinline__ void append3_if(uint32_t on, uint32_t& at, uint32_t a, float u, float v,
                                           uint32_t w) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.f32 [%2], %3;\n\t"
        "@p st.shared.f32 [%2+%6], %4;\n\t@p st.shared.u32 [%2+%7], %5;\n\t"
        "@p add.u32 %0, %0, 4;\n\t}"
        : "+r"(at) : "r"(on), "r"(a), "f"(u), "f"(v), "r"(w), "n"(4 * kStride), "n"(8 * kStride)
        : "memory");
}
__device__ __forceinline__ void append_if(uint32_t on, uint32_t& at, uint32_t a, uint32_t w) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.u32 [%2], %3;\n\t"
        "@p add.u32 %0, %0, 4;\n\t}" : "+r"(at) : "r"(on), "r"(a), "r"(w) : "memory");
}

// Walks the tile's stencil, 64 candidates at a time.  put(hit, n4, d2, m, j) stores,
// if hit, the (n4 / 4)-th neighbour of the lane's particle in its queue and adds 4 to n4; turn(false) takes neighbours off the queues: it is
// called while one of them (kQueue entries) has no room left for a chunk.  B, xi, i, valid: the
// tile's box, the lane's particle (the team's).  nn: its neighbours, itself included.
template <int kQueue, class Smem, class Put, class Turn>
__device__ __forceinline__ void team_walk(const Buffers& b, const Geom& g, const Tile& T,
                                          const TileBox& B, int i, const float4& xi, bool valid,
                                          float r2, int lane, Smem* S, F2 neg0, TeamQueue& Q,
                                          uint32_t& nn, Put&& put, Turn&& turn) {
    const uint32_t lt = (1u << lane) - 1u;
    const int sub = lane & (kTeam - 1);
    const float r2m = r2 * 1.0001f;
    const F2 X = f2(xi.x), Y = f2(xi.y), Z = f2(xi.z);
    // the tile's own particles lie between these positions
    const int own_lo = __reduce_min_sync(kFull, valid ? i : 0x7fffffff);
    const int own_hi = __reduce_max_sync(kFull, valid ? i : -1);
    __syncwarp();  // the previous tile's segments are read
    const int nseg = build_segments(b, g, T, lane, S->seg);
    __syncwarp();
    int sg = 0, s = 0, e = 0;
    if (nseg) {
        s = S->seg[0].x;
        e = S->seg[0].y;
    }
    float4 na = make_float4(0.f, 0.f, 0.f, 0.f), nb = na;  // the next candidates, read ahead
    if (s + lane < e) na = b.pos4_s[s + lane];
    if (s + 32 + lane < e) nb = b.pos4_s[s + 32 + lane];
    int kept = 0, tested = 0, self = -1;
    while (sg < nseg) {
        const float4 pa = na, pb = nb;
        const int at = s + lane;
        const bool ia = at < e, ib = at + 32 < e;
        const int first = s, end = e;
        s += 64;
        if (s >= e && ++sg < nseg) {
            s = S->seg[sg].x;
            e = S->seg[sg].y;
        }
        if (s + lane < e) na = b.pos4_s[s + lane];
        if (s + 32 + lane < e) nb = b.pos4_s[s + 32 + lane];
        const uint32_t ka = __ballot_sync(kFull, ia && box_near(B, pa, r2m));
        const uint32_t kb = __ballot_sync(kFull, ib && box_near(B, pb, r2m));
        const int mid = kept + __popc(ka);
        auto keep = [&](uint32_t mask, int base, const float4& p, int j) {
            const uint32_t on = mask & (1u << lane);
            const uint32_t a = smem_u32(&S->cx[(base + __popc(mask & lt)) & 127]);
            store5_if(on, a, p, j);
        };
        keep(ka, kept, pa, at);
        keep(kb, mid, pb, at + 32);
        if (first <= own_hi && own_lo < first + 64) {
            const int o = i < end ? i - first : -1;
            if ((unsigned)o < 32u) self = kept + __popc(ka & ((1u << o) - 1u));
            else if ((unsigned)o < 64u) self = mid + __popc(kb & ((1u << (o - 32)) - 1u));
        }
        kept = mid + __popc(kb);
        while (kept - tested >= 32 || (sg >= nseg && kept > tested)) {
            __syncwarp();  // the chunk is complete; the queues' last entries are read
            // the lane's 8 candidates of the chunk: the reference's rounded test, two per
            // packed instruction (see ring_hits)
            const int f = (tested & 96) + sub * 8;
            float d2[8];
            uint32_t mask = 0;
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(S->cx + f + h);
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(S->cy + f + h);
                const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(S->cz + f + h);
                const float2 a = upk2(pair_d2(X - F2{x.x}, Y - F2{y.x}, Z - F2{z.x}, neg0).v);
                const float2 c = upk2(pair_d2(X - F2{x.y}, Y - F2{y.y}, Z - F2{z.y}, neg0).v);
                d2[h] = a.x;
                d2[h + 1] = a.y;
                d2[h + 2] = c.x;
                d2[h + 3] = c.y;
            }
            const float4 m0 = *reinterpret_cast<const float4*>(S->cm + f),
                         m1 = *reinterpret_cast<const float4*>(S->cm + f + 4);
            const uint4 j0 = *reinterpret_cast<const uint4*>(S->cj + f),
                        j1 = *reinterpret_cast<const uint4*>(S->cj + f + 4);
            const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            const uint32_t j[8] = {j0.x, j0.y, j0.z, j0.w, j1.x, j1.y, j1.z, j1.w};
#pragma unroll
            for (int h = 0; h < 8; ++h) mask |= d2[h] <= r2 ? 1u << h : 0u;
            if (kept - tested < 32) {  // the last chunk
                const int left = kept - tested - sub * 8;
                if (left < 8) mask &= left <= 0 ? 0u : (1u << left) - 1u;
            }
            if (!valid) mask = 0;
            const int own = self - tested - sub * 8;
            if ((unsigned)own < 8u) mask &= ~(1u << own);
            // the team's masks, 8 bits a lane, in the chunk's order
            uint32_t all = mask << (8 * sub);
            all |= __shfl_xor_sync(kFull, all, 1);
            all |= __shfl_xor_sync(kFull, all, 2);
            uint32_t n4 = 4u * (Q.have + __popc(all & ((1u << (8 * sub)) - 1u)));
#pragma unroll
            for (int h = 0; h < 8; ++h) put(mask & (1u << h), n4, d2[h], m[h], j[h]);
            Q.have += __popc(all);
            tested += 32;
            __syncwarp();  // entries are in place, the chunk is read
            while (__any_sync(kFull, Q.have - Q.done > (uint32_t)(kQueue - 32))) turn(false);
        }
    }
    nn = Q.have + (self >= 0 && valid ? 1u : 0u);
}

}  // namespace sphx
