// Standalone spatial hash on the GPU: the device side of SpatialHash::build / query /
// query_squared / get_cell_particles (src/spatial_hash.cpp:15-63).
//
// build() runs the step's grid pipeline (bbox, cell keys, stable radix sort, cell
// offsets) on the given positions with the hash's cell size.  A query visits the
// reference's stencil -- cells cq + (dx, dy, dz), each of dx, dy, dz in
// [-cell_radius, cell_radius] with cell_radius = ceil(sqrt(r2) * inv_cell) + 1, in
// lexicographic order -- and each cell's particles in insertion order, keeping those with
// dot(p - x_j, p - x_j) <= r2: the reference's list, element for element.
#include <cmath>
#include <mutex>
#include <utility>
#include <vector>

#include "sphx_internal.cuh"

using namespace sphx;

// Device blocks of one query, grown as needed.
struct QueryWork {
    void* p[4] = {};         // query points, counts, list offsets, lists
    size_t bytes[4] = {};
};

struct sphx_grid {
    int device = 0;
    cudaStream_t stream = nullptr;
    size_t capacity = 0;
    size_t n = 0;
    float cell_size = 0.0f;
    bool built = false;
    StepConst sc{};
    Buffers b{};
    DevState* ds = nullptr;
    float* stage = nullptr;  // 4 * capacity floats
    LaunchCtx L{};
    DevState host{};         // copy of the device state after the last build
    // The query workspace of the last call, for the next one (each allocation and release of the
    // result array synchronises and takes 0.1 ms).  A call takes it out of the grid for as long
    // as it runs, so that calls from several threads never share a block: those that find it
    // gone allocate their own.
    QueryWork kept;
    std::mutex kept_mutex;
};

constexpr size_t kKeepBytes = (size_t)256 << 20;  // of each block: a larger one is given back

namespace {

struct QueryArgs {
    const float* q;       // 3 floats per query
    int nq;
    float r2;
    int cr;               // stencil half-width in cells
    float inv_cell, cell_size;
};

// Lower bound of |p - x| on one axis over the particles x of cell `c` (p lies in cell `own`);
// the guard covers the rounding of x * inv_cell and of this bound.
__device__ __forceinline__ float axis_gap(float p, long long own, long long c, float cell,
                                          float guard) {
    const float d = c > own ? (float)c * cell - p : (c < own ? p - (float)(c + 1) * cell : 0.0f);
    return fmaxf(d - guard, 0.0f);
}

// One warp per query; kFill = false counts, kFill = true writes insertion indices.  The lanes
// take the candidates of a stencil row (dx, dy, *), one contiguous range of the sorted array,
// 32 at a time, and keep the row's order by their ranks.  Cells that lie farther than r from
// the query are skipped (the reference's outer layer, but for queries at a cell face).  Bound
// by L2 reads of the candidates (20,011 unordered queries of 250 neighbours among 200,003
// particles: 0.7 GB, 0.088 ms to count and 0.098 to fill; with a thread per query over the
// whole stencil 0.68 and 2.14 ms).
template <bool kFill>
__global__ void __launch_bounds__(128) k_grid_query(const QueryArgs a, const Buffers b,
                                                    const DevState* ds, uint32_t* counts,
                                                    const uint64_t* offsets, int64_t* out) {
    const int lane = threadIdx.x & 31;
    const long long qi = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (qi >= a.nq) return;
    const float p[3] = {a.q[3 * qi], a.q[3 * qi + 1], a.q[3 * qi + 2]};
    uint32_t found = 0;
    const uint64_t at = kFill ? offsets[qi] : 0;
    if (finite3(p[0], p[1], p[2]) && ds->status == 0) {
        // r^2 with a margin that covers the rounding of the exact test
        const float r2m = a.r2 * 1.0001f;
        long long own[3];
        float guard[3];
        int dim[3];
        bool wrap[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            own[k] = cell_coord(p[k], a.inv_cell);
            guard[k] = a.cell_size * 1.52587890625e-5f + fabsf(p[k]) * 9.5367431640625e-7f;
            dim[k] = ds->dim[k];
            wrap[k] = ds->wrap[k];
        }
        // grid index of the true cell coordinate c; false: outside the grid
        auto index = [&](int k, long long c, long long& g) {
            g = c - ds->cmin[k];
            if (wrap[k]) g = ((g % dim[k]) + dim[k]) % dim[k];
            return wrap[k] || (g >= 0 && g < dim[k]);
        };
        auto range = [&](uint32_t k0, uint32_t k1) {
            for (uint32_t s = k0; s < k1; s += 32) {
                const uint32_t k = s + (uint32_t)lane;
                bool hit = false;
                if (k < k1) {
                    const float4 x = b.pos4_s[k];
                    hit = xdot3(xsub(p[0], x.x), xsub(p[1], x.y), xsub(p[2], x.z)) <= a.r2;
                }
                const uint32_t hits = __ballot_sync(0xffffffffu, hit);
                if (kFill && hit)
                    out[at + found + __popc(hits & ((1u << lane) - 1u))] = (int64_t)b.id_s[k];
                found += __popc(hits);
            }
        };
        for (int dx = -a.cr; dx <= a.cr; ++dx) {
            long long X;
            const float gx = axis_gap(p[0], own[0], own[0] + dx, a.cell_size, guard[0]);
            if (gx * gx > r2m || !index(0, own[0] + dx, X)) continue;
            for (int dy = -a.cr; dy <= a.cr; ++dy) {
                long long Y;
                const float gy = axis_gap(p[1], own[1], own[1] + dy, a.cell_size, guard[1]);
                const float g2 = gx * gx + gy * gy;
                if (g2 > r2m || !index(1, own[1] + dy, Y)) continue;
                int z0 = -a.cr, z1 = a.cr;  // the row's cells within reach
                auto far = [&](int dz) {
                    const float gz = axis_gap(p[2], own[2], own[2] + dz, a.cell_size, guard[2]);
                    return g2 + gz * gz > r2m;
                };
                while (z0 < 0 && far(z0)) ++z0;
                while (z1 > 0 && far(z1)) --z1;
                const uint32_t* off = b.off + ((uint32_t)X * (uint32_t)dim[1] + (uint32_t)Y) *
                                                  (uint32_t)dim[2];
                const long long first = own[2] + z0 - ds->cmin[2], last = own[2] + z1 - ds->cmin[2];
                if (!wrap[2]) {
                    const long long c0 = first < 0 ? 0 : first;
                    const long long c1 = last >= dim[2] ? dim[2] - 1 : last;
                    if (c0 <= c1) range(off[c0], off[c1 + 1]);
                } else {  // cell by cell, in the stencil's order
                    for (int dz = z0; dz <= z1; ++dz) {
                        long long Z;
                        index(2, own[2] + dz, Z);
                        range(off[Z], off[Z + 1]);
                    }
                }
            }
        }
    }
    if (!kFill && lane == 0) counts[qi] = found;
}

// (the runtime's record of the error is cleared: it is this call's to report, not the next one's)
int cuda_err(cudaError_t e) {
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? SPHX_ERR_OOM : SPHX_ERR_CUDA;
}

#define GRID_CUDA(call)                             \
    do {                                            \
        cudaError_t e_ = (call);                    \
        if (e_ != cudaSuccess) return cuda_err(e_); \
    } while (0)

template <class T>
int galloc(T** p, size_t count) {
    *p = nullptr;
    if (cudaMalloc(reinterpret_cast<void**>(p), (count ? count : 1) * sizeof(T)) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return SPHX_ERR_OOM;
    }
    return SPHX_OK;
}

// block k with room for count elements
template <class T>
int workspace(QueryWork& w, int k, size_t count, T** p) {
    const size_t bytes = (count ? count : 1) * sizeof(T);
    if (bytes > w.bytes[k]) {
        if (w.p[k]) cudaFree(w.p[k]);
        w.p[k] = nullptr;
        w.bytes[k] = 0;
        unsigned char* q = nullptr;
        const int rc = galloc(&q, bytes);
        if (rc) return rc;
        w.p[k] = q;
        w.bytes[k] = bytes;
    }
    *p = static_cast<T*>(w.p[k]);
    return SPHX_OK;
}
// gives back the blocks of more than `keep` bytes
void trim(QueryWork& w, size_t keep) {
    for (int k = 0; k < 4; ++k)
        if (w.p[k] && w.bytes[k] > keep) {
            cudaFree(w.p[k]);
            w.p[k] = nullptr;
            w.bytes[k] = 0;
        }
}

// The grid's workspace for the duration of a call.
struct QueryWorkLease {
    sphx_grid* g;
    QueryWork w;
    explicit QueryWorkLease(sphx_grid* grid) : g(grid) {
        std::lock_guard<std::mutex> lock(g->kept_mutex);
        std::swap(w, g->kept);
    }
    ~QueryWorkLease() {
        trim(w, kKeepBytes);
        {
            std::lock_guard<std::mutex> lock(g->kept_mutex);
            std::swap(w, g->kept);
        }
        trim(w, 0);  // another call's, given back in the meantime
    }
    QueryWorkLease(const QueryWorkLease&) = delete;
    QueryWorkLease& operator=(const QueryWorkLease&) = delete;
};

void grid_free(sphx_grid* g) {
    trim(g->kept, 0);
    Buffers& b = g->b;
    void* ptrs[] = {b.pos4, b.vel4, b.pos4_s, b.vel4_s, b.key[0], b.key[1], b.val[0], b.val[1],
                    b.key_s, b.id_s, b.off, b.tiles, b.sync, g->ds, g->stage};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (g->stream) cudaStreamDestroy(g->stream);
}

// the stencil half-width of SpatialHash::query_squared (spatial_hash.cpp:35)
int cell_radius(float r2, float inv_cell) {
    return static_cast<int>(std::ceil(std::sqrt(r2) * inv_cell)) + 1;
}

}  // namespace

extern "C" {

int sphx_grid_create(sphx_grid** out, size_t capacity) {
    if (!out) return SPHX_ERR_INVALID_ARG;
    *out = nullptr;
    if (capacity == 0 || capacity > (size_t)0x7fffffff - 64) return SPHX_ERR_INVALID_ARG;
    int devs = 0;
    if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) return SPHX_ERR_CUDA;
    sphx_grid* g = new sphx_grid();
    auto fail = [&](int rc) {
        grid_free(g);
        delete g;
        return rc;
    };
    if (cudaGetDevice(&g->device) != cudaSuccess) return fail(SPHX_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking) != cudaSuccess)
        return fail(SPHX_ERR_CUDA);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
    g->L.stream = g->stream;
    g->L.device = g->device;
    g->L.num_sms = sms > 0 ? sms : 1;
    g->L.warps_per_block = 4;
    g->capacity = capacity;
    int64_t max_cells = (int64_t)capacity * 4;
    if (max_cells < ((int64_t)1 << 24)) max_cells = (int64_t)1 << 24;
    if (max_cells > ((int64_t)1 << 31) - 4) max_cells = ((int64_t)1 << 31) - 4;
    g->sc.max_cells = (uint32_t)max_cells;
    Buffers& b = g->b;
    const size_t C = capacity;
    int rc;
    if ((rc = galloc(&b.pos4, C)) || (rc = galloc(&b.vel4, C)) || (rc = galloc(&b.pos4_s, C)) ||
        (rc = galloc(&b.vel4_s, C)) || (rc = galloc(&b.key[0], C)) || (rc = galloc(&b.key[1], C)) ||
        (rc = galloc(&b.val[0], C)) || (rc = galloc(&b.val[1], C)) || (rc = galloc(&b.key_s, C)) ||
        (rc = galloc(&b.id_s, C)) || (rc = galloc(&b.off, (size_t)max_cells + 2)) ||
        (rc = galloc(&b.tiles, C)) ||  (rc = galloc(&g->ds, 1)) ||
        (rc = galloc(&g->stage, 4 * C)))
        return fail(rc);
    unsigned char* scratch = nullptr;
    if ((rc = galloc(&scratch, grid_scratch_bytes(C)))) return fail(rc);
    set_grid_scratch(b, scratch);
    if (cudaMemset(g->ds, 0, sizeof(DevState)) != cudaSuccess ||
        cudaMemset(scratch, 0, grid_scratch_bytes(C)) != cudaSuccess)
        return fail(SPHX_ERR_CUDA);
    *out = g;
    return SPHX_OK;
}

void sphx_grid_destroy(sphx_grid* g) {
    if (!g) return;
    cudaSetDevice(g->device);
    cudaStreamSynchronize(g->stream);
    grid_free(g);
    delete g;
}

int sphx_grid_build(sphx_grid* g, size_t n, const float* pos_xyz, float cell_size) {
    if (!g) return SPHX_ERR_INVALID_ARG;
    if (n > g->capacity) return SPHX_ERR_CAPACITY;
    if (n > 0 && !pos_xyz) return SPHX_ERR_INVALID_ARG;
    if (!(cell_size > 0.0f) || !std::isfinite(cell_size) || !std::isfinite(1.0f / cell_size))
        return SPHX_ERR_INVALID_ARG;
    GRID_CUDA(cudaSetDevice(g->device));
    g->n = n;
    g->cell_size = cell_size;
    g->built = true;
    g->sc.n = (int)n;
    g->sc.inv_cell = 1.0f / cell_size;  // SpatialHash::set_cell_size (spatial_hash.h:63-66)
    if (n == 0) return SPHX_OK;
    float* s_pos = g->stage;
    float* s_mass = g->stage + 3 * g->capacity;
    GRID_CUDA(cudaMemcpyAsync(s_pos, pos_xyz, 3 * n * sizeof(float), cudaMemcpyHostToDevice, g->stream));
    GRID_CUDA(cudaMemsetAsync(s_mass, 0, n * sizeof(float), g->stream));
    launch_pack(g->L, (int)n, s_pos, nullptr, s_mass, g->b.pos4, g->b.vel4);
    launch_grid(g->L, g->sc, g->b, g->ds, kNoStep, 0.0f);
    GRID_CUDA(cudaGetLastError());
    GRID_CUDA(cudaStreamSynchronize(g->stream));
    GRID_CUDA(cudaMemcpy(&g->host, g->ds, sizeof(DevState), cudaMemcpyDeviceToHost));
    return g->host.status;
}

int sphx_grid_query(sphx_grid* g, size_t nq, const float* q_xyz, float radius_squared,
                    int64_t* counts, int64_t* idx, size_t* total_inout) {
    if (!g || !counts || !total_inout || (nq > 0 && !q_xyz)) return SPHX_ERR_INVALID_ARG;
    if (nq > (size_t)0x7fffffff) return SPHX_ERR_INVALID_ARG;
    GRID_CUDA(cudaSetDevice(g->device));
    const size_t cap = *total_inout;
    *total_inout = 0;
    if (nq == 0) return SPHX_OK;
    if (!g->built || g->n == 0 || !(radius_squared >= 0.0f) || !std::isfinite(radius_squared)) {
        for (size_t i = 0; i < nq; ++i) counts[i] = 0;  // nothing can be within r
        return SPHX_OK;
    }
    const int cr = cell_radius(radius_squared, g->sc.inv_cell);
    // a folded axis may not wrap the stencil onto itself
    for (int a = 0; a < 3; ++a)
        if (g->host.wrap[a] && 2 * (long long)cr + 1 > g->host.dim[a]) return SPHX_ERR_DOMAIN;
    float* d_q = nullptr;
    uint32_t* d_cnt = nullptr;
    uint64_t* d_off = nullptr;
    int64_t* d_out = nullptr;
    int rc = SPHX_OK;
    QueryWorkLease lease(g);
    QueryWork& work = lease.w;
    if ((rc = workspace(work, 0, 3 * nq, &d_q)) || (rc = workspace(work, 1, nq, &d_cnt))) return rc;
    QueryArgs qa{d_q, (int)nq, radius_squared, cr, g->sc.inv_cell, g->cell_size};
    const int threads = 128, blocks = (int)((nq + threads / 32 - 1) / (threads / 32));
    std::vector<uint32_t> h_cnt(nq);
    cudaError_t e = cudaMemcpyAsync(d_q, q_xyz, 3 * nq * sizeof(float), cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) {
        k_grid_query<false><<<blocks, threads, 0, g->stream>>>(qa, g->b, g->ds, d_cnt, nullptr, nullptr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(h_cnt.data(), d_cnt, nq * sizeof(uint32_t), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) return cuda_err(e);
    std::vector<uint64_t> off(nq);
    uint64_t total = 0;
    for (size_t i = 0; i < nq; ++i) {
        counts[i] = h_cnt[i];
        off[i] = total;
        total += h_cnt[i];
    }
    *total_inout = (size_t)total;
    if (!idx || total == 0) return SPHX_OK;
    if (cap < total) return SPHX_ERR_OVERFLOW;
    if ((rc = workspace(work, 2, nq, &d_off)) || (rc = workspace(work, 3, total, &d_out))) return rc;
    e = cudaMemcpyAsync(d_off, off.data(), nq * sizeof(uint64_t), cudaMemcpyHostToDevice, g->stream);
    if (e == cudaSuccess) {
        k_grid_query<true><<<blocks, threads, 0, g->stream>>>(qa, g->b, g->ds, nullptr, d_off, d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(idx, d_out, total * sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
    return e == cudaSuccess ? SPHX_OK : cuda_err(e);
}

int sphx_grid_info(sphx_grid* g, size_t* occupied_cells, size_t* max_per_cell) {
    if (!g) return SPHX_ERR_INVALID_ARG;
    const bool any = g->built && g->n > 0;
    if (occupied_cells) *occupied_cells = any ? g->host.occupied : 0;
    if (max_per_cell) *max_per_cell = any ? g->host.max_occ : 0;
    return SPHX_OK;
}

int sphx_grid_cell(sphx_grid* g, int x, int y, int z, int64_t* idx, size_t* count_inout) {
    if (!g || !count_inout) return SPHX_ERR_INVALID_ARG;
    GRID_CUDA(cudaSetDevice(g->device));
    const size_t cap = *count_inout;
    *count_inout = 0;
    if (!g->built || g->n == 0) return SPHX_OK;
    const DevState& s = g->host;
    const int c[3] = {x, y, z};
    long long r[3];
    for (int a = 0; a < 3; ++a) {
        if (c[a] < s.cmin[a] || c[a] > s.cmax[a]) return SPHX_OK;  // no particle there
        r[a] = (long long)c[a] - s.cmin[a];
        if (s.wrap[a]) r[a] %= s.dim[a];
    }
    const uint32_t key = (uint32_t)((r[0] * s.dim[1] + r[1]) * s.dim[2] + r[2]);
    uint32_t range[2];
    GRID_CUDA(cudaMemcpy(range, g->b.off + key, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (range[1] <= range[0]) return SPHX_OK;
    const size_t cnt = range[1] - range[0];
    std::vector<uint32_t> ids(cnt);
    std::vector<float4> pos(cnt);
    GRID_CUDA(cudaMemcpy(ids.data(), g->b.id_s + range[0], cnt * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    GRID_CUDA(cudaMemcpy(pos.data(), g->b.pos4_s + range[0], cnt * sizeof(float4), cudaMemcpyDeviceToHost));
    // a folded grid cell can hold several true cells: keep the requested one
    size_t m = 0;
    std::vector<int64_t> keep;
    keep.reserve(cnt);
    const float inv = g->sc.inv_cell;
    for (size_t k = 0; k < cnt; ++k) {
        const float p[3] = {pos[k].x, pos[k].y, pos[k].z};
        bool same = true;
        for (int a = 0; a < 3 && same; ++a) {
            float f = std::floor(p[a] * inv);
            f = std::fmin(std::fmax(f, -(float)kCellClamp), (float)(kCellClamp - 1));
            same = (int)f == c[a];
        }
        if (same) keep.push_back(ids[k]);
    }
    m = keep.size();
    *count_inout = m;
    if (!idx) return SPHX_OK;
    if (cap < m) return SPHX_ERR_OVERFLOW;
    for (size_t k = 0; k < m; ++k) idx[k] = keep[k];
    return SPHX_OK;
}

}  // extern "C"
