// Internal declarations of the sm_103a SPH step: device-resident state, per-step
// constants, exact-arithmetic helpers and the launch wrappers shared by the .cu files.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "sphx.h"

namespace sphx {

constexpr int kWarp = 32;
constexpr int kTile = 32;              // particles of one cell handled by one warp
constexpr int kTeam = 4;                // lanes per particle of the small sets' exact passes
constexpr int kTeamTile = kWarp / kTeam;
constexpr int kTeamMax = 1 << 16, kTeamMaxDensity = 40000;  // see pass_tile
constexpr int kRadixBits = 8;
constexpr int kRadixBuckets = 1 << kRadixBits;
constexpr int kRadixThreads = 256;
constexpr int kRadixItems = 16;
constexpr int kRadixTileN = kRadixThreads * kRadixItems;  // keys per radix block
constexpr int kMaxPasses = 4;                             // 32-bit keys
constexpr int kSmallSort = 1 << 18;                       // keys: see launch_radix_sort
constexpr int kSmallMax = 1 << 16;     // particles: see k_grid_small
constexpr int kPrepThreads = 256, kMaxPrepBlocks = 608;   // first kernel of a step
constexpr int kDiagThreads = 256;
constexpr int kDiagSums = 8;
constexpr float kCoincident = 1e-30f;  // see sweep_d2
// A nonzero coordinate below kTiny (in magnitude) sets DevState::general: without one x_i - x_j
// is 0 or at least kLeastStep, on which the pair forms rely.
constexpr float kTiny = 0x1p-45f, kLeastStep = 0x1p-68f;
constexpr int kCellClamp = 1 << 30;    // |cell coordinate| clamp for finite positions

// Operands of the packed pair arithmetic (F2), both halves equal: read as 64-bit operands from
// the kernel parameters, where a pair built from a scalar would cost two moves at each use.
typedef unsigned long long f32x2;
struct PairLits {  // numbers
    f32x2 neg0;    // -0: see F2
    f32x2 half, one, two, neg2, three, onehalf, neg2p40, p2p20, neg2p20, p2p21, two_thirds,
        one_sixth, neg5, five, neg_half, neg1, neg3, coincident;
};
struct PairConst {  // of the step's parameters
    f32x2 neg_h, h, rcp_h, neg_hsq, rcp_hsq, sigma, neg_sigma, gas, rest, wnorm, wl;
};

// Constants of one step, computed on the host in float exactly as the reference does
// (SpatialHash::set_cell_size, spatial_hash.h:63-66; CubicSplineKernel ctor,
// kernels.cpp:12-14, 23-36) and passed to the kernels by value.
struct StepConst {
    int n;                 // particles loaded
    float inv_cell;        // 1.0f / neighbor_search_radius
    float r2;              // neighbor_search_radius * neighbor_search_radius
    float h, h_sq, sigma;  // kernel constants
    float w0;              // W(vec3(0)) -- the self term factor
    float rest, gas, visc, grav, damping, cfl, timestep;
    float lo[3], hi[3];    // box
    uint32_t max_cells;    // capacity of the dense cell grid
    // precision mode (positions = integer cell + FP32 in-cell offset)
    int precise;           // 1: cell + offset storage, compensated sums, FP64 CFL/time
    int fp16;              // 1: offsets rounded to binary16 at every write
    float cs;              // cell size of the storage and of the search grid (= r_search)
    double cs_d;           // the same, as double
    // division by the fixed divisors h and h*h (see xdiv_fixed)
    float rcp_h, rcp_hsq;  // RN(1/h), RN(1/h^2)
    // the precision sweeps' units (lengths in units of h), read from the kernel parameters
    // rather than held in registers: cs / h, r^2 / h^2, the same with the box cull's margin,
    // (1e-6 m / h)^2
    float sw_cs, sw_r2, sw_r2m, sw_skip2;
    int fast_div_h, fast_div_hsq;  // 1: the one-correction sequence is verified for it
    // smoothing kernel (SPHX_KERNEL_*) and the constants its constructor computes in float
    PairLits lit;
    PairConst pair;
    int kern;
    float wnorm;  // Wendland norm_factor_ 21/(2 pi h^3); Gaussian norm_ 1/(pi h^2)^1.5
    float wl;     // Wendland norm_factor_ * (5 / h_sq)
    float gs;     // Gaussian sigma_sq_inv_ = 1 / (h h)
    float gg;     // Gaussian -2 sigma_sq_inv_ norm_
    float gl;     // Gaussian 2 sigma_sq_inv_ norm_
    float g2s;    // Gaussian 2 sigma_sq_inv_
    // 1: the pair forms' divisions by h and h^2 (div_fixed2) are in range: |r| of a hit is +0
    // or in [2^-74.5, r (1 + 2^-23)] (div_nz); the Laplacian's dividends are, too (force_nz = 1),
    // and the gradient's of all pairs without tiny coordinates (2)
    int div_nz, force_nz;
    // the precision force sweep's factors (sphx_sweep.cu); sw_kappa also as a packed operand
    float sw_kg, sw_kappa;
    f32x2 sw_kappa2;
};

// Device-resident scalars written and read by the kernels of a step.
struct DevState {
    int status;                 // 0 or SPHX_ERR_* raised on the device
    int cmin[3], cmax[3];       // box of occupied cells (finite particles)
    int dim[3];                 // grid extent in cells per axis
    int wrap[3];                // 1: the axis is folded (cell index taken modulo dim)
    uint32_t ncells;            // dim product; also the key of non-finite particles
    uint32_t passes;            // radix passes needed this step
    uint32_t n_tiles;           // warp work items
    uint32_t nonfinite;         // particles with a NaN/inf coordinate
    uint32_t occupied;          // occupied cells
    uint32_t max_occ;           // particles in the fullest cell
    uint32_t work[2];           // tile counters of the density and force passes
    float dt;                   // dt of the current step
    float time;                 // current_time_
    float a0[4];                // accelerations_[0] (persists across steps)
    unsigned long long max_nn;  // max |N(i)| since the last stats reset
    double sums[kDiagSums];     // FP64 diagnostics of the state after the last step
    double dt64, time64;        // precision mode: dt and current time in FP64
    uint32_t n_spread;          // precision mode: spread tiles listed this step
    uint32_t spread_work[2];    // precision mode: tile counters of the spread-tile kernels
    uint32_t general;           // exact mode: 1 if a particle lies outside the pair forms' ranges
};

// What blocks of one grid-build kernel tell each other; not part of the step's state (never
// saved or restored, zero once at creation).
struct GridSync {
    uint32_t done;               // blocks of the step's first kernel that have finished
    uint32_t epoch;              // sorts started: tags the look-back words (sphx_sort.cu)
    uint32_t tile[kMaxPasses];   // sort tickets of each pass
    uint32_t general;            // batched mode: see DevState::general
};
// One block's share of the first kernel's reductions.
struct PrepPart {
    int mn[3], mx[3];
    uint32_t bad, general;
    unsigned long long vmax;     // max |v|: float or (precision mode) double bits
};

// Batched mode: one record per scene (device memory).  Scenes are contiguous ranges of
// the insertion order; each owns a dense block of grid cells starting at `base`.
struct SceneInfo {
    StepConst c;                // the scene's parameters and constants (c.n = count)
    uint32_t start, count;      // particle range in insertion order
    // reductions of the step's first kernel, reset when they have been read
    int acc_min[3], acc_max[3];
    uint32_t acc_bad, acc_vmax;
    int cmin[3], cmax[3];       // box of occupied cells
    int dim[3];                 // grid extent of the scene
    uint32_t base, ncells;      // first grid cell, number of cells
    float dt, time;             // the scene's dt of the current step and current_time_
    float a0[4];                // acceleration of the scene's first particle
    double sums[kDiagSums];     // FP64 diagnostics of the scene after the last step
};

// Grid geometry of one tile: the whole grid (single scene) or the tile's scene block.
struct Geom {
    int dim[3];
    int wrap[3];
    uint32_t base;      // first cell of the block
    uint32_t sentinel;  // key of the non-finite group (total number of cells)
};

struct Buffers {
    float4* pos4;     // insertion order: x, y, z, mass
    float4* vel4;     // insertion order: vx, vy, vz, 0
    float4* pos4_s;   // cell-sorted copies
    float4* vel4_s;
    float4* aux4_s;   // cell-sorted: rho, P, (m/rho) mu, 1/(2 rho) or 0 (pair_range);
                      // precision mode: rho, P, m/(2 rho)
    float4* acc4_s;   // cell-sorted accelerations of the last step/eval
    int4* cell4;      // precision mode, insertion order: cell (x, y, z), w = 1 if not finite
    int4* cell4_s;    // precision mode, cell-sorted copy
    uint32_t* key[2]; // radix ping-pong
    uint32_t* val[2];
    uint32_t* key_s;  // sorted cell keys
    uint32_t* id_s;   // sorted position -> insertion index
    uint32_t* rank = nullptr;  // insertion index -> sorted position (a context's steps)
    uint32_t* off;    // dense cell grid: first sorted position of each cell (max_cells + 2)
    uint2* tiles;     // warp work items: first target position and number of targets
    // Target order: the particle of target position k is sorted position tgt[k]; null: k.
    // (k_order_tiles: a permutation within each cell, so position k's cell is key_s[k].)
    uint32_t* tgt = nullptr;
    uint32_t* hist;   // radix digit histograms, one per pass
    unsigned long long* look;  // radix look-back words: one per (tile, digit)
    GridSync* sync;
    PrepPart* prep;   // kMaxPrepBlocks
    double* diag_part;
    uint32_t* scene_of;  // batched mode: scene of each particle (insertion order)
    uint32_t* scene_s;   // batched mode: scene of each particle (cell-sorted)
    SceneInfo* scenes;   // batched mode: per-scene records
    int nscenes;         // 0: single scene
    // What the density pass tells the force pass of the same step about each tile, in records
    // of 32 words: exact mode, per chunk of 32 candidates that the tile's box keeps their
    // sorted positions and the lanes' neighbour masks (word = lane: bit 31 - j set if the j-th
    // of them is a neighbour of the lane's particle), on tiles of up to 8 the neighbours
    // themselves, rows of 16 per particle (4 records: sphx_team.cuh); precision mode, the
    // sorted positions of the kept candidates that are a neighbour of some lane.  Every warp of the density grid
    // owns an equal region of the pool and stores its tiles one after another; tile_list[t] =
    // first record and candidates (or rows), or kNoSlot when the tile did not fit in what was left of
    // the region (the force pass then walks and tests that tile itself).
    uint32_t* records = nullptr;
    uint2* tile_list = nullptr;
    unsigned long long record_cap = 0;
    int diag_blocks;
    int num_sms = 1;
    int tile_n = kTile;  // particles per warp work item (1 .. kTile)
    // 1: the tiles run along cell columns (x, y, *), spanning cells, with each cell's particles
    // taken in z order; 0: insertion order within each cell and tiles within one cell
    int columns = 0;
    // precision mode: the tiles whose particles lie in cells far apart (listed by the density
    // sweep, swept by the spread-tile kernels), one entry per tile at most
    uint32_t* spread_tiles = nullptr;
};
// A column's tiles restart at cell z when z is a multiple of kRunAlign and the kRunWindow
// cells below z hold fewer particles than a tile (tile_starts): no tile then reaches more
// than kRunCells = kRunWindow + kRunAlign - 1 cells past its first one.
constexpr int kRunWindow = 2, kRunAlign = 3;
constexpr int kRunCells = kRunWindow + kRunAlign - 1;
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint64_t kNoPairs = ~0ull;  // pair fill: this particle's list is not wanted

// Device generation of initial conditions (sphx_gen.cu): one shape, its constants derived
// on the host with the generator's float operations.
struct GenShape {
    int kind;                 // SPHX_SHAPE_*
    uint32_t offset, count;   // first staged particle; particles (balls: after counting)
    float start[3], center[3], r2, spacing, mass, vel[3];
    int n[3];                 // lattice extents (balls: points per axis of the cube)
    uint32_t face_off[7];     // box: first particle of each face
    int face_n2[6];
    int face_a[6][3];         // box: (axis1, axis2, axis3) per face
    float face_val[6];
    float jitter;             // benchmark lattice
    uint64_t seed;
    float origin[3];
    int has_origin;
    double c64[3], sp64, R2;  // FP64 ball
    int kmax;
};
struct GenArgs {
    GenShape s;
    float* pos;   // staging: 3 floats per particle
    float* vel;
    float* mass;
};

// Headless rendering (sphx_render.cu): the shader pair's uniforms, derived on the host.
struct RenderConst {
    float pvm[16];          // projection * view * model, column-major
    float right[3], up[3];  // camera right / up: rows 0 and 1 of the view matrix
    float size;             // particleSize
    int mode;               // colorMode: 0 velocity, 1 density, 2 pressure, 3 type
    float diffuse;          // max(dot(normal, lightDir), 0) of the fragment shader
    int width, height;      // viewport = image
    float bg[3];            // clear colour
};
struct RenderArgs {
    int n;
    const float4* pos4;   // insertion order (precision mode: in-cell offsets)
    const float4* vel4;
    const int4* cell4;    // precision mode: cells (else null)
    double cs;            // precision mode: cell size
    const float* colors;  // per-particle colour (3 floats) or null (0, 0.5, 1)
};

// ---- exact float arithmetic: IEEE round-to-nearest, never contracted into FMA ---------
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float xsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float xdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float xsqrt(float a) { return __fsqrt_rn(a); }

// a / b for a fixed divisor b, correctly rounded: q0 = RN(a*y), r = a - q0*b (exact, by
// FMA), q = RN(q0 + r*y) with y = RN(1/b) -- Markstein's FMA correction (as in
// Brisebarre, Muller & Raina, "Accelerating correctly rounded floating-point division
// when the divisor is known in advance", IEEE TC 53(8), 2004).  The host verifies the
// sequence for the divisor against IEEE division over every dividend significand of one
// binade (`verified`); the sequence commutes with power-of-two scaling while every
// intermediate stays normal, which |a| in [2^-60, 2^60] and b in [2^-48, 2^40] ensure.
// Anything else (zero, subnormal, huge, NaN/inf dividend, unverified divisor) takes the
// IEEE division.
__device__ __forceinline__ float xdiv_fixed(float a, float b, float y, int verified) {
    const float aa = fabsf(a);
    if (verified && aa >= 0x1p-60f && aa <= 0x1p60f) {
        const float q0 = __fmul_rn(a, y);
        const float r = __fmaf_rn(-q0, b, a);
        return __fmaf_rn(r, y, q0);
    }
    return __fdiv_rn(a, b);
}

// Packed FP32 pairs (Blackwell f32x2 instructions): two IEEE round-to-nearest operations in
// one instruction, each element rounded exactly as the scalar __f*_rn would.
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 upk2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 xsub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 xmul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 xadd2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ f32x2 xfma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// ---- packed FP32 pairs as a value type ------------------------------------------------
// Two pair terms, or two components, side by side: half the instructions of the scalar form
// (the FP32 pipe still spends a cycle on each half).
//
// The compiler (CUDA 13.0) contracts a packed product and the packed addition that uses it
// into one fma.rn.f32x2 although both are written with .rn (found by comparing sums of
// products in a loop with the scalar form: 68% differed).  Exact code therefore forms a
// product that is added or subtracted by pmul, an FMA with a -0 addend which the compiler
// cannot see through (PairLits::neg0): RN(a b + -0) = RN(a b), zeros' signs included, and
// an FMA's result is not contracted further.  Unpacked halves added by __fadd_rn are safe.
struct F2 {
    f32x2 v;
};
__device__ __forceinline__ F2 f2(float a) { return {pk2(a, a)}; }
__device__ __forceinline__ F2 f2(float a, float b) { return {pk2(a, b)}; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return {xadd2(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return {xsub2(a.v, b.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return {xmul2(a.v, b.v)}; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return {xfma2(a.v, b.v, c.v)}; }
__device__ __forceinline__ F2 pmul(F2 a, F2 b, F2 neg0) { return {xfma2(a.v, b.v, neg0.v)}; }
__device__ __forceinline__ F2 select2(bool ka, bool kb, F2 a, F2 b) {
    const float2 u = upk2(a.v), w = upk2(b.v);
    return f2(ka ? u.x : w.x, kb ? u.y : w.y);
}

__device__ __forceinline__ F2 max0(F2 a) {
    const float2 u = upk2(a.v);
    return f2(fmaxf(u.x, 0.0f), fmaxf(u.y, 0.0f));
}

// xdiv_fixed of both halves without the range test, nb = -b, y = RN(1/b), for dividends known
// to be +-0 or of magnitude in [2^-100, 2^100], with a verified divisor b in [2^-48, 2^40] and
// a normal quotient.  Then q0 is normal, too, and the residual r is exact (a multiple of
// 2^(e_a - 46) >= 2^-146, at most about 2^-22 |a|), so the sequence scales exactly with powers
// of two of a and the verification on one binade covers every binade.  A zero dividend gives
// a zero whose sign is not kept.
__device__ __forceinline__ F2 div_fixed2(F2 a, F2 nb, F2 y) {
    const F2 q0 = a * y;
    return fma2(fma2(q0, nb, a), y, q0);
}

// a / b, correctly rounded, from the correctly rounded reciprocal y = RN(1/b), nb = -b: two
// FMA corrections.  The first brings RN(a y) (at most 1.5 ulp off) within an ulp of a / b;
// the second is then correctly rounded (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990: with y the correctly
// rounded reciprocal and q within an ulp of a / b, RN(q + RN(a - q b) y) = RN(a / b)).  For
// dividends that are 0 or at least 2^-100 in magnitude and quotients in the normal range (a
// zero's sign is not kept).
__device__ __forceinline__ F2 div_rcp2(F2 a, F2 nb, F2 y) {
    const F2 q0 = a * y;
    const F2 q1 = fma2(fma2(q0, nb, a), y, q0);
    return fma2(fma2(q1, nb, a), y, q1);
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Correctly rounded square roots of a pair in [0, 2^86], by Goldschmidt's iteration with a
// final residual correction (Markstein, "Software division and square root using
// Goldschmidt's algorithms", RNC6, 2004): from y0 ~ 1/sqrt(x), g ~ sqrt(x) and h ~ 1/(2
// sqrt(x)) are refined once and g gets the correction (x - g g) h.  x is scaled by 2^40 (the
// result by 2^-20, both exact), which keeps the residuals of all x that occur out of the
// subnormal range; the clamp gives sqrt(0) = 0.  Equal to sqrt.rn for every float in the
// range (all of them compared, test_gpu_kernels).  h: 1/(2 sqrt(2^40 x)), a few ulp.
// ns: the negated roots (the iteration runs on -g and -x: an FMA needs no negated operand).
__device__ __forceinline__ F2 sqrt2_exact(const PairLits& k, F2 x, F2& h, F2& ns) {
    const F2 nx = x * F2{k.neg2p40};
    const float2 u = upk2(nx.v);
    const F2 y0 = f2(rsqrt_approx(fmaxf(-u.x, 0x1p-126f)), rsqrt_approx(fmaxf(-u.y, 0x1p-126f)));
    const F2 ng0 = nx * y0, h0 = y0 * F2{k.half};
    const F2 r = fma2(ng0, h0, F2{k.half});
    const F2 ng = fma2(ng0, r, ng0);
    h = fma2(h0, r, h0);
    const F2 t = fma2(fma2(ng, ng, nx), h, ng);  // -(g + (x - g g) h)
    ns = t * F2{k.p2p20};
    return t * F2{k.neg2p20};
}

// Correctly rounded reciprocals of b = -nb from approximations y1 within a few ulp: two
// Newton steps (the first leaves less than an ulp, after which the second is correctly
// rounded for every significand but all ones, where it ends an ulp below: Markstein 1990).
__device__ __forceinline__ F2 rcp2_exact(const PairLits& k, F2 nb, F2 y1) {
    const F2 one{k.one};
    const F2 y2 = fma2(fma2(nb, y1, one), y1, y1);
    const float2 y = upk2(fma2(fma2(nb, y2, one), y2, y2).v), s = upk2(nb.v);
    auto fix = [](float q, float b) {
        return __uint_as_float(__float_as_uint(q) +
                               (((__float_as_uint(b) & 0x7fffffu) + 1u) >> 23));
    };
    return f2(fix(y.x, s.x), fix(y.y, s.y));
}

// glm::dot(v, v) = (x*x + y*y) + z*z (products rounded first)
__device__ __forceinline__ float xdot3(float x, float y, float z) {
    return xadd(xadd(xmul(x, x), xmul(y, y)), xmul(z, z));
}

// float(2)/float(3) and float(1)/float(6), the constants the reference folds at compile
// time in W_3d (kernels.cpp:58-66)
constexpr float kTwoThirds = 0x1.555556p-1f;
constexpr float kOneSixth = 0x1.555556p-3f;

// CubicSplineKernel::W_3d (kernels.cpp:58-66).  Both branches are evaluated and one is
// selected: the lanes of a warp hold q on both sides of 1, so a branch would run both
// paths anyway, plus the divergence handling.
__device__ __forceinline__ float cubic_w(const StepConst& c, float q) {
    const float w1 =
        xmul(c.sigma, xadd(xsub(kTwoThirds, xmul(q, q)), xmul(xmul(xmul(0.5f, q), q), q)));
    const float tmp = xsub(2.0f, q);
    const float w2 = xmul(c.sigma, xmul(xmul(xmul(kOneSixth, tmp), tmp), tmp));
    return (q >= 0.0f && q <= 1.0f) ? w1 : ((q > 1.0f && q <= 2.0f) ? w2 : 0.0f);
}

// scalar factor of CubicSplineKernel::gradW_3d (kernels.cpp:96-108):
// grad = factor * (r / |r|) / h ; r_len >= 1e-6 is the caller's business.  Branch-free
// like cubic_w.
__device__ __forceinline__ float cubic_grad_factor(const StepConst& c, float q) {
    const float f1 = xmul(c.sigma, xadd(xmul(-2.0f, q), xmul(xmul(1.5f, q), q)));
    const float tmp = xsub(2.0f, q);
    const float f2 = xmul(-c.sigma, xmul(xmul(0.5f, tmp), tmp));
    return (q >= 0.0f && q <= 1.0f) ? f1 : ((q > 1.0f && q <= 2.0f) ? f2 : 0.0f);
}

// CubicSplineKernel::laplacianW_3d (kernels.cpp:130-138).  The branch picks the
// numerator, one division follows: lanes of a warp hold q on both sides of 1, and a
// division per branch would run twice.  Outside both ranges (and for NaN q) the numerator
// is 0 and 0 / h_sq = +0, the reference's 0.0f.
__device__ __forceinline__ float cubic_lap(const StepConst& c, float q) {
    const float a = (q > 1.0f) ? xsub(2.0f, q) : xadd(-2.0f, xmul(3.0f, q));
    const bool in = (q >= 0.0f && q <= 1.0f) || (q > 1.0f && q <= 2.0f);
    const float num = in ? xmul(c.sigma, a) : 0.0f;
    return xdiv_fixed(num, c.h_sq, c.rcp_hsq, c.fast_div_hsq);
}

// WendlandC2Kernel::W after q = length(r)/h (kernels.cpp:172-178):
// norm * tmp^4 * (2q + 1), tmp = 1 - q/2, 0 for q >= 2
__device__ __forceinline__ float wendland_w(const StepConst& c, float q) {
    if (q >= 2.0f) return 0.0f;
    const float tmp = xsub(1.0f, xmul(0.5f, q));
    return xmul(xmul(xmul(xmul(xmul(c.wnorm, tmp), tmp), tmp), tmp), xadd(xmul(2.0f, q), 1.0f));
}

// WendlandC2Kernel::laplacianW after q (kernels.cpp:194-200):
// norm * (5 / h_sq) * tmp * tmp * (5q - 3), 0 for q >= 2
__device__ __forceinline__ float wendland_lap(const StepConst& c, float q) {
    if (q >= 2.0f) return 0.0f;
    const float tmp = xsub(1.0f, xmul(0.5f, q));
    return xmul(xmul(xmul(c.wl, tmp), tmp), xsub(xmul(5.0f, q), 3.0f));
}

__device__ __forceinline__ bool finite3(float x, float y, float z) {
    return isfinite(x) && isfinite(y) && isfinite(z);
}

// Cell coordinate of one axis: floor(x * inv_cell) as SpatialHash::get_grid_coords
// computes it (spatial_hash.h:30-36), clamped to +-2^30 so that every finite position
// has a well-defined cell (clamping keeps neighbouring cells neighbouring).
__device__ __forceinline__ int cell_coord(float x, float inv_cell) {
    float f = floorf(xmul(x, inv_cell));
    f = fminf(fmaxf(f, -(float)kCellClamp), (float)(kCellClamp - 1));
    return (int)f;
}

// Density and pressure in the ranges of the force pass's pair forms (pair_terms): P_i + P_j is
// then 0 or in [2^-74, 2^61] and its quotient by 2 rho_j in [2^-115, 2^120].
__device__ __forceinline__ bool pair_range(float rho, float P) {
    return rho >= 0x1p-60f && rho <= 0x1p40f &&
           (P == 0.0f || (fabsf(P) >= 0x1p-50f && fabsf(P) <= 0x1p60f));
}

// a nonzero coordinate below kTiny in magnitude
__device__ __forceinline__ bool tiny_coord(float x) { return x != 0.0f && fabsf(x) < kTiny; }

// ---- pieces of the step's first kernel (single scene and batched) -----------------------

// true in every thread of the block that finishes last; its reads then see what the other
// blocks wrote before their call
__device__ __forceinline__ bool last_block(GridSync* sync) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(&sync->done, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}
__device__ __forceinline__ void reset_counters(DevState* ds) {
    ds->status = 0;
    ds->occupied = 0;
    ds->max_occ = 0;
    ds->n_tiles = 0;
    ds->work[0] = ds->work[1] = 0;
    ds->spread_work[0] = ds->spread_work[1] = 0;
    ds->n_spread = 0;
}
// resets what the step's kernels count in (one block, all threads)
__device__ __forceinline__ void reset_step(DevState* ds, const Buffers& b) {
    for (int i = threadIdx.x; i < kMaxPasses * kRadixBuckets; i += blockDim.x) b.hist[i] = 0;
    if (threadIdx.x != 0) return;
    reset_counters(ds);
    b.sync->epoch++;
    for (int p = 0; p < kMaxPasses; ++p) b.sync->tile[p] = 0;
}
// dt = min({dt_cfl, dt_force, timestep}) with std::min's first-smallest rule
// (SPHEngine::compute_cfl_timestep, sph_engine.cpp:312-333)
__device__ __forceinline__ float cfl_dt(const StepConst& c, float vmax, const float* a0) {
    const float dt_cfl = xdiv(xmul(c.cfl, c.h), xadd(vmax, 1e-6f));
    const float alen = xsqrt(xdot3(a0[0], a0[1], a0[2]));
    const float dt_force = xmul(c.cfl, xsqrt(xdiv(c.h, xadd(alen, 1e-6f))));
    float dt = dt_cfl;
    if (dt_force < dt) dt = dt_force;
    if (c.timestep < dt) dt = c.timestep;
    return dt;
}
// digit counts of a key for the sort's passes, gathered in shared memory; the lanes of a warp
// that all hold the same digit (the high digits of neighbouring particles) count once
__device__ __forceinline__ void count_digits(uint32_t (*h)[kRadixBuckets], uint32_t key, bool ok,
                                             uint32_t passes) {
    const uint32_t act = __ballot_sync(0xffffffffu, ok);
    if (!act) return;
    const int first = __ffs(act) - 1;
    for (uint32_t p = 0; p < passes; ++p) {
        const uint32_t d = (key >> (p * kRadixBits)) & (kRadixBuckets - 1);
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, first);
        if (__all_sync(0xffffffffu, !ok || d == d0)) {
            if ((threadIdx.x & 31) == (unsigned)first) atomicAdd(&h[p][d0], (uint32_t)__popc(act));
        } else if (ok) {
            atomicAdd(&h[p][d], 1u);
        }
    }
}
__device__ __forceinline__ void add_digits(uint32_t (*h)[kRadixBuckets], uint32_t* hist,
                                           uint32_t passes) {
    for (uint32_t i = threadIdx.x; i < passes * kRadixBuckets; i += blockDim.x)
        if ((&h[0][0])[i]) atomicAdd(&hist[i], (&h[0][0])[i]);
}

// ---- asynchronous copies of single elements, global to shared memory -------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
// closes a group of this thread's copies; waits until at most N groups are outstanding
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// waits for this thread's copies
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---- precision mode helpers ----------------------------------------------------------

// Neumaier's compensated summation (Neumaier 1974): sum + running correction.
struct KSum {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x;
        if (fabsf(s) >= fabsf(x)) c += (s - t) + x;
        else c += (x - t) + s;
        s = t;
    }
    __device__ __forceinline__ float value() const { return s + c; }
};

__device__ __forceinline__ float round_half(float x) { return __half2float(__float2half_rn(x)); }

// ---- host-side constants -------------------------------------------------------------
// The StepConst of one parameter block, for `n` particles, smoothing kernel `kernel`
// (SPHX_KERNEL_*) and mode `mode` (SPHX_MODE_*): every constant computed with the
// reference's float operations, the fixed-divisor checks run (cached per divisor).
void step_const_from_params(const sphx_params& p, size_t n, int kernel, int mode,
                            uint32_t max_cells, StepConst& s);

// ---- launch wrappers (host) --------------------------------------------------------
struct LaunchCtx {
    cudaStream_t stream;
    int device;  // CUDA device the launches go to (keys per-device launch-shape caches)
    int num_sms;
    int warps_per_block;
    int blocks_per_sm;
};

// A flag per device, filled by whichever thread comes first.
constexpr int kMaxCacheDevices = 64;
struct LaunchShapeFlag {
    std::atomic<int> v[kMaxCacheDevices];
    std::atomic<int>& at(int device) {
        return v[device >= 0 && device < kMaxCacheDevices ? device : 0];
    }
};

// How a step gets its dt.
constexpr int kNoStep = 0, kHostDt = 1, kCflDt = 2;
// The grid build (single scene): resets the step's counters, finds the box of occupied cells,
// lays out the grid, sorts the particles and lists the tiles; how != kNoStep: sets dt and
// advances the time.
int launch_grid(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds, int how,
                float host_dt);
// the same in one launch, for sets of 1 to kSmallMax particles; false: the device cannot
bool launch_grid_small(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                       int how, float host_dt);
int launch_grid_sort(const LaunchCtx& L, const Buffers& b, DevState* ds, int n, const StepConst& c);
int launch_density(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds);
int launch_force(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                  int integrate);
// Particles per tile where the caller leaves the choice: the exact passes take tiles of 8, four
// lanes a particle, on sets too small to fill the GPU with a lane per particle.  Density +
// force with tiles of 8 and of 32, lattice, us: 4k 45 and 122, 10k 57 and 133, 33k 138 and
// 179, 47k 178 and 199, 64k 234 and 243; the density pass alone, which has no list to gain
// by: 22k 55 and 77, 33k 73 and 79, 47k 94 and 91, 64k 122 and 105.
inline int pass_tile(int n, bool precise, bool density_only = false) {
    return !precise && n <= (density_only ? kTeamMaxDensity : kTeamMax) ? kTeamTile : kTile;
}
// the same passes with four lanes per particle (sphx_team_density.cu, sphx_team_force.cu)
int launch_density_team(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds);
int launch_force_team(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                      int integrate);
int launch_diag(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds);
// precision mode (single scene): the tile-sweep passes (sphx_sweep.cu)
int launch_density_sweep(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                         DevState* ds);
int launch_force_sweep(const LaunchCtx& L, const StepConst& c, const Buffers& b, DevState* ds,
                       int integrate);
void launch_pair_counts(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                        DevState* ds, uint32_t* counts_by_id);
void launch_pair_fill(const LaunchCtx& L, const StepConst& c, const Buffers& b,
                      DevState* ds, const uint64_t* offsets_by_id, int64_t* out_idx);

// batched mode (sphx_batch.cu)
int launch_batch_prepare(const LaunchCtx& L, const Buffers& b, DevState* ds, int n, int how,
                         float host_dt, uint32_t max_cells);
int launch_batch_grid(const LaunchCtx& L, const Buffers& b, DevState* ds, int n);
int launch_batch_diag(const LaunchCtx& L, const Buffers& b, DevState* ds);

// The grid build's working memory besides the per-particle arrays, one block: GridSync (first),
// PrepPart, digit histograms and the sort's look-back words; zero once at creation (sphx_sort.cu).
size_t grid_scratch_bytes(size_t capacity);
void set_grid_scratch(Buffers& b, unsigned char* base);
// radix sort (sphx_sort.cu)
int launch_radix_sort(const LaunchCtx& L, const Buffers& b, DevState* ds, int n);

// io (sphx_grid.cu)
void launch_pack(const LaunchCtx& L, int n, const float* pos3, const float* vel3,
                 const float* mass, float4* pos4, float4* vel4);
void launch_unpack_state(const LaunchCtx& L, int n, const float4* pos4, const float4* vel4,
                         float* pos3, float* vel3);
void launch_unpack_direct(const LaunchCtx& L, int n, const Buffers& b, const DevState* ds,
                          double cs, float* pos3, float* vel3, float* rho, float* pressure, float* acc3,
                          int* status);
void launch_unpack_sorted(const LaunchCtx& L, int n, const uint32_t* id_s,
                          const float4* aux4_s, const float4* acc4_s, float* rho,
                          float* pressure, float* acc3);
// precision mode: absolute positions (float or double) <-> cell + offset
int launch_ball_count(const LaunchCtx& L, const GenArgs& g, uint32_t* rows);
int launch_generate(const LaunchCtx& L, const GenArgs& g, const uint32_t* rows);
int launch_render_instances(const LaunchCtx& L, const RenderConst& r, const RenderArgs& a,
                            float* out);
int launch_render_image(const LaunchCtx& L, const RenderConst& r, const RenderArgs& a,
                        unsigned long long* keys, uchar4* rgba);
void launch_pack_cells(const LaunchCtx& L, const StepConst& c, int n, const float* pos3f,
                       const double* pos3d, const float* vel3, const float* mass, int4* cell4,
                       float4* pos4, float4* vel4);
void launch_unpack_cells(const LaunchCtx& L, const StepConst& c, int n, const int4* cell4,
                         const float4* pos4, float* pos3f, double* pos3d);

}  // namespace sphx
