// Stable LSD radix sort of 32-bit cell keys (8-bit digits).
//
// One launch per pass: a block takes the next tile of keys (a ticket), ranks them, publishes
// its digit counts and learns from the blocks before it where its keys go (decoupled
// look-back, Merrill & Garland, "Single-pass parallel prefix scan with decoupled look-back",
// NVR-2016-002, 2016; Adinets & Merrill, "Onesweep", arXiv:2206.01784, 2022).  The digit
// histograms of all passes come from the kernel that makes the keys.  Against a histogram, a
// three-launch scan and a scatter per pass: 3 active passes of 1M keys 0.10 -> 0.04 ms, and 5
// launches instead of 20 where the launches count.
//
// The number of passes is decided on the device (DevState::passes, from the number of
// significant key bits of this step's cell grid), so a whole step can be enqueued -- or
// captured -- without a host round trip: kMaxPasses pass launches are issued and the
// inactive ones return at once.  Pass p reads buffer (p & 1) and writes (p + 1) & 1; the
// result is in buffer (passes & 1).
//
// Stability: within a tile, warp w owns a contiguous sub-range and walks it in rounds of 32
// consecutive keys; ranks inside a round come from __match_any_sync, ranks across rounds from
// a per-warp running count per digit, and ranks across warps from an exclusive scan of those
// counts.  Equal digits therefore keep their input order, which is what makes the cell-sorted
// order (cell, insertion index): the keys are produced in insertion order.
#include "sphx_internal.cuh"

namespace sphx {

// Published state of a (tile, digit): epoch << 34 | flag << 32 | count.  The epoch (one per
// step and pass, GridSync::epoch) marks words of earlier sorts as absent, so the array is
// never cleared.
constexpr uint32_t kLookCount = 1, kLookPrefix = 2;
__device__ __forceinline__ unsigned long long look_word(uint32_t epoch, uint32_t flag,
                                                        uint32_t count) {
    return (unsigned long long)((epoch << 2) | flag) << 32 | count;
}
// Polls of a predecessor's word before giving up (seconds): the predecessors took their
// tickets earlier, so they are running and will publish.
constexpr uint32_t kLookPolls = 1u << 22;

// kItems keys per thread.  kFirst: pass 0, whose values are the keys' indices.
template <int kItems, bool kFirst>
__global__ void __launch_bounds__(kRadixThreads) k_radix_pass(const Buffers b, int n, int pass,
                                                              DevState* ds) {
    if (ds->status || (uint32_t)pass >= ds->passes) return;
    constexpr int kWarps = kRadixThreads / 32;
    __shared__ uint32_t cnt[kWarps][kRadixBuckets];
    __shared__ uint32_t warp_sums[kWarps];
    __shared__ uint32_t s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t* __restrict__ keys_in = b.key[pass & 1];
    const uint32_t* __restrict__ vals_in = b.val[pass & 1];
    uint32_t* __restrict__ keys_out = b.key[(pass & 1) ^ 1];
    uint32_t* __restrict__ vals_out = b.val[(pass & 1) ^ 1];
    if (tid == 0) s_tile = atomicAdd(&b.sync->tile[pass], 1u);
    for (int i = tid; i < kWarps * kRadixBuckets; i += kRadixThreads) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t epoch = b.sync->epoch * kMaxPasses + (uint32_t)pass;
    const int shift = pass * kRadixBits;
    const long long wbase =
        (long long)tile * (kRadixThreads * kItems) + (long long)warp * (kItems * 32);
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const long long i = wbase + r * 32 + lane;
        key[r] = i < n ? keys_in[i] : 0u;
        val[r] = i < n ? (kFirst ? (uint32_t)i : vals_in[i]) : 0u;
    }
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const bool ok = wbase + r * 32 + lane < n;
        // lanes past the end get a digit value that no real key has
        const uint32_t d = ok ? ((key[r] >> shift) & (kRadixBuckets - 1)) : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t before = ok ? cnt[warp][d] : 0u;
        __syncwarp();
        if (ok && (peers & lt_mask) == 0) cnt[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[r] = before + __popc(peers & lt_mask);
    }
    __syncthreads();
    {
        const int d = tid;  // kRadixThreads == kRadixBuckets: a digit per thread
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) total += cnt[w][d];
        volatile unsigned long long* look = b.look;
        const size_t at = (size_t)tile * kRadixBuckets + d;
        look[at] = look_word(epoch, tile ? kLookCount : kLookPrefix, total);
        // first position of the digit: exclusive scan of the pass's histogram
        const uint32_t h = b.hist[pass * kRadixBuckets + d];
        uint32_t x = h;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        uint32_t run = x - h;
        for (int w = 0; w < warp; ++w) run += warp_sums[w];
        // keys of this digit in the tiles before
        uint32_t before = 0;
        for (uint32_t t = tile; t > 0;) {
            const volatile unsigned long long* p = look + (size_t)(t - 1) * kRadixBuckets + d;
            unsigned long long word = *p;
            for (uint32_t k = 0; (uint32_t)(word >> 34) != (epoch & 0x3fffffffu); ++k) {
                if (k == kLookPolls) {
                    atomicCAS(&ds->status, 0, SPHX_ERR_TIMEOUT);
                    break;
                }
                word = *p;
            }
            before += (uint32_t)word;
            if ((uint32_t)(word >> 32 & 3u) != kLookCount) break;  // a prefix (or a timeout)
            --t;
        }
        if (tile) look[at] = look_word(epoch, kLookPrefix, before + total);
        run += before;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = cnt[w][d];
            cnt[w][d] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        if (wbase + r * 32 + lane < n) {
            const uint32_t d = (key[r] >> shift) & (kRadixBuckets - 1);
            const uint32_t dst = cnt[warp][d] + rank[r];
            if (dst < (uint32_t)n) {  // always true for a consistent histogram
                keys_out[dst] = key[r];
                vals_out[dst] = val[r];
            }
        }
    }
}

// look-back words for sorts of up to `capacity` keys
static size_t look_words(size_t capacity) {
    const size_t big = (capacity + kRadixTileN - 1) / kRadixTileN;
    const size_t small_n = capacity < (size_t)kSmallSort ? capacity : (size_t)kSmallSort;
    const size_t small = (small_n + kRadixThreads * 4 - 1) / (kRadixThreads * 4);
    return (big > small ? big : small) * kRadixBuckets;
}

static size_t align256(size_t x) { return (x + 255) / 256 * 256; }

size_t grid_scratch_bytes(size_t capacity) {
    return align256(sizeof(GridSync)) + align256(kMaxPrepBlocks * sizeof(PrepPart)) +
           align256((size_t)kMaxPasses * kRadixBuckets * sizeof(uint32_t)) +
           align256(look_words(capacity) * sizeof(unsigned long long));
}

void set_grid_scratch(Buffers& b, unsigned char* base) {
    b.sync = reinterpret_cast<GridSync*>(base);
    base += align256(sizeof(GridSync));
    b.prep = reinterpret_cast<PrepPart*>(base);
    base += align256(kMaxPrepBlocks * sizeof(PrepPart));
    b.hist = reinterpret_cast<uint32_t*>(base);
    base += align256((size_t)kMaxPasses * kRadixBuckets * sizeof(uint32_t));
    b.look = reinterpret_cast<unsigned long long*>(base);
}

// Keys per block: 4096 once they fill the GPU, else 1024, so that a small sort spreads over
// more SMs (a tile's time is its serial ranking rounds: 4 against 16).
template <int kItems>
static void radix_passes(const LaunchCtx& L, const Buffers& b, DevState* ds, int n) {
    const int nb = (int)(((long long)n + kRadixThreads * kItems - 1) / (kRadixThreads * kItems));
    k_radix_pass<kItems, true><<<nb, kRadixThreads, 0, L.stream>>>(b, n, 0, ds);
    for (int pass = 1; pass < kMaxPasses; ++pass)
        k_radix_pass<kItems, false><<<nb, kRadixThreads, 0, L.stream>>>(b, n, pass, ds);
}

int launch_radix_sort(const LaunchCtx& L, const Buffers& b, DevState* ds, int n) {
    if (n <= kSmallSort) radix_passes<4>(L, b, ds, n);
    else radix_passes<kRadixItems>(L, b, ds, n);
    return kMaxPasses;
}

}  // namespace sphx
