// k_sort.cu - stable LSD radix sort of (u64 Morton key, u32 position) pairs,
// one "onesweep" launch per 8-bit digit.
//
// Replaces cub::DeviceRadixSort::SortPairs (cuda_engine.cu:272,397).  The
// method is the single-pass LSD sort of Adinets & Merrill (2022): per pass,
// every tile of keys ranks its keys locally, publishes its per-digit counts,
// and learns the counts of all earlier tiles by decoupled look-back, so each
// key moves exactly once per pass.  This implementation:
//
//  * global digit histograms of all passes come from the encode kernel
//    (k_stream.cu), so no counting pass over the keys is needed;
//  * tiles are taken in launch order from an atomic ticket, so a tile only
//    ever waits on tiles that are already resident (forward progress);
//  * ranking is warp-local with 8 ballots per key (lanes with equal digits
//    are found by intersecting per-bit ballots) and a per-warp shared-memory
//    histogram that only its own warp touches; keys of warp w precede those
//    of warp w+1 and items are ranked in input order, so equal digits keep
//    their input order (the sort is stable, which makes position the
//    tie-break, karras_bvh.cuh:40);
//  * a tile's keys and values are loaded right after its ticket, and the
//    global digit starts are scanned while those loads are in flight;
//  * a tile publishes its counts as soon as it has ranked, moves its pairs to
//    shared memory in digit order, and only then looks back, so the earlier
//    tiles' counts travel while it works and the look-back has the registers
//    that held the pairs;
//  * the look-back has two levels: a tile reads the counts of the earlier
//    tiles of its own group of kLookGroup directly (all loads in flight
//    together), the group's last tile publishes the group's sum, and the
//    groups before it are read a window at a time until an inclusive prefix.
//    All tiles of up to about 1.2 M keys are resident at once and publish
//    together, so a one-level look-back was a serial chain of tiles / 8
//    windows;
//  * look-back waits are bounded: a wait that runs out sets
//    GCS_DEV_SORT_LOOKBACK_TIMEOUT, the tile still publishes (so later tiles
//    finish) and skips its scatter, so nothing is written out of bounds;
//  * keys are scattered through shared memory so global writes come out as
//    runs of equal digits.
//
// A pass is bound by the latency of one tile (launch, ticket, loads, ranking,
// look-back, write-out), not by bytes.  An eighth of the sort stage (CUDA events
// around it alone, plain launches, two memsets included): 14.2 us at 1,048,576
// pairs (25 MB, 1.8 TB/s), 7.2 at 45,056; 19.3 and 11.3 with the one-level
// look-back and launches that do not overlap (pdl.cuh).
//
// With more than one segment, one or two further stable passes order by the
// segment id of each element's source position; the result is every segment
// sorted by key with position as the tie-break, as if sorted alone.
#include <algorithm>
#include <type_traits>

#include "gcs_internal.h"
#include "pdl.cuh"

namespace gcs {

namespace {

constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagInclusive = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr int kLookWindow = 8;   // groups read together

template <int kThreads, int kItems, bool kSegPass>
struct SortSmem {
    static constexpr int kTile = kThreads * kItems;
    static constexpr int kWarps = kThreads / 32;
    uint64_t keys[kTile];
    uint32_t vals[kTile];
    uint8_t dig[kSegPass ? kTile : 1];  // a segment digit is not in the key
    uint32_t whist[kWarps][kRadix];
    uint32_t gbase[kRadix];
    uint32_t tstart[kRadix];
    int32_t final_base[kRadix];
    uint32_t warp_sums[kRadix / 32];
    uint32_t tile;
    int bad;
};

// Exclusive scan over the first kRadix threads of the block (one value each;
// every thread of the block calls it).
__device__ __forceinline__ uint32_t digit_exclusive_scan(uint32_t v, uint32_t* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31 && warp < kRadix / 32) warp_sums[warp] = x;
    __syncthreads();
    uint32_t off = 0;
#pragma unroll
    for (int w = 0; w < kRadix / 32; ++w) off += w < warp ? warp_sums[w] : 0u;
    __syncthreads();
    return off + x - v;
}

// One look-back step: reads `count` (<= K) published words nearest first
// (word k at base - k * kRadix) and waits, boundedly, until each is there.
// Returns false when the wait ran out.
template <int K>
__device__ __forceinline__ bool read_published(const volatile uint32_t* base, int count, uint32_t (&v)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = k < count ? base[-(int64_t)k * kRadix] : kFlagAggregate;
    for (uint32_t spins = 0;; ++spins) {
        bool empty = false;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if ((v[k] & ~kCountMask) == 0u) {
                v[k] = base[-(int64_t)k * kRadix];
                empty |= (v[k] & ~kCountMask) == 0u;
            }
        if (!empty) return true;
        if (spins > kSpinLimit) return false;
        __nanosleep(20);
    }
}

template <int kThreads, int kItems, bool kSegPass>
__global__ void __launch_bounds__(kThreads, kThreads == kSortThreads ? 2 : 4)
onesweep_kernel(Layout L, int shift, const uint64_t* __restrict__ keys_in,
                const uint32_t* __restrict__ vals_in, uint64_t* __restrict__ keys_out,
                uint32_t* __restrict__ vals_out, const uint32_t* __restrict__ hist,
                uint32_t* __restrict__ tile_counter, uint32_t* __restrict__ lookback,
                uint32_t* __restrict__ status, int n_tiles) {
    using Smem = SortSmem<kThreads, kItems, kSegPass>;
    constexpr int kTile = Smem::kTile;
    constexpr int kWarps = Smem::kWarps;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n = L.n;

    let_next_start();
    for (int i = t; i < kWarps * kRadix; i += kThreads) (&S.whist[0][0])[i] = 0;
    wait_for_previous();
    if (t == 0) {
        S.tile = atomicAdd(tile_counter, 1u);
        S.bad = 0;
    }
    const uint32_t h = t < kRadix ? hist[t] : 0u;  // t == digit
    __syncthreads();
    const int tile = (int)S.tile;
    const int tile_base = tile * kTile;
    const int warp_base = tile_base + warp * (kItems * 32);

    // ---- load (warp-striped: item j of lane l is warp_base + 32j + l); the
    // values come with the keys and the global digit starts are scanned while
    // the loads are in flight, so no later phase waits on global memory
    // except the look-back
    uint64_t key[kItems];
    uint32_t val[kItems];
    uint32_t rank[kItems];  // digit << 16 | rank within the warp's items
    const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = warp_base + 32 * j + lane;
        const bool valid = i < n;
        key[j] = valid ? keys_in[i] : 0ull;
        val[j] = valid ? vals_in[i] : 0u;
    }
    const uint32_t gbase = digit_exclusive_scan(h, S.warp_sums);
    if (t < kRadix) S.gbase[t] = gbase;

    // ---- rank
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const bool valid = warp_base + 32 * j + lane < n;
        uint32_t d;
        if (kSegPass) {
            d = valid ? (((uint32_t)__ldg(L.seg_id + val[j]) >> shift) & (kRadix - 1)) : 0u;
        } else {
            d = (uint32_t)(key[j] >> shift) & (kRadix - 1);
        }
        uint32_t peers = __ballot_sync(0xFFFFFFFFu, valid);
#pragma unroll
        for (int b = 0; b < kRadixBits; ++b) {
            const bool bit = (d >> b) & 1u;
            const uint32_t bb = __ballot_sync(0xFFFFFFFFu, bit);
            peers &= bit ? bb : ~bb;
        }
        // the warp's own histogram: every lane reads its digit's count so
        // far, then the last of the digit's lanes (the one with all the
        // others below it) adds the lanes of this item
        const uint32_t before = (uint32_t)__popc(peers & lt_mask);
        const uint32_t prev = S.whist[warp][d];
        __syncwarp();
        if (valid && (peers >> lane) == 1u) S.whist[warp][d] = prev + before + 1u;
        __syncwarp();
        rank[j] = (d << 16) | (prev + before);
    }
    __syncthreads();

    // ---- per-digit tile totals and warp prefixes (thread t owns digit t)
    uint32_t total = 0;
    volatile uint32_t* lb = lookback + (size_t)tile * kRadix + t;
    if (t < kRadix) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = S.whist[w][t];
            S.whist[w][t] = total;
            total += c;
        }
        *lb = kFlagAggregate | total;  // early, so later tiles can proceed
    }
    const uint32_t tstart = digit_exclusive_scan(total, S.warp_sums);
    if (t < kRadix) S.tstart[t] = tstart;
    __syncthreads();

    // ---- scatter into shared memory in digit order (needs only the tile's
    // own counts)
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (warp_base + 32 * j + lane < n) {
            const uint32_t d = rank[j] >> 16;
            const uint32_t lp = S.tstart[d] + S.whist[warp][d] + (rank[j] & 0xFFFFu);
            S.keys[lp] = key[j];
            S.vals[lp] = val[j];
            if (kSegPass) S.dig[lp] = (uint8_t)d;
        }
    }

    // ---- two-level decoupled look-back for digit t
    if (t < kRadix) {
        const int group = tile / kLookGroup, in_group = tile % kLookGroup;
        volatile uint32_t* lg = lookback + (size_t)n_tiles * kRadix + (size_t)group * kRadix + t;
        bool ok = true;
        uint32_t excl = 0;
        if (in_group > 0) {
            uint32_t v[kLookGroup - 1];
            ok = read_published<kLookGroup - 1>(lb - kRadix, in_group, v);
#pragma unroll
            for (int k = 0; k < kLookGroup - 1; ++k) excl += v[k] & kCountMask;
        }
        const bool last = in_group == kLookGroup - 1;
        if (last) *lg = (group == 0 ? kFlagInclusive : kFlagAggregate) | ((excl + total) & kCountMask);
        for (int g = group - 1; g >= 0 && ok;) {
            uint32_t v[kLookWindow];
            ok = read_published<kLookWindow>(lg - (int64_t)(group - g) * kRadix, min(kLookWindow, g + 1), v);
            bool done = false;
#pragma unroll
            for (int k = 0; k < kLookWindow; ++k)
                if (!done) {
                    excl += v[k] & kCountMask;
                    done = (v[k] & ~kCountMask) == kFlagInclusive;
                }
            if (done) break;
            g -= kLookWindow;
        }
        if (last && group > 0) *lg = kFlagInclusive | ((excl + total) & kCountMask);
        if (!ok) {
            S.bad = 1;
            atomicOr(status, GCS_DEV_SORT_LOOKBACK_TIMEOUT);
        }
        S.final_base[t] = (int)(S.gbase[t] + excl) - (int)tstart;
    }
    __syncthreads();

    // ---- write out: runs of equal digits land contiguously
    if (!S.bad) {
        const int valid = min(n - tile_base, kTile);
        for (int q = t; q < valid; q += kThreads) {
            const uint64_t k = S.keys[q];
            const uint32_t d = kSegPass ? S.dig[q] : (uint32_t)(k >> shift) & (kRadix - 1);
            const int g = S.final_base[d] + q;
            if (g >= 0 && g < n) {
                keys_out[g] = k;
                vals_out[g] = S.vals[q];
            }
        }
    }
}

template <int kThreads, int... kItems>
void configure_tiles() {
    (cudaFuncSetAttribute(onesweep_kernel<kThreads, kItems, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)sizeof(SortSmem<kThreads, kItems, false>)), ...);
    (cudaFuncSetAttribute(onesweep_kernel<kThreads, kItems, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)sizeof(SortSmem<kThreads, kItems, true>)), ...);
}

template <int kThreads, int kItems>
void launch_tiles(const Layout& L, int pass, int tiles, const uint64_t* keys_in, const uint32_t* vals_in,
                  uint64_t* keys_out, uint32_t* vals_out, const uint32_t* hist, uint32_t* tile_counter,
                  uint32_t* lookback, uint32_t* status, cudaStream_t st) {
    constexpr size_t smem_key = sizeof(SortSmem<kThreads, kItems, false>);
    constexpr size_t smem_seg = sizeof(SortSmem<kThreads, kItems, true>);
    if (pass < kKeyPasses) {
        launch_after(onesweep_kernel<kThreads, kItems, false>, (unsigned)tiles, kThreads, smem_key, st, L,
                     kRadixBits * pass, keys_in, vals_in, keys_out, vals_out, hist, tile_counter, lookback, status,
                     tiles);
    } else {
        launch_after(onesweep_kernel<kThreads, kItems, true>, (unsigned)tiles, kThreads, smem_seg, st, L,
                     kRadixBits * (pass - kKeyPasses), keys_in, vals_in, keys_out, vals_out, hist, tile_counter,
                     lookback, status, tiles);
    }
}

size_t pass_words(int64_t n) {
    const int tile = sort_tile(n);
    const int64_t tiles = n > 0 ? (n + tile - 1) / tile : 1;
    return (size_t)(tiles + tiles / kLookGroup) * kRadix;  // (only whole groups publish a sum)
}

}  // namespace

size_t sort_lookback_words(int64_t n, int passes) { return pass_words(n) * passes; }

size_t sort_lookback_words_upto(int64_t n, int passes) {
    // one wave of tiles at most while the tile grows with n, then n / kSortTile
    const size_t wave = (size_t)(kSortWave + kSortWave / kLookGroup) * kRadix;
    return std::max(pass_words(n), n > kSortSmallMax ? wave : pass_words(std::min(n, kSortSmallMax))) * passes;
}

void launch_sort_pass(const Layout& L, int pass, const uint64_t* keys_in, const uint32_t* vals_in,
                      uint64_t* keys_out, uint32_t* vals_out, const uint32_t* hist,
                      uint32_t* tile_counter, uint32_t* lookback, uint32_t* status,
                      cudaStream_t st) {
    if (L.n <= 0) return;
    // every tile size at the first call on a device, which may be a captured one
    // (the attribute is set at once, not on the stream): no call after it sets
    // anything
    static std::once_flag configured[kMaxDevices];
    once_per_device(configured, [] {
        configure_tiles<256, kSortSmallTile / 256>();
        configure_tiles<kSortThreads, 2, 3, 4, 5, 6, 7, kSortMaxItems>();
    });
    const int tile = sort_tile(L.n);
    const int tiles = (L.n + tile - 1) / tile;
    uint32_t* lb = lookback + (size_t)pass * pass_words(L.n);
    hist += pass * kRadix;
    tile_counter += pass;
    const auto go = [&](auto threads, auto items) {
        launch_tiles<decltype(threads)::value, decltype(items)::value>(
            L, pass, tiles, keys_in, vals_in, keys_out, vals_out, hist, tile_counter, lb, status, st);
    };
    using std::integral_constant;
    const integral_constant<int, kSortThreads> wide{};
    if (L.n <= kSortSmallMax) go(integral_constant<int, 256>{}, integral_constant<int, kSortSmallTile / 256>{});
    else switch (tile / kSortThreads) {
        case 2: go(wide, integral_constant<int, 2>{}); break;
        case 3: go(wide, integral_constant<int, 3>{}); break;
        case 4: go(wide, integral_constant<int, 4>{}); break;
        case 5: go(wide, integral_constant<int, 5>{}); break;
        case 6: go(wide, integral_constant<int, 6>{}); break;
        case 7: go(wide, integral_constant<int, 7>{}); break;
        default: go(wide, integral_constant<int, kSortMaxItems>{}); break;
    }
}

}  // namespace gcs
