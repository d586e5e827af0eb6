// k_front.cu - bounds, Morton encode and radix sort of a small scenario in
// one launch: one thread-block cluster holds all keys in shared memory.
//
// The three stages of up to kFrontMax particles of one segment are eleven
// launches on their own, each as long as its latency chain: together 56, 62, 63
// and 64 us at 1,408, 8,192, 32,768 and 49,152 particles (CUDA events, plain
// launches), 29, 37, 54 and 66 in one (1,024 threads a block took 3 to 7 us
// more).  Here a cluster of 8 or 16 blocks keeps every (key, position) pair in
// its shared memory for all eight passes of the same stable LSD sort
// (k_sort.cu): a block ranks its own pairs with warp ballots and puts them in
// digit order, the blocks exchange digit counts through distributed shared
// memory, and each run of a digit moves to its place in the block that owns it
// in the next pass.  Two cluster barriers a pass; nothing but the particles, the
// sorted keys and the positions touches global memory.
//
// Keys, order and bounds are bit for bit those of the separate stages.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "gcs_internal.h"
#include "device_math.cuh"
#include "pdl.cuh"

namespace gcs {

namespace {

namespace cg = cooperative_groups;

constexpr int kFrontThreads = 512;
constexpr int kFrontWarps = kFrontThreads / 32;
constexpr uint32_t kAll = 0xFFFFFFFFu;

template <int kItems>
struct FrontSmem {
    static constexpr int kTile = kFrontThreads * kItems;  // pairs a block owns
    uint64_t keys[2][kTile];
    uint16_t idx[2][kTile];
    uint32_t whist[kFrontWarps][kRadix];
    uint32_t count[kRadix];         // this block's keys of each digit (read by the others)
    uint32_t sums[2][2][kRadix];    // by half of the blocks: all keys of a digit, those of earlier blocks
    uint32_t start[kRadix];         // where a digit starts in this block's own order
    int32_t shift[kRadix];          // from there to its place among all blocks
    uint32_t warp_sums[kRadix / 32];
    float lo[kFrontWarps], hi[kFrontWarps];
    float2 range;                   // this block's min and max (read by the others)
};

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, x, o);
        if (lane >= o) x += y;
    }
    return x;
}
__device__ __forceinline__ uint32_t warps_before(const uint32_t* sums, int warp) {
    uint32_t off = 0;
#pragma unroll
    for (int w = 0; w < kRadix / 32; ++w) off += w < warp ? sums[w] : 0u;
    return off;
}

template <int kItems>
__global__ void __launch_bounds__(kFrontThreads, 1)
front_kernel(const float4* __restrict__ pos, int n, int front_bounds, float gmin, float gmax,
             float2* __restrict__ seg_bounds, uint64_t* __restrict__ keys_out, uint32_t* __restrict__ idx_out,
             uint32_t* __restrict__ status) {
    using Smem = FrontSmem<kItems>;
    constexpr int kTile = Smem::kTile;
    extern __shared__ __align__(16) unsigned char front_smem[];
    Smem& S = *reinterpret_cast<Smem*>(front_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int tile_base = rank * kTile;
    const int warp_at = warp * (kItems * 32);  // the warp's first pair in the tile
    const uint32_t lt_mask = (1u << lane) - 1u;

    let_next_start();
    wait_for_previous();

    // ---- particles, bounds, keys
    float4 p[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = tile_base + warp_at + 32 * j + lane;
        p[j] = i < n ? __ldg(pos + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float lo = gmin, hi = gmax;
    if (front_bounds == kFrontBoundsReduce) {
        float l = INFINITY, h = -INFINITY;
        bool bad = false;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            if (tile_base + warp_at + 32 * j + lane < n) {
                bad |= !(isfinite(p[j].x) && isfinite(p[j].y) && isfinite(p[j].z));
                l = fminf(l, fminf(p[j].x, fminf(p[j].y, p[j].z)));
                h = fmaxf(h, fmaxf(p[j].x, fmaxf(p[j].y, p[j].z)));
            }
        }
        if (__any_sync(kAll, bad) && lane == 0) atomicOr(status, GCS_DEV_NONFINITE_POSITION);
        for (int o = 16; o > 0; o >>= 1) {
            l = fminf(l, __shfl_xor_sync(kAll, l, o));
            h = fmaxf(h, __shfl_xor_sync(kAll, h, o));
        }
        if (lane == 0) {
            S.lo[warp] = l;
            S.hi[warp] = h;
        }
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < kFrontWarps; ++w) {
                l = fminf(l, S.lo[w]);
                h = fmaxf(h, S.hi[w]);
            }
            S.range = make_float2(l, h);
        }
        cluster.sync();
        // every thread combines the blocks' ranges (as bounds_kernel's ordered
        // maxima do: min of mins, max of maxes)
        uint32_t el = 0u, eh = 0u;
        for (int r = 0; r < blocks; ++r) {
            const float2 b = *cluster.map_shared_rank(&S.range, r);
            el = max(el, ~float_to_ordered(b.x));
            eh = max(eh, float_to_ordered(b.y));
        }
        lo = ordered_to_float(~el);
        hi = ordered_to_float(eh);
        if (rank == 0 && t == 0) seg_bounds[0] = make_float2(lo, hi);
    } else if (front_bounds == kFrontBoundsGiven) {
        const float2 b = __ldg(seg_bounds);
        lo = b.x;
        hi = b.y;
    }
    const float scale = morton_scale(lo, hi);
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int at = warp_at + 32 * j + lane;
        S.keys[0][at] = morton63(p[j].x, p[j].y, p[j].z, lo, scale);
        S.idx[0][at] = (uint16_t)(tile_base + at);
    }
    __syncwarp();  // a warp reads what it wrote in the first pass

    // ---- eight stable passes
    for (int pass = 0; pass < kKeyPasses; ++pass) {
        const int cur = pass & 1, shift = kRadixBits * pass;
        uint64_t key[kItems];
        uint32_t idx[kItems], rk[kItems];
        uint4* h4 = reinterpret_cast<uint4*>(S.whist[warp]);
        h4[lane] = h4[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const int at = warp_at + 32 * j + lane;
            key[j] = S.keys[cur][at];
            idx[j] = S.idx[cur][at];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const bool valid = tile_base + warp_at + 32 * j + lane < n;
            const uint32_t d = (uint32_t)(key[j] >> shift) & (kRadix - 1);
            uint32_t peers = __ballot_sync(kAll, valid);
#pragma unroll
            for (int b = 0; b < kRadixBits; ++b) {
                const bool bit = (d >> b) & 1u;
                const uint32_t bb = __ballot_sync(kAll, bit);
                peers &= bit ? bb : ~bb;
            }
            const uint32_t before = (uint32_t)__popc(peers & lt_mask);
            const uint32_t prev = S.whist[warp][d];
            __syncwarp();
            if (valid && (peers >> lane) == 1u) S.whist[warp][d] = prev + before + 1u;
            __syncwarp();
            rk[j] = prev + before;
        }
        __syncthreads();
        // this block's counts, and where its digits start in its own order
        uint32_t mine = 0, scan = 0;
        if (t < kRadix) {
#pragma unroll
            for (int w = 0; w < kFrontWarps; ++w) {
                const uint32_t c = S.whist[w][t];
                S.whist[w][t] = mine;
                mine += c;
            }
            S.count[t] = mine;
            scan = warp_inclusive(mine, lane);
            if (lane == 31) S.warp_sums[warp] = scan;
        }
        cluster.barrier_arrive();  // the counts are out; the others' are waited for below
        __syncthreads();
        if (t < kRadix) S.start[t] = scan - mine + warps_before(S.warp_sums, warp);
        __syncthreads();
        // the pairs in digit order within the block, so that what goes to
        // another block goes in runs: single 8-byte stores to random places of
        // 16 blocks were most of a pass (2.8 cycles each)
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            if (tile_base + warp_at + 32 * j + lane < n) {
                const uint32_t d = (uint32_t)(key[j] >> shift) & (kRadix - 1);
                const uint32_t at = S.start[d] + S.whist[warp][d] + rk[j];
                S.keys[cur][at] = key[j];
                S.idx[cur][at] = (uint16_t)idx[j];
            }
        }
        cluster.barrier_wait();
        // digit t % 256 over one half of the blocks
        {
            const int d = t & (kRadix - 1), half = t / kRadix, per = blocks / 2;
            uint32_t all = 0, earlier = 0;
            for (int r = half * per; r < half * per + per; ++r) {
                const uint32_t c = cluster.map_shared_rank(S.count, r)[d];
                all += c;
                earlier += r < rank ? c : 0u;
            }
            S.sums[half][0][d] = all;
            S.sums[half][1][d] = earlier;
        }
        __syncthreads();
        uint32_t all = 0;
        if (t < kRadix) {
            all = S.sums[0][0][t] + S.sums[1][0][t];
            scan = warp_inclusive(all, lane);
            if (lane == 31) S.warp_sums[warp] = scan;
        }
        __syncthreads();
        if (t < kRadix)  // global place of a pair minus its place in the block
            S.shift[t] = (int)(scan - all + warps_before(S.warp_sums, warp) + S.sums[0][1][t] + S.sums[1][1][t]) -
                         (int)S.start[t];
        __syncthreads();
        const int here = min(kTile, n - tile_base);
        for (int at = t; at < here; at += kFrontThreads) {
            const uint64_t k = S.keys[cur][at];
            const uint32_t to = (uint32_t)(at + S.shift[(uint32_t)(k >> shift) & (kRadix - 1)]);
            const uint32_t block = to / kTile, place = to % kTile;
            cluster.map_shared_rank(S.keys[cur ^ 1], block)[place] = k;
            cluster.map_shared_rank(S.idx[cur ^ 1], block)[place] = S.idx[cur][at];
        }
        cluster.sync();
    }

    // ---- out (an even number of passes ends in buffer 0)
    static_assert(kKeyPasses % 2 == 0, "the sorted pairs end in buffer 0");
    for (int at = t; at < kTile && tile_base + at < n; at += kFrontThreads) {
        keys_out[tile_base + at] = S.keys[0][at];
        idx_out[tile_base + at] = S.idx[0][at];
    }
}

template <int kItems>
void configure_front() {
    static std::once_flag done[kMaxDevices];
    once_per_device(done, [] {
        cudaFuncSetAttribute(front_kernel<kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(FrontSmem<kItems>));
        cudaFuncSetAttribute(front_kernel<kItems>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    });
}

template <int kItems>
cudaLaunchConfig_t front_config(int blocks, cudaLaunchAttribute (&attr)[2], cudaStream_t st) {
    configure_front<kItems>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kFrontThreads);
    cfg.dynamicSmemBytes = sizeof(FrontSmem<kItems>);
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (pdl.cuh)
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

// Blocks and items a thread for n particles: the fewest pairs a block that
// the cluster holds.
struct FrontShape {
    int blocks, items;
};
FrontShape front_shape(int n) {
    constexpr int k = kFrontThreads;
    if (n <= 8 * k) return {8, 1};
    if (n <= 16 * k) return {16, 1};
    if (n <= 32 * k) return {16, 2};
    if (n <= 48 * k) return {16, 3};
    if (n <= 64 * k) return {16, 4};
    return {16, 6};
}
static_assert(kFrontMax == 16 * kFrontThreads * 6, "front_shape covers kFrontMax");

template <class F>
void with_items(int items, F&& f) {
    using std::integral_constant;
    switch (items) {
        case 1: f(integral_constant<int, 1>{}); break;
        case 2: f(integral_constant<int, 2>{}); break;
        case 3: f(integral_constant<int, 3>{}); break;
        case 4: f(integral_constant<int, 4>{}); break;
        default: f(integral_constant<int, 6>{}); break;
    }
}

}  // namespace

bool front_available() {
    // a cluster of 16 blocks is beyond the portable size: ask the device
    bool ok = true;
    for (int items : {1, 2, 3, 4, 6})
        with_items(items, [&](auto k) {
            constexpr int kItems = decltype(k)::value;
            cudaLaunchAttribute attr[2];
            const cudaLaunchConfig_t cfg = front_config<kItems>(16, attr, nullptr);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, front_kernel<kItems>, &cfg) != cudaSuccess || clusters < 1)
                ok = false;
        });
    cudaGetLastError();
    return ok;
}

void launch_front(const float4* pos, int n, int front_bounds, float gmin, float gmax, float2* seg_bounds,
                  uint64_t* keys, uint32_t* idx, uint32_t* status, cudaStream_t st) {
    if (n <= 0 || n > kFrontMax) return;
    const FrontShape shape = front_shape(n);
    with_items(shape.items, [&](auto k) {
        constexpr int kItems = decltype(k)::value;
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = front_config<kItems>(shape.blocks, attr, st);
        cudaLaunchKernelEx(&cfg, front_kernel<kItems>, pos, n, front_bounds, gmin, gmax, seg_bounds, keys, idx, status);
    });
}

}  // namespace gcs
