// k_tree.cu - Karras (2012) binary radix tree over each segment's sorted
// Morton keys, and the bottom-up aggregation of bounds, mass and centre of
// mass.
//
// Build: one thread per internal node, as in karras_bvh.cuh:73-131.  The
// steps of the published algorithm (direction from the neighbours' common
// prefixes, exponential then binary search for the far end, binary search
// for the split) decide the topology, so they are the same steps; the
// common-prefix function is the reference's, including its duplicate-key
// rule (equal keys compare their positions, karras_bvh.cuh:23-31).  Indices
// are local to the segment, so a segment's tree is the tree the reference
// builds for that segment alone.  Each node also records the far end of its
// particle range, which gives the walk the node's particle count.
//
// Aggregation: a climb starts at every particle's leaf and goes up as long as
// both children of a node are known (karras_bvh.cuh:175-225).  Nodes inside a
// block's run of particles are climbed in shared memory; above them the left
// child's values are handed to the right child's climber through global
// memory word by word (the relay below), so, unlike in the reference, a node
// is never computed from values its children have not written.  Centres of
// mass are either the reference's FP32 formula or FP64 mass-weighted sums
// carried up the tree (exact for leaf terms, no cancellation at the top of
// the tree), rounded once to FP32.
#include "gcs_internal.h"
#include "device_math.cuh"
#include "pdl.cuh"

namespace gcs {

namespace {

constexpr int kAggThreads = 128;     // threads of an aggregation block
constexpr int kAggRange = 256;       // particles a block owns (measured at aggregate_kernel)
constexpr uint32_t kRelayPolls = 1u << 22;  // turns a climber waits for its left child (seconds)
constexpr int kAggMaxLevels = 96;    // internal levels of a valid tree (strictly increasing prefix lengths)

// ---- relay ------------------------------------------------------------------
// A node whose particles lie in more than one block's run (aggregate_kernel)
// is computed by its right child's climber, which gets the left child's
// values from the node's own records, before they hold the node's values:
//   wn     lo.x lo.y lo.z hi.x       (32-bit words, in place of cm)
//   tr     hi.y hi.z com.x com.y     (in place of com and mass)
//   bd     com.z mass                (in place of min x and y)
//   com64  the FP64 sums, of a left child that has them (64-bit words)
// (never in place of a walk record's codes: a walk that follows a failed
// climb must still read inside its arrays)
// The build (or launch_relay_reset) sets every word of these to all ones, the
// left child's climber writes them, and a word that is not all ones is there:
// each is a single relaxed access and needs no fence, counter or order among
// the others.  All ones is a NaN no arithmetic gives; a value with those bits
// (a NaN position of the caller's) is handed on as another NaN.
__device__ __forceinline__ uint4 load_relaxed(const void* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint2 load_relaxed2(const void* p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ ulonglong2 load_relaxed64(const void* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_relaxed(uint4* p, uint4 v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void store_relaxed(uint2* p, uint2 v) {
    asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" :: "l"(p), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void store_relaxed(ulonglong2* p, ulonglong2 v) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" :: "l"(p), "l"(v.x), "l"(v.y) : "memory");
}
__device__ __forceinline__ uint32_t relay_word(float f) {
    const uint32_t u = __float_as_uint(f);
    return u == 0xFFFFFFFFu ? 0x7FFFFFFFu : u;
}
__device__ __forceinline__ unsigned long long relay_word(double f) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(f);
    return u == ~0ull ? 0x7FFFFFFFFFFFFFFFull : u;
}
__device__ __forceinline__ void relay_clear(WalkNode* wn, BvhNodeTraverse* tr, BvhNodeBuild* bd, double4* com64,
                                            int node) {
    const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    *reinterpret_cast<uint4*>(wn + node) = ones;
    *reinterpret_cast<uint4*>(tr + node) = ones;
    *reinterpret_cast<uint2*>(bd + node) = make_uint2(~0u, ~0u);
    uint4* q = reinterpret_cast<uint4*>(com64 + node);
    q[0] = ones;
    q[1] = ones;
}
// Whether particles [lo, hi] lie in more than one aggregation block's run.
__device__ __forceinline__ bool above_blocks(int lo, int hi) { return lo / kAggRange != hi / kAggRange; }

// Common prefix length of sorted keys i and j of one segment (local indices);
// -1 when j falls outside the segment.
__device__ __forceinline__ int lcp(int i, int j, int n, const uint64_t* __restrict__ k,
                                   uint64_t ki) {
    if (j < 0 || j >= n) return -1;
    const uint64_t kj = __ldg(k + j);
    if (ki == kj) return 64 + __clz(i ^ j);
    return __clzll(ki ^ kj);
}

__global__ void build_kernel(Layout L, const uint64_t* __restrict__ keys,
                             BvhNodeTraverse* __restrict__ tr, BvhNodeBuild* __restrict__ bd,
                             int32_t* __restrict__ leaf_parent, WalkNode* __restrict__ wn,
                             double4* __restrict__ com64, uint32_t* __restrict__ agg_ticket,
                             uint32_t* __restrict__ status) {
    let_next_start();
    wait_for_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) *agg_ticket = 0u;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < L.n; g += gridDim.x * blockDim.x) {
        const int s = L.nseg > 1 ? __ldg(L.seg_id + g) : 0;
        const int off = (int)__ldg(L.seg_off + s);
        const int n = (int)__ldg(L.seg_off + s + 1) - off;
        const int i = g - off;                  // local index
        const int node_base = off - s;          // first internal node of the segment
        const int leaf_base = L.n_internal + off;
        const uint64_t* k = keys + off;
        if (n == 1) {                           // single particle: its leaf is the root
            leaf_parent[g] = -1;
            continue;
        }
        if (i >= n - 1) continue;
        const uint64_t ki = __ldg(k + i);
        const int d = (lcp(i, i + 1, n, k, ki) - lcp(i, i - 1, n, k, ki)) > 0 ? 1 : -1;
        const int dmin = lcp(i, i - d, n, k, ki);
        int lmax = 2;
        while (lcp(i, i + lmax * d, n, k, ki) > dmin) lmax *= 2;
        int l = 0;
        for (int t = lmax / 2; t >= 1; t /= 2)
            if (lcp(i, i + (l + t) * d, n, k, ki) > dmin) l += t;
        const int j = i + l * d;
        const int dnode = lcp(i, j, n, k, ki);
        int s_ = 0, step = l;
        do {
            step = (step + 1) >> 1;
            if (lcp(i, i + (s_ + step) * d, n, k, ki) > dnode) s_ += step;
        } while (step > 1);
        const int split = i + s_ * d + (d > 0 ? 0 : -1);
        const int lo = min(i, j), hi = max(i, j);
        if (split < lo || split + 1 > hi) {  // cannot happen for sorted keys; never write out of range
            atomicOr(status, GCS_DEV_BUILD_RANGE);
            continue;
        }
        const int node = node_base + i;
        const int cl = (lo == split) ? leaf_base + split : node_base + split;
        const int cr = (hi == split + 1) ? leaf_base + split + 1 : node_base + split + 1;
        BvhNodeTraverse* nt = tr + node;
        nt->child_left = cl;
        nt->child_right = cr;
        nt->range_end = off + j;
        if (lo == split) leaf_parent[off + split] = node;
        else bd[cl].parent = node;
        if (hi == split + 1) leaf_parent[off + split + 1] = node;
        else bd[cr].parent = node;
        bd[node].flag = 0;
        if (i == 0) bd[node].parent = -1;       // segment root
        if (above_blocks(off + lo, off + hi)) relay_clear(wn, tr, bd, com64, node);
    }
}

struct ChildData {
    float3 lo, hi, com;
    float m;
    double3 mx;   // FP64 mass-weighted position sums
    double md;    // FP64 mass sum
};

// FP64 centre-of-mass sums (com_fp64) are kept for the top of the tree:
// nodes of at least this many particles, where the mass-weighted positions
// of many particles are summed.  A child below the size (or a particle)
// enters its parent's sums as the exact double product of its FP32 mass and
// centre of mass (position).  Block-local nodes hold at most kAggRange
// particles, so they are never FP64 nodes.
constexpr int kComFp64Min = 1024;
static_assert(kComFp64Min > kAggRange, "block-local nodes are never FP64 nodes");

// A child's terms in its parent's FP64 sums: its own sums if it is an FP64
// node, else the double product of its FP32 mass and centre of mass.
__device__ __forceinline__ void fp64_terms(const ChildData& c, bool big, double3& mx, double& md) {
    if (big) {
        mx = c.mx;
        md = c.md;
    } else {
        md = (double)c.m;
        mx = make_double3(md * (double)c.com.x, md * (double)c.com.y, md * (double)c.com.z);
    }
}

// Walk record of internal node `node` (links already range-checked): the
// particle range [min(own, re), max(own, re)] clipped to the segment
// [seg_lo, seg_hi]; <= leaf_size particles make a bucket, else the children
// are coded as internal node or ~particle.
__device__ __forceinline__ void write_walk_node(const WalkNodeParams& wnp, int node, float3 com, float m,
                                                float width, int cl, int cr, int own, int re, int seg_lo,
                                                int seg_hi, int n_internal) {
    const int lo = max(min(own, re), seg_lo);
    const int cnt = min(max(own, re), seg_hi) - lo + 1;
    int ca, cb;
    if (cnt <= wnp.leaf_size) {
        ca = lo;
        cb = kWalkBucketTag + max(cnt, 0);
    } else {
        ca = cl >= n_internal ? ~(cl - n_internal) : cl;
        cb = cr >= n_internal ? ~(cr - n_internal) : cr;
    }
    float4* w = reinterpret_cast<float4*>(wnp.wn + node);
    w[0] = make_float4(com.x, com.y, com.z, __fmul_rn(wnp.G, m));
    reinterpret_cast<int4*>(w)[1] = make_int4(__float_as_int(__fmul_rn(width, width)), ca, cb, 0);
}

// Walk records from the traverse records: one thread per particle g; the
// internal node g - s exists for every particle but the last of segment s.
__global__ void walk_nodes_kernel(Layout L, const BvhNodeTraverse* __restrict__ tr, WalkNodeParams wnp,
                                  uint32_t* __restrict__ status) {
    let_next_start();
    wait_for_previous();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= L.n) return;
    const int s = L.nseg > 1 ? __ldg(L.seg_id + g) : 0;
    const int seg_lo = (int)__ldg(L.seg_off + s), seg_hi = (int)__ldg(L.seg_off + s + 1) - 1;
    if (g >= seg_hi) return;
    const int node = g - s;
    const float4* np = reinterpret_cast<const float4*>(tr + node);
    const float4 a = __ldg(np);
    const float4 c = __ldg(np + 1);
    const int cl = __float_as_int(c.y), cr = __float_as_int(c.z);
    const int lim = L.n_internal + L.n;
    if (cl >= 0 && cl < lim && cr >= 0 && cr < lim) {
        write_walk_node(wnp, node, make_float3(a.x, a.y, a.z), a.w, c.x, cl, cr, node + s, __float_as_int(c.w),
                        seg_lo, seg_hi, L.n_internal);
    } else {
        atomicOr(status, GCS_DEV_BUILD_RANGE);
        float4* w = reinterpret_cast<float4*>(wnp.wn + node);
        w[0] = make_float4(a.x, a.y, a.z, __fmul_rn(wnp.G, a.w));
        reinterpret_cast<int4*>(w)[1] = make_int4(__float_as_int(__fmul_rn(c.x, c.x)), 0, kWalkSkipTag, 0);
    }
}

// A node's own values from its two children's: box, width, mass, and the
// centre of mass in the reference's FP32 formula (of FP64 nodes the caller
// replaces it).
__device__ __forceinline__ float merge_children(const ChildData& A, const ChildData& B, ChildData& out) {
    out.lo = make_float3(fminf(A.lo.x, B.lo.x), fminf(A.lo.y, B.lo.y), fminf(A.lo.z, B.lo.z));
    out.hi = make_float3(fmaxf(A.hi.x, B.hi.x), fmaxf(A.hi.y, B.hi.y), fmaxf(A.hi.z, B.hi.z));
    out.m = __fadd_rn(A.m, B.m);
    return fmaxf(__fsub_rn(out.hi.x, out.lo.x),
                 fmaxf(__fsub_rn(out.hi.y, out.lo.y), __fsub_rn(out.hi.z, out.lo.z)));
}
__device__ __forceinline__ float3 merged_com_fp32(const ChildData& A, const ChildData& B, const ChildData& n) {
    if (n.m > 0.0f)
        return make_float3(com_fp32(A.com.x, A.m, B.com.x, B.m, n.m), com_fp32(A.com.y, A.m, B.com.y, B.m, n.m),
                           com_fp32(A.com.z, A.m, B.com.z, B.m, n.m));
    return make_float3(__fmul_rn(__fadd_rn(n.lo.x, n.hi.x), 0.5f), __fmul_rn(__fadd_rn(n.lo.y, n.hi.y), 0.5f),
                       __fmul_rn(__fadd_rn(n.lo.z, n.hi.z), 0.5f));
}

// A block's nodes in shared memory, by the particle at the node's own end of
// its range (slot 0 is the block's first particle).
template <int kRange>
struct AggSmem {
    float4 pos[kRange];        // the particles
    int4 link[kRange];         // children, far end of the range, parent (-2: not a node of this block)
    float4 com_m[kRange];      // finished nodes
    float4 box_a[kRange];      // min x y z, max x
    float2 box_b[kRange];      // max y z
    int32_t arrived[kRange];
    uint16_t queue[3][kRange / 2 + 1];  // nodes whose children are both finished, by step
    int n_queue[3];
    int32_t root[kRange == kAggRange ? kRange : 1];  // finished subtree whose parent lies above the block, at
                                                     // its first particle (-1: none starts here)
};
constexpr int kNotLocal = -2;
constexpr int kAggWholeMax = 2048;   // particles one block takes whole
constexpr int kAggWholeThreads = 512;
// A child's FP64 sums, written by this block before its last barrier.
__device__ __forceinline__ void load_sums(const double4* q, ChildData& c) {
    const double2 a = *reinterpret_cast<const double2*>(q), b = *(reinterpret_cast<const double2*>(q) + 1);
    c.mx = make_double3(a.x, a.y, b.x);
    c.md = b.y;
}

template <int kRange>
__device__ __forceinline__ ChildData smem_particle(const AggSmem<kRange>& S, int slot) {
    ChildData r;
    const float4 p = S.pos[slot];
    r.lo = r.hi = r.com = make_float3(p.x, p.y, p.z);
    r.m = p.w;
    return r;
}
template <int kRange>
__device__ __forceinline__ ChildData smem_node(const AggSmem<kRange>& S, int slot) {
    ChildData r;
    const float4 c = S.com_m[slot], a = S.box_a[slot];
    const float2 b = S.box_b[slot];
    r.com = make_float3(c.x, c.y, c.z);
    r.m = c.w;
    r.lo = make_float3(a.x, a.y, a.z);
    r.hi = make_float3(a.w, b.x, b.y);
    return r;
}

// Block b owns particles [kAggRange b, kAggRange (b + 1)).  A node is local
// to the block when its whole particle range lies inside; both children are
// then finished by this block.
//
//   load    the block's particles, leaf parents and node links, coalesced;
//   climb   local nodes, in shared memory alone, in block-wide steps: each
//           step computes the nodes whose two children are finished, packed
//           into whole warps (a step waits on no global load, store or
//           fence, and a climb by every particle's own lane keeps 8 lanes of
//           a warp busy).  A subtree whose parent is not local is marked at
//           its first particle;
//   list    the marked subtrees, by position (rise_kernel relies on it);
//   store   the finished nodes' records, whole and coalesced.
// The nodes above the blocks are rise_kernel's.
// A context of up to kAggWholeMax particles is one block's run: no node is
// above it, and its FP64 nodes are summed here too (1,408 particles: build and
// aggregation 48.1 us with rise_kernel, 17 levels above the blocks, 37.9 so).
template <int kRange, int kThreads, bool kWhole>
__global__ void __launch_bounds__(kThreads)
aggregate_kernel(Layout L, const float4* __restrict__ pos, BvhNodeTraverse* __restrict__ tr,
                 BvhNodeBuild* __restrict__ bd, double4* com64, const int32_t* __restrict__ leaf_parent,
                 int com_fp64, WalkNodeParams wnp,
                 int2* __restrict__ roots, uint32_t* __restrict__ n_roots, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char agg_smem[];
    AggSmem<kRange>& S = *reinterpret_cast<AggSmem<kRange>*>(agg_smem);
    const int ni = L.n_internal;
    const int lim = ni + L.n;
    if (threadIdx.x == 0) S.n_queue[0] = S.n_queue[1] = S.n_queue[2] = 0;
    if (!kWhole)
        for (int j = threadIdx.x; j < kRange; j += kThreads) S.root[j] = -1;
    const int b0 = blockIdx.x * kRange;
    const int count = min(kRange, L.n - b0);
    let_next_start();
    const auto seg_of = [&](int g) { return L.nseg > 1 ? (int)__ldg(L.seg_id + g) : 0; };
    const auto seg_end = [&](int s) { return L.nseg > 1 ? (int)__ldg(L.seg_off + s + 1) : L.n; };

    // ---- load
    int my_parent[kRange / kThreads];  // of the thread's particles
#pragma unroll
    for (int u = 0; u < kRange / kThreads; ++u) {
        const int j = threadIdx.x + u * kThreads;
        my_parent[u] = -1;
        if (j >= count) break;
        const int g = b0 + j, s = seg_of(g);
        S.pos[j] = __ldg(pos + g);
        my_parent[u] = __ldg(leaf_parent + g);
        S.arrived[j] = 0;
        int4 k = make_int4(-1, -1, 0, kNotLocal);
        if (g + 1 < seg_end(s)) {  // node g - s exists
            const int node = g - s;
            const int4 t = __ldg(reinterpret_cast<const int4*>(tr + node) + 1);  // width, left, right, range end
            const int up = __ldg(&bd[node].parent);
            const int lo = min(g, t.w), hi = max(g, t.w);
            if (lo >= b0 && hi < b0 + count) {
                if (t.y < 0 || t.z < 0 || t.y >= lim || t.z >= lim) atomicOr(status, GCS_DEV_TREE_MALFORMED);
                else k = make_int4(t.y, t.z, t.w, up);
            }
        }
        S.link[j] = k;
    }
    __syncthreads();

    // ---- climb
    // arrive: `from` (its first particle in slot `first`) is finished; the
    // second child to arrive at a local parent queues it for the next step, a
    // subtree under any other parent is a root
    const auto arrive = [&](int from, int first, int up, int sg, int q) {
        if (up < 0) return;  // the segment's root (or a one-particle segment)
        const int slot = up + sg - b0;
        if (slot < 0 || slot >= count || S.link[slot].w == kNotLocal) {
            if (!kWhole) S.root[first] = from;
        } else if (atomicAdd(&S.arrived[slot], 1) == 1) {
            S.queue[q][atomicAdd(&S.n_queue[q], 1)] = (uint16_t)slot;
        }
    };
#pragma unroll
    for (int u = 0; u < kRange / kThreads; ++u) {
        const int j = threadIdx.x + u * kThreads;
        if (j < count) arrive(ni + b0 + j, j, my_parent[u], seg_of(b0 + j), 0);
    }
    __syncthreads();
    for (int step = 0; S.n_queue[step % 3] > 0; ++step) {
        const int q = step % 3, n_ready = S.n_queue[q];
        if (threadIdx.x == 0) S.n_queue[(step + 2) % 3] = 0;
        for (int e = threadIdx.x; e < n_ready; e += kThreads) {
            const int slot = S.queue[q][e];
            const int4 k = S.link[slot];
            const int sg = seg_of(b0 + slot);
            const int sl = k.x >= ni ? k.x - ni - b0 : k.x + sg - b0, sr = k.y >= ni ? k.y - ni - b0 : k.y + sg - b0;
            if (sl < 0 || sr < 0 || sl >= count || sr >= count) {
                atomicOr(status, GCS_DEV_TREE_MALFORMED);
                continue;
            }
            const ChildData A = k.x >= ni ? smem_particle(S, sl) : smem_node(S, sl);
            const ChildData B = k.y >= ni ? smem_particle(S, sr) : smem_node(S, sr);
            ChildData node;
            merge_children(A, B, node);
            bool sums = false;
            if (kWhole && com_fp64) {  // (as rise_kernel)
                const int own = b0 + slot, lo = min(own, k.z), hi = max(own, k.z);
                const int split = k.x >= ni ? k.x - ni : k.x + sg;
                if (hi - lo + 1 >= kComFp64Min) {
                    const bool big_l = split - lo + 1 >= kComFp64Min, big_r = hi - split >= kComFp64Min;
                    ChildData C = A, D = B;
                    if (big_l) load_sums(com64 + k.x, C);
                    if (big_r) load_sums(com64 + k.y, D);
                    node.mx = make_double3(0.0, 0.0, 0.0);
                    node.md = 0.0;
                    sums = node.m > 0.0f;
                    if (sums) {
                        double3 amx, bmx;
                        double amd, bmd;
                        fp64_terms(C, big_l, amx, amd);
                        fp64_terms(D, big_r, bmx, bmd);
                        node.md = amd + bmd;
                        node.mx = make_double3(amx.x + bmx.x, amx.y + bmx.y, amx.z + bmx.z);
                        node.com = make_float3((float)(node.mx.x / node.md), (float)(node.mx.y / node.md),
                                               (float)(node.mx.z / node.md));
                    }
                    com64[own - sg] = make_double4(node.mx.x, node.mx.y, node.mx.z, node.md);
                }
            }
            if (!sums) node.com = merged_com_fp32(A, B, node);
            S.com_m[slot] = make_float4(node.com.x, node.com.y, node.com.z, node.m);
            S.box_a[slot] = make_float4(node.lo.x, node.lo.y, node.lo.z, node.hi.x);
            S.box_b[slot] = make_float2(node.hi.y, node.hi.z);
            arrive(b0 + slot - sg, min(b0 + slot, k.z) - b0, k.w, sg, (step + 1) % 3);
        }
        __syncthreads();
    }

    // ---- list
    if (!kWhole && threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int listed = 0;
#pragma unroll
        for (int j0 = 0; j0 < kRange; j0 += 32) {
            const int from = S.root[j0 + lane];
            const uint32_t marked = __ballot_sync(0xFFFFFFFFu, from >= 0);
            if (from >= 0)
                roots[b0 + listed + __popc(marked & ((1u << lane) - 1u))] = make_int2(from, seg_of(b0 + j0 + lane));
            listed += __popc(marked);
        }
        if (lane == 0) n_roots[blockIdx.x] = (uint32_t)listed;
    }

    // ---- store
    for (int j = threadIdx.x; j < count; j += kThreads) {
        const int4 k = S.link[j];
        if (k.w == kNotLocal || S.arrived[j] < 2) continue;
        const int g = b0 + j, s = seg_of(g), node = g - s;
        const float4 c = S.com_m[j], a = S.box_a[j];
        const float2 b = S.box_b[j];
        const float width = fmaxf(__fsub_rn(a.w, a.x), fmaxf(__fsub_rn(b.x, a.y), __fsub_rn(b.y, a.z)));
        float4* t4 = reinterpret_cast<float4*>(tr + node);
        t4[0] = c;
        reinterpret_cast<int4*>(t4)[1] = make_int4(__float_as_int(width), k.x, k.y, k.z);
        float4* b4 = reinterpret_cast<float4*>(bd + node);
        b4[0] = a;
        reinterpret_cast<int4*>(b4)[1] = make_int4(__float_as_int(b.x), __float_as_int(b.y), 0, k.w);
        write_walk_node(wnp, node, make_float3(c.x, c.y, c.z), c.w, width, k.x, k.y, g, k.z,
                            L.nseg > 1 ? (int)__ldg(L.seg_off + s) : 0, seg_end(s) - 1, ni);
    }
}

// Climbs on from the subtrees the blocks' climbs left, one warp for each run
// of kAggRange particles: lane l takes the subtrees l, l + 32, ... of the run's
// list one after another (a run has one subtree per level of the paths at its
// two ends: up to 18 in a smooth collision, above 60 in a steep profile).  A
// left child hands its values to the relay and stops, a right child waits for
// the left one's, computes the node and goes on.
//
// No wait is for something that has not started.  A climber waits only for a
// left sibling of its own subtree, and that sibling's values come from a
// climber that started at a lower position.  Lists are in the order of
// position, so within a run that climber is an earlier entry: in the same turn
// of the warp, on another lane, or in a turn that is over.  Between runs it is
// one of an earlier run, and blocks take their runs in launch order from a
// ticket.  So the lowest waiting climber can always go on.  The wait is
// bounded all the same.
// A node above the blocks: its links, and which of it and its children are
// FP64 nodes.
struct RiseNode {
    int node, cl, cr, re, up;  // node < 0: none
    bool big, big_l, big_r;
};
__device__ __forceinline__ RiseNode rise_node(const BvhNodeTraverse* __restrict__ tr,
                                              const BvhNodeBuild* __restrict__ bd, int node, int s, int ni, bool fp64) {
    RiseNode r;
    r.node = node < ni ? node : -1;
    r.cl = r.cr = r.up = -1;
    r.re = 0;
    r.big = r.big_l = r.big_r = false;
    if (r.node < 0) return r;
    r.cl = __ldg(&tr[node].child_left);
    r.cr = __ldg(&tr[node].child_right);
    r.re = __ldg(&tr[node].range_end);
    r.up = __ldg(&bd[node].parent);
    // particles of the node and of its two children (the split is the left
    // child's end of the range)
    const int own = node + s, lo = min(own, r.re), hi = max(own, r.re);
    const int split = r.cl >= ni ? r.cl - ni : r.cl + s;
    r.big = fp64 && hi - lo + 1 >= kComFp64Min;
    r.big_l = r.big && split - lo + 1 >= kComFp64Min;
    r.big_r = r.big && hi - split >= kComFp64Min;
    return r;
}
__device__ __forceinline__ bool valid_links(const RiseNode& n, int from, int lim) {
    return n.cl >= 0 && n.cr >= 0 && n.cl < lim && n.cr < lim && (n.cl == from || n.cr == from);
}
struct RelayWords {
    uint4 w0, w1;
    uint2 w2;
    ulonglong2 q0, q1;
};
__device__ __forceinline__ void relay_load(const WalkNode* wn, const BvhNodeTraverse* tr, const BvhNodeBuild* bd,
                                           const double4* com64, const RiseNode& n, RelayWords& r) {
    r.w0 = load_relaxed(wn + n.node);
    r.w1 = load_relaxed(tr + n.node);
    r.w2 = load_relaxed2(bd + n.node);
    r.q0 = r.q1 = make_ulonglong2(0ull, 0ull);
    if (n.big_l) {
        r.q0 = load_relaxed64(com64 + n.node);
        r.q1 = load_relaxed64(reinterpret_cast<const ulonglong2*>(com64 + n.node) + 1);
    }
}
__device__ __forceinline__ bool relay_there(const RelayWords& r) {
    return r.w0.x != ~0u && r.w0.y != ~0u && r.w0.z != ~0u && r.w0.w != ~0u && r.w1.x != ~0u && r.w1.y != ~0u &&
           r.w1.z != ~0u && r.w1.w != ~0u && r.w2.x != ~0u && r.w2.y != ~0u && r.q0.x != ~0ull && r.q0.y != ~0ull &&
           r.q1.x != ~0ull && r.q1.y != ~0ull;
}
__device__ __forceinline__ ChildData relay_values(const RelayWords& r) {
    ChildData A;
    A.lo = make_float3(__uint_as_float(r.w0.x), __uint_as_float(r.w0.y), __uint_as_float(r.w0.z));
    A.hi = make_float3(__uint_as_float(r.w0.w), __uint_as_float(r.w1.x), __uint_as_float(r.w1.y));
    A.com = make_float3(__uint_as_float(r.w1.z), __uint_as_float(r.w1.w), __uint_as_float(r.w2.x));
    A.m = __uint_as_float(r.w2.y);
    A.mx = make_double3(__longlong_as_double((long long)r.q0.x), __longlong_as_double((long long)r.q0.y),
                        __longlong_as_double((long long)r.q1.x));
    A.md = __longlong_as_double((long long)r.q1.y);
    return A;
}
// The values of node n's left child, to its right child's climber.
__device__ __forceinline__ void hand_over(WalkNode* wn, BvhNodeTraverse* tr, BvhNodeBuild* bd, double4* com64,
                                          const RiseNode& n, const ChildData& c) {
    store_relaxed(reinterpret_cast<uint4*>(wn + n.node),
                  make_uint4(relay_word(c.lo.x), relay_word(c.lo.y), relay_word(c.lo.z), relay_word(c.hi.x)));
    store_relaxed(reinterpret_cast<uint4*>(tr + n.node),
                  make_uint4(relay_word(c.hi.y), relay_word(c.hi.z), relay_word(c.com.x), relay_word(c.com.y)));
    store_relaxed(reinterpret_cast<uint2*>(bd + n.node), make_uint2(relay_word(c.com.z), relay_word(c.m)));
    if (n.big_l) {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(com64 + n.node);
        store_relaxed(q, make_ulonglong2(relay_word(c.mx.x), relay_word(c.mx.y)));
        store_relaxed(q + 1, make_ulonglong2(relay_word(c.mx.z), relay_word(c.md)));
    }
}

constexpr int kRiseWarps = 2;

__global__ void __launch_bounds__(kRiseWarps * 32)
rise_kernel(Layout L, const float4* __restrict__ pos, BvhNodeTraverse* __restrict__ tr, BvhNodeBuild* __restrict__ bd,
            double4* __restrict__ com64, const int32_t* __restrict__ leaf_parent, const int2* __restrict__ roots,
            const uint32_t* __restrict__ n_roots, int n_runs, int com_fp64, WalkNodeParams wnp,
            uint32_t* __restrict__ ticket, uint32_t* __restrict__ status) {
    __shared__ int s_block;
    let_next_start();
    wait_for_previous();
    if (threadIdx.x == 0) s_block = (int)atomicAdd(ticket, 1u);
    __syncthreads();
    const int run = s_block * kRiseWarps + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (run >= n_runs) return;
    const int ni = L.n_internal;
    const int lim = ni + L.n;
    const int count = min((int)__ldg(n_roots + run), kAggRange);
    const bool fp64 = com_fp64 != 0;
    // the finished subtree `from`: its values, and the node above it
    const auto start = [&](int from, int s, ChildData& mine) {
        int node;
        if (from >= ni) {
            const float4 p = __ldg(pos + (from - ni));
            mine.lo = mine.hi = mine.com = make_float3(p.x, p.y, p.z);
            mine.m = p.w;
            node = __ldg(leaf_parent + (from - ni));
        } else {
            const float4 c = *reinterpret_cast<const float4*>(tr + from);
            const float4 b_0 = *reinterpret_cast<const float4*>(bd + from);
            const float4 b_1 = *(reinterpret_cast<const float4*>(bd + from) + 1);
            mine.com = make_float3(c.x, c.y, c.z);
            mine.m = c.w;
            mine.lo = make_float3(b_0.x, b_0.y, b_0.z);
            mine.hi = make_float3(b_0.w, b_1.x, b_1.y);
            node = __float_as_int(b_1.w);
        }
        mine.mx = make_double3(0.0, 0.0, 0.0);
        mine.md = 0.0;
        return rise_node(tr, bd, node, s, ni, fp64);
    };
    // left children of the later turns hand over before any wait of the first
    for (int r = lane + 32; r < count; r += 32) {
        const int2 root = roots[run * kAggRange + r];
        ChildData mine;
        const RiseNode N = start(root.x, root.y, mine);
        if (N.node >= 0 && valid_links(N, root.x, lim) && N.cl == root.x) hand_over(wnp.wn, tr, bd, com64, N, mine);
    }
    for (int r = lane; r < count; r += 32) {
        const int2 root = roots[run * kAggRange + r];
        const int s = root.y;
        ChildData mine;
        RiseNode N = start(root.x, s, mine);
        const int seg_lo = L.nseg > 1 ? (int)__ldg(L.seg_off + s) : 0;
        const int seg_hi = (L.nseg > 1 ? (int)__ldg(L.seg_off + s + 1) : L.n) - 1;
        bool ok = N.node >= 0 && valid_links(N, root.x, lim);
        if (ok && N.cl == root.x) {
            if (r < 32) hand_over(wnp.wn, tr, bd, com64, N, mine);
            continue;
        }
        RelayWords w;
        if (ok) relay_load(wnp.wn, tr, bd, com64, N, w);
        RiseNode up = rise_node(tr, bd, ok ? N.up : -1, s, ni, fp64);
        uint32_t polls = 0;
        int levels = 0;
        // a waiting lane polls once a turn, one that has its left child's
        // values moves up one level
        while (ok) {
            if (!relay_there(w)) {
                ok = ++polls < kRelayPolls;
                relay_load(wnp.wn, tr, bd, com64, N, w);
                continue;
            }
            const ChildData A = relay_values(w);
            ChildData next;
            const float width = merge_children(A, mine, next);
            next.md = 0.0;
            next.mx = make_double3(0.0, 0.0, 0.0);
            const bool sums = N.big && next.m > 0.0f;
            if (sums) {
                double3 amx, bmx;
                double amd, bmd;
                fp64_terms(A, N.big_l, amx, amd);
                fp64_terms(mine, N.big_r, bmx, bmd);
                next.md = amd + bmd;
                next.mx = make_double3(amx.x + bmx.x, amx.y + bmx.y, amx.z + bmx.z);
                next.com = make_float3(0.0f, 0.0f, 0.0f);  // below: a parent takes the sums instead
            } else {
                next.com = merged_com_fp32(A, mine, next);
            }
            // the parent first: its other child may be waiting, and its words
            // and links travel while this node's record is finished
            const RiseNode cur = N;
            const bool more = up.node >= 0 && cur.up >= 0;
            ok = !more ? cur.up < 0 : valid_links(up, cur.node, lim) && ++levels <= kAggMaxLevels;
            const bool hand = ok && more && up.cl == cur.node;
            if (sums && ok && more && !(hand ? up.big_l : up.big_r)) ok = false;  // FP64 nodes have FP64 parents
            if (hand && ok) hand_over(wnp.wn, tr, bd, com64, up, next);
            N = up;
            if (ok && more && !hand) {
                relay_load(wnp.wn, tr, bd, com64, N, w);
                up = rise_node(tr, bd, N.up, s, ni, fp64);
            }
            if (sums)
                next.com = make_float3((float)(next.mx.x / next.md), (float)(next.mx.y / next.md),
                                       (float)(next.mx.z / next.md));
            com64[cur.node] = make_double4(next.mx.x, next.mx.y, next.mx.z, next.md);
            reinterpret_cast<float4*>(tr + cur.node)[0] = make_float4(next.com.x, next.com.y, next.com.z, next.m);
            tr[cur.node].width = width;
            float4* b4 = reinterpret_cast<float4*>(bd + cur.node);
            b4[0] = make_float4(next.lo.x, next.lo.y, next.lo.z, next.hi.x);
            reinterpret_cast<float2*>(b4 + 1)[0] = make_float2(next.hi.y, next.hi.z);
            write_walk_node(wnp, cur.node, next.com, next.m, width, cur.cl, cur.cr, cur.node + s, cur.re, seg_lo,
                            seg_hi, ni);
            if (!ok || !more || hand) break;
            mine = next;
            polls = 0;
        }
        if (!ok) atomicOr(status, GCS_DEV_TREE_MALFORMED);
    }
}

// Empty relay words of every node above the blocks, and the block ticket, for
// an aggregation that does not follow a build (one thread per particle, as in
// walk_nodes_kernel).
__global__ void relay_reset_kernel(Layout L, BvhNodeTraverse* __restrict__ tr, BvhNodeBuild* __restrict__ bd,
                                   WalkNode* __restrict__ wn, double4* __restrict__ com64,
                                   uint32_t* __restrict__ ticket) {
    let_next_start();
    wait_for_previous();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g == 0) *ticket = 0u;
    if (g >= L.n) return;
    const int s = L.nseg > 1 ? __ldg(L.seg_id + g) : 0;
    if (g + 1 >= (int)__ldg(L.seg_off + s + 1)) return;
    const int re = tr[g - s].range_end;
    if (above_blocks(min(g, re), max(g, re))) relay_clear(wn, tr, bd, com64, g - s);
}

int tree_grid(int64_t n) {
    int64_t b = (n + 255) / 256;
    return (int)(b < 1 ? 1 : b);
}

}  // namespace

void launch_build(const Layout& L, const uint64_t* keys, BvhNodeTraverse* tr, BvhNodeBuild* bd,
                  int32_t* leaf_parent, WalkNode* wn, double4* com64, uint32_t* agg_ticket, uint32_t* status,
                  cudaStream_t st) {
    if (L.n <= 0) return;
    launch_after(build_kernel, tree_grid(L.n), 256, 0, st, L, keys, tr, bd, leaf_parent, wn, com64, agg_ticket, status);
}

void launch_relay_reset(const Layout& L, BvhNodeTraverse* tr, BvhNodeBuild* bd, WalkNode* wn, double4* com64,
                        uint32_t* agg_ticket, cudaStream_t st) {
    if (L.n <= 0) return;
    launch_after(relay_reset_kernel, tree_grid(L.n), 256, 0, st, L, tr, bd, wn, com64, agg_ticket);
}

void launch_aggregate(const Layout& L, const float4* pos, BvhNodeTraverse* tr, BvhNodeBuild* bd,
                      double4* com64, const int32_t* leaf_parent, int com_fp64, const WalkNodeParams& wnp,
                      int2* roots, uint32_t* n_roots, uint32_t* agg_ticket, uint32_t* status, cudaStream_t st) {
    if (L.n <= 0) return;
    if (L.n <= kAggWholeMax) {
        constexpr size_t smem = sizeof(AggSmem<kAggWholeMax>);
        static std::once_flag configured[kMaxDevices];
        once_per_device(configured, [] {
            cudaFuncSetAttribute(aggregate_kernel<kAggWholeMax, kAggWholeThreads, true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        });
        aggregate_kernel<kAggWholeMax, kAggWholeThreads, true><<<1, kAggWholeThreads, smem, st>>>(
            L, pos, tr, bd, com64, leaf_parent, com_fp64, wnp, roots, n_roots, status);
        return;
    }
    const int runs = (L.n + kAggRange - 1) / kAggRange;
    // (launched plainly: early blocks would hold shared memory that the gather
    // beside the build needs; 344 against 351 us a step of 45,056 particles)
    aggregate_kernel<kAggRange, kAggThreads, false><<<(unsigned)runs, kAggThreads, sizeof(AggSmem<kAggRange>), st>>>(
        L, pos, tr, bd, com64, leaf_parent, com_fp64, wnp, roots, n_roots, status);
    if (runs > 1)
        launch_after(rise_kernel, (unsigned)((runs + kRiseWarps - 1) / kRiseWarps), kRiseWarps * 32, 0, st, L, pos, tr,
                     bd, com64, leaf_parent, roots, n_roots, runs, com_fp64, wnp, agg_ticket, status);
}

void launch_walk_nodes(const Layout& L, const BvhNodeTraverse* tr, WalkNodeParams wnp, uint32_t* status,
                       cudaStream_t st) {
    if (L.n <= 0 || !wnp.wn) return;
    launch_after(walk_nodes_kernel, tree_grid(L.n), 256, 0, st, L, tr, wnp, status);
}

}  // namespace gcs
