// k_stream.cu - the HBM-streaming stages: Star <-> SoA transposes, per-segment
// bounds, Morton encode (+ sort histograms), gather, kick+drift+colour,
// FP64 diagnostics and the FP64 direct sum.
//
// All particle records are float4 (16-byte) loads/stores; grids are sized
// as a multiple of the SM count with grid-stride loops.
#include <algorithm>
#include <atomic>

#include "gcs_internal.h"
#include "device_math.cuh"
#include "digits.cuh"
#include "pdl.cuh"

namespace gcs {

int current_device() {
    int dev = -1;
    return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

int current_sm_count() {
    static std::atomic<int> cached[kMaxDevices] = {};
    const int dev = current_device();
    if (dev >= 0 && dev < kMaxDevices) {
        const int v = cached[dev].load(std::memory_order_relaxed);
        if (v > 0) return v;
    }
    int sms = 0;
    if (dev < 0 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    if (dev >= 0 && dev < kMaxDevices) cached[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

namespace {

constexpr int kStreamThreads = 256;

int stream_grid(int64_t n) {
    const int sms = current_sm_count();
    int64_t want = (n + kStreamThreads - 1) / kStreamThreads;
    int64_t cap = (int64_t)sms * 8;
    if (want > cap) want = cap;
    if (want < 1) want = 1;
    return (int)want;
}

// seg_id[i] = the segment s with seg_off[s] <= i < seg_off[s+1] (binary
// search over the nseg+1 offsets, which stay in L1).
__global__ void fill_segment_ids_kernel(const int64_t* __restrict__ seg_off, int nseg,
                                        int32_t* __restrict__ seg_id, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = nseg - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(seg_off + mid) <= i) lo = mid;
            else hi = mid - 1;
        }
        seg_id[i] = lo;
    }
}

// Star (x,y,z,vx | vy,vz,m,tcol) <-> pos (x,y,z,m), vel (vx,vy,vz,tcol).
__global__ void unpack_stars_kernel(const float4* __restrict__ stars, float4* __restrict__ pos,
                                    float4* __restrict__ vel, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 a = __ldg(stars + 2 * i);
        const float4 b = __ldg(stars + 2 * i + 1);
        pos[i] = make_float4(a.x, a.y, a.z, b.z);
        vel[i] = make_float4(a.w, b.x, b.y, b.w);
    }
}

__global__ void pack_stars_kernel(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                  float4* __restrict__ stars, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        store_star(stars, i, pos[i], vel[i]);
    }
}

// PlaybackStar = x, y, z, r, g, b, type (main.cpp:266 writes type into the
// padding byte).
__global__ void pack_playback_kernel(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                     float4* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        const uint32_t tcol = __float_as_uint(vel[i].w);
        const uint32_t rgbt = (tcol >> 8) | ((tcol & 0xFFu) << 24);
        out[i] = make_float4(p.x, p.y, p.z, __uint_as_float(rgbt));
    }
}

// Per-segment min/max over x, y and z of every particle (main.cpp:152-166
// reduces one scalar min and max over all three axes).  min/max is exact in
// any precision, so the reduction runs in FP32.  Each block takes chunks
// that never straddle a segment, reduces in registers and warp shuffles, and
// publishes with one atomicMax per chunk on order-preserving encodings
// (min stored as the max of ~enc), so a zeroed buffer is a valid start.
__global__ void bounds_kernel(const float4* __restrict__ pos, const Chunk* __restrict__ chunks,
                              int n_chunks, uint32_t* __restrict__ bounds_enc,
                              uint32_t* __restrict__ status) {
    let_next_start();
    wait_for_previous();
    constexpr int kInFlight = 8;  // independent loads per thread per sweep
    __shared__ float s_lo[kStreamThreads / 32], s_hi[kStreamThreads / 32];
    for (int c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const Chunk ch = chunks[c];
        float lo = INFINITY, hi = -INFINITY;
        bool bad = false;
        for (int i0 = threadIdx.x; i0 < ch.count; i0 += kInFlight * blockDim.x) {
            float4 p[kInFlight];
#pragma unroll
            for (int k = 0; k < kInFlight; ++k) {
                const int i = i0 + k * blockDim.x;
                p[k] = i < ch.count ? __ldg(pos + ch.start + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < kInFlight; ++k) {
                if (i0 + k * (int)blockDim.x < ch.count) {
                    bad |= !(isfinite(p[k].x) && isfinite(p[k].y) && isfinite(p[k].z));
                    lo = fminf(lo, fminf(p[k].x, fminf(p[k].y, p[k].z)));
                    hi = fmaxf(hi, fmaxf(p[k].x, fmaxf(p[k].y, p[k].z)));
                }
            }
        }
        if (__any_sync(0xFFFFFFFFu, bad) && (threadIdx.x & 31) == 0)
            atomicOr(status, GCS_DEV_NONFINITE_POSITION);
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
        }
        const int w = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) {
            s_lo[w] = lo;
            s_hi[w] = hi;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
                lo = fminf(lo, s_lo[k]);
                hi = fmaxf(hi, s_hi[k]);
            }
            atomicMax(bounds_enc + 2 * ch.seg, ~float_to_ordered(lo));
            atomicMax(bounds_enc + 2 * ch.seg + 1, float_to_ordered(hi));
        }
        __syncthreads();
    }
}

__global__ void bounds_decode_kernel(const uint32_t* __restrict__ enc, float2* __restrict__ out,
                                     int nseg) {
    let_next_start();
    wait_for_previous();
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x)
        out[s] = make_float2(ordered_to_float(~enc[2 * s]), ordered_to_float(enc[2 * s + 1]));
}

// keys[i] = 63-bit Morton code of particle i in its segment's cube; idx[i] = i
// (karras_bvh.cuh:34-41).  The radix sort's global digit histograms (8 key
// digits, plus the segment-id digits when there is more than one segment)
// are accumulated here in shared memory, so the sort needs no separate
// counting pass over the keys.
__global__ void __launch_bounds__(kCountThreads, 2)
encode_kernel(Layout L, const float4* __restrict__ pos, int bounds_mode,
                              float gmin, float gmax, const float2* __restrict__ seg_bounds,
                              uint64_t* __restrict__ keys, uint32_t* __restrict__ idx,
                              uint32_t* __restrict__ hist, int n_seg_passes) {
    __shared__ uint32_t s_hist[kMaxPasses][kRadix];
    const int passes = kKeyPasses + n_seg_passes;
    let_next_start();
    for (int t = threadIdx.x; t < passes * kRadix; t += blockDim.x) (&s_hist[0][0])[t] = 0;
    __syncthreads();
    wait_for_previous();
    float lo = gmin, scale = 0.0f;
    int cur_seg = -1;
    if (bounds_mode == GCS_BOUNDS_CALLER) scale = morton_scale(gmin, gmax);
    // whole warps go round together (count_digits)
    for (int base = blockIdx.x * kCountThreads + (threadIdx.x & ~31); base < L.n; base += gridDim.x * kCountThreads) {
        const int i = base + (threadIdx.x & 31);
        const bool valid = i < L.n;
        uint64_t k = 0ull;
        int seg = 0;
        if (valid) {
            const float4 p = __ldg(pos + i);
            seg = (L.nseg > 1) ? __ldg(L.seg_id + i) : 0;
            if (bounds_mode != GCS_BOUNDS_CALLER && seg != cur_seg) {
                const float2 b = __ldg(seg_bounds + seg);
                lo = b.x;
                scale = morton_scale(b.x, b.y);
                cur_seg = seg;
            }
            k = morton63(p.x, p.y, p.z, lo, scale);
            keys[i] = k;
            idx[i] = (uint32_t)i;
        }
        count_digits(s_hist, k, valid);
        if (valid)
            for (int d = 0; d < n_seg_passes; ++d)
                atomicAdd(&s_hist[kKeyPasses + d][((uint32_t)seg >> (kRadixBits * d)) & (kRadix - 1)], 1u);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < passes * kRadix; t += blockDim.x) {
        const uint32_t c = (&s_hist[0][0])[t];
        if (c) atomicAdd(hist + t, c);
    }
}

// Permute the particle state into sorted order (karras_bvh.cuh:44-70):
// out[k] = in[idx[k]] for the two 16-byte records.
__global__ void gather_kernel(const uint32_t* __restrict__ idx, const float4* __restrict__ pos_in,
                              const float4* __restrict__ vel_in, float4* __restrict__ pos_out,
                              float4* __restrict__ vel_out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t s = __ldg(idx + i);
        if ((int64_t)s >= n) continue;  // only after a sort that timed out (in the status word)
        pos_out[i] = __ldg(pos_in + s);
        vel_out[i] = __ldg(vel_in + s);
    }
}

// v += a dt; x += v dt; recolour types 0/2 by speed (kick_drift,
// cuda_engine.cu:164-216), in place.
__global__ void integrate_kernel(float4* __restrict__ pos, float4* __restrict__ vel,
                                 const float4* __restrict__ acc, float dt, int recolor, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 a = __ldg(acc + i);
        float4 v = vel[i];
        float4 p = pos[i];
        kick_drift(p, v, a, dt, recolor);
        vel[i] = v;
        pos[i] = p;
    }
}

__global__ void kick_kernel(float4* __restrict__ vel, const float4* __restrict__ acc, float dt,
                            int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 a = __ldg(acc + i);
        float4 v = vel[i];
        v.x = __fmaf_rn(a.x, dt, v.x);
        v.y = __fmaf_rn(a.y, dt, v.y);
        v.z = __fmaf_rn(a.z, dt, v.z);
        vel[i] = v;
    }
}

// FP64 kinetic energy, momentum, mass and potential energy of particles
// [first, first+n).  out = {KE, px, py, pz, M, PE}; PE = 0.5 sum m phi with
// phi from the walk's potential lane (acc.w).  Blocks reduce in shared
// memory and add with FP64 atomics.
// Velocities enter as v + a * kick (in FP64): kick = dt/2 turns the stored
// half-step velocities of the leapfrog into synchronised ones.
__global__ void diag_kernel(const float4* __restrict__ pos, const float4* __restrict__ vel,
                            const float4* __restrict__ accp, int64_t first, int64_t n, double kick,
                            double* __restrict__ out) {
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = __ldg(pos + first + i);
        const float4 v = __ldg(vel + first + i);
        const float4 a = __ldg(accp + first + i);
        const double m = p.w;
        const double vx = (double)v.x + (double)a.x * kick;
        const double vy = (double)v.y + (double)a.y * kick;
        const double vz = (double)v.z + (double)a.z * kick;
        acc[0] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        acc[1] += m * vx;
        acc[2] += m * vy;
        acc[3] += m * vz;
        acc[4] += m;
        acc[5] += 0.5 * m * (double)a.w;
    }
    __shared__ double s[6][kStreamThreads / 32];
    for (int k = 0; k < 6; ++k) {
        double x = acc[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
        if ((threadIdx.x & 31) == 0) s[k][threadIdx.x >> 5] = x;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double x = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += s[threadIdx.x][w];
        atomicAdd(out + threadIdx.x, x);
    }
}

// g x^(-3/2) to double precision: the hardware estimate y of x^(-1/2), with
// e = 1 - x y^2, and the first terms of the binomial series
// x^(-3/2) = y^3 (1 - e)^(-3/2) = y^3 (1 + 3/2 e + 15/8 e^2 + ...).  The
// estimate is good to about 2^-20, which leaves a term below 2^-55.  An
// infinite or zero x and an infinite g give NaN (direct_nonfinite_kernel).
__device__ __forceinline__ double times_inv_r3(double g, double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double y2 = y * y;
    const double e = fma(-x, y2, 1.0);
    const double a = (g * y) * y2;
    return fma(a * e, fma(e, 1.875, 1.5), a);
}

// FP64 direct sum, excluding only the target itself: a block takes
// kTargets targets (held in registers, with their sums) and every
// kDirectThreads-th source of its split of the segment; the splits' sums are
// added in order by direct_sum_kernel.  Only sources between the block's
// first and last target can be one of its targets; the others are summed
// without the test.
//
// Bound by the FP64 pipe: 16 instructions a pair (the earlier kernel, a block
// per target with a software square root and divide and four conversions for
// every pair, needed about three times as many).  4,096 targets of 262,144
// particles: 2.86 ms before, 1.41 ms now (800 G pairs/s at 65,536
// targets, 69 % of the pipe at 1,965 MHz); 3, 6 and 8 targets a block 1.46, 1.35
// and 2.1 ms, 6 slower where targets are few.  Up to eight targets an SM the
// chip is not full and a call takes as long as a block: two a block then
// (16 targets of 1,000 particles, whole call: 35.5 us with four, 28.9 with two,
// 30.5 with the earlier kernel; 1,000 of 262,144: 403 and 394; 4,000 of 30,000:
// 213 and 224).
constexpr int kDirectThreads = 128;
constexpr int kDirectTargets = 4;
constexpr int kDirectFewTargets = 2;

template <int kTargets>
__global__ void __launch_bounds__(kDirectThreads)
direct_fp64_kernel(const float4* __restrict__ pos, int64_t seg_first, int64_t seg_n,
                   const int64_t* __restrict__ targets, int64_t n_targets, int64_t per_split, double G, double eps2,
                   double* __restrict__ sums) {
    double tx[kTargets], ty[kTargets], tz[kTargets];
    double ax[kTargets] = {}, ay[kTargets] = {}, az[kTargets] = {};
    const int64_t first = (int64_t)blockIdx.x * kTargets;
    const auto target = [&](int t) { return __ldg(targets + (first + t < n_targets ? first + t : n_targets - 1)); };
    int64_t t_min = seg_n, t_max = -1;
#pragma unroll
    for (int t = 0; t < kTargets; ++t) {
        const int64_t ti = target(t);
        t_min = ti < t_min ? ti : t_min;
        t_max = ti > t_max ? ti : t_max;
        const float4 p = __ldg(pos + seg_first + ti);
        tx[t] = p.x;
        ty[t] = p.y;
        tz[t] = p.z;
    }
    const int64_t begin = per_split * blockIdx.y, end = begin + per_split < seg_n ? begin + per_split : seg_n;
    for (int64_t j = begin + threadIdx.x; j < end; j += kDirectThreads) {
        const float4 p = __ldg(pos + seg_first + j);
        const double sx = p.x, sy = p.y, sz = p.z, gm = G * (double)p.w;
        if (j < t_min || j > t_max) {
#pragma unroll
            for (int t = 0; t < kTargets; ++t) {
                const double dx = sx - tx[t], dy = sy - ty[t], dz = sz - tz[t];
                const double f = times_inv_r3(gm, fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
                ax[t] = fma(f, dx, ax[t]);
                ay[t] = fma(f, dy, ay[t]);
                az[t] = fma(f, dz, az[t]);
            }
        } else {
#pragma unroll
            for (int t = 0; t < kTargets; ++t) {
                const double dx = sx - tx[t], dy = sy - ty[t], dz = sz - tz[t];
                const double f = times_inv_r3(gm, fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
                if (j != target(t)) {
                    ax[t] = fma(f, dx, ax[t]);
                    ay[t] = fma(f, dy, ay[t]);
                    az[t] = fma(f, dz, az[t]);
                }
            }
        }
    }
    __shared__ double s[3 * kTargets][kDirectThreads / 32];
#pragma unroll
    for (int t = 0; t < kTargets; ++t) {
        for (int o = 16; o > 0; o >>= 1) {
            ax[t] += __shfl_xor_sync(0xFFFFFFFFu, ax[t], o);
            ay[t] += __shfl_xor_sync(0xFFFFFFFFu, ay[t], o);
            az[t] += __shfl_xor_sync(0xFFFFFFFFu, az[t], o);
        }
        if ((threadIdx.x & 31) == 0) {
            s[3 * t][threadIdx.x >> 5] = ax[t];
            s[3 * t + 1][threadIdx.x >> 5] = ay[t];
            s[3 * t + 2][threadIdx.x >> 5] = az[t];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 * kTargets && first + threadIdx.x / 3 < n_targets) {
        double x = 0;
        for (int w = 0; w < kDirectThreads / 32; ++w) x += s[threadIdx.x][w];
        sums[3 * (n_targets * blockIdx.y + first) + threadIdx.x] = x;
    }
}

// Sums with a NaN component again, a block per target, term by term as written
// down: a source infinitely far away adds NaN to the components in which it is
// and nothing to the others, where times_inv_r3 makes all three NaN.  Launched
// only where the caller has seen a NaN (the choice made inside
// direct_fp64_kernel, by pair, by source or after its loop: 1,545 us in place
// of 1,395).
__global__ void __launch_bounds__(kStreamThreads)
direct_nonfinite_kernel(const float4* __restrict__ pos, int64_t seg_first, int64_t seg_n,
                        const int64_t* __restrict__ targets, int64_t n_targets, double G, double eps2,
                        double* __restrict__ out) {
    __shared__ double s[3][kStreamThreads / 32];
    for (int64_t t = blockIdx.x; t < n_targets; t += gridDim.x) {
        if (!isnan(out[3 * t]) && !isnan(out[3 * t + 1]) && !isnan(out[3 * t + 2])) continue;  // the same in all threads
        const int64_t ti = __ldg(targets + t);
        const float4 q = __ldg(pos + seg_first + ti);
        double a[3] = {0.0, 0.0, 0.0};
        for (int64_t j = threadIdx.x; j < seg_n; j += kStreamThreads) {
            if (j == ti) continue;
            const float4 p = __ldg(pos + seg_first + j);
            const double dx = (double)p.x - q.x, dy = (double)p.y - q.y, dz = (double)p.z - q.z;
            const double inv = 1.0 / sqrt(dx * dx + dy * dy + dz * dz + eps2);
            const double f = G * (double)p.w * inv * inv * inv;
            a[0] += f * dx;
            a[1] += f * dy;
            a[2] += f * dz;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xFFFFFFFFu, a[k], o);
            if ((threadIdx.x & 31) == 0) s[k][threadIdx.x >> 5] = a[k];
        }
        __syncthreads();  // (also: every thread has read out)
        if (threadIdx.x < 3) {
            double x = 0.0;
            for (int w = 0; w < kStreamThreads / 32; ++w) x += s[threadIdx.x][w];
            out[3 * t + threadIdx.x] = x;
        }
        __syncthreads();
    }
}

__global__ void direct_sum_kernel(const double* __restrict__ sums, int splits, int64_t n, double* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x = sums[i];
    for (int k = 1; k < splits; ++k) x += sums[n * k + i];
    out[i] = x;
}

}  // namespace

void launch_fill_segment_ids(const int64_t* seg_off, int nseg, int32_t* seg_id, int64_t n,
                             cudaStream_t st) {
    if (n <= 0) return;
    fill_segment_ids_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(seg_off, nseg, seg_id, n);
}

void launch_unpack_stars(const Star* stars, float4* pos, float4* vel, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    unpack_stars_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(
        reinterpret_cast<const float4*>(stars), pos, vel, n);
}

void launch_pack_stars(const float4* pos, const float4* vel, Star* out, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    pack_stars_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(pos, vel,
                                                                 reinterpret_cast<float4*>(out), n);
}

void launch_pack_playback(const float4* pos, const float4* vel, PlaybackStar* out, int64_t n,
                          cudaStream_t st) {
    if (n <= 0) return;
    pack_playback_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(
        pos, vel, reinterpret_cast<float4*>(out), n);
}

void launch_bounds(const Layout& L, const float4* pos, const Chunk* chunks, int n_chunks,
                   uint32_t* bounds_enc, uint32_t* status, cudaStream_t st) {
    if (n_chunks <= 0) return;
    int grid = stream_grid(L.n);
    if (grid > n_chunks) grid = n_chunks;
    launch_after(bounds_kernel, grid, kStreamThreads, 0, st, pos, chunks, n_chunks, bounds_enc, status);
}

void launch_bounds_decode(const uint32_t* bounds_enc, float2* bounds, int nseg, cudaStream_t st) {
    launch_after(bounds_decode_kernel, (nseg + 255) / 256, 256, 0, st, bounds_enc, bounds, nseg);
}

void launch_encode(const Layout& L, const float4* pos, int bounds_mode, float gmin, float gmax,
                   const float2* seg_bounds, uint64_t* keys, uint32_t* idx, uint32_t* hist,
                   int n_seg_passes, cudaStream_t st) {
    if (L.n <= 0) return;
    launch_after(encode_kernel, count_grid(L.n, current_sm_count()), kCountThreads, 0, st, L, pos, bounds_mode, gmin, gmax, seg_bounds,
                 keys, idx, hist, n_seg_passes);
}

void launch_gather(const uint32_t* idx, const float4* pos_in, const float4* vel_in, float4* pos_out,
                   float4* vel_out, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    gather_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(idx, pos_in, vel_in, pos_out, vel_out,
                                                             n);
}

void launch_integrate(float4* pos, float4* vel, const float4* acc, float dt, int recolor,
                      int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    integrate_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(pos, vel, acc, dt, recolor, n);
}

void launch_kick(float4* vel, const float4* acc, float dt, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    kick_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(vel, acc, dt, n);
}

void launch_diag(const float4* pos, const float4* vel, const float4* acc, int64_t first, int64_t n,
                 double kick, double* out6, cudaStream_t st) {
    if (n <= 0) return;
    diag_kernel<<<stream_grid(n), kStreamThreads, 0, st>>>(pos, vel, acc, first, n, kick, out6);
}

// Splits of the sources: enough blocks for several waves (three 128-thread
// blocks are resident on an SM), but at least 1,024 sources for each.
int direct_splits(int64_t seg_n, int64_t n_targets) {
    const int64_t tiles = (n_targets + kDirectTargets - 1) / kDirectTargets;
    const int64_t want = ((int64_t)current_sm_count() * 24 + tiles - 1) / tiles;
    return (int)std::max<int64_t>(1, std::min<int64_t>({want, seg_n / 1024, kDirectMaxSplits}));
}

void launch_direct_fp64(const float4* pos, int64_t seg_first, int64_t seg_n, const int64_t* targets,
                        int64_t n_targets, int splits, double G, double eps2, double* sums, double* out,
                        cudaStream_t st) {
    if (n_targets <= 0) return;
    double* to = splits > 1 ? sums : out;
    const int64_t per_split = (seg_n + splits - 1) / splits;
    const auto blocks = [&](int per) { return dim3((unsigned)((n_targets + per - 1) / per), (unsigned)splits); };
    if (n_targets <= (int64_t)current_sm_count() * 8)
        direct_fp64_kernel<kDirectFewTargets><<<blocks(kDirectFewTargets), kDirectThreads, 0, st>>>(
            pos, seg_first, seg_n, targets, n_targets, per_split, G, eps2, to);
    else
        direct_fp64_kernel<kDirectTargets><<<blocks(kDirectTargets), kDirectThreads, 0, st>>>(
            pos, seg_first, seg_n, targets, n_targets, per_split, G, eps2, to);
    if (splits > 1)
        direct_sum_kernel<<<(unsigned)((3 * n_targets + 255) / 256), 256, 0, st>>>(sums, splits, 3 * n_targets, out);
}

void launch_direct_nonfinite(const float4* pos, int64_t seg_first, int64_t seg_n, const int64_t* targets,
                             int64_t n_targets, double G, double eps2, double* out, cudaStream_t st) {
    const int64_t cap = (int64_t)current_sm_count() * 16;
    direct_nonfinite_kernel<<<(unsigned)std::min(n_targets, cap), kStreamThreads, 0, st>>>(pos, seg_first, seg_n, targets,
                                                                                         n_targets, G, eps2, out);
}

}  // namespace gcs
