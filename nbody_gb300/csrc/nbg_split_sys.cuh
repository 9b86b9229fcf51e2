// nbg_split_sys.cuh -- a body system prepared for two-word arithmetic
// (nbg_split.cuh): scaled bodies and, per body, the scale of its sum.  Used by
// the FP64 direct sum (nbg_direct.cu), the FP64 Barnes-Hut walk (nbg_bh.cu) and
// the potential energy (nbg_stats.cu).
#pragma once

#include <cmath>

#include "nbg_internal.cuh"
#include "nbg_split.cuh"

namespace nbg {
namespace {

constexpr float kSplitNear = 1.f / 1024.f;   // of a body's scale: larger terms go to FP64
constexpr float kSplitFarP = 1.0995116e12f;  // 2^40: 1 / r^2 of the closest two-word pair
constexpr int kSplitT = 128;                 // threads per CTA, 2 bodies each
constexpr int kSplitTile = 64;               // j-bodies per shared-memory tile
constexpr int kSplitQ = 16;                  // queued FP64 pairs per body
constexpr int kSplitChunk = 8;               // j-bodies between two looks at the queues
constexpr int kSplitExtents = 64;            // CTAs of split_extent_kernel
constexpr int kSplitEst = 8;                 // ranges of split_estimate_kernel
constexpr int kSplitMaxSample = 256;         // least sample: 32 of every 8192 bodies

// One body of the FP64 sum: a += m_j d r^-3, r^2 at least kMinDistance (16 FP64
// operations; the reference's pair force, nbody/nbody_data.cpp:35-44, without
// its multiplication and division by m_i).
__device__ __forceinline__ void pair_fp64(double dx, double dy, double dz, double m, double& ax,
                                          double& ay, double& az) {
    const double r2 = fmax(fma(dx, dx, fma(dy, dy, dz * dz)), kMinDistance);
    const double w = m * rcube_fp64(r2);
    ax = fma(dx, w, ax);
    ay = fma(dy, w, ay);
    az = fma(dz, w, az);
}

// The reference forms the force with m_i and divides by m_i again: for a
// massless or non-finite m_i that is NaN, but for a lone body, whose force is 0.
__device__ __forceinline__ double fp64_result(double a, double m, int n) {
    if (m != 0.0 && fabs(m) <= 1.7976931348623157e308) return a;
    return (n == 1 ? 0.0 : a * m) / m;
}

struct SplitBody {  // 48 bytes
    float4 a;       // xh xm xl yh
    float4 b;       // ym yl zh zm
    float4 c;       // zl mh ml |m|
};

struct SplitSystem {
    const double* y;             // [3][n] coordinates
    const double* mass;
    SplitBody* bodies;           // [n_pad], padding far away and massless
    float* est;                  // [kSplitEst][n_pad] sampled scales, scaled units
    unsigned long long* extent;  // [kSplitExtents] bits of max |coordinate|
    double eps2;                 // softening, 0 = none
    double mass_scale;           // power of two: largest |m| into [1/2, 1)
    int mass_exp;                // mass_scale = 2^-mass_exp
    int n, n_pad;                // n_pad: a multiple of 2 kSplitT
    int sample;                  // the estimate takes 32 of every 32 sample bodies
};

__global__ void __launch_bounds__(256) split_extent_kernel(SplitSystem a) {
    if (!after_previous()) return;
    unsigned long long m = 0;
    const size_t n3 = 3 * (size_t)a.n;
    for (size_t i = blockIdx.x * 256 + threadIdx.x; i < n3; i += (size_t)gridDim.x * 256)
        m = max(m, (unsigned long long)__double_as_longlong(fabs(a.y[i])));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ unsigned long long w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) m = max(m, w[k]);
        a.extent[blockIdx.x] = m;
    }
}

// exponent E with every |coordinate| < 2^E (in every thread; 2048 for a
// coordinate that is not finite)
__device__ __forceinline__ int split_exponent(const SplitSystem& a) {
    unsigned long long m = 0;
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < kSplitExtents; k += 32) m = max(m, __ldg(a.extent + k));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int ex = (int)(m >> 52);
    return ex == 0x7ff ? 2048 : ex - 1022;
}

// |m| of a scaled mass as the near test reads it: NaN, so that FP64 takes all of
// its terms, for a mass far below the largest and for one that is not finite
// (whose two words would be inf - inf).
__device__ __forceinline__ float split_mass_size(double ms) {
    const double a = fabs(ms);
    const bool words = ms == 0.0 || (a >= 9.313225746154785e-10 && a <= 1.7976931348623157e308);  // 2^-30
    return words ? (float)a : __int_as_float(0x7fffffff);
}

__global__ void __launch_bounds__(256) split_pack_kernel(SplitSystem a) {
    if (!after_previous()) return;
    const int ex = split_exponent(a);
    for (int i = blockIdx.x * 256 + threadIdx.x; i < a.n_pad; i += gridDim.x * 256) {
        SplitBody b;
        if (i < a.n) {
            float h[3], m[3], l[3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                split3(ex == 2048 ? nan("") : scalbn(a.y[(size_t)c * a.n + i], -ex), h[c], m[c], l[c]);
            const double ms = a.mass[i] * a.mass_scale;
            const float mh = (float)ms, ml = split_word(ms - (double)mh, (unsigned)i);
            b.a = make_float4(h[0], m[0], l[0], h[1]);
            b.b = make_float4(m[1], l[1], h[2], m[2]);
            b.c = make_float4(l[2], mh, ml, split_mass_size(ms));
        } else {
            // padding: massless, and so far away that r^-3 underflows to 0
            b.a = make_float4(1e18f, 0.f, 0.f, 1e18f);
            b.b = make_float4(0.f, 0.f, 1e18f, 0.f);
            b.c = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        a.bodies[i] = b;
    }
}

// Per body, the sum of |m_j| / r^2 (POT: of |m_j| / r, softened) over a sample of
// the others, 32 bodies of every 32 a.sample (a sum without cancellation, so
// neither the sample nor a body in the middle of a symmetric system changes its
// scale much).  256 bodies per CTA against one of kSplitEst ranges, in FP32x2.
// A close neighbour in the sample stands for a.sample bodies and raises the
// limit: it is above it itself as long as a.sample kSplitNear < 1, but other
// terms up to that fraction of it are then taken in two words (a quarter of it
// from 2^20 bodies on: 1 / 4 of 1e-14, what a serial FP64 sum of 5000 terms rounds
// off).  Counting it once lowers the limit of all bodies: no smaller errors at
// 1536 to 20011 bodies and up to 10 % more time (1536: 85 -> 94 us).
template <bool POT>
__global__ void __launch_bounds__(kSplitT) split_estimate_kernel(SplitSystem a) {
    if (!after_previous()) return;
    __shared__ __align__(16) float4 tile[kSplitT][2];
    const int tid = threadIdx.x;
    const int i0 = blockIdx.x * 2 * kSplitT + tid, i1 = i0 + kSplitT;  // < n_pad
    const SplitBody p = a.bodies[i0], q = a.bodies[i1];
    const f2_t xi = f2_pack(p.a.x, q.a.x), yi = f2_pack(p.a.w, q.a.w), zi = f2_pack(p.b.z, q.b.z);
    constexpr float kLeast = 1.f / kSplitFarP;  // closer pairs (the body itself) do not count
    const float eps2 = POT ? (float)scalbn(a.eps2, -2 * min(split_exponent(a), 1000)) : 0.f;
    f2_t sum = f2_pack(0.f, 0.f);
    const uint32_t base = smem_addr(tile);
    // 4 runs of 32 bodies per tile
    const int runs = a.n_pad / 32, tiles = (runs / a.sample + 3) / 4;
    for (int q = blockIdx.y; q < max(tiles, 1); q += gridDim.y) {
        const int run = (q * 4 + (tid >> 5)) * a.sample;
        __syncthreads();
        SplitBody b = a.bodies[min(run, runs - 1) * 32 + (tid & 31)];
        if (run >= runs) b.c.y = 0.f;
        // (a mass that is not finite does not count: the scale stays finite)
        const float m = fabsf(b.c.y) <= 1.f ? fabsf(b.c.y) : 0.f;
        tile[tid][0] = make_float4(b.a.x, b.a.x, b.a.w, b.a.w);
        tile[tid][1] = make_float4(b.b.z, b.b.z, m, m);
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kSplitT; ++k) {
            const float4 u = lds128(base + 32u * k), v = lds128(base + 32u * k + 16u);
            const f2_t dx = f2_sub(f2_pack(u.x, u.y), xi), dy = f2_sub(f2_pack(u.z, u.w), yi);
            const f2_t dz = f2_sub(f2_pack(v.x, v.y), zi);
            float r0, r1;
            f2_unpack(f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz))), r0, r1);
            const float t0 = r0 <= kLeast ? 0.f : POT ? rsqrt_mufu(r0 + eps2) : rcp_mufu(r0);
            const float t1 = r1 <= kLeast ? 0.f : POT ? rsqrt_mufu(r1 + eps2) : rcp_mufu(r1);
            sum = f2_fma(f2_pack(v.z, v.w), f2_pack(t0, t1), sum);
        }
    }
    float s0, s1;
    f2_unpack(sum, s0, s1);
    a.est[(size_t)blockIdx.y * a.n_pad + i0] = s0;
    a.est[(size_t)blockIdx.y * a.n_pad + i1] = s1;
}

__device__ __forceinline__ float split_limit(const SplitSystem& a, int i) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < kSplitEst; ++r) s += __ldg(a.est + (size_t)r * a.n_pad + i);
    return kSplitNear * (float)a.sample * s;
}

// The three words of two bodies, packed.
__device__ __forceinline__ void split_words(const SplitBody& p, const SplitBody& q, f2_t* h, f2_t* m,
                                            f2_t* l) {
    h[0] = f2_pack(p.a.x, q.a.x);
    m[0] = f2_pack(p.a.y, q.a.y);
    l[0] = f2_pack(p.a.z, q.a.z);
    h[1] = f2_pack(p.a.w, q.a.w);
    m[1] = f2_pack(p.b.x, q.b.x);
    l[1] = f2_pack(p.b.y, q.b.y);
    h[2] = f2_pack(p.b.z, q.b.z);
    m[2] = f2_pack(p.b.w, q.b.w);
    l[2] = f2_pack(p.c.x, q.c.x);
}
__device__ __forceinline__ void split_load(const SplitSystem& a, int i0, int i1, f2_t* h, f2_t* m,
                                           f2_t* l) {
    split_words(a.bodies[i0], a.bodies[i1], h, m, l);
}

// A shared-memory tile holds every word twice, for FP32x2: the first
// kSplitTile threads of the CTA write one body each.
__device__ __forceinline__ void split_store_tile(float4 (*tile)[6], const SplitBody& b) {
    float4* t = tile[threadIdx.x];
    t[0] = make_float4(b.a.x, b.a.x, b.a.y, b.a.y);
    t[1] = make_float4(b.a.z, b.a.z, b.a.w, b.a.w);
    t[2] = make_float4(b.b.x, b.b.x, b.b.y, b.b.y);
    t[3] = make_float4(b.b.z, b.b.z, b.b.w, b.b.w);
    t[4] = make_float4(b.c.x, b.c.x, b.c.y, b.c.y);
    t[5] = make_float4(b.c.z, b.c.z, b.c.w, b.c.w);
}

// One body of a tile against two: the difference vectors; its mass words.
struct SplitPair {
    f2_t d1[3], d2[3], mh, ml, mabs;
};
__device__ __forceinline__ SplitPair split_pair(uint32_t at, const f2_t* h, const f2_t* m,
                                                const f2_t* l) {
    const float4 w0 = lds128(at), w1 = lds128(at + 16), w2 = lds128(at + 32);
    const float4 w3 = lds128(at + 48), w4 = lds128(at + 64), w5 = lds128(at + 80);
    SplitPair s;
    split_diff(f2_pack(w0.x, w0.y), f2_pack(w0.z, w0.w), f2_pack(w1.x, w1.y), h[0], m[0], l[0],
               s.d1[0], s.d2[0]);
    split_diff(f2_pack(w1.z, w1.w), f2_pack(w2.x, w2.y), f2_pack(w2.z, w2.w), h[1], m[1], l[1],
               s.d1[1], s.d2[1]);
    split_diff(f2_pack(w3.x, w3.y), f2_pack(w3.z, w3.w), f2_pack(w4.x, w4.y), h[2], m[2], l[2],
               s.d1[2], s.d2[2]);
    s.mh = f2_pack(w4.z, w4.w);
    s.ml = f2_pack(w5.x, w5.y);
    s.mabs = f2_pack(w5.z, w5.w);
    return s;
}

// Scratch of a system of n bodies, in bytes (a multiple of 16), and its place.
size_t split_bytes(SplitSystem* a, int n) {
    a->n = n;
    a->n_pad = (n + 2 * kSplitT - 1) / (2 * kSplitT) * (2 * kSplitT);
    a->sample = 4;
    while (a->n_pad / a->sample > 4096 && a->sample < kSplitMaxSample) a->sample *= 2;
    return (size_t)a->n_pad * (sizeof(SplitBody) + kSplitEst * sizeof(float)) +
           kSplitExtents * sizeof(unsigned long long);
}

// The system at `at` (split_bytes of scratch): three launches.
template <bool POT>
nbg_status split_prepare(nbg_engine* e, SplitSystem* a, const double* y, const double* mass,
                         double eps2, void* at) {
    a->y = y;
    a->mass = mass;
    a->eps2 = eps2;
    a->mass_exp = e->mass_exp;
    a->mass_scale = std::ldexp(1.0, -e->mass_exp);
    a->bodies = static_cast<SplitBody*>(at);
    a->extent = reinterpret_cast<unsigned long long*>(a->bodies + a->n_pad);
    a->est = reinterpret_cast<float*>(a->extent + kSplitExtents);
    queued(split_extent_kernel, kSplitExtents, 256, 0, e->stream)(*a);
    NBG_LAUNCHED(e, "split_extent_kernel");
    queued(split_pack_kernel, grid_for(a->n_pad, 256, (unsigned)e->sm_count * 8u), 256, 0, e->stream)(*a);
    NBG_LAUNCHED(e, "split_pack_kernel");
    const dim3 grid((unsigned)(a->n_pad / (2 * kSplitT)), kSplitEst);
    queued(split_estimate_kernel<POT>, grid, kSplitT, 0, e->stream)(*a);
    NBG_LAUNCHED(e, "split_estimate_kernel");
    return NBG_OK;
}

}  // namespace
}  // namespace nbg
