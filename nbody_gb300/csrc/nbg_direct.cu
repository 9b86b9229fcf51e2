// nbg_direct.cu -- direct O(N^2) gravity: f = [v ; a(y)].
//
// Four paths share the engine entry point:
//
//  * FP64 (parity) -- the reference 'simple' engine's sum
//    (nbody/nbody_engine_simple.cpp:143-172 with nbody_data::force,
//    nbody/nbody_data.cpp:35-44) to FP64 rounding, self pair skipped.  Its
//    rounding errors are smaller than those of the reference's serial sum
//    (measured against extended precision), because the partial sums are.
//    Small systems: one warp per body on the FP64 pipe (direct_fp64_kernel);
//    larger ones: two-word FP32 arithmetic, with the terms that matter taken
//    in FP64 (split_force_kernel).  Both repeat bit for bit.
//
//  * mixed (throughput) -- FP32 pair math on the FP32 pipe, FP64 state.
//    A pack kernel turns y into a tile-padded array of bodies in
//    (x x y y | z z m m) form and writes f = [v ; 0].  The force kernel is
//    persistent: the (i-block, j-tile) units are split evenly over one wave
//    of CTAs (stream-K), thread 0 streams j-tiles global -> shared with 1-D
//    bulk async copies (TMA) through a 4-stage mbarrier ring, and the 4 warps
//    each hold 2G i-bodies per lane (G = 2 or 4 packed pairs) in FP32x2
//    registers.  Per
//    tile the FP32 partial sums are folded into a (hi, lo) two-sum pair; at
//    the end of an i-block segment hi + lo is added into the FP64 a-part of f
//    with one atomicAdd per component.  Pair term:
//        a_i += m_j (r_j - r_i) / (|r_j - r_i|^2 + eps^2)^{3/2}
//    with r^2 clamped to >= 1e-8 when eps = 0 (the reference clamp).
//
//  * mixed, symmetric (the default, tuning key direct.symmetric = 1) -- the
//    same arithmetic with every unordered pair evaluated once and applied to
//    both bodies (details at direct_sym_kernel).
//
//  * mixed, small systems (tuning key direct.small) -- ordered pairs again, a
//    block of bodies' sums leaving its CTA once (direct_small_kernel).
#include <algorithm>
#include <cmath>
#include <mutex>

#include "nbg_internal.cuh"
#include "nbg_pair.cuh"
#include "nbg_ptx.cuh"
#include "nbg_split_sys.cuh"

namespace nbg {
namespace {

template <bool CLAMP>
__device__ __forceinline__ void pair2(f2_t xj, f2_t yj, f2_t zj, f2_t mj, f2_t xi, f2_t yi,
                                      f2_t zi, f2_t eps2, f2_t& ax, f2_t& ay, f2_t& az) {
    const f2_t dx = f2_sub(xj, xi);
    const f2_t dy = f2_sub(yj, yi);
    const f2_t dz = f2_sub(zj, zi);
    f2_t r2 = f2_fma(dz, dz, eps2);
    r2 = f2_fma(dy, dy, r2);
    r2 = f2_fma(dx, dx, r2);
    float r2a, r2b;
    f2_unpack(r2, r2a, r2b);
    if (CLAMP) {
        r2a = fmaxf(r2a, 1e-8f);
        r2b = fmaxf(r2b, 1e-8f);
    }
    const f2_t inv = f2_pack(rsqrt_mufu(r2a), rsqrt_mufu(r2b));
    const f2_t inv2 = f2_mul(inv, inv);
    const f2_t s = f2_mul(mj, inv);
    const f2_t s3 = f2_mul(s, inv2);
    ax = f2_fma(dx, s3, ax);
    ay = f2_fma(dy, s3, ay);
    az = f2_fma(dz, s3, az);
}

// ---------------------------------------------------------------------------
// FP64 kernels
// ---------------------------------------------------------------------------
// Small systems (and any size, where the split path's scratch cannot be had):
// one warp per body, the other bodies across its lanes, the 32 partial sums
// added by shuffles in a fixed order.
constexpr int kF64Threads = 32;  // one warp per CTA: the fewest idle SMs in the last wave

__global__ void __launch_bounds__(kF64Threads)
direct_fp64_kernel(const double* __restrict__ y, const double* __restrict__ mass,
                   double* __restrict__ f, int n) {
    if (!after_previous()) return;
    const int lane = threadIdx.x & 31;
    const int i = (int)((blockIdx.x * kF64Threads + threadIdx.x) >> 5);
    if (i >= n) return;
    const size_t sn = (size_t)n;
    const double x1 = y[i], y1 = y[sn + i], z1 = y[2 * sn + i];
    double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll 4
    for (int j = lane; j < n; j += 32) {
        if (j == i) continue;  // nbody/nbody_engine_simple.cpp:155-158
        pair_fp64(__ldg(y + j) - x1, __ldg(y + sn + j) - y1, __ldg(y + 2 * sn + j) - z1,
                  __ldg(mass + j), ax, ay, az);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (lane < 3) {
        f[lane * sn + i] = y[(3 + lane) * sn + i];
        f[(3 + lane) * sn + i] = fp64_result(lane == 0 ? ax : lane == 1 ? ay : az, mass[i], n);
    }
}

// The FP64 sum on the FP32 pipe (nbg_split.cuh), for all but small systems.
// Terms above kSplitNear of the sum of a body's |m_j| / r^2, and pairs closer
// than 2^-20 of the system's extent or than the clamp, are queued and taken
// in FP64: some 45 of 20011 bodies.  The rest are in two words, each off by
// up to 1e-14 of itself at random; as none of them is large, that adds up to
// a few 1e-16 of the sum, below what a serial FP64 sum of as many terms
// rounds off.
//   split_extent_kernel    max |coordinate|
//   split_pack_kernel      scaled three-word coordinates, two-word masses
//   split_estimate_kernel  the scale of each body's sum
//   split_force_kernel     the sums of every (256 bodies) x (range of bodies)
//   split_reduce_kernel    their total in range order: equal states give
//                          equal forces
//
// Bound by the FP32 pipe: about 101 packed operations a pair (two bodies at
// once), 79 % of the pipe's cycles used, the FP64 pipe 24 % beside it.  At
// 20011 bodies 1.49 ms (the FP64 pipe alone, 16 operations a pair: 12.3 ms;
// the reference's divide and square root in body order: 46.7 ms), RMS error
// 8e-16 of |a| against 3.6e-15 for the serial FP64 sum.  Taking terms above
// 1 / 2048 or 1 / 4096 in FP64 instead costs 3 % and 15 % at that size (35 %
// and 100 % at 2048 bodies) for an error of 7e-16 and 6e-16.
struct SplitArgs {
    SplitSystem s;
    double* f;
    double* part;       // [ranges][3][n]
    int range, ranges;  // range: j-bodies per CTA, a multiple of kSplitTile
};

template <bool UNI>
__global__ void __launch_bounds__(kSplitT, 4) split_force_kernel(SplitArgs a) {
    if (!after_previous()) return;
    __shared__ __align__(16) float4 tile[kSplitTile][6];  // every word twice, for FP32x2
    __shared__ unsigned queue[2][kSplitQ][kSplitT];
    const int tid = threadIdx.x;
    const SplitSystem& s = a.s;
    const size_t sn = (size_t)s.n;
    const int i0 = blockIdx.x * 2 * kSplitT + tid, i1 = i0 + kSplitT;  // < n_pad
    f2_t ih[3], im[3], il[3];
    split_load(s, i0, i1, ih, im, il);
    const float lim0 = split_limit(s, i0), lim1 = split_limit(s, i1);
    const int ex = split_exponent(s);
    // pairs at or below the clamp are taken in FP64
    const float far_p = fminf(kSplitFarP, (float)scalbn(0.999 / kMinDistance, 2 * min(max(ex, -400), 400)));
    const f2_t zero = f2_pack(0.f, 0.f);
    f2_t hi[3] = {zero, zero, zero}, lo[3] = {zero, zero, zero};
    double far0[3] = {0, 0, 0}, far1[3] = {0, 0, 0}, near0[3] = {0, 0, 0}, near1[3] = {0, 0, 0};
    int c0 = 0, c1 = 0;  // queued pairs of this thread's two bodies
    const int j_begin = blockIdx.y * a.range, j_end = min(j_begin + a.range, s.n_pad);

    auto flush_queue = [&](int half, int i, int& cnt, double* acc) {
        const int k = min(i, s.n - 1);
        const double x1 = __ldg(s.y + k), y1 = __ldg(s.y + sn + k), z1 = __ldg(s.y + 2 * sn + k);
        while (__any_sync(0xffffffffu, cnt > 0)) {
            if (cnt > 0) {
                const int j = (int)queue[half][--cnt][tid];
                if (j != i && j < s.n)
                    pair_fp64(__ldg(s.y + j) - x1, __ldg(s.y + sn + j) - y1,
                              __ldg(s.y + 2 * sn + j) - z1, __ldg(s.mass + j), acc[0], acc[1],
                              acc[2]);
            }
        }
    };

    for (int j0 = j_begin; j0 < j_end; j0 += kSplitTile) {
        __syncthreads();
        if (tid < kSplitTile) split_store_tile(tile, s.bodies[j0 + tid]);
        __syncthreads();
        const uint32_t base = smem_addr(tile);
#pragma unroll 1
        for (int jc = 0; jc < kSplitTile; jc += kSplitChunk) {
#pragma unroll 2
            for (int j = jc; j < jc + kSplitChunk; ++j) {
                const SplitPair p = split_pair(base + 96u * j, ih, im, il);
                f2_t r1, r2, w, wl;
                split_norm2(p.d1, p.d2, r1, r2);
                const SplitRsqrt v = split_rsqrt(r1, r2);
                split_cube(v, w, wl);
                if (!UNI) {
                    const f2_t c = w;
                    w = f2_mul_rn(p.mh, c);
                    wl = f2_fma(p.ml, c, f2_fma(p.mh, wl, f2_fma(p.mh, c, f2_neg(w))));
                }
                float p0, p1, t0, t1;
                f2_unpack(v.p, p0, p1);
                f2_unpack(f2_mul(v.p, p.mabs), t0, t1);
                const bool is0 = !(t0 <= lim0 && p0 <= far_p);  // NaN counts as near
                const bool is1 = !(t1 <= lim1 && p1 <= far_p);
                if (is0 || is1) {
                    float u0, u1, l0, l1;
                    f2_unpack(w, u0, u1);
                    f2_unpack(wl, l0, l1);
                    if (is0) {
                        queue[0][c0++][tid] = (unsigned)(j0 + j);
                        u0 = l0 = 0.f;
                    }
                    if (is1) {
                        queue[1][c1++][tid] = (unsigned)(j0 + j);
                        u1 = l1 = 0.f;
                    }
                    w = f2_pack(u0, u1);
                    wl = f2_pack(l0, l1);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) split_axpy(hi[k], lo[k], w, wl, p.d1[k], p.d2[k]);
            }
            // the sums join the FP64 totals every 32 bodies: the error of lo grows
            // with the square of their number (the FP64 pipe is idle otherwise)
            if ((jc & 31) == 32 - kSplitChunk) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    float h0, h1, l0, l1;
                    f2_unpack(hi[k], h0, h1);
                    f2_unpack(lo[k], l0, l1);
                    far0[k] += (double)h0 + (double)l0;
                    far1[k] += (double)h1 + (double)l1;
                    hi[k] = lo[k] = zero;
                }
            }
            if (__any_sync(0xffffffffu, c0 > kSplitQ - kSplitChunk)) flush_queue(0, i0, c0, near0);
            if (__any_sync(0xffffffffu, c1 > kSplitQ - kSplitChunk)) flush_queue(1, i1, c1, near1);
        }
    }
    flush_queue(0, i0, c0, near0);
    flush_queue(1, i1, c1, near1);
    // back to the caller's units: lengths 2^ex, masses 2^mass_exp
    const int un = s.mass_exp - 2 * ex;
    const double mu = UNI ? s.mass[0] * s.mass_scale : 1.0;
    double* out = a.part + (size_t)blockIdx.y * 3 * sn;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // (with a coordinate that is not finite every pair is in near)
        if (i0 < s.n) out[k * sn + i0] = near0[k] + (ex == 2048 ? 0.0 : scalbn(far0[k] * mu, un));
        if (i1 < s.n) out[k * sn + i1] = near1[k] + (ex == 2048 ? 0.0 : scalbn(far1[k] * mu, un));
    }
}

__global__ void __launch_bounds__(128) split_reduce_kernel(SplitArgs a) {
    if (!after_previous()) return;
    const size_t sn = (size_t)a.s.n, at = (size_t)blockIdx.x * 128 + threadIdx.x;
    if (at >= 3 * sn) return;
    double s = 0.0;
#pragma unroll 16
    for (int r = 0; r < a.ranges; ++r) s += __ldg(a.part + (size_t)r * 3 * sn + at);
    a.f[at] = a.s.y[3 * sn + at];
    a.f[3 * sn + at] = fp64_result(s, a.s.mass[at % sn], a.s.n);
}

// ---------------------------------------------------------------------------
// mixed kernel
// ---------------------------------------------------------------------------
constexpr int kWarps = 4;                      // warps per CTA (all compute)
constexpr int kThreadsMixed = kWarps * 32;
constexpr int kMinBlocksMixed = 6;             // resident CTAs per SM targeted
constexpr int kT = 128;                        // j-bodies per tile
constexpr int kStages = 4;                     // tiles in flight
constexpr uint32_t kTileBytes = kT * 32;       // 32 bytes per body (x x y y z z m m)

struct Body2 {  // one body in duplicated form, 32 bytes
    float4 xxyy;
    float4 zzmm;
};

__global__ void pack_mixed_kernel(const double* __restrict__ y, const double* __restrict__ mass,
                                  Body2* __restrict__ out, double* __restrict__ f, int n,
                                  int n_pad) {
    if (!after_previous()) return;
    int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += stride) {
        Body2 b;
        if (i < n) {
            float x = (float)y[i], yy = (float)y[n + i], z = (float)y[2 * n + i];
            float m = (float)mass[i];
            b.xxyy = make_float4(x, x, yy, yy);
            b.zzmm = make_float4(z, z, m, m);
            f[i] = y[3 * n + i];
            f[n + i] = y[4 * n + i];
            f[2 * n + i] = y[5 * n + i];
            f[3 * n + i] = 0.0;
            f[4 * n + i] = 0.0;
            f[5 * n + i] = 0.0;
        } else {
            b.xxyy = make_float4(0.f, 0.f, 0.f, 0.f);
            b.zzmm = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        out[i] = b;
    }
}

struct MixedArgs {
    const Body2* bodies;  // [n_pad]
    double* acc;          // a-part of f: [3][n]
    int n;
    int n_jt;             // j-tiles
    long long units;      // n_iblocks * n_jt
    float eps2;
    unsigned* err;
};

// Issue the bulk copy of j-tile `jt` into stage `s` (one thread).
__device__ __forceinline__ void issue_tile(Body2* tiles, uint64_t* full, int s, int jt,
                                           const Body2* bodies) {
    mbar_arrive_expect_tx(&full[s], kTileBytes);
    bulk_g2s(tiles + s * kT, bodies + (size_t)jt * kT, kTileBytes, &full[s]);
}

// G packed pairs (2G i-bodies) per lane; the j loop is unrolled UNR times.
// i-body of lane `lane`, warp `warp`, slot r in [0, 2G):
//     i = ib * IB + r * 128 + warp * 32 + lane,   IB = 128 * 2G,
// so every slot is a coalesced row of 128 consecutive bodies.
template <bool CLAMP, int G, int UNR>
__global__ void __launch_bounds__(kThreadsMixed, G >= 4 ? 4 : kMinBlocksMixed)
direct_mixed_kernel(MixedArgs a) {
    if (!after_previous()) return;
    constexpr int kIB = kThreadsMixed * 2 * G;
    constexpr int kSlots = 6 * G;  // (hi, lo) x 3 components x G pairs
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Body2* tiles = reinterpret_cast<Body2*>(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + kStages * kTileBytes);
    uint64_t* empty = full + kStages;
    // Compensated per-body accumulators (hi, lo) live in shared memory: they
    // are touched once per tile, and keeping them out of registers lets more
    // CTAs stay resident.  Slot q = 2 * (3 * g + c) + {0: hi, 1: lo}.
    f2_t* acc_sm = reinterpret_cast<f2_t*>(smem_raw + kStages * kTileBytes +
                                           2 * kStages * sizeof(uint64_t));

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const long long per = a.units / gridDim.x;
    const long long rem = a.units % gridDim.x;
    const long long u0 = blockIdx.x * per + min((long long)blockIdx.x, rem);
    const long long u1 = u0 + per + ((long long)blockIdx.x < rem ? 1 : 0);
    const long long cnt = u1 - u0;
    const bool producer = threadIdx.x == 0;
    auto acc_at = [&](int q) -> f2_t& { return acc_sm[q * kThreadsMixed + threadIdx.x]; };

    if (producer) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kWarps);
        }
        mbar_fence_init();
    }
    __syncthreads();
    if (producer) {  // prologue: fill the ring
        for (long long k = 0; k < kStages && k < cnt; ++k)
            issue_tile(tiles, full, (int)k, (int)((u0 + k) % a.n_jt), a.bodies);
    }

    const f2_t eps2 = f2_pack(a.eps2, a.eps2);
    const f2_t zero = f2_pack(0.f, 0.f);
    f2_t xi[G], yi[G], zi[G];
    long long cur_ib = -1;
    bool ok = true;
    const uint32_t tiles_addr = smem_addr(tiles);

    auto flush = [&](long long ib) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float h0, h1, l0, l1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f2_unpack(acc_at(2 * (3 * g + c)), h0, h1);
                f2_unpack(acc_at(2 * (3 * g + c) + 1), l0, l1);
                const int i0 = (int)(ib * kIB) + (2 * g) * kThreadsMixed + warp * 32 + lane;
                const int i1 = i0 + kThreadsMixed;
                if (i0 < a.n) atomicAdd(a.acc + (size_t)c * a.n + i0, (double)h0 + (double)l0);
                if (i1 < a.n) atomicAdd(a.acc + (size_t)c * a.n + i1, (double)h1 + (double)l1);
            }
        }
    };

    for (long long k = 0; k < cnt; ++k) {
        const long long u = u0 + k;
        // Refill the stage that iteration k-1 freed, once every warp is done with it.
        if (producer && k >= 1 && k - 1 + kStages < cnt) {
            const int sp = (int)((k - 1) % kStages);
            const uint32_t par = (uint32_t)(((k - 1) / kStages) & 1);
            if (!mbar_wait(&empty[sp], par, a.err)) {
                ok = false;
                break;
            }
            issue_tile(tiles, full, sp, (int)((u - 1 + kStages) % a.n_jt), a.bodies);
        }
        const long long ib = u / a.n_jt;
        if (ib != cur_ib) {
            if (cur_ib >= 0) flush(cur_ib);
            cur_ib = ib;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int i0 = (int)(ib * kIB) + (2 * g) * kThreadsMixed + warp * 32 + lane;
                const int i1 = i0 + kThreadsMixed;
                float x0 = 0.f, y0 = 0.f, z0 = 0.f, x1 = 0.f, y1 = 0.f, z1 = 0.f;
                if (i0 < a.n) {
                    const float4 b = __ldg(&a.bodies[i0].xxyy);
                    x0 = b.x; y0 = b.z; z0 = __ldg(&a.bodies[i0].zzmm.x);
                }
                if (i1 < a.n) {
                    const float4 b = __ldg(&a.bodies[i1].xxyy);
                    x1 = b.x; y1 = b.z; z1 = __ldg(&a.bodies[i1].zzmm.x);
                }
                xi[g] = f2_pack(x0, x1);
                yi[g] = f2_pack(y0, y1);
                zi[g] = f2_pack(z0, z1);
            }
#pragma unroll
            for (int q = 0; q < kSlots; ++q) acc_at(q) = zero;
        }
        const int s = (int)(k % kStages);
        if (!mbar_wait(&full[s], (uint32_t)((k / kStages) & 1), a.err)) {
            ok = false;
            break;
        }
        const uint32_t tbase = tiles_addr + (uint32_t)s * kTileBytes;
        f2_t ax[G], ay[G], az[G];
#pragma unroll
        for (int g = 0; g < G; ++g) ax[g] = ay[g] = az[g] = zero;
#pragma unroll UNR
        for (int j = 0; j < kT; ++j) {
            const float4 p0 = lds128(tbase + 32u * j);
            const float4 p1 = lds128(tbase + 32u * j + 16u);
            const f2_t xj = f2_pack(p0.x, p0.y);
            const f2_t yj = f2_pack(p0.z, p0.w);
            const f2_t zj = f2_pack(p1.x, p1.y);
            const f2_t mj = f2_pack(p1.z, p1.w);
#pragma unroll
            for (int g = 0; g < G; ++g)
                pair2<CLAMP>(xj, yj, zj, mj, xi[g], yi[g], zi[g], eps2, ax[g], ay[g], az[g]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            f2_two_sum(acc_at(2 * (3 * g + 0)), acc_at(2 * (3 * g + 0) + 1), ax[g]);
            f2_two_sum(acc_at(2 * (3 * g + 1)), acc_at(2 * (3 * g + 1) + 1), ay[g]);
            f2_two_sum(acc_at(2 * (3 * g + 2)), acc_at(2 * (3 * g + 2) + 1), az[g]);
        }
    }
    if (ok && cur_ib >= 0) flush(cur_ib);
}

size_t mixed_smem_bytes(int G) {
    return (size_t)kStages * kTileBytes + 2 * kStages * sizeof(uint64_t) +
           6 * G * kThreadsMixed * sizeof(f2_t);
}

using MixedKernel = void (*)(MixedArgs);

template <bool CLAMP>
MixedKernel pick_mixed(int G, int unr) {
    if (G == 4) {
        if (unr <= 2) return direct_mixed_kernel<CLAMP, 4, 2>;
        return direct_mixed_kernel<CLAMP, 4, 4>;
    }
    if (unr <= 2) return direct_mixed_kernel<CLAMP, 2, 2>;
    if (unr >= 8) return direct_mixed_kernel<CLAMP, 2, 8>;
    return direct_mixed_kernel<CLAMP, 2, 4>;
}

// ---------------------------------------------------------------------------
// symmetric mixed kernel: every unordered pair evaluated once
// ---------------------------------------------------------------------------
// Bodies are split into ranges of 256 G bodies.  A CTA holds one range in
// registers (the A bodies: 2 G per lane as G packed FP32x2 pairs, G = 4 by
// default, 3 with 5 CTAs per SM) and streams
// 128-body B tiles through the same TMA ring as above.  Unit (R, t) pairs
// range R with tile t for t >= the first tile of R:
//   * t inside R: one-sided, all ordered pairs, A side only (the self pair
//     contributes d = 0);
//   * t after R: symmetric.  Each pair adds m_B d / r^3 to A and
//     -m_A d / r^3 to B (Newton's third law), so tiles before R are covered
//     by the units of their own ranges.
// Symmetric chunks of 32 B bodies rotate through the warp: at step k lane l
// meets B body (l + k) mod 32 with its 2 G A bodies, and the B accumulator
// follows its body one lane down per step (a shuffle), so after 32 steps lane
// l holds the complete warp sum for B body l and adds it to f with FP64
// reductions.  Per pair this costs 16 FP32 operations and one reciprocal
// square root for two interactions, against 12 and one per interaction in
// the one-sided kernel.
constexpr int kSymWarps = 4;
constexpr int kSymThreads = kSymWarps * 32;
constexpr int kSymT = 128;  // B bodies per tile
// G packed pairs of A bodies per lane (4 by default, 3 with "direct.sym_g");
// a range is 256 G bodies, 2 G tiles
__host__ __device__ constexpr int sym_range(int G) { return kSymThreads * 2 * G; }
constexpr int kSymStages = 4;
constexpr uint32_t kSymTileBytes = kSymT * 32;  // (x x y y | z z m m) FP32 per body

struct SymArgs {
    const float4* bodies;  // [2 n_pad], tile-split layout
    double* acc;           // a-part of f: [3][n]
    double m_uni;          // the common mass (uniform-mass kernel)
    int n;
    int n_jt;              // tiles = n_pad / kSymT
    int n_ranges;          // n_pad / range
    long long units;
    float eps2;
    unsigned* err;
};

// Tile-split layout: tile t holds [(x x y y) x 128 | (z z m m) x 128], so a
// lane's two LDS.128 of one body return both packed operands ready for the
// FP32x2 arithmetic, and 32 lanes reading 32 different bodies touch 512
// contiguous bytes per load.
__device__ __forceinline__ size_t sym_xy(int i) { return (size_t)(i >> 7) * 256 + (i & 127); }

__global__ void pack_sym_kernel(const double* __restrict__ y, const double* __restrict__ mass,
                                float4* __restrict__ out, double* __restrict__ f, int n,
                                int n_pad) {
    if (!after_previous()) return;
    int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += stride) {
        // padding bodies: zero mass, and parked at 1e18 on every axis, where
        // r^-3 underflows to exactly 0 in FP32, so that they add nothing in
        // the uniform-mass kernel, which does not weight pairs by mass either
        float4 xy = make_float4(1e18f, 1e18f, 1e18f, 1e18f);
        float4 zm = make_float4(1e18f, 1e18f, 0.f, 0.f);
        if (i < n) {
            const float x = (float)y[i], yy = (float)y[n + i], z = (float)y[2 * n + i];
            const float m = (float)mass[i];
            xy = make_float4(x, x, yy, yy);
            zm = make_float4(z, z, m, m);
            f[i] = y[3 * n + i];
            f[n + i] = y[4 * n + i];
            f[2 * n + i] = y[5 * n + i];
            f[3 * n + i] = 0.0;
            f[4 * n + i] = 0.0;
            f[5 * n + i] = 0.0;
        }
        out[sym_xy(i)] = xy;
        out[sym_xy(i) + kSymT] = zm;
    }
}

// First unit of range R: sum over R' < R of (n_jt - tpr R'), tpr = tiles per range.
__host__ __device__ __forceinline__ long long sym_range_start(long long R, long long n_jt,
                                                              int tpr) {
    return R * n_jt - (long long)tpr * (R * (R - 1) / 2);
}

template <int TPR>
struct SymCursor {
    int R, t;
    __device__ void locate(long long u, int n_jt, int n_ranges) {
        int lo = 0, hi = n_ranges - 1;  // largest R with start(R) <= u
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sym_range_start(mid, n_jt, TPR) <= u) lo = mid;
            else hi = mid - 1;
        }
        R = lo;
        t = (int)(u - sym_range_start(lo, n_jt, TPR)) + TPR * lo;
    }
    __device__ void next(int n_jt) {
        if (++t == n_jt) {
            ++R;
            t = TPR * R;
        }
    }
};

template <bool CLAMP>
__device__ __forceinline__ void pair_uni(f2_t xj, f2_t yj, f2_t zj, f2_t xi, f2_t yi, f2_t zi,
                                         f2_t eps2, f2_t& ax, f2_t& ay, f2_t& az) {
    const f2_t dx = f2_sub(xj, xi);
    const f2_t dy = f2_sub(yj, yi);
    const f2_t dz = f2_sub(zj, zi);
    f2_t r2 = f2_fma(dz, dz, eps2);
    r2 = f2_fma(dy, dy, r2);
    r2 = f2_fma(dx, dx, r2);
    float r2a, r2b;
    f2_unpack(r2, r2a, r2b);
    if (CLAMP) {
        r2a = fmaxf(r2a, 1e-8f);
        r2b = fmaxf(r2b, 1e-8f);
    }
    const f2_t inv = f2_pack(rsqrt_mufu(r2a), rsqrt_mufu(r2b));
    const f2_t inv3 = f2_mul(f2_mul(inv, inv), inv);
    ax = f2_fma(dx, inv3, ax);
    ay = f2_fma(dy, inv3, ay);
    az = f2_fma(dz, inv3, az);
}

__device__ __forceinline__ void sym_issue(float4* tiles, uint64_t* full, int s, int t,
                                          const float4* bodies) {
    mbar_arrive_expect_tx(&full[s], kSymTileBytes);
    bulk_g2s(tiles + s * 2 * kSymT, bodies + (size_t)t * 2 * kSymT, kSymTileBytes, &full[s]);
}

template <bool CLAMP, int MINB, int RUNR, int G = 4, bool UNI = false>
__global__ void __launch_bounds__(kSymThreads, MINB)
direct_sym_kernel(SymArgs a) {
    if (!after_previous()) return;
    constexpr int kSymRange = sym_range(G);
    constexpr int kSymTilesPerRange = kSymRange / kSymT;
    constexpr int kSlots = 6 * G;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4* tiles = reinterpret_cast<float4*>(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + kSymStages * kSymTileBytes);
    uint64_t* empty = full + kSymStages;
    f2_t* acc_sm = reinterpret_cast<f2_t*>(smem_raw + kSymStages * kSymTileBytes +
                                           2 * kSymStages * sizeof(uint64_t));
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const long long per = a.units / gridDim.x;
    const long long rem = a.units % gridDim.x;
    const long long u0 = blockIdx.x * per + min((long long)blockIdx.x, rem);
    const long long cnt = per + ((long long)blockIdx.x < rem ? 1 : 0);
    const bool producer = threadIdx.x == 0;
    auto acc_at = [&](int q) -> f2_t& { return acc_sm[q * kSymThreads + threadIdx.x]; };

    if (producer) {
        for (int s = 0; s < kSymStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kSymWarps);
        }
        mbar_fence_init();
    }
    __syncthreads();
    SymCursor<kSymTilesPerRange> cons, prod;
    cons.locate(u0, a.n_jt, a.n_ranges);
    prod = cons;
    if (producer) {
        for (long long k = 0; k < kSymStages && k < cnt; ++k) {
            sym_issue(tiles, full, (int)k, prod.t, a.bodies);
            prod.next(a.n_jt);
        }
    }

    const f2_t eps2 = f2_pack(a.eps2, a.eps2);
    const f2_t zero = f2_pack(0.f, 0.f);
    f2_t xi[G], yi[G], zi[G], mi[G];
    int cur_R = -1;
    bool ok = true;
    const uint32_t tiles_addr = smem_addr(tiles);

    auto flush = [&](int R) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float h0, h1, l0, l1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f2_unpack(acc_at(2 * (3 * g + c)), h0, h1);
                f2_unpack(acc_at(2 * (3 * g + c) + 1), l0, l1);
                const int i0 = R * kSymRange + (2 * g) * kSymThreads + warp * 32 + lane;
                const int i1 = i0 + kSymThreads;
                const double w = UNI ? a.m_uni : 1.0;  // the common mass, applied once
                if (i0 < a.n) atomicAdd(a.acc + (size_t)c * a.n + i0, w * ((double)h0 + (double)l0));
                if (i1 < a.n) atomicAdd(a.acc + (size_t)c * a.n + i1, w * ((double)h1 + (double)l1));
            }
        }
    };

    for (long long k = 0; k < cnt; ++k) {
        if (producer && k >= 1 && k - 1 + kSymStages < cnt) {
            const int sp = (int)((k - 1) % kSymStages);
            const uint32_t par = (uint32_t)(((k - 1) / kSymStages) & 1);
            if (!mbar_wait(&empty[sp], par, a.err)) {
                ok = false;
                break;
            }
            sym_issue(tiles, full, sp, prod.t, a.bodies);
            prod.next(a.n_jt);
        }
        if (cons.R != cur_R) {
            if (cur_R >= 0) flush(cur_R);
            cur_R = cons.R;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int i0 = cur_R * kSymRange + (2 * g) * kSymThreads + warp * 32 + lane;
                const float4 p0 = __ldg(&a.bodies[sym_xy(i0)]);
                const float4 q0 = __ldg(&a.bodies[sym_xy(i0) + kSymT]);
                const float4 p1 = __ldg(&a.bodies[sym_xy(i0 + kSymThreads)]);
                const float4 q1 = __ldg(&a.bodies[sym_xy(i0 + kSymThreads) + kSymT]);
                xi[g] = f2_pack(p0.x, p1.x);
                yi[g] = f2_pack(p0.z, p1.z);
                zi[g] = f2_pack(q0.x, q1.x);
                mi[g] = f2_pack(q0.z, q1.z);
            }
#pragma unroll
            for (int q = 0; q < kSlots; ++q) acc_at(q) = zero;
        }
        const int s = (int)(k % kSymStages);
        if (!mbar_wait(&full[s], (uint32_t)((k / kSymStages) & 1), a.err)) {
            ok = false;
            break;
        }
        const uint32_t tbase = tiles_addr + (uint32_t)s * kSymTileBytes;
        f2_t ax[G], ay[G], az[G];
#pragma unroll
        for (int g = 0; g < G; ++g) ax[g] = ay[g] = az[g] = zero;
        if (cons.t < kSymTilesPerRange * (cons.R + 1)) {
            // own range: one-sided, broadcast loads
#pragma unroll 4
            for (int j = 0; j < kSymT; ++j) {
                const float4 p = lds128(tbase + 16u * j);
                const float4 q = lds128(tbase + 16u * (j + kSymT));
                const f2_t xj = f2_pack(p.x, p.y);
                const f2_t yj = f2_pack(p.z, p.w);
                const f2_t zj = f2_pack(q.x, q.y);
                const f2_t mj = f2_pack(q.z, q.w);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    if constexpr (UNI)
                        pair_uni<CLAMP>(xj, yj, zj, xi[g], yi[g], zi[g], eps2, ax[g], ay[g], az[g]);
                    else
                        pair2<CLAMP>(xj, yj, zj, mj, xi[g], yi[g], zi[g], eps2, ax[g], ay[g],
                                     az[g]);
                }
            }
        } else {
#pragma unroll 1
            for (int c = 0; c < kSymT / 32; ++c) {
                const uint32_t cbase = tbase + (uint32_t)c * 512u;
                float bx = 0.f, by = 0.f, bz = 0.f;
#pragma unroll RUNR
                for (int r = 0; r < 32; ++r) {
                    const uint32_t off = cbase + ((uint32_t)((lane + r) & 31) << 4);
                    const float4 p = lds128(off);
                    const float4 q = lds128(off + 16u * kSymT);
                    const f2_t xj = f2_pack(p.x, p.y);
                    const f2_t yj = f2_pack(p.z, p.w);
                    const f2_t zj = f2_pack(q.x, q.y);
                    const f2_t mj = f2_pack(q.z, q.w);
                    f2_t px = zero, py = zero, pz = zero;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        if constexpr (UNI)
                            sym_pair_uni<CLAMP>(xj, yj, zj, xi[g], yi[g], zi[g], eps2, ax[g],
                                                ay[g], az[g], px, py, pz);
                        else
                            sym_pair<CLAMP>(xj, yj, zj, mj, xi[g], yi[g], zi[g], mi[g], eps2,
                                            ax[g], ay[g], az[g], px, py, pz);
                    }
                    float l, h;
                    f2_unpack(px, l, h);
                    bx += l + h;
                    f2_unpack(py, l, h);
                    by += l + h;
                    f2_unpack(pz, l, h);
                    bz += l + h;
                    // the accumulator of B body (lane + r) moves to lane - 1,
                    // which meets that body at step r + 1
                    const int src = (lane + 1) & 31;
                    bx = __shfl_sync(0xffffffffu, bx, src);
                    by = __shfl_sync(0xffffffffu, by, src);
                    bz = __shfl_sync(0xffffffffu, bz, src);
                }
                // after 32 steps and shifts lane l holds the sum for B body l
                const int jb = cons.t * kSymT + c * 32 + lane;
                if (jb < a.n) {
                    const double w = UNI ? -a.m_uni : -1.0;
                    atomicAdd(a.acc + jb, w * (double)bx);
                    atomicAdd(a.acc + (size_t)a.n + jb, w * (double)by);
                    atomicAdd(a.acc + 2 * (size_t)a.n + jb, w * (double)bz);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            f2_two_sum(acc_at(2 * (3 * g + 0)), acc_at(2 * (3 * g + 0) + 1), ax[g]);
            f2_two_sum(acc_at(2 * (3 * g + 1)), acc_at(2 * (3 * g + 1) + 1), ay[g]);
            f2_two_sum(acc_at(2 * (3 * g + 2)), acc_at(2 * (3 * g + 2) + 1), az[g]);
        }
        cons.next(a.n_jt);
    }
    if (ok && cur_R >= 0) flush(cur_R);
}

size_t sym_smem_bytes(int G) {
    return (size_t)kSymStages * kSymTileBytes + 2 * kSymStages * sizeof(uint64_t) +
           6 * G * kSymThreads * sizeof(f2_t);
}

nbg_status direct_sym_launch(nbg_engine* e, const double* y, double* f) {
    const int n = (int)e->count;
    const int G = e->tune_get("direct.sym_g", 4) == 3 ? 3 : 4;
    const int range = sym_range(G);
    const int n_ranges = (n + range - 1) / range;
    const int n_pad = n_ranges * range;
    const size_t need = 2 * (size_t)n_pad * sizeof(float4);
    if (!reserve_scratch(e, need))
        return cuda_error(e, cudaErrorMemoryAllocation, "the packed bodies' buffer");
    float4* bodies = reinterpret_cast<float4*>(e->d_xyzm);
    queued(pack_sym_kernel, grid_for(n_pad, 256, (unsigned)e->sm_count * 8u), 256, 0, e->stream)(
        y, e->d_mass, bodies, f, n, n_pad);
    NBG_LAUNCHED(e, "pack_sym_kernel");
    const bool clamp = !(e->params.softening > 0.0);
    // "direct.sym_blocks": CTAs per SM the register budget is set for
    // (4: 128 registers, 5: 102)
    // "direct.sym_unroll": unroll of the 32-step rotation loop (1, 2, 4 or 8)
    const bool b5 = e->tune_get("direct.sym_blocks", 4) >= 5;
    // (an RK4 step with 4 / 8: 8000 bodies 74.0 / 74.5 us, 20000 424 / 423,
    // 131072 16.91 / 16.81 ms)
    const int64_t ru = e->tune_get("direct.sym_unroll", n >= 16384 ? 8 : 4);
    using SymKernel = void (*)(SymArgs);
    SymKernel kern;
    // "direct.uniform_mass" (1, the default): with equal masses the kernel
    // that scales the pair sums by the common mass once
    const bool uni = e->uniform_mass && e->tune_get("direct.uniform_mass", 1) != 0;
#define NBG_SYM(MB, RU, GG)                                                                  \
    (uni ? (clamp ? direct_sym_kernel<true, MB, RU, GG, true> : direct_sym_kernel<false, MB, RU, GG, true>) \
         : (clamp ? direct_sym_kernel<true, MB, RU, GG> : direct_sym_kernel<false, MB, RU, GG>))
    if (G == 3)  // 6 A bodies per lane: fewer registers, 5 CTAs per SM
        kern = NBG_SYM(5, 4, 3);
    else if (b5)
        kern = NBG_SYM(5, 2, 4);
    else if (ru >= 8)
        kern = NBG_SYM(4, 8, 4);
    else if (ru >= 4)
        kern = NBG_SYM(4, 4, 4);
    else if (ru <= 1)
        kern = NBG_SYM(4, 1, 4);
    else
        kern = NBG_SYM(4, 2, 4);
#undef NBG_SYM
    const size_t smem = sym_smem_bytes(G);
    NBG_CUDA(e, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    int occ = 0;
    NBG_CUDA(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kSymThreads, smem));
    if (occ < 1) occ = 1;
    const int64_t bps = e->tune_get("direct.blocks_per_sm", 0);
    if (bps > 0 && bps < occ) occ = (int)bps;
    SymArgs a;
    a.bodies = bodies;
    a.acc = f + 3 * (size_t)n;
    a.m_uni = e->mass_value;
    a.n = n;
    a.n_jt = n_pad / kSymT;
    a.n_ranges = n_ranges;
    a.units = sym_range_start(n_ranges, a.n_jt, range / kSymT);
    a.eps2 = (float)(e->params.softening * e->params.softening);
    a.err = e->d_err;
    long long grid = (long long)e->sm_count * occ;
    if (grid > a.units) grid = a.units;
    ProfScope ps(e, NBG_K_DIRECT);
    queued(kern, (unsigned)grid, kSymThreads, smem, e->stream)(a);
    NBG_LAUNCHED(e, "direct_sym_kernel");
    return NBG_OK;
}

// ---------------------------------------------------------------------------
// mixed kernel for small systems
// ---------------------------------------------------------------------------
// The symmetric kernel's units (1024 bodies times 128) are too few for a small
// system: 120 at 5003 bodies, one CTA of four warps each, 23 us for what the
// FP32 pipe does in 5.  Smaller units cost it an FP64 conversion and atomic
// per A body and unit (the FP64 pipe takes 16 cycles a warp instruction).
// Here all ordered pairs are evaluated: the sixteen warps of a CTA hold the
// same 64 bodies, two a lane, and each takes every sixteenth quad of the
// others, so the block's sums leave the CTA once.  The (block, quad) pairs are
// divided evenly over one CTA per SM, whose segments begin and end anywhere.
// Pairs are packed over the quad's bodies, whose records of four float4 need
// no duplication.  Bound by the FP32 pipe (11 packed operations a pair with
// equal masses, 12 else) and, below 4000 bodies, by its two launches.
constexpr int kSmallWarps = 16;
constexpr int kSmallThreads = kSmallWarps * 32;
constexpr int kSmallB = 2;        // bodies per lane, 32 kSmallB a block
constexpr int kSmallFold = 16;    // quads a warp sums before the sums are folded
constexpr long long kSmallMin = 32;  // at least so many quads per CTA
// Up to this size the small-system kernel: fcompute 16 / 5.9 us at 1000 bodies
// (symmetric / small), 20 / 8.7 at 3000, 20 / 15 at 5003.  It does twice the
// symmetric kernel's pairs, which an engine that has the GPU to itself does not
// notice and several side by side do.  An RK4 step of a Plummer sphere alone, and
// of three engines side by side, us: 4096 bodies 111 / 75 and 42 / 42, 5003
// 114 / 87 and 47 / 54, 5120 114 / 89 and 47 / 56, 5500 146 / 98 and 55 / 62, 6000
// 146 / 99 and 55 / 71, 7000 150 / 126 and 64 / 90, 8000 152 / 148 and 75 / 113.  So
// no limit serves both: side by side it would be 4096, alone 8000; at this one
// (five of the symmetric kernel's ranges of 1024 bodies) the small kernel gains
// 22 % alone and costs 19 % side by side.
constexpr int kSmallMax = 5120;

struct SmallArgs {
    const float4* quads;  // 4 bodies: (x x x x) (y y y y) (z z z z) (m m m m)
    double* acc;          // a-part of f: [3][n]
    double m_uni;         // the common mass (uniform-mass kernel)
    int n;
    int nq;               // quads of the n bodies
    long long units;      // blocks * nq
    float eps2;
};

__global__ void pack_small_kernel(const double* __restrict__ y, const double* __restrict__ mass,
                                  float* __restrict__ out, double* __restrict__ f, int n, int n_pad) {
    if (!after_previous()) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    // padding bodies as in pack_sym_kernel
    float x = 1e18f, yy = 1e18f, z = 1e18f, m = 0.f;
    if (i < n) {
        x = (float)y[i];
        yy = (float)y[n + i];
        z = (float)y[2 * n + i];
        m = (float)mass[i];
        f[i] = y[3 * n + i];
        f[n + i] = y[4 * n + i];
        f[2 * n + i] = y[5 * n + i];
        f[3 * n + i] = 0.0;
        f[4 * n + i] = 0.0;
        f[5 * n + i] = 0.0;
    }
    float* q = out + (size_t)(i >> 2) * 16 + (i & 3);
    q[0] = x;
    q[4] = yy;
    q[8] = z;
    q[12] = m;
}

template <bool CLAMP, bool UNI>
__global__ void __launch_bounds__(kSmallThreads, 1)
direct_small_kernel(SmallArgs a) {
    if (!after_previous()) return;
    constexpr int B = kSmallB;
    __shared__ float2 red[kSmallWarps][3 * B][32];  // sums as hi + lo
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* scalars = reinterpret_cast<const float*>(a.quads);
    const long long per = a.units / gridDim.x, rem = a.units % gridDim.x;
    long long u = blockIdx.x * per + min((long long)blockIdx.x, rem);
    const long long u1 = u + per + ((long long)blockIdx.x < rem ? 1 : 0);
    const f2_t eps2 = f2_pack(a.eps2, a.eps2), zero = f2_pack(0.f, 0.f);
    while (u < u1) {
        const int blk = (int)(u / a.nq), qa = (int)(u % a.nq);
        const int qb = (int)min((long long)a.nq, qa + (u1 - u));
        u += qb - qa;
        f2_t xi[B], yi[B], zi[B], hi[3 * B], lo[3 * B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int i = (blk * B + b) * 32 + lane;
            const float* q = scalars + (size_t)(i >> 2) * 16 + (i & 3);
            const float x = __ldg(q), y = __ldg(q + 4), z = __ldg(q + 8);
            xi[b] = f2_pack(x, x);
            yi[b] = f2_pack(y, y);
            zi[b] = f2_pack(z, z);
        }
#pragma unroll
        for (int k = 0; k < 3 * B; ++k) hi[k] = lo[k] = zero;
        float4 nX, nY, nZ, nM = make_float4(0.f, 0.f, 0.f, 0.f);
        auto load = [&](int q) {
            const float4* p = a.quads + 4 * (size_t)q;
            nX = __ldg(p);
            nY = __ldg(p + 1);
            nZ = __ldg(p + 2);
            if (!UNI) nM = __ldg(p + 3);
        };
        load(min(qa + warp, a.nq - 1));
        for (int q0 = qa + warp; q0 < qb; q0 += kSmallFold * kSmallWarps) {
            const int q1 = min(qb, q0 + kSmallFold * kSmallWarps);
            f2_t ax[B], ay[B], az[B];
#pragma unroll
            for (int b = 0; b < B; ++b) ax[b] = ay[b] = az[b] = zero;
#pragma unroll 2
            for (int q = q0; q < q1; q += kSmallWarps) {
                const float4 X = nX, Y = nY, Z = nZ, M = nM;
                load(min(q + kSmallWarps, a.nq - 1));  // in flight over this quad's terms
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const f2_t x0 = f2_pack(X.x, X.y), x1 = f2_pack(X.z, X.w);
                    const f2_t y0 = f2_pack(Y.x, Y.y), y1 = f2_pack(Y.z, Y.w);
                    const f2_t z0 = f2_pack(Z.x, Z.y), z1 = f2_pack(Z.z, Z.w);
                    if constexpr (UNI) {
                        pair_uni<CLAMP>(x0, y0, z0, xi[b], yi[b], zi[b], eps2, ax[b], ay[b], az[b]);
                        pair_uni<CLAMP>(x1, y1, z1, xi[b], yi[b], zi[b], eps2, ax[b], ay[b], az[b]);
                    } else {
                        pair2<CLAMP>(x0, y0, z0, f2_pack(M.x, M.y), xi[b], yi[b], zi[b], eps2,
                                     ax[b], ay[b], az[b]);
                        pair2<CLAMP>(x1, y1, z1, f2_pack(M.z, M.w), xi[b], yi[b], zi[b], eps2,
                                     ax[b], ay[b], az[b]);
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < B; ++b) {
                f2_two_sum(hi[3 * b + 0], lo[3 * b + 0], ax[b]);
                f2_two_sum(hi[3 * b + 1], lo[3 * b + 1], ay[b]);
                f2_two_sum(hi[3 * b + 2], lo[3 * b + 2], az[b]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3 * B; ++k) {
            float h0, h1, l0, l1;
            f2_unpack(hi[k], h0, h1);
            f2_unpack(lo[k], l0, l1);
            // (in FP32: the FP64 pipe takes 16 cycles per warp instruction)
            const float s1 = h0 + h1, b1 = s1 - h0;
            red[warp][k][lane] = make_float2(s1, ((h0 - (s1 - b1)) + (h1 - b1)) + (l0 + l1));
        }
        __syncthreads();
        for (int t = threadIdx.x; t < 96 * B; t += kSmallThreads) {
            const int k = t >> 5, i = (blk * B + k / 3) * 32 + lane;
            float2 s = red[0][k][lane];
#pragma unroll
            for (int w = 1; w < kSmallWarps; ++w) {
                const float2 p = red[w][k][lane];
                const float s1 = s.x + p.x, b1 = s1 - s.x;
                s = make_float2(s1, s.y + (((s.x - (s1 - b1)) + (p.x - b1)) + p.y));
            }
            const double v = two_word_value(s.x, s.y);
            if (i < a.n) atomicAdd(a.acc + (size_t)(k % 3) * a.n + i, UNI ? a.m_uni * v : v);
        }
        __syncthreads();
    }
}

nbg_status direct_small_launch(nbg_engine* e, const double* y, double* f) {
    const int n = (int)e->count;
    constexpr int B = kSmallB;
    const int n_pad = (n + 32 * B - 1) / (32 * B) * (32 * B);
    if (!reserve_scratch(e, (size_t)n_pad * sizeof(float4)))
        return cuda_error(e, cudaErrorMemoryAllocation, "the packed bodies' buffer");
    queued(pack_small_kernel, (unsigned)(n_pad + 127) / 128, 128, 0, e->stream)(
        y, e->d_mass, reinterpret_cast<float*>(e->d_xyzm), f, n, n_pad);
    NBG_LAUNCHED(e, "pack_small_kernel");
    const bool clamp = !(e->params.softening > 0.0);
    const bool uni = e->uniform_mass && e->tune_get("direct.uniform_mass", 1) != 0;
    using SmallKernel = void (*)(SmallArgs);
    SmallKernel kern =
        uni ? (clamp ? direct_small_kernel<true, true> : direct_small_kernel<false, true>)
            : (clamp ? direct_small_kernel<true, false> : direct_small_kernel<false, false>);
    int occ = 0;
    NBG_CUDA(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kSmallThreads, 0));
    SmallArgs a;
    a.quads = e->d_xyzm;
    a.acc = f + 3 * (size_t)n;
    a.m_uni = e->mass_value;
    a.n = n;
    a.nq = (n + 3) / 4;
    a.units = (long long)(n_pad / (32 * B)) * a.nq;
    a.eps2 = (float)(e->params.softening * e->params.softening);
    // at least kSmallMin quads a CTA
    const long long fit = (a.units + kSmallMin - 1) / kSmallMin;
    const long long grid = std::min((long long)e->sm_count * std::max(occ, 1), std::max(fit, 1LL));
    ProfScope ps(e, NBG_K_DIRECT);
    queued(kern, (unsigned)grid, kSmallThreads, 0, e->stream)(a);
    NBG_LAUNCHED(e, "direct_small_kernel");
    return NBG_OK;
}

// Which FP64 kernel: the split path from kSplitMin bodies on, where its five
// launches and the FP64 share of its pairs cost less than the FP64 pipe's 16
// operations a pair (1024 bodies: 37 us against 94; 1280: 60 against 78; 1536:
// 83 against 72; 2048: 140 against 78).
constexpr int kSplitMin = 1536;

nbg_status direct_fp64_launch(nbg_engine* e, const double* y, double* f) {
    const int n = (int)e->count;
    ProfScope ps(e, NBG_K_DIRECT);
    SplitArgs a;
    const size_t system = split_bytes(&a.s, n);
    const int blocks = a.s.n_pad / (2 * kSplitT);
    // ranges: about 8 waves of 4 CTAs per SM (the last one weighs little; 2
    // waves measured 2.2 ms instead of 1.5 at 20011 bodies), at least a tile each
    const int want = (e->sm_count * 4 * 8 + blocks - 1) / blocks;
    const int tiles = a.s.n_pad / kSplitTile;
    const int per = std::max(1, tiles / std::max(1, want));
    a.range = per * kSplitTile;
    a.ranges = (tiles + per - 1) / per;
    bool split = e->tune_get("direct.fp64_split", n >= kSplitMin) != 0;
    // without scratch (or with none to be had while the stream is being
    // captured): the kernel that needs none
    split = split && reserve_scratch(e, system + (size_t)a.ranges * 3 * n * sizeof(double));
    if (!split) {
        const unsigned warps = kF64Threads / 32;
        queued(direct_fp64_kernel, ((unsigned)n + warps - 1) / warps, kF64Threads, 0, e->stream)(
            y, e->d_mass, f, n);
        NBG_LAUNCHED(e, "direct_fp64_kernel");
        return NBG_OK;
    }
    a.f = f;
    a.part = reinterpret_cast<double*>(reinterpret_cast<char*>(e->d_xyzm) + system);
    nbg_status s = split_prepare<false>(e, &a.s, y, e->d_mass, 0.0, e->d_xyzm);
    if (s != NBG_OK) return s;
    const dim3 grid((unsigned)blocks, (unsigned)a.ranges);
    if (e->uniform_mass)
        queued(split_force_kernel<true>, grid, kSplitT, 0, e->stream)(a);
    else
        queued(split_force_kernel<false>, grid, kSplitT, 0, e->stream)(a);
    NBG_LAUNCHED(e, "split_force_kernel");
    queued(split_reduce_kernel, (unsigned)((3 * (size_t)n + 127) / 128), 128, 0, e->stream)(a);
    NBG_LAUNCHED(e, "split_reduce_kernel");
    return NBG_OK;
}

}  // namespace

nbg_status direct_fcompute(nbg_engine* e, const double* y, double* f) {
    const int n = (int)e->count;
    if (e->params.precision == NBG_PREC_FP64) return direct_fp64_launch(e, y, f);

    // ---- mixed precision ----
    if (e->tune_get("direct.symmetric", 1) != 0) {
        // ("direct.sym_g" asks for the symmetric kernel of that shape)
        const bool small = n <= kSmallMax && e->tune_get("direct.sym_g", 0) == 0;
        return e->tune_get("direct.small", small) != 0 ? direct_small_launch(e, y, f)
                                                       : direct_sym_launch(e, y, f);
    }
    const int n_jt = (n + kT - 1) / kT;
    const int n_pad = n_jt * kT;
    const size_t need = (size_t)n_pad * sizeof(Body2);
    if (!reserve_scratch(e, need))
        return cuda_error(e, cudaErrorMemoryAllocation, "the packed bodies' buffer");
    Body2* bodies = reinterpret_cast<Body2*>(e->d_xyzm);
    queued(pack_mixed_kernel, grid_for(n_pad, 256, (unsigned)e->sm_count * 8u), 256, 0, e->stream)(
        y, e->d_mass, bodies, f, n, n_pad);
    NBG_LAUNCHED(e, "pack_mixed_kernel");

    const bool clamp = !(e->params.softening > 0.0);
    const int G = e->tune_get("direct.pairs_per_lane", 4) >= 4 ? 4 : 2;
    const int unr = (int)e->tune_get("direct.unroll", 4);
    MixedKernel kern = clamp ? pick_mixed<true>(G, unr) : pick_mixed<false>(G, unr);
    const size_t smem = mixed_smem_bytes(G);
    NBG_CUDA(e, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    int occ = 0;
    NBG_CUDA(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreadsMixed, smem));
    if (occ < 1) occ = 1;
    const int64_t bps = e->tune_get("direct.blocks_per_sm", 0);
    if (bps > 0 && bps < occ) occ = (int)bps;
    MixedArgs a;
    a.bodies = bodies;
    a.acc = f + 3 * (size_t)n;
    a.n = n;
    a.n_jt = n_jt;
    const int ib_size = kThreadsMixed * 2 * G;
    const long long n_ib = (n + ib_size - 1) / ib_size;
    a.units = n_ib * n_jt;
    a.eps2 = (float)(e->params.softening * e->params.softening);
    a.err = e->d_err;
    long long grid = (long long)e->sm_count * occ;
    if (grid > a.units) grid = a.units;
    ProfScope ps(e, NBG_K_DIRECT);
    queued(kern, (unsigned)grid, kThreadsMixed, smem, e->stream)(a);
    NBG_LAUNCHED(e, "direct_mixed_kernel");
    return NBG_OK;
}

}  // namespace nbg

// ---------------------------------------------------------------------------
// Allocation-free variant of the mixed-precision direct sum
// ---------------------------------------------------------------------------
// Some callers cannot call cudaMalloc: a host application that owns all GPU
// memory through its own arena and forbids allocations behind its back, or a
// time-stepping loop with a hard latency budget where an allocation (and the
// device synchronisation it implies) is not allowed.  For them the packed-body
// scratch of the kernel above lives in a fixed file-scope device array instead
// of an engine allocation.  The array is created with this module on every GPU
// that loads the library and stays there until the process exits, so its size
// is capped: NBG_NOALLOC_MAX_BODIES bodies x 32 bytes = 4 MiB, plus one error
// word.
namespace nbg {
namespace {

static __device__ __align__(256) Body2 g_noalloc_bodies[NBG_NOALLOC_MAX_BODIES];
static __device__ __align__(256) unsigned g_noalloc_err;

constexpr int kNoallocMaxDevices = 64;
struct NoallocDevice {
    bool ready;
    Body2* bodies;  // device address of g_noalloc_bodies on this device
    unsigned* err;  // device address of g_noalloc_err on this device
    int sm_count;
};
std::mutex g_noalloc_mu;
NoallocDevice g_noalloc_dev[kNoallocMaxDevices];

}  // namespace
}  // namespace nbg

extern "C" nbg_status nbg_direct_mixed_noalloc(const double* y, const double* mass, double* f,
                                               size_t n, double softening, void* stream) {
    using namespace nbg;
    if (y == nullptr || mass == nullptr || f == nullptr || n == 0 || !(softening >= 0.0))
        return NBG_ERR_INVALID_ARG;
    if (n > (size_t)NBG_NOALLOC_MAX_BODIES) return NBG_ERR_TOO_LARGE;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices)
        return NBG_ERR_CUDA;

    // One-time set-up per device, on the current device: host code cannot use
    // the array's name as a device address, so look the address up.
    NoallocDevice d;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        NoallocDevice& slot = g_noalloc_dev[dev];
        if (!slot.ready) {
            void* pb = nullptr;
            void* pe = nullptr;
            if (cudaGetSymbolAddress(&pb, g_noalloc_bodies) != cudaSuccess ||
                cudaGetSymbolAddress(&pe, g_noalloc_err) != cudaSuccess ||
                cudaDeviceGetAttribute(&slot.sm_count, cudaDevAttrMultiProcessorCount, dev) !=
                    cudaSuccess) {
                cudaGetLastError();
                return NBG_ERR_CUDA;
            }
            slot.bodies = static_cast<Body2*>(pb);
            slot.err = static_cast<unsigned*>(pe);
            slot.ready = true;
        }
        d = slot;
    }

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nn = (int)n;
    const int n_jt = (nn + kT - 1) / kT;
    const int n_pad = n_jt * kT;
    const bool clamp = !(softening > 0.0);
    constexpr int G = 4;
    MixedKernel kern = clamp ? pick_mixed<true>(G, 4) : pick_mixed<false>(G, 4);
    const size_t smem = mixed_smem_bytes(G);
    int occ = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreadsMixed, smem) !=
            cudaSuccess) {
        cudaGetLastError();
        return NBG_ERR_CUDA;
    }
    if (occ < 1) occ = 1;

    // The error word must start at zero; the pack kernel rewrites every
    // scratch entry the force kernel reads (padding included) and zeroes the
    // acceleration half of f, so nothing else carries over from earlier calls.
    if (cudaMemsetAsync(d.err, 0, sizeof(unsigned), st) != cudaSuccess) {
        cudaGetLastError();
        return NBG_ERR_CUDA;
    }
    queued(pack_mixed_kernel, grid_for(n_pad, 256, (unsigned)d.sm_count * 8u), 256, 0, st)(
        y, mass, d.bodies, f, nn, n_pad);
    MixedArgs a;
    a.bodies = d.bodies;
    a.acc = f + 3 * n;
    a.n = nn;
    a.n_jt = n_jt;
    const long long n_ib = (nn + kThreadsMixed * 2 * G - 1) / (kThreadsMixed * 2 * G);
    a.units = n_ib * n_jt;
    a.eps2 = (float)(softening * softening);
    a.err = d.err;
    long long grid = (long long)d.sm_count * occ;
    if (grid > a.units) grid = a.units;
    queued(kern, (unsigned)grid, kThreadsMixed, smem, st)(a);
    if (cudaGetLastError() != cudaSuccess) return NBG_ERR_CUDA;

    // Synchronous: the result is in f when this returns, and a device-side
    // wait that timed out is reported here.  The error word is read on the
    // caller's stream, so the call waits for that stream only (a plain
    // cudaMemcpy would go through the legacy default stream and wait for
    // unrelated work on other blocking streams).
    unsigned err_host = 0;
    if (cudaMemcpyAsync(&err_host, d.err, sizeof(unsigned), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return NBG_ERR_CUDA;
    }
    return err_host != 0 ? NBG_ERR_DEVICE_TIMEOUT : NBG_OK;
}
