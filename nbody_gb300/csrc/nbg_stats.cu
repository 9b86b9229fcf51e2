// nbg_stats.cu -- conservation checks on the GPU (FP64).
//
// The reference computes momentum P, angular momentum L, kinetic and
// potential energy E and the mass centre V on the host with Kahan sums,
// including an O(N^2) single-threaded potential-energy loop
// (nbody/nbody_data.cpp:57-145, nbody/summation_proxy.h).  Here the same
// quantities come from FP64 reductions on the device, for one system or for
// every system of an ensemble (segments of a concatenated body array).
// Per system the 12 outputs are P[3], L[3], KE, PE, centre[3], mass; KE and
// PE are halved as print_statistics does, and pairs closer than the
// reference's MinDistance contribute no potential (nbody/nbody_data.cpp:46-55).
// With a Plummer softening eps the pair potential is -m_i m_j / sqrt(r^2 + eps^2),
// the potential of the softened force the engine integrates; eps = 0 is the
// reference's form.  The potential of one large system is summed in two-word
// FP32 arithmetic (split_potential_kernel), of small ones and of ensembles on
// the FP64 pipe (stats_potential_kernel).
#include <algorithm>

#include "nbg_internal.cuh"
#include "nbg_split_sys.cuh"
#include "nbg_stats.cuh"

namespace nbg {
namespace {

constexpr int kStatThreads = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    return r;  // valid in thread 0
}

// The O(N) sums: CTA (s, p) takes every gridDim.y-th 256 bodies of system s;
// lin[s][p] receives its 11 sums.
constexpr int kLinSums = 11;

__global__ void __launch_bounds__(kStatThreads)
stats_linear_kernel(const double* __restrict__ y, const double* __restrict__ mass, size_t stride,
                    const long long* __restrict__ off, const int* __restrict__ cnt, int n_single,
                    double* __restrict__ lin) {
    if (!after_previous()) return;
    __shared__ double sh[kStatThreads / 32];
    const int s = blockIdx.x;
    const long long o = off != nullptr ? off[s] : 0;
    const int n = cnt != nullptr ? cnt[s] : n_single;
    double acc[kLinSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int k = blockIdx.y * kStatThreads + threadIdx.x; k < n; k += gridDim.y * kStatThreads) {
        const size_t i = (size_t)(o + k);
        const double m = mass[i];
        const double rx = y[i], ry = y[stride + i], rz = y[2 * stride + i];
        const double px = y[3 * stride + i] * m, py = y[4 * stride + i] * m, pz = y[5 * stride + i] * m;
        acc[0] += px;
        acc[1] += py;
        acc[2] += pz;
        acc[3] += ry * pz - rz * py;
        acc[4] += rz * px - rx * pz;
        acc[5] += rx * py - ry * px;
        acc[6] += (y[3 * stride + i] * y[3 * stride + i] + y[4 * stride + i] * y[4 * stride + i] +
                   y[5 * stride + i] * y[5 * stride + i]) * m;
        acc[7] += rx * m;
        acc[8] += ry * m;
        acc[9] += rz * m;
        acc[10] += m;
    }
    double* out = lin + ((size_t)s * gridDim.y + blockIdx.y) * kLinSums;
    for (int q = 0; q < kLinSums; ++q) {
        const double r = block_sum(acc[q], sh);
        if (threadIdx.x == 0) out[q] = r;
    }
}

// Totals of `parts` partial sums per quantity, one warp per quantity, and the
// 12 outputs; with pot != null the potential is the (negated) sum of pot[0 ..
// npot), else out[7] is left to stats_potential_kernel.
__global__ void __launch_bounds__(32 * (kLinSums + 1))
stats_finish_kernel(const double* __restrict__ lin, int parts, const double* __restrict__ pot,
                    int npot, double* __restrict__ out) {
    if (!after_previous()) return;
    __shared__ double res[kLinSums + 1];
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0.0;
    if (q < kLinSums)
        for (int p = lane; p < parts; p += 32)
            v += lin[((size_t)blockIdx.x * parts + p) * kLinSums + q];
    else if (pot != nullptr)
        for (int p = lane; p < npot; p += 32) v += pot[p];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) res[q] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double* r = out + 12 * (size_t)blockIdx.x;
        for (int k = 0; k < 6; ++k) r[k] = res[k];
        r[6] = res[6] / 2;
        if (pot != nullptr) r[7] = -res[kLinSums];
        r[8] = res[7] / res[10];
        r[9] = res[8] / res[10];
        r[10] = res[9] / res[10];
        r[11] = res[10];
    }
}

struct PairUnit {
    int sys;
    int i0;  // first body (system-local) of the 256-body block
};

// 1 / sqrt(x) in FP64: the FP32 hardware estimate y0 (about 23 correct
// bits) refined by one second-order step of the series
// (1 - e)^(-1/2) = 1 + e/2 + 3e^2/8 + ..., e = 1 - x y0^2 (Householder's
// iteration of order 2), which leaves a truncation error of order e^3,
// below 2^-60 relative: the result is within a few ulp of the correctly
// rounded value, for 5 FP64 operations.  Inputs whose FP32 image is not a
// positive normal number (zero, subnormal, infinite, NaN, negative) take
// the division form; the test is integer arithmetic on the FP32 bits.
// The conversions between the formats move bits in integer registers: the
// conversion instructions run at the FP64 pipe's rate, which is what bounds
// the sums.
__device__ __forceinline__ double rsqrt_fp64(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    if (h - 0x38100000u >= 0x0fd00000u) return 1.0 / sqrt(x);
    const unsigned b =
        __float_as_uint(rsqrtf(__uint_as_float(((h - 0x38000000u) << 3) | (l >> 29))));
    const double y0 = __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
    const double e = fma(-x * y0, y0, 1.0);
    return fma(y0 * e, fma(e, 0.375, 0.5), y0);
}

// Potential energy: one CTA per (system, 256 i-bodies); FP64 pair sums over
// j-tiles in shared memory, each unordered pair once.  With B blocks in a
// system, block b takes the tiles b, b+1, ..., b+B/2 (mod B): its own tile
// (both orders of each pair, weight 1), then tiles at distances 1 .. B/2
// (one order, weight 2, the potential being symmetric); for even B the tile
// at distance B/2 is shared by two blocks and only the lower one takes it.
// Every CTA of a system does the same work.  One atomicAdd per CTA into
// PE[s] (pre-halved).
template <bool SOFT>
__global__ void __launch_bounds__(kStatThreads)
stats_potential_kernel(const double* __restrict__ y, const double* __restrict__ mass, size_t stride,
                       const long long* __restrict__ off, const int* __restrict__ cnt,
                       const PairUnit* __restrict__ units, double eps2,
                       double* __restrict__ out) {
    if (!after_previous()) return;
    __shared__ double tx[kStatThreads], ty[kStatThreads], tz[kStatThreads], tm[kStatThreads];
    __shared__ double sh[kStatThreads / 32];
    const PairUnit u = units[blockIdx.x];
    const long long o = off[u.sys];
    const int n = cnt[u.sys];
    const int li = u.i0 + threadIdx.x;
    const bool live = li < n;
    const size_t i = (size_t)(o + (live ? li : 0));
    const double xi = y[i], yi = y[stride + i], zi = y[2 * stride + i], mi = live ? mass[i] : 0.0;
    double pe = 0.0;
    const int nb = (n + kStatThreads - 1) / kStatThreads;
    const int bi = u.i0 / kStatThreads;
    const int last = (nb % 2 == 0 && bi >= nb / 2) ? nb / 2 - 1 : nb / 2;
    for (int t = 0; t <= last; ++t) {
        const int j0 = ((bi + t) % nb) * kStatThreads;
        const int lj = j0 + threadIdx.x;
        __syncthreads();
        if (lj < n) {
            const size_t j = (size_t)(o + lj);
            tx[threadIdx.x] = y[j];
            ty[threadIdx.x] = y[stride + j];
            tz[threadIdx.x] = y[2 * stride + j];
            tm[threadIdx.x] = mass[j];
        }
        __syncthreads();
        const int c = min(kStatThreads, n - j0);
        const bool own = t == 0;
        double tile = 0.0;
        // the own tile skips the self pair; without softening, pairs closer
        // than kMinDistance add nothing
        auto add = [&](int k) {
            const double dx = xi - tx[k], dy = yi - ty[k], dz = zi - tz[k];
            // (unsoftened: in the order that decides at the minimum distance)
            const double r2 = SOFT ? fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)))
                                   : dx * dx + dy * dy + dz * dz;
            if (!SOFT && r2 < kMinDistance) return;
            tile = fma(-tm[k], rsqrt_fp64(r2), tile);
        };
        if (own) {
            for (int k = 0; k < c; ++k)
                if (j0 + k != li) add(k);
            pe += tile;
        } else {
#pragma unroll 4
            for (int k = 0; k < c; ++k) add(k);
            pe += 2.0 * tile;
        }
    }
    const double tot = block_sum(pe * mi, sh);
    if (threadIdx.x == 0) atomicAdd(out + 12 * (size_t)u.sys + 7, tot / 2);
}

// The potential of one system on the FP32 pipe (nbg_split.cuh): CTA (b, c)
// holds block b (256 bodies, 2 per thread) and takes the c-th share of the
// blocks b, b + 1, ..., b + B/2 (mod B), the schedule of
// stats_potential_kernel with 256-body blocks.  As in the direct sum, terms
// above kSplitNear of the body's own sum of |m_j| / r (and pairs closer than
// 2^-20 of the extent, which covers the minimum distance) are queued and
// taken in FP64, the two-word sums join FP64 totals every 32 bodies.  part
// receives the CTA's share of -PE; its order and every sum are fixed.
// Bound by the FP32 pipe: 72 packed operations (80 softened) for two pairs,
// against 12 operations a pair on the FP64 pipe, which issues 1/64 as many:
// 50000 bodies in 3.55 ms (3.83 softened), 29.9 ms (27.3) on the FP64 pipe;
// 54.0 ms with 256-thread CTAs, format conversions and 15 FP64 operations.
struct PotArgs {
    SplitSystem s;
    double* part;      // [shares][blocks]
    int blocks, dist;  // 256-body blocks; distances of blocks per CTA
};

template <bool SOFT>
__global__ void __launch_bounds__(kSplitT, 4) split_potential_kernel(PotArgs a) {
    if (!after_previous()) return;
    __shared__ __align__(16) float4 tile[kSplitTile][6];
    __shared__ unsigned queue[2][kSplitQ][kSplitT];
    __shared__ double sh[kSplitT / 32];
    const int tid = threadIdx.x;
    const SplitSystem& s = a.s;
    const size_t sn = (size_t)s.n;
    const int bi = blockIdx.x, nb = a.blocks;
    const int i0 = bi * 2 * kSplitT + tid, i1 = i0 + kSplitT;  // < n_pad
    f2_t ih[3], im[3], il[3];
    split_load(s, i0, i1, ih, im, il);
    const float lim0 = split_limit(s, i0), lim1 = split_limit(s, i1);
    const int ex = split_exponent(s);
    const int exc = min(max(ex, -400), 400);
    // unsoftened: pairs at or below the minimum distance are taken in FP64
    const float far_p = SOFT ? kSplitFarP : fminf(kSplitFarP, (float)scalbn(0.999 / kMinDistance, 2 * exc));
    const double e2 = SOFT ? scalbn(s.eps2, -2 * exc) : 0.0;
    const float e2h = (float)e2, e2l = split_word(e2 - (double)e2h, blockIdx.y * gridDim.x + blockIdx.x);
    const f2_t zero = f2_pack(0.f, 0.f);
    f2_t hi = zero, lo = zero;
    double far0 = 0.0, far1 = 0.0, near0 = 0.0, near1 = 0.0;
    int c0 = 0, c1 = 0;
    const int last = (nb % 2 == 0 && bi >= nb / 2) ? nb / 2 - 1 : nb / 2;
    const int t_begin = blockIdx.y * a.dist, t_end = min(t_begin + a.dist, last + 1);

    auto flush_queue = [&](int half, int i, int& cnt, double& acc) {
        const int k = min(i, s.n - 1);
        const double x1 = __ldg(s.y + k), y1 = __ldg(s.y + sn + k), z1 = __ldg(s.y + 2 * sn + k);
        while (__any_sync(0xffffffffu, cnt > 0)) {
            if (cnt > 0) {
                const int j = (int)queue[half][--cnt][tid];
                if (j != i && j < s.n) {
                    const double dx = x1 - __ldg(s.y + j), dy = y1 - __ldg(s.y + sn + j);
                    const double dz = z1 - __ldg(s.y + 2 * sn + j);
                    const double r2 = SOFT ? fma(dx, dx, fma(dy, dy, fma(dz, dz, s.eps2)))
                                           : dx * dx + dy * dy + dz * dz;
                    if (SOFT || !(r2 < kMinDistance)) acc = fma(__ldg(s.mass + j), rsqrt_fp64(r2), acc);
                }
            }
        }
    };

    for (int t = t_begin; t < t_end; ++t) {
        const int block0 = ((bi + t) % nb) * 2 * kSplitT;
        for (int j0 = block0; j0 < block0 + 2 * kSplitT; j0 += kSplitTile) {
            __syncthreads();
            if (tid < kSplitTile) split_store_tile(tile, s.bodies[j0 + tid]);
            __syncthreads();
            const uint32_t base = smem_addr(tile);
#pragma unroll 1
            for (int jc = 0; jc < kSplitTile; jc += kSplitChunk) {
#pragma unroll 2
                for (int j = jc; j < jc + kSplitChunk; ++j) {
                    const SplitPair p = split_pair(base + 96u * j, ih, im, il);
                    f2_t r1, r2;
                    split_norm2(p.d1, p.d2, r1, r2);
                    if (SOFT) {
                        f2_t g;
                        r1 = f2_sum_err(r1, f2_pack(e2h, e2h), g);
                        r2 = f2_add(r2, f2_add(g, f2_pack(e2l, e2l)));
                    }
                    const SplitRsqrt v = split_rsqrt(r1, r2);
                    // 1 / r = y + y (e / 2 + 3/8 e^2)
                    const f2_t yl = f2_mul(v.y, f2_mul(f2_fma(v.e, f2_pack(0.375f, 0.375f),
                                                              f2_pack(0.5f, 0.5f)), v.e));
                    f2_t w = f2_mul_rn(p.mh, v.y);
                    f2_t wl = f2_fma(p.ml, v.y, f2_fma(p.mh, yl, f2_fma(p.mh, v.y, f2_neg(w))));
                    float p0, p1, t0, t1;
                    f2_unpack(v.p, p0, p1);
                    f2_unpack(f2_mul(v.y, p.mabs), t0, t1);
                    const bool is0 = !(t0 <= lim0 && p0 <= far_p) || j0 + j == i0;
                    const bool is1 = !(t1 <= lim1 && p1 <= far_p) || j0 + j == i1;
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
                    f2_two_sum(hi, lo, w);
                    lo = f2_add(lo, wl);
                }
                if ((jc & 31) == 32 - kSplitChunk) {
                    float h0, h1, l0, l1;
                    f2_unpack(hi, h0, h1);
                    f2_unpack(lo, l0, l1);
                    far0 += (double)h0 + (double)l0;
                    far1 += (double)h1 + (double)l1;
                    hi = lo = zero;
                }
                if (__any_sync(0xffffffffu, c0 > kSplitQ - kSplitChunk)) flush_queue(0, i0, c0, near0);
                if (__any_sync(0xffffffffu, c1 > kSplitQ - kSplitChunk)) flush_queue(1, i1, c1, near1);
            }
        }
        if (t == 0) {  // the own block holds both orders of its pairs
            flush_queue(0, i0, c0, near0);
            flush_queue(1, i1, c1, near1);
            far0 *= 0.5;
            far1 *= 0.5;
            near0 *= 0.5;
            near1 *= 0.5;
        }
    }
    flush_queue(0, i0, c0, near0);
    flush_queue(1, i1, c1, near1);
    // back to the caller's units: lengths 2^ex, masses 2^mass_exp (with a
    // coordinate that is not finite every pair is in near)
    const int un = s.mass_exp - ex;
    double v = 0.0;
    if (i0 < s.n) v += s.mass[i0] * (near0 + (ex == 2048 ? 0.0 : scalbn(far0, un)));
    if (i1 < s.n) v += s.mass[i1] * (near1 + (ex == 2048 ? 0.0 : scalbn(far1, un)));
    v = block_sum(v, sh);
    if (tid == 0) a.part[(size_t)blockIdx.y * nb + bi] = v;
}

// The potential of one small system on the FP64 pipe: a warp per body i, its
// lanes on the bodies i + 1 .. i + n / 2 (mod n; the last distance of an even
// n belongs to the lower half), so each unordered pair is met once.
// part[i] receives the body's share of -PE.
template <bool SOFT>
__global__ void __launch_bounds__(32)
pot_fp64_kernel(const double* __restrict__ y, const double* __restrict__ mass, int n, double eps2,
                double* __restrict__ part) {
    if (!after_previous()) return;
    const int i = blockIdx.x, lane = threadIdx.x;
    const size_t sn = (size_t)n;
    const double x1 = y[i], y1 = y[sn + i], z1 = y[2 * sn + i];
    const int last = n % 2 == 0 && i >= n / 2 ? n / 2 - 1 : n / 2;
    double acc = 0.0;
#pragma unroll 4
    for (int d = 1 + lane; d <= last; d += 32) {
        const int j = i + d < n ? i + d : i + d - n;
        const double dx = x1 - __ldg(y + j), dy = y1 - __ldg(y + sn + j), dz = z1 - __ldg(y + 2 * sn + j);
        const double r2 = SOFT ? fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))) : dx * dx + dy * dy + dz * dz;
        if (SOFT || !(r2 < kMinDistance)) acc = fma(__ldg(mass + j), rsqrt_fp64(r2), acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) part[i] = mass[i] * acc;
}

// From this many bodies on the two-word path: below, many terms are above
// kSplitNear of their sum and the FP64 pipe is done first (2048 bodies: 99 us
// against 173; 3000: 150 against 148; 4096: 240 against 126).
constexpr int kPotSplitMin = 3072;

// Statistics of one system of n bodies, with the masses the engine was
// initialised with; *done false when there is no scratch for it.
nbg_status stats_single(nbg_engine* e, const double* y, const double* mass, int n, double eps2,
                        double* out, bool* done) {
    const bool split = n >= e->tune_get("statistics.split_min", kPotSplitMin);
    PotArgs a;
    const size_t system = split_bytes(&a.s, n);
    a.blocks = a.s.n_pad / (2 * kSplitT);
    // CTAs for about 8 waves of 4 per SM
    const int dists = a.blocks / 2 + 1;
    const int shares = std::min(dists, std::max(1, (e->sm_count * 32 + a.blocks - 1) / a.blocks));
    a.dist = (dists + shares - 1) / shares;
    const int rows = (dists + a.dist - 1) / a.dist;
    const int parts = std::max(1, std::min(e->sm_count, n / kStatThreads));
    const int npot = split ? rows * a.blocks : n;
    const size_t doubles = (size_t)npot + (size_t)parts * kLinSums + 12;
    *done = reserve_scratch(e, system + doubles * sizeof(double));
    if (!*done) return NBG_OK;
    a.part = reinterpret_cast<double*>(reinterpret_cast<char*>(e->d_xyzm) + system);
    double* lin = a.part + npot;
    double* res = lin + (size_t)parts * kLinSums;
    queued(stats_linear_kernel, dim3(1, (unsigned)parts), kStatThreads, 0, e->stream)(
        y, mass, (size_t)n, nullptr, nullptr, n, lin);
    NBG_LAUNCHED(e, "stats_linear_kernel");
    if (split) {
        nbg_status s = split_prepare<true>(e, &a.s, y, mass, eps2, e->d_xyzm);
        if (s != NBG_OK) return s;
        const dim3 grid((unsigned)a.blocks, (unsigned)rows);
        if (eps2 > 0.0)
            queued(split_potential_kernel<true>, grid, kSplitT, 0, e->stream)(a);
        else
            queued(split_potential_kernel<false>, grid, kSplitT, 0, e->stream)(a);
        NBG_LAUNCHED(e, "split_potential_kernel");
    } else {
        if (eps2 > 0.0)
            queued(pot_fp64_kernel<true>, (unsigned)n, 32, 0, e->stream)(y, mass, n, eps2, a.part);
        else
            queued(pot_fp64_kernel<false>, (unsigned)n, 32, 0, e->stream)(y, mass, n, eps2, a.part);
        NBG_LAUNCHED(e, "pot_fp64_kernel");
    }
    queued(stats_finish_kernel, 1, 32 * (kLinSums + 1), 0, e->stream)(lin, parts, a.part,
                                                                  npot, res);
    NBG_LAUNCHED(e, "stats_finish_kernel");
    NBG_CUDA(e, cudaMemcpyAsync(out, res, 12 * sizeof(double), cudaMemcpyDeviceToHost, e->stream));
    NBG_CUDA(e, cudaStreamSynchronize(e->stream));
    return NBG_OK;
}

}  // namespace

nbg_status stats_segments(nbg_engine* e, const double* y, const double* mass, size_t stride,
                          int nsys, const long long* d_off, const int* d_cnt,
                          const long long* h_off, const int* h_cnt, double eps2,
                          double* d_out) {
    std::vector<PairUnit> units;
    for (int s = 0; s < nsys; ++s)
        for (int i0 = 0; i0 < h_cnt[s]; i0 += kStatThreads) units.push_back(PairUnit{s, i0});
    (void)h_off;
    DevScratch units_buf;
    NBG_CUDA(e, cudaMalloc(&units_buf.p, units.size() * sizeof(PairUnit) + 16));
    PairUnit* d_units = units_buf.as<PairUnit>();
    NBG_CUDA(e, cudaMemcpyAsync(d_units, units.data(), units.size() * sizeof(PairUnit),
                                cudaMemcpyHostToDevice, e->stream));
    NBG_CUDA(e, cudaMemsetAsync(d_out, 0, 12 * (size_t)nsys * sizeof(double), e->stream));
    DevScratch lin;
    NBG_CUDA(e, cudaMalloc(&lin.p, (size_t)nsys * kLinSums * sizeof(double)));
    queued(stats_linear_kernel, nsys, kStatThreads, 0, e->stream)(y, mass, stride, d_off, d_cnt, 0,
                                                              lin.as<double>());
    NBG_LAUNCHED(e, "stats_linear_kernel");
    queued(stats_finish_kernel, nsys, 32 * (kLinSums + 1), 0, e->stream)(lin.as<double>(), 1, nullptr, 0,
                                                                     d_out);
    NBG_LAUNCHED(e, "stats_finish_kernel");
    if (!units.empty()) {
        auto kern = eps2 > 0.0 ? stats_potential_kernel<true> : stats_potential_kernel<false>;
        queued(kern, (unsigned)units.size(), kStatThreads, 0, e->stream)(y, mass, stride, d_off, d_cnt,
                                                                     d_units, eps2, d_out);
        NBG_LAUNCHED(e, "stats_potential_kernel");
    }
    NBG_CUDA(e, cudaStreamSynchronize(e->stream));  // before units_buf is freed
    return NBG_OK;
}

}  // namespace nbg

extern "C" nbg_status nbg_statistics(nbg_engine* e, const nbg_buffer* y, double out[12]) {
    using namespace nbg;
    if (e == nullptr || out == nullptr) return NBG_ERR_INVALID_ARG;
    if (y == nullptr || e->buffers.count(y) == 0)
        return set_error(e, NBG_ERR_FOREIGN_BUFFER, "y is not gb300 memory");
    if (e->count == 0) return set_error(e, NBG_ERR_NOT_INITIALIZED, "engine not initialized");
    if (y->bytes < 6 * e->count * sizeof(double))
        return set_error(e, NBG_ERR_SIZE_MISMATCH, "y smaller than 6N doubles");
    bool done = false;
    nbg_status s = stats_single(e, static_cast<const double*>(y->dptr), e->d_mass, (int)e->count,
                                e->params.softening * e->params.softening, out, &done);
    if (s != NBG_OK || done) return s;
    // no scratch for it: the kernels of ensembles
    long long h_off = 0;
    int h_cnt = (int)e->count;
    DevScratch off, cnt, res;
    NBG_CUDA(e, cudaMalloc(&off.p, sizeof(long long)));
    NBG_CUDA(e, cudaMalloc(&cnt.p, sizeof(int)));
    NBG_CUDA(e, cudaMalloc(&res.p, 12 * sizeof(double)));
    NBG_CUDA(e, cudaMemcpyAsync(off.p, &h_off, sizeof(h_off), cudaMemcpyHostToDevice, e->stream));
    NBG_CUDA(e, cudaMemcpyAsync(cnt.p, &h_cnt, sizeof(h_cnt), cudaMemcpyHostToDevice, e->stream));
    s = stats_segments(e, static_cast<const double*>(y->dptr), e->d_mass, e->count, 1,
                                  off.as<long long>(), cnt.as<int>(), &h_off, &h_cnt,
                                  e->params.softening * e->params.softening, res.as<double>());
    if (s == NBG_OK) {
        NBG_CUDA(e, cudaMemcpy(out, res.p, 12 * sizeof(double), cudaMemcpyDeviceToHost));
    }
    return s;
}
