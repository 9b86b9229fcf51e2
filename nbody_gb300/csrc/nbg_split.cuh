// nbg_split.cuh -- FP64-accurate gravity arithmetic on the FP32 pipe.
//
// The FP64 pipe of sm_103a issues 2 operations per clock and SM, the FP32
// pipe 128.  A pair term in FP64 needs 16 FP64 operations (256 clocks per
// warp); the same term in two-word FP32 arithmetic (an unevaluated sum of two
// floats, error-free transforms of Knuth and Dekker) needs about 110 FP32
// operations (28 clocks).  Two words carry 48 bits, so a single term is off
// by up to about 1e-14 of itself; the callers therefore take the few terms
// that make up much of a body's sum in FP64, and everything a sum is formed
// from is kept to 2^-48 of the sum or better.
//
// Coordinates are scaled by a power of two into (-1, 1) and written as three
// words on fixed grids, x = h + m + l: h a multiple of 2^-22, m of 2^-45, l
// the rest.  The differences of two h and of two m are then exact in FP32,
// whatever the cancellation, and cost one operation each.
#pragma once

#include "nbg_ptx.cuh"

namespace nbg {

// A product that an addition must see rounded: ptxas contracts mul.rn.f32x2
// into a following add (the scalar form it leaves alone), which breaks the
// error terms below; an fma with +0 it cannot.
__device__ __forceinline__ f2_t f2_mul_rn(f2_t a, f2_t b) {
    return f2_fma(a, b, f2_pack(0.f, 0.f));
}

// -a, 2 a and a / 2 in integer registers: the FP32 pipe is what bounds the
// kernels that use them.  They add to the exponent field: 2 a of a zero comes out
// as 2^-126, which the sums below do not see, and a / 2 wants a normal number (a
// zero gives an infinity; split_rsqrt meets one only for an infinite r^2, whose
// NaN the callers' near test sends to FP64).
__device__ __forceinline__ f2_t f2_neg(f2_t a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ f2_t f2_scale_exp(f2_t a, int exp_bits) {
    float l, h;
    f2_unpack(a, l, h);
    return f2_pack(__int_as_float(__float_as_int(l) + exp_bits),
                   __int_as_float(__float_as_int(h) + exp_bits));
}
__device__ __forceinline__ f2_t f2_twice(f2_t a) { return f2_scale_exp(a, 0x00800000); }
__device__ __forceinline__ f2_t f2_half(f2_t a) { return f2_scale_exp(a, -0x00800000); }

// hi + a b = s + u + v to 2^-48 (Knuth's two-sum of hi and the rounded
// product, whose own rounding error v takes in).
__device__ __forceinline__ f2_t f2_two_fma(f2_t a, f2_t b, f2_t hi, f2_t& u, f2_t& v) {
    const f2_t s = f2_add(hi, f2_mul_rn(a, b));
    const f2_t n = f2_sub(hi, s);
    u = f2_sub(hi, f2_add(s, n));
    v = f2_fma(a, b, n);
    return s;
}

__device__ __forceinline__ void split3(double x, float& h, float& m, float& l) {
    const double hd = rint(x * 4194304.0) * (1.0 / 4194304.0);                // 2^22
    const double r = x - hd;
    const double md = rint(r * 35184372088832.0) * (1.0 / 35184372088832.0);  // 2^45
    h = (float)hd;
    m = (float)md;
    l = (float)(r - md);
}

// The second word of a value that many terms share, r the value less its first
// word.  Two words are off by up to 2^-49 of the value; rounded alike, equal
// masses (or the softening) would be off by the same in every term, up to 1.8e-15
// that no sum averages out (1.2e-15 of the potential of 20011 bodies of mass
// 1 / 20011).  So the k-th of them is rounded down after a share of FP32's last
// place has been added, the shares being the multiples of the golden ratio.
// (Three FP64 operations, the last place's exponent and the share put together in
// integers.)
__device__ __forceinline__ float split_word(double r, unsigned k) {
    const unsigned h = k * 2654435769u;
    const double share = __hiloint2double((int)(0x3ff00000u | h >> 12), (int)(h << 20));  // + 1
    const double last = __hiloint2double(max((__double2hiint(r) & 0x7ff00000) - (23 << 20), 0), 0);
    return __double2float_rd(fma(share, last, r) - last);
}

// Packed difference of one coordinate, d = d1 + d2 with |d2| <= ulp(d1) / 2
// up to the l words (|h| >= |m| or h = 0 makes the two-operation sum exact).
__device__ __forceinline__ void split_diff(f2_t hj, f2_t mj, f2_t lj, f2_t hi, f2_t mi, f2_t li,
                                           f2_t& d1, f2_t& d2) {
    const f2_t s = f2_sub(hj, hi), t = f2_sub(mj, mi), l = f2_sub(lj, li);
    d1 = f2_add(s, t);
    d2 = f2_add(f2_sub(t, f2_sub(d1, s)), l);
}

// a + b = s + e, exactly (Knuth).
__device__ __forceinline__ f2_t f2_sum_err(f2_t a, f2_t b, f2_t& e) {
    const f2_t s = f2_add(a, b);
    const f2_t bp = f2_sub(s, a);
    e = f2_add(f2_sub(a, f2_sub(s, bp)), f2_sub(b, bp));
    return s;
}

// r^2 = r1 + r2 of a two-word difference vector.  2 d1 d2 + d2^2 joins the
// (exact) rounding error of d1^2 before anything else does: on its own d2^2
// is below the last place of the other terms and always rounds away, and the
// last bits of squares are not random, so that rounding them alone leaves a
// bias (1e-15 and 3e-16 of r^2 measured).
__device__ __forceinline__ void split_norm2(const f2_t* d1, const f2_t* d2, f2_t& r1, f2_t& r2) {
    f2_t p[3], er[3], f, g;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        p[c] = f2_mul_rn(d1[c], d1[c]);
        er[c] = f2_add(f2_fma(d1[c], d1[c], f2_neg(p[c])),
                       f2_fma(d2[c], f2_twice(d1[c]), f2_mul(d2[c], d2[c])));
    }
    r1 = f2_sum_err(f2_sum_err(p[0], p[1], f), p[2], g);
    r2 = f2_add(f2_add(f2_add(er[0], er[1]), er[2]), f2_add(f, g));
}

// From r^2 = r1 + r2: y = 1/r to FP32 accuracy (the hardware estimate and
// one Newton step, so that e is small and its rounding with it),
// y^2 = p + q, and the relative residual e = 1 - r^2 y^2.
struct SplitRsqrt {
    f2_t y, p, q, e;
};
__device__ __forceinline__ SplitRsqrt split_rsqrt(f2_t r1, f2_t r2) {
    SplitRsqrt s;
    const f2_t one = f2_pack(1.f, 1.f);
    float a, b;
    f2_unpack(r1, a, b);
    const f2_t y0 = f2_pack(rsqrt_mufu(a), rsqrt_mufu(b));
    const f2_t nr1 = f2_neg(r1);
    const f2_t z = f2_fma(f2_mul(nr1, y0), y0, one);
    s.y = f2_fma(f2_half(y0), z, y0);
    s.p = f2_mul_rn(s.y, s.y);
    const f2_t np = f2_neg(s.p);
    s.q = f2_fma(s.y, s.y, np);
    s.e = f2_fma(nr1, s.p, one);
    s.e = f2_fma(nr1, s.q, s.e);
    s.e = f2_fma(r2, np, s.e);
    return s;
}

// r^-3 = c + cl: y^3 (1 + 3/2 e + 15/8 e^2).
__device__ __forceinline__ void split_cube(const SplitRsqrt& s, f2_t& c, f2_t& cl) {
    c = f2_mul_rn(s.p, s.y);
    cl = f2_fma(s.q, s.y, f2_fma(s.p, s.y, f2_neg(c)));
    const f2_t t = f2_mul(f2_fma(s.e, f2_pack(1.875f, 1.875f), f2_pack(1.5f, 1.5f)), s.e);
    cl = f2_fma(c, t, f2_fma(cl, t, cl));
}

// (hi, lo) += (w + wl) (d1 + d2).  (wl d2, whose mean is -4e-16 of a term, falls
// below the last place of the sum it joins once hi has grown: with 32 terms to a
// fold forces come out 4e-16 to 6e-16 too large.  An order that keeps it costs an
// operation a component, 3 %; the serial FP64 sum's error is 5e-16 to 2e-15.)
__device__ __forceinline__ void split_axpy(f2_t& hi, f2_t& lo, f2_t w, f2_t wl, f2_t d1, f2_t d2) {
    f2_t u, v;
    hi = f2_two_fma(w, d1, hi, u, v);
    v = f2_fma(wl, d1, f2_fma(wl, d2, f2_fma(w, d2, v)));
    lo = f2_add(f2_add(lo, u), v);
}

// r^-3 in FP64 to a few 2^-53: the FP32 estimate y of 1/r and
// y^3 (1 + 3/2 e + 15/8 e^2), e = 1 - x y^2 (6 FP64 operations; the next term
// of the series is below 2^-63).  The conversions between the two formats
// move bits in integer registers, because the conversion instructions run at
// the FP64 pipe's rate; x outside FP32's normal range takes the division form.
__device__ __forceinline__ double rcube_fp64(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    if (h - 0x38100000u >= 0x0fd00000u) return 1.0 / (x * sqrt(x));
    const unsigned b =
        __float_as_uint(rsqrt_mufu(__uint_as_float(((h - 0x38000000u) << 3) | (l >> 29))));
    const double y = __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
    const double q = y * y;
    const double e = fma(-x, q, 1.0);
    const double c = q * y;
    return fma(c * e, fma(e, 1.875, 1.5), c);
}

}  // namespace nbg
