// bw_arith.cuh -- exact modular arithmetic for the two prime paths.
//
// Residues are kept lazily reduced (Harvey).  On the 32-bit path the forward
// Cooley-Tukey butterfly keeps values in [0, 4p) and the inverse
// Gentleman-Sande butterfly in [0, 2p), which needs 4p < 2^32 (primes below
// 2^30).  The 64-bit path's primes are below 2^58, which leaves its forward
// transform 64x headroom (see Ar64).
//
// Multiplication by a precomputed constant w uses Shoup's method with the
// companion wq = floor(w * 2^bits / p): q = hi(x * wq), r = x*w - q*p lies in
// [0, 2p) for every x < 2^bits.  Products of two variables (the pointwise
// step) use Montgomery multiplication; its 2^-bits factor is cancelled by a
// 2^bits folded into the inverse transform's scale constant.
//
// The reference computes these products with a plain `%` on 64/128-bit
// values (pointwise_mul_kernel, src/gpu_ntt.cu:216-238; mulmod64,
// src/crt_gpu.cu:47-67), which is a software division on the GPU.
#pragma once
#include <cstdint>
#include <type_traits>

namespace bw {

template <typename T>
struct alignas(2 * sizeof(T)) Tw {
    T w;
    T wq;
};
// double precision: the quotient comes from the rounded product (ArD), so an
// entry is the constant alone and two fit in a 16-byte load
template <>
struct Tw<double> {
    double w;
};

struct Ar32 {
    using T = uint32_t;
    static constexpr int BITS = 32;
    static constexpr bool kF64 = false;
    uint32_t p;
    uint32_t p2;    // 2p
    uint32_t pinv;  // -p^-1 mod 2^32
    uint32_t r32;   // 2^32 mod p
    uint32_t r32q;  // Shoup companion of r32
    uint32_t oneq;  // floor(2^32 / p): Shoup companion of 1
    double pinv_d;  // 2^32 / p, for companions of twiddles built on the device

    __device__ __forceinline__ T red2(T a) const { return min(a, a - p2); }
    __device__ __forceinline__ T red1(T a) const { return min(a, a - p); }
    // x < 2^32, w < p: returns x*w mod p in [0, 2p)
    __device__ __forceinline__ T shoup(T x, T w, T wq) const {
        const uint32_t q = __umulhi(x, wq);
        return x * w - q * p;
    }
    // a, b < 2p: returns a*b*2^-32 mod p in [0, 2p)
    __device__ __forceinline__ T mont(T a, T b) const {
        const uint64_t t = (uint64_t)a * b;
        const uint32_t m = (uint32_t)t * pinv;
        return (uint32_t)((t + (uint64_t)m * p) >> 32);
    }
    // the pointwise product: a any forward output, b reduced to [0, 2p)
    __device__ __forceinline__ T pointwise(T a, T b) const { return mont(fwd_to_2p(a), b); }
    // forward CT butterfly, inputs/outputs in [0, 4p)
    __device__ __forceinline__ void ct(T& a, T& b, const Tw<T>& w) const {
        const T x = red2(a);
        const T t = shoup(b, w.w, w.wq);
        a = x + t;
        b = x - t + p2;
    }
    // inverse GS butterfly, inputs/outputs in [0, 2p)
    __device__ __forceinline__ void gs(T& a, T& b, const Tw<T>& w) const {
        const T u = a + b;
        const T v = a - b + p2;
        a = red2(u);
        b = shoup(v, w.w, w.wq);
    }
    // twiddle-1 butterflies of stage 0 (inputs known to be in [0, 2p))
    __device__ __forceinline__ void ct1(T& a, T& b) const {
        const T x = a;
        a = x + b;
        b = x - b + p2;
    }
    __device__ __forceinline__ void gs1(T& a, T& b) const {
        const T x = a;
        a = red2(x + b);
        b = red2(x - b + p2);
    }
    // forward-transform output range [0, 4p) -> [0, 2p)
    __device__ __forceinline__ T fwd_to_2p(T a) const { return red2(a); }
    // inverse-transform output range [0, 2p) -> [0, p)
    __device__ __forceinline__ T inv_out(T a) const { return red1(a); }
    // x * w for a twiddle applied between transform passes, in [0, 2p)
    __device__ __forceinline__ T mulc(T x, const Tw<T>& w) const { return shoup(x, w.w, w.wq); }
    // a 16- or 32-bit coefficient as a residue
    static __device__ __forceinline__ T from_u32(uint32_t x) { return (T)x; }
    // last scaling of a single-pass transform, in [0, p)
    __device__ __forceinline__ T scale_out(T x, const Tw<T>& w) const {
        return red1(shoup(x, w.w, w.wq));
    }
    // the product of two table constants, with its companion
    __device__ __forceinline__ Tw<T> mul_tw(const Tw<T>& a, const Tw<T>& b) const {
        const T w = red1(shoup(a.w, b.w, b.wq));
        return Tw<T>{w, companion(w)};
    }
    // Shoup companion floor(w 2^32 / p) of w < p: a double-precision estimate
    // w (2^32 / p) is within 2^-20 of the quotient (below 2^32, relative error
    // under 2^-51), so its floor is exact or one off, and the exact remainder
    // w 2^32 - q p (in [-p, 2p)) decides the correction
    __device__ __forceinline__ T companion(T w) const {
        uint32_t q = (uint32_t)((double)w * pinv_d);
        const int64_t r = (int64_t)((((uint64_t)w) << 32) - (uint64_t)q * p);
        if (r < 0) {
            --q;
        } else if (r >= (int64_t)p) {
            ++q;
        }
        return q;
    }
    // a 64-bit coefficient x = h 2^32 + l reduced to [0, 2p): h (2^32 mod p)
    // and l * 1 by Shoup, each in [0, 2p), their sum below 4p
    __device__ __forceinline__ T from_u64(uint64_t x) const {
        const T h = shoup((uint32_t)(x >> 32), r32, r32q);
        const T l = shoup((uint32_t)x, 1u, oneq);
        return red2(h + l);
    }
};

// The 64-bit path's primes are p = c 2^32 + 1 below 2^58, so 64p < 2^64.
// Every multiplication by a constant inside and between the transforms uses
// the truncated Shoup quotient, which omits the x0*v0 partial product (q may
// be 2 short, so the product lies in [0, 3p)).  The forward (CT) butterfly
// adds without reducing: from inputs below 3p its stage-0 sums stay below 6p
// and every later stage adds less than 3p, so s stages stay below 3p (s + 1)
// -- below 64p for 20 stages, as many as the fixed-length row pass reaches when
// it continues the column pass's values up to its first multiplication of each
// (bw_plan_setup keeps longer sums on the any-length rows).  It is the headroom
// the 58-bit primes buy: with primes near 2^62 every butterfly reduced its input.
// The inverse (GS) transform keeps values in [0, 3p): sums are reduced by one
// conditional subtraction of 3p, differences are offset by 3p (6p < 2^64).
// A forward output enters the pointwise product reduced to [0, 2p) by an
// exact Shoup multiplication by 1.  Garner and the final scalings use the
// exact quotient.
struct Ar64 {
    using T = uint64_t;
    static constexpr int BITS = 64;
    static constexpr bool kF64 = false;
    uint64_t p;
    uint64_t p2;    // 2p
    uint64_t pinv;  // -p^-1 mod 2^64
    uint32_t c;     // p = c * 2^32 + 1
    uint32_t c3;    // 3c
    uint64_t p3;    // 3p
    uint64_t p4;    // 4p
    uint64_t mu_lo; // floor(2^128 / p) = mu_hi 2^64 + mu_lo
    uint32_t mu_hi;
    uint64_t oneq;  // floor(2^64 / p): Shoup companion of 1

    __device__ __forceinline__ T red2(T a) const { return min(a, a - p2); }
    __device__ __forceinline__ T red1(T a) const { return min(a, a - p); }
    // x < 2^64, w < p: x*w mod p in [0, 2p).  The quotient q = hi64(x * wq)
    // is exact and built from 32x32->64 multiply-adds (mad.wide.u32) whose
    // 64-bit addends never overflow:
    //   T = x0 v1 + hi(x0 v0),  W = x1 v0 + lo(T),  q = x1 v1 + hi(W) + hi(T).
    // Because p = c 2^32 + 1, q*p mod 2^64 = q + (q0 c) 2^32 costs one
    // multiply-add; r = lo64(x w) - lo64(q p).
    __device__ __forceinline__ T shoup(T x, T w, T wq) const {
        uint64_t r;
        asm("{\n\t"
            ".reg .u32 x0, x1, v0, v1, w0, w1, h, t0, t1, s0, s1, f0, f1, q0, q1, l0, l1, qh, r0, r1;\n\t"
            ".reg .u64 A, TT, WW, F, Q, L;\n\t"
            "mov.b64 {x0, x1}, %1;\n\t"
            "mov.b64 {w0, w1}, %2;\n\t"
            "mov.b64 {v0, v1}, %3;\n\t"
            "mul.hi.u32 h, x0, v0;\n\t"
            "mov.b64 A, {h, 0};\n\t"
            "mad.wide.u32 TT, x0, v1, A;\n\t"
            "mov.b64 {t0, t1}, TT;\n\t"
            "mov.b64 A, {t0, 0};\n\t"
            "mad.wide.u32 WW, x1, v0, A;\n\t"
            "mov.b64 {s0, s1}, WW;\n\t"
            "add.cc.u32 f0, s1, t1;\n\t"
            "addc.u32 f1, 0, 0;\n\t"
            "mov.b64 F, {f0, f1};\n\t"
            "mad.wide.u32 Q, x1, v1, F;\n\t"
            "mov.b64 {q0, q1}, Q;\n\t"
            "mul.wide.u32 L, x0, w0;\n\t"
            "mov.b64 {l0, l1}, L;\n\t"
            "mad.lo.u32 l1, x0, w1, l1;\n\t"
            "mad.lo.u32 l1, x1, w0, l1;\n\t"
            "mad.lo.u32 qh, q0, %4, q1;\n\t"
            "sub.cc.u32 r0, l0, q0;\n\t"
            "subc.u32 r1, l1, qh;\n\t"
            "mov.b64 %0, {r0, r1};\n\t"
            "}"
            : "=l"(r)
            : "l"(x), "l"(w), "l"(wq), "r"(c));
        return r;
    }
    // a, b < 2p: returns a*b*2^-64 mod p in [0, 2p).  The low word of
    // t + m*p is zero by construction, so its carry is (lo != 0).
    __device__ __forceinline__ T mont(T a, T b) const {
        const uint64_t lo = a * b;
        const uint64_t hi = __umul64hi(a, b);
        const uint64_t m = lo * pinv;
        const uint64_t mh = __umul64hi(m, p);
        return hi + mh + (lo != 0 ? 1ull : 0ull);
    }
    // the pointwise product: a any forward output, b reduced to [0, 2p)
    __device__ __forceinline__ T pointwise(T a, T b) const { return mont(fwd_to_2p(a), b); }
    // x < 2^64, w < p: x*w mod p in [0, 3p) from the truncated quotient
    // q' = x1 v1 + hi(x0 v1 + x1 v0) (the dropped x0 v0 term and the dropped
    // low bits make q' at most 2 below hi64(x * wq)).
    __device__ __forceinline__ T shoup3(T x, T w, T wq) const {
        uint64_t r;
        asm("{\n\t"
            ".reg .u32 x0, x1, v0, v1, w0, w1, t0, t1, s0, s1, f0, f1, q0, q1, l0, l1, qh, r0, r1;\n\t"
            ".reg .u64 A, TT, WW, F, Q, L;\n\t"
            "mov.b64 {x0, x1}, %1;\n\t"
            "mov.b64 {w0, w1}, %2;\n\t"
            "mov.b64 {v0, v1}, %3;\n\t"
            "mul.wide.u32 TT, x0, v1;\n\t"
            "mov.b64 {t0, t1}, TT;\n\t"
            "mov.b64 A, {t0, 0};\n\t"
            "mad.wide.u32 WW, x1, v0, A;\n\t"
            "mov.b64 {s0, s1}, WW;\n\t"
            "add.cc.u32 f0, s1, t1;\n\t"
            "addc.u32 f1, 0, 0;\n\t"
            "mov.b64 F, {f0, f1};\n\t"
            "mad.wide.u32 Q, x1, v1, F;\n\t"
            "mov.b64 {q0, q1}, Q;\n\t"
            "mul.wide.u32 L, x0, w0;\n\t"
            "mov.b64 {l0, l1}, L;\n\t"
            "mad.lo.u32 l1, x0, w1, l1;\n\t"
            "mad.lo.u32 l1, x1, w0, l1;\n\t"
            "mad.lo.u32 qh, q0, %4, q1;\n\t"
            "sub.cc.u32 r0, l0, q0;\n\t"
            "subc.u32 r1, l1, qh;\n\t"
            "mov.b64 %0, {r0, r1};\n\t"
            "}"
            : "=l"(r)
            : "l"(x), "l"(w), "l"(wq), "r"(c));
        return r;
    }
    // forward CT butterfly: a + t and a - t + 3p with t = b w in [0, 3p), no
    // reduction (each stage grows the bound by less than 3p)
    __device__ __forceinline__ void ct(T& a, T& b, const Tw<T>& w) const {
        const T x = a;
        const T t = shoup3(b, w.w, w.wq);  // [0, 3p)
        a = x + t;
        b = x - t + p3;
    }
    // inverse GS butterfly, inputs/outputs in [0, 3p)
    __device__ __forceinline__ void gs(T& a, T& b, const Tw<T>& w) const {
        const T u = a + b;       // [0, 6p)
        const T v = a - b + p3;  // (0, 6p)
        a = min(u, u - p3);
        b = shoup3(v, w.w, w.wq);
    }
    // twiddle-1 butterflies of stage 0 (inputs in [0, 3p))
    __device__ __forceinline__ void ct1(T& a, T& b) const {
        const T x = a;
        a = x + b;
        b = x - b + p3;
    }
    __device__ __forceinline__ void gs1(T& a, T& b) const {
        const T u = a + b, v = a - b + p3;
        a = min(u, u - p3);
        b = min(v, v - p3);
    }
    // forward-transform output (any value below 2^64) -> [0, 2p)
    __device__ __forceinline__ T fwd_to_2p(T a) const { return shoup(a, 1, oneq); }
    // a 64-bit coefficient -> [0, 2p): the path's primes are c 2^32 + 1 with
    // 2^25 < c < 2^26, so q = x >> 58 is floor(x / p) or one less (x / p - q
    // < 1 + 2^-13), and x - q p = (x - q) - (q c) 2^32
    __device__ __forceinline__ T from_u64(T x) const {
        const uint32_t q = (uint32_t)(x >> 58);
        return x - q - ((uint64_t)(q * c) << 32);
    }
    // inverse-transform output range [0, 3p) -> [0, p)
    __device__ __forceinline__ T inv_out(T a) const { return red1(min(a, a - p2)); }
    // x * w for a twiddle applied between transform passes, in [0, 3p)
    __device__ __forceinline__ T mulc(T x, const Tw<T>& w) const { return shoup3(x, w.w, w.wq); }
    // a 16- or 32-bit coefficient as a residue
    static __device__ __forceinline__ T from_u32(uint32_t x) { return (T)x; }
    // last scaling of a single-pass transform, in [0, p)
    __device__ __forceinline__ T scale_out(T x, const Tw<T>& w) const {
        return red1(shoup(x, w.w, w.wq));
    }
    // the product of two table constants, with its companion
    __device__ __forceinline__ Tw<T> mul_tw(const Tw<T>& a, const Tw<T>& b) const {
        const T w = red1(shoup(a.w, b.w, b.wq));
        return Tw<T>{w, companion(w)};
    }
    // Shoup companion floor(w 2^64 / p) of w < p by a Barrett step with
    // mu = floor(2^128 / p): the estimate is at most 2 short.
    __device__ __forceinline__ T companion(T w) const {
        uint64_t q = w * (uint64_t)mu_hi + __umul64hi(w, mu_lo);
        uint64_t r = 0 - q * p;
        if (r >= p) {
            ++q;
            r -= p;
        }
        if (r >= p) ++q;
        return q;
    }
};

// Exact modular arithmetic in double precision, for the 64-bit path's 64-bit
// coefficients.  A residue is a double holding an integer of either sign below
// 2^53 in magnitude, so sums and differences are exact, and a product by a
// constant w (|w| <= p/2) takes six operations:
//
//   h = x w (rounded), l = x w - h (exact, one FMA), q = round(h / p),
//   r = (h - q p) + l = x w - q p.
//
// q comes from adding and subtracting 1.5 2^52, which rounds to an integer
// while |q| <= 2^51.  The primes are chosen so that 1 / p is within 2^-58 of a
// double, so q is within 1/2 + |x w / p| 2^-53 (1 + 2^-5) of x w / p, and with
// |x| = X p, |r| <= p (1/2 + X p 2^-54 (1 + 2^-5)).  h - q p is an integer below
// 2^53, so the FMA and the last addition are exact.  The FP64 pipe of an SM
// takes 64 such operations per cycle, beside the integer pipe's addressing: a
// butterfly is 8 of them against about 40 integer instructions for a 58-bit
// prime (measured 6.5 against 2.83 butterflies per SM-cycle).  A companion
// w / p per constant would shorten the chain by one operation and measured 6.7,
// but doubles the twiddle loads, and those bound the last round of a row.
//
// POL 0: primes within 1% above 2^50: q needs X <= 3.96, |r| <= p (1/2 + 0.066
//   X).  Forward: a round reduces the half it does not multiply in its first
//   stage and then adds four stages: from X = 3.1 at most 1.21, 1.79, 2.41,
//   3.07.  A row's last round starts from products instead (0.71) and ends at
//   3.12, an any-length row, whose first stage has no multiplication, at 3.31.
//   Inverse: the sums of every second stage, and of a round's last, are reduced:
//   from E a difference of 4 E and an output of 1/2 + 0.27 E, so from the
//   pointwise product's 0.72 E stays below that, and differences below 2.9.
// POL 1: primes just above 2^51.67 (X <= 1.24 for q, 2.4 for exact sums, |r| <=
//   p (1/2 + 0.21 X)), for transforms whose coefficients need three such
//   primes: a forward round reduces all its values before its first and third
//   stage (at most 1.11, then 1.85), an inverse stage reduces both outputs.
template <int POL>
struct ArD {
    using T = double;
    static constexpr int BITS = 0;  // products carry no power of two to cancel
    static constexpr bool kF64 = true;
    double p;
    double pinv;  // 1 / p

    static __device__ __forceinline__ double rnd(double t) {
        return __dadd_rn(t, -6755399441055744.0);
    }
    static constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52
    // x - p round(x / p): at most p/2 (1 + 2^-49) in magnitude
    __device__ __forceinline__ T red(T x) const {
        const double q = rnd(__fma_rn(x, pinv, kMagic));
        return __fma_rn(-q, p, x);
    }
    __device__ __forceinline__ T mul(T x, T w) const {
        const double h = __dmul_rn(x, w);
        const double q = rnd(__fma_rn(h, pinv, kMagic));
        const double l = __fma_rn(x, w, -h);
        return __dadd_rn(__fma_rn(-q, p, h), l);
    }
    // the pointwise product: a any forward output, b reduced (POL 0: |a b| <=
    // 3.31 p * p/2, so |q| < 2^51 and the result is below 0.72 p)
    __device__ __forceinline__ T pointwise(T a, T b) const {
        return POL ? red(mul(red(a), b)) : mul(a, b);
    }
    // value u of a round of half width h before its stage l; ent: the round's
    // inputs may be any forward output (else they are reduced)
    __device__ __forceinline__ T ct_enter(T x, int u, int h, int l, bool ent) const {
        if (l == 0 && !ent) return x;
        return (POL == 0 ? l == 0 && u < h : (l & 1) == 0) ? red(x) : x;
    }
    __device__ __forceinline__ void ct(T& a, T& b, const Tw<T>& w) const {
        const T x = a;
        const T t = mul(b, w.w);
        a = __dadd_rn(x, t);
        b = __dsub_rn(x, t);
    }
    __device__ __forceinline__ void ct1(T& a, T& b) const {
        const T x = a;
        a = __dadd_rn(x, b);
        b = __dsub_rn(x, b);
    }
    // RED: this stage's sums are reduced
    template <bool RED>
    __device__ __forceinline__ void gs(T& a, T& b, const Tw<T>& w) const {
        const T u = __dadd_rn(a, b);
        const T v = __dsub_rn(a, b);
        a = RED || POL ? red(u) : u;
        const T r = mul(v, w.w);
        b = POL ? red(r) : r;
    }
    __device__ __forceinline__ void gs1(T& a, T& b) const {
        const T u = __dadd_rn(a, b);
        const T v = __dsub_rn(a, b);
        a = red(u);
        b = red(v);
    }
    __device__ __forceinline__ T fwd_to_2p(T a) const { return red(a); }
    // twiddles between passes: any forward or inverse output in, below p out
    // (POL 1: reduced)
    __device__ __forceinline__ T mulc(T x, const Tw<T>& w) const {
        return POL ? red(mul(red(x), w.w)) : mul(x, w.w);
    }
    // the product of two table constants
    __device__ __forceinline__ Tw<T> mul_tw(const Tw<T>& a, const Tw<T>& b) const {
        return Tw<T>{red(mul(a.w, b.w))};
    }
    // an integer below 2^32 or 2^64 as a residue: its words land in the
    // mantissas of 2^52 and 2^84; the high word's multiple of 2^32 is reduced
    // (|hi - q p| < 2^51 is exact) before the low word is added
    static __device__ __forceinline__ T from_u32(uint32_t x) {
        return __dsub_rn(__hiloint2double(0x43300000, (int)x), 4503599627370496.0);
    }
    __device__ __forceinline__ T from_u64(uint64_t x) const {
        const double lo = from_u32((uint32_t)x);
        const double hi = __dsub_rn(__hiloint2double(0x45300000, (int)(x >> 32)),
                                    19342813113834066795298816.0);
        const double q = rnd(__fma_rn(hi, pinv, kMagic));
        return __dadd_rn(__fma_rn(-q, p, hi), lo);
    }
    // an inverse output (|x| < p) in [0, p)
    __device__ __forceinline__ T inv_out(T x) const { return x < 0.0 ? __dadd_rn(x, p) : x; }
    __device__ __forceinline__ T scale_out(T x, const Tw<T>& w) const { return inv_out(mulc(x, w)); }
};

// Twiddle load from shared memory (generic pointer into the CTA's tables).
template <typename T>
__device__ __forceinline__ Tw<T> ld_tw_s(const Tw<T>* p) {
    return *p;
}

template <typename T>
__device__ __forceinline__ Tw<T> ld_tw(const Tw<T>* p) {
    Tw<T> r;
    if constexpr (std::is_same<T, double>::value) {
        r.w = __ldg(reinterpret_cast<const double*>(p));
    } else if constexpr (sizeof(T) == 8) {
        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p));
        r.w = v.x;
        r.wq = v.y;
    } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
        r.w = v.x;
        r.wq = v.y;
    }
    return r;
}

}  // namespace bw
