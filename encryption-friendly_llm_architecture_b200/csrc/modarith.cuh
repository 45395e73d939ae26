// Device-side modular arithmetic for word-sized primes q < 2^61 (sm_100a).
// All helpers are exact: whichever reduction strategy a kernel uses (Shoup with a
// precomputed quotient, 128-bit Barrett, lazy ranges), stored results are the
// canonical residues in [0, q).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace hb {

using u32 = uint32_t;
using u64 = unsigned long long;
using i64 = long long;

constexpr int kMaxPrimes = 32;   // Q limbs + special limbs
constexpr int kMaxDigitLimbs = 8; // alpha upper bound
constexpr int kMaxList = 96;     // limb instances named by one launch

// Per-prime constants, one array per context in global memory.
struct PrimeConst {
    u64 q;
    u64 mu_hi, mu_lo;   // floor(2^128 / q)
    u64 n_inv, n_inv_sh; // N^-1 mod q and its Shoup companion
    u64 n_inv_w[2], n_inv_c[2]; // N^-1 and N^-1 psi^(-N/2) in the form the 2^16 transforms multiply by: (w, companion)
    u64 iu, iu_sh;      // psi^(N/2): the image of the imaginary unit
    u64 small;          // 1 when q < 2^44 and N = 2^16: the transforms carry its residues as doubles
    double q_inv_f;     // 1/q
    u64 fp;             // 1 when q < 2^44: element-wise kernels take quotients from the FP64 pipe
    u32 fold_shift;     // primes of b >= 45 bits: b - 32 (every such prime of a context lies within 2^(b-12) below 2^b)
    u32 fold_d;         //   and 2^b - q
    u32 d60;            // 2^60 - q when that is positive and below 2^26, else 0
    u64 q7;             // 7q of the primes of 45 bits and more
};

// Limb instances of a launch: instance li (0 <= li < count) uses prime[li % n].
struct LimbMap {
    int n;
    unsigned char prime[kMaxList];
};

__device__ __forceinline__ u64 mul_hi(u64 a, u64 b) { return __umul64hi(a, b); }

// x*w mod q in [0, 2q) for any x < 2^64, w < q, wsh = floor(w * 2^64 / q)
__device__ __forceinline__ u64 mul_shoup_lazy(u64 x, u64 w, u64 wsh, u64 q) {
    return x * w - mul_hi(x, wsh) * q;
}
__device__ __forceinline__ u64 mul_shoup(u64 x, u64 w, u64 wsh, u64 q) {
    u64 r = mul_shoup_lazy(x, w, wsh, q);
    return r >= q ? r - q : r;
}
// ---- cheaper lazy forms for the primes of 45 to 60 bits --------------------------------------------------------
// Measured here (cycles per warp instruction and SM sub-partition, chains that use both words of a product): a low product with a 32-bit addend 2, a
// 32 x 32 -> 64 product 4, with a 64-bit addend 5 to 6, a high word 4, a 64-bit add 2; products overlap with separate adds, shifts and FP64
// instructions (product and FMA 4.4 together), those with a 64-bit addend hardly (7.2).  The quotient of a Shoup product does not need the exact high
// product: h = x1 s1 + hi(x0 s1) + hi(x1 s0) is low by less than three, so x*w - h*q lies in [0, 4q) for any x < 2^64.  A radix-16 round of
// butterflies with it takes 37 (Cooley-Tukey) and 39 (Gentleman-Sande) cycles per warp butterfly; with the exact high
// product and a conditional subtraction per butterfly 49.  Primes next to 2^60 have a cheaper form (LongPm in ntt16.cuh).
__device__ __forceinline__ u64 mul_shoup4(u64 x, u64 w, u64 wsh, u64 nq /* 2^64 - q */) {
    const u32 x0 = (u32)x, x1 = (u32)(x >> 32), s0 = (u32)wsh, s1 = (u32)(wsh >> 32), w0 = (u32)w, w1 = (u32)(w >> 32), n0 = (u32)nq, n1 = (u32)(nq >> 32);
    const u64 h = (u64)x1 * s1 + (u64)__umulhi(x0, s1) + __umulhi(x1, s0);
    const u32 h0 = (u32)h, h1 = (u32)(h >> 32);
    const u64 r = (u64)x0 * w0 + (u64)h0 * n0;
    u32 hi = (u32)(r >> 32);
    hi = x0 * w1 + hi; hi = x1 * w0 + hi; hi = h0 * n1 + hi; hi = h1 * n0 + hi;
    return ((u64)hi << 32) | (u32)r;
}
// x < 16 q  ->  congruent value below (1 + 2^-7) * 2^b, b = fold_shift + 32: replaces k * 2^b (k = x >> b) by k * (2^b - q)
struct FoldQ { u32 shift, mask, d; };
__device__ __forceinline__ u64 fold_q(u64 x, const FoldQ &f) {
    const u32 hi = (u32)(x >> 32);
    return (((u64)(hi & f.mask) << 32) | (u32)x) + (u64)(hi >> f.shift) * f.d;
}
__device__ __forceinline__ u64 canon_q(u64 x, u64 q, const FoldQ &f) { // x < 16 q -> [0, q)
    const u64 r = fold_q(x, f);
    return r >= q ? r - q : r;
}
// (z1:z0) mod q, any 128-bit input.  The quotient estimate is low by at most 4.
__device__ __forceinline__ u64 barrett128(u64 z1, u64 z0, const PrimeConst &m) {
    u64 qh = z1 * m.mu_hi + mul_hi(z1, m.mu_lo) + mul_hi(z0, m.mu_hi);
    u64 r = z0 - qh * m.q;
    u64 q4 = m.q << 2, q2 = m.q << 1;
    if (r >= q4) r -= q4;
    if (r >= q2) r -= q2;
    if (r >= m.q) r -= m.q;
    return r;
}
__device__ __forceinline__ u64 mul_mod(u64 a, u64 b, const PrimeConst &m) {
    return barrett128(mul_hi(a, b), a * b, m);
}
__device__ __forceinline__ u64 add_mod(u64 a, u64 b, u64 q) { u64 s = a + b; return s >= q ? s - q : s; }
__device__ __forceinline__ u64 sub_mod(u64 a, u64 b, u64 q) { return a >= b ? a - b : a + q - b; }
__device__ __forceinline__ u64 reduce_u64(u64 x, const PrimeConst &m) { return barrett128(0, x, m); }
__device__ __forceinline__ u64 reduce_i64(i64 v, const PrimeConst &m) {
    if (v >= 0) return reduce_u64((u64)v, m);
    u64 r = reduce_u64((u64)(-(v + 1)), m);
    return m.q - 1 - r;
}
// ---- FP64-assisted product for primes below 2^44 ------------------------------------------
// B200 issues 64-bit integer adds, compares and selects on a half-rate ALU pipe, and that pipe is
// what bounds a Shoup butterfly (17 ALU instructions each).  For small primes the quotient
// floor(y*w/q) is taken from the FP64 pipe instead: y < 2^52 converts exactly through the 2^52
// magic constant, fma(y, w/q, 2^52) leaves round(y*w/q) in the mantissa (error well below 1),
// and the remainder y*w - qh*q is exact in 64-bit integer arithmetic.  The result is congruent
// to y*w and lies in (0.4q, 1.6q); final stores reduce to the canonical residue, so the bits
// that reach memory are those of any other exact method.
constexpr double kTwo52 = 4503599627370496.0;
__device__ __forceinline__ double u52_to_double(u64 v) { return __longlong_as_double((long long)(v | 0x4330000000000000ull)) - kTwo52; }
__device__ __forceinline__ u64 mantissa52(double d) { return (u64)__double_as_longlong(d) & 0x000FFFFFFFFFFFFFull; }
// low 64 bits of a*b + c*d + e as one chain of integer multiply-adds (no separate add instructions)
__device__ __forceinline__ u64 mad2_lo64(u64 a, u64 b, u64 c, u64 d, u64 e) {
    const u32 a0 = (u32)a, a1 = (u32)(a >> 32), b0 = (u32)b, b1 = (u32)(b >> 32);
    const u32 c0 = (u32)c, c1 = (u32)(c >> 32), d0 = (u32)d, d1 = (u32)(d >> 32);
    u64 r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a0), "r"(b0), "l"(e));
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(r) : "r"(c0), "r"(d0));
    u32 lo = (u32)r, hi = (u32)(r >> 32);
    asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(a0), "r"(b1));
    asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(a1), "r"(b0));
    asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(c0), "r"(d1));
    asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(c1), "r"(d0));
    return ((u64)hi << 32) | lo;
}
// v < 2^52 -> residue in (0.4q, 1.6q)
__device__ __forceinline__ u64 reduce_fp_lazy(u64 v, double q_inv, u64 q) {
    const u64 qh = mantissa52(__fma_rn(u52_to_double(v), q_inv, kTwo52));
    return v - qh * q + q;
}
// v < 2^52 -> canonical residue
__device__ __forceinline__ u64 reduce_fp(u64 v, double q_inv, u64 q) {
    const u64 r = reduce_fp_lazy(v, q_inv, q); // (0.4q, 1.6q)
    return r >= q ? r - q : r;
}

// a*b for a, b < 2^44 and q < 2^44: result congruent to a*b in (0.4q, 1.6q).  The double product is only
// used for the quotient estimate (relative error 2^-52, far below one unit); the remainder is exact.
__device__ __forceinline__ u64 mul_small_lazy_d(u64 a, double ad, u64 b, double bd, double q_inv, u64 q) {
    const u64 qh = mantissa52(__fma_rn(ad * bd, q_inv, kTwo52));
    return mad2_lo64(a, b, qh, 0ull - q, q);
}
__device__ __forceinline__ u64 mul_small_lazy(u64 a, u64 b, double q_inv, u64 q) {
    return mul_small_lazy_d(a, u52_to_double(a), b, u52_to_double(b), q_inv, q);
}
// canonical a*b mod q, choosing the FP64-assisted form for small primes
__device__ __forceinline__ u64 mul_mod_any(u64 a, u64 b, const PrimeConst &m) {
    if (m.fp) { const u64 r = mul_small_lazy(a, b, m.q_inv_f, m.q); return r >= m.q ? r - m.q : r; }
    return mul_mod(a, b, m);
}
// canonical residue of a signed value
__device__ __forceinline__ u64 reduce_i64_any(i64 v, const PrimeConst &m) {
    const u64 a = v < 0 ? (u64)(-(v + 1)) + 1 : (u64)v;
    if (m.fp && a < (1ull << 51)) {
        u64 r = reduce_fp(a, m.q_inv_f, m.q);
        return (v < 0 && r) ? m.q - r : r;
    }
    return reduce_i64(v, m);
}

// ---- the product of two residues of a prime below 2^44 entirely on the FP64 pipe ---------------------------------
// a, w: integer-valued doubles, |a| < 2^44, |w| < 2^44.  p + e = a * w exactly (rounded product and its error, one FMA),
// the quotient estimate rint(p / q) is off by far less than one, p - qh * q is an integer below 2^45 and so is its sum
// with e: the result is congruent to a * w and lies within 0.51 q of zero.  Seven FP64 instructions with the running
// sum, no conversions, against about eleven mixed ones for the integer-assisted form.
constexpr double kMagicS = 6755399441055744.0; // 2^52 + 2^51
__device__ __forceinline__ double mul_fp64_lazy(double a, double w, double q_inv, double qd) {
    const double p = __dmul_rn(a, w);
    const double e = __fma_rn(a, w, -p);
    const double qh = __dadd_rn(__fma_rn(p, q_inv, kMagicS), -kMagicS);
    return __dadd_rn(__fma_rn(-qh, qd, p), e);
}
// integer-valued double, |v| < 2^50  ->  canonical residue in [0, q)
__device__ __forceinline__ u64 canon_fp64(double v, double q_inv, double qd) {
    const double k = __dadd_rn(__fma_rn(v, q_inv, kMagicS), -kMagicS);
    double r = __fma_rn(-k, qd, v);        // within 0.51 q of zero, exact
    if (r < 0.0) r = __dadd_rn(r, qd);
    return mantissa52(__dadd_rn(r, kTwo52));
}

// ---- exact sums of a few such products -------------------------------------------------------------------------
// h collects the products rounded to multiples of 2^40 (it starts at 1.5 * 2^92, whose ulp that is), l the remainders: four FP64
// instructions per product instead of seven, one quotient for the sum.  a, w >= 0, or a within 0.6 q of zero (ks_rows); the products must add up to less than 2^91 in magnitude:
// 2^7 of them for primes below 2^42, eight below 2^44.
constexpr double kGrid40 = 1.5 * 0x1p92;
struct FpAcc {
    double h, l;
    __device__ __forceinline__ void zero() { h = kGrid40; l = 0.0; }
    __device__ __forceinline__ void first(double a, double w) {
        h = __fma_rn(a, w, kGrid40);
        l = __fma_rn(a, w, -__dadd_rn(h, -kGrid40));
    }
    __device__ __forceinline__ void mac(double a, double w) {
        const double t = __fma_rn(a, w, h), d = __dadd_rn(t, -h);
        h = t;
        l = __dadd_rn(l, __fma_rn(a, w, -d));
    }
    // The quotient is below 2^49 and off by less than 0.2 beyond its rounding; t - k q is an integer below 2^48, so exact.
    __device__ __forceinline__ double reduced(double q_inv, double qd) const { // within 0.7 q of zero
        const double t = __dadd_rn(h, -kGrid40);
        const double k = __dadd_rn(__dadd_rn(__fma_rn(t, q_inv, __dmul_rn(l, q_inv)), kMagicS), -kMagicS);
        return __dadd_rn(__fma_rn(-k, qd, t), l);
    }
    __device__ __forceinline__ void relax(double q_inv, double qd) { l = reduced(q_inv, qd); h = kGrid40; } // makes room for as many products again
    __device__ __forceinline__ u64 finish(double q_inv, double qd) const { // canonical
        double r = reduced(q_inv, qd);
        if (r < 0.0) r = __dadd_rn(r, qd);
        return mantissa52(__dadd_rn(r, kTwo52));
    }
    // of residues, and with the constants of a prime: the names that PieceAcc has them under
    __device__ __forceinline__ void product(u64 a, u64 w) { mac(u52_to_double(a), u52_to_double(w)); }
    __device__ __forceinline__ void relax(const PrimeConst &m) { relax(m.q_inv_f, (double)m.q); }
    __device__ __forceinline__ u64 canonical(const PrimeConst &m) const { return finish(m.q_inv_f, (double)m.q); }
};

// ---- sums of products modulo the primes of 45 to 60 bits ---------------------------------------------------------
// A full 64 x 64 -> 128-bit product with its carries costs about 34 cycles here.  For sums of a few products the operands are cut
// into two pieces of 30 bits instead: a product is three 32 x 32 -> 64-bit multiply-adds into three carry-free accumulators (12
// cycles, 4 more per operand that is cut), and the sum  a0 + a1 * 2^30 + a2 * 2^60  is reduced once per output residue with
// 2^60 = d60 modulo q (a 128-bit Barrett reduction takes 65 cycles).  Eight products fit the accumulators.
// The pair mad.lo.cc / madc.hi is a little cheaper in a chain of its own (4.1 against 5.0 cycles), but not inside the kernels: part sums of 48
// polynomials 6.5 against 5.9 ms, one limb of them 1.3 against 0.9 ms.
__device__ __forceinline__ u64 mad_wide(u32 a, u32 b, u64 c) {
    u64 r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// the same as two instructions that the compiler does not join
__device__ __forceinline__ u64 mul_add_wide(u32 a, u32 b, u64 c) {
    u64 t, r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(t) : "r"(a), "r"(b));
    asm volatile("add.u64 %0, %1, %2;" : "=l"(r) : "l"(t), "l"(c));
    return r;
}
// a0 + a1 * 2^30 + a2 * 2^60 modulo a prime of 45 to 60 bits (a0, a1 + 2^34, a2 + 2^34 < 2^64): below 3q
__device__ __forceinline__ u64 finish_wide(u64 a0, u64 a1, u64 a2, const PrimeConst &m) {
    const u32 m30 = 0x3FFFFFFFu;
    if (m.d60) { // 2^60 = d60 modulo q
        const u64 u = a1 + (a0 >> 30), v = a2 + (u >> 30);
        u64 r = mad_wide((u32)u & m30, 1u << 30, (u64)((u32)a0 & m30)); // < 2^60
        r = mad_wide((u32)v, m.d60, r);                                 // + 2^58
        const u64 t = (u64)(u32)(v >> 32) * m.d60;                      // < 2^58, weight 2^32
        r = mad_wide((u32)(t >> 28), m.d60, r);                         // + 2^56
        return r + ((u64)((u32)t & 0x0FFFFFFFu) << 32);                 // + 2^60
    }
    u64 lo = a0, hi = 0, x = a1 << 30;
    lo += x; hi += (a1 >> 34) + (lo < x);
    x = a2 << 60;
    lo += x; hi += (a2 >> 4) + (lo < x);
    return barrett128(hi, lo, m);
}
// Karatsuba: the middle products come from one product of the sums of the pieces, from which the outer two are taken off at the end (modulo
// 2^64, which the true sum a1 does not reach): three multiply-adds and two 32-bit additions, of which the compiler makes one per factor.
// SPLIT: products and additions apart, which lets FP64 products of other warps in between (see mul_shoup4) and takes more registers.  Layer pass:
// masked sums 62.4 -> 57.9 ms, inner products of three digits 8.9 -> 8.7; but part sums (which then spill) 32.3 -> 37.0, rotation sums 7.1 -> 7.6.
template <bool SPLIT> struct PieceAccT {
    u64 a0, am, a2; // weights 1 and 2^60 of the outer products; am = a0 + a1 + a2 modulo 2^64, a1 of weight 2^30
    __device__ __forceinline__ void zero() { a0 = am = a2 = 0; }
    __device__ __forceinline__ void mac(u32 v0, u32 v1, u32 k0, u32 k1) { // 30-bit pieces of the factors
        if (SPLIT) { a0 = mul_add_wide(v0, k0, a0); am = mul_add_wide(v0 + v1, k0 + k1, am); a2 = mul_add_wide(v1, k1, a2); }
        else { a0 = mad_wide(v0, k0, a0); am = mad_wide(v0 + v1, k0 + k1, am); a2 = mad_wide(v1, k1, a2); }
    }
    __device__ __forceinline__ void mac(u64 v, u64 k) { mac((u32)v & 0x3FFFFFFFu, (u32)(v >> 30), (u32)k & 0x3FFFFFFFu, (u32)(k >> 30)); } // v, k < 2^60
    // after at most eight products: makes room for eight more
    __device__ __forceinline__ void relax(const PrimeConst &m) {
        const u64 r = finish_wide(a0, am - a0 - a2, a2, m);
        a0 = r & 0x3FFFFFFFu; am = a0 + (r >> 30); a2 = 0;
    }
    __device__ __forceinline__ u64 finish(const PrimeConst &m) const { // canonical
        const u64 r = finish_wide(a0, am - a0 - a2, a2, m);
        return canon_q(r, m.q, FoldQ{m.fold_shift, (1u << m.fold_shift) - 1u, m.fold_d});
    }
    __device__ __forceinline__ void product(u64 a, u64 w) { mac(a, w); }
    __device__ __forceinline__ u64 canonical(const PrimeConst &m) const { return finish(m); }
};
using PieceAcc = PieceAccT<false>;

// index of the source slot of the automorphism X -> X^g on an NTT-form limb:
//   out[i] = in[ntt_perm(i)], exponents 2*bitrev(i)+1 multiply by g modulo 2N
__device__ __forceinline__ u32 ntt_perm(u32 i, u32 g, int logn) {
    u32 e = ((__brev(i) >> (32 - logn)) << 1) | 1u;
    u32 ej = (g * e) & ((2u << logn) - 1u);
    return __brev(ej >> 1) >> (32 - logn);
}

} // namespace hb
