// Negacyclic NTT / inverse NTT of 2^16-coefficient limbs for sm_100a.
//
// Output order of the forward transform: a_hat[i] = a(psi^(2*bitrev(i)+1)) -- the order of the tables psi^bitrev(k).
//
// The limb is a 256 x 256 matrix (index = row*256 + col).  The forward transform is a column pass (stages 1-8,
// butterfly distance >= 256) followed by a row pass (stages 9-16); the inverse runs the row pass first.  A pass moves
// a limb through HBM once: a CTA of 256 threads owns 16 columns (or 16 rows), every thread keeps 16 coefficients in
// registers and performs four butterfly stages at a time (radix 16), exchanging through shared memory once.  The threads of a row are half a
// warp, so the row passes exchange behind a warp barrier: with a barrier of the CTA its warps loaded, computed and stored together (scores of twelve
// heads: forward row passes 221 -> 191 us a launch, inverse ones 130 -> 122, with the last step of a division 247 -> 233).
//
// Two things set these kernels apart from a textbook radix-2 transform:
//
//  * Twiddles are stored in the order the kernels read them (Ntt16Layout): 16-byte entries (w, companion) so that one
//    128-bit load fetches both words, at offsets that are compile-time constants from one per-thread base pointer.
//    The 15 twiddles a thread owns alone in the last four stages sit 16 entries apart, so the 16 threads of a row
//    read 256 contiguous bytes per load.
//
//  * For primes below 2^44 the coefficients are carried as integer-valued doubles ("double storage") from the first
//    load of a transform to its last store, signed and unreduced.  A butterfly is then
//        p  = y*w, e = fma(y, w, -p)              product and its rounding error
//        qh = fma(y, w/q, M) - M                  quotient estimate, M = 2^52 + 2^51, off by less than 0.02
//        t  = fma(-qh, q, p) + e                  exact remainder in (-0.52 q, 0.52 q)
//        x' = x + t,  y' = x - t
//    eight instructions, all on the FP64 pipe (which runs beside the integer pipe).  Values grow by at most 0.52 q per
//    forward stage (|x| < 9.4 q after 16 stages from a canonical start, far below 2^51).
//    The pass boundary stores the doubles as they are (the intermediate array is private to the transform); the last
//    store reduces to the canonical residue, so the bits that reach memory are those of any other exact method.
//    Primes of 44 bits and more use butterflies on integers below 16 q (LongPm, LongShoup).
#pragma once
#include "modarith.cuh"
#include "pdl.cuh"
#include <cstring>

namespace hb {

constexpr int kN16 = 65536;
constexpr int kRowStride = 272; // 256 + one pad word per 16: conflict-free 16-consecutive reads

// Where twiddle psi^bitrev((base << s) + g) of a four-stage round sits in the per-prime table; j = (1 << s) - 1 + g.
struct Ntt16Layout {
    static constexpr int kColsA = 0;                // column pass, first round: base 1, shared by everybody
    static constexpr int kColsB = 16;               // column pass, second round: base 16 + sub, 16 entries per sub
    static constexpr int kRowsA = 16 + 16 * 16;     // row pass, first round: base 256 + row, 16 entries per row
    static constexpr int kRowsB = kRowsA + 256 * 16; // row pass, second round: base (256 + row) * 16 + clo, entry j of lane clo at (row * 15 + j) * 16 + clo
    static constexpr int kEntries = kRowsB + 256 * 15 * 16;
    static __host__ __device__ constexpr int colsA(int j) { return kColsA + j; }
    static __host__ __device__ constexpr int colsB(int sub, int j) { return kColsB + sub * 16 + j; }
    static __host__ __device__ constexpr int rowsA(int row, int j) { return kRowsA + row * 16 + j; }
    static __host__ __device__ constexpr int rowsB(int row, int j, int clo) { return kRowsB + (row * 15 + j) * 16 + clo; }
};
// entry: x = w, y = companion, as scale_words makes them: below 2^44 the bits of the doubles w and w/q, otherwise what LongPm or LongShoup multiply by
struct Ntt16Tables {
    const ulonglong2 *fwd, *inv; // each [nprimes][Ntt16Layout::kEntries]
    // the last round of the row pass for primes below 2^44: the twiddle alone as a double, [nprimes][kRowsB8], entry j of
    // lane clo of row `row` at (row * 15 + j) * 16 + clo -- half the bytes of the 16-byte entries, and in that round every
    // thread reads 15 twiddles nobody else uses (more bytes than the coefficients themselves)
    const double *fwdB8, *invB8;
    bool pm; // the constants of the primes of 45 bits and more are those of LongPm
    u32 below44; // bit i: prime i is below 2^44.  An argument, so that a kernel knows its branch, and asks for its operands, before PrimeConst has come from memory
    __device__ __forceinline__ bool small(int prime) const { return below44 >> prime & 1; }
};
constexpr int kRowsB8 = 256 * 15 * 16;

// Fills one prime's table from psi^bitrev(k) (k < 2^16) and the companion words; host side.
template <class F> inline void ntt16_fill_table(ulonglong2 *out, F entry /* (index into the bit-reversed table) -> ulonglong2 */) {
    auto put = [&](int off, unsigned base) {
        for (int s = 0; s < 4; ++s)
            for (int g = 0; g < (1 << s); ++g) out[off + (1 << s) - 1 + g] = entry((base << s) + (unsigned)g);
    };
    put(Ntt16Layout::colsA(0), 1u);
    for (int sub = 0; sub < 16; ++sub) put(Ntt16Layout::colsB(sub, 0), 16u + (unsigned)sub);
    for (int row = 0; row < 256; ++row) put(Ntt16Layout::rowsA(row, 0), 256u + (unsigned)row);
    for (int row = 0; row < 256; ++row)
        for (int clo = 0; clo < 16; ++clo) {
            const unsigned base = ((256u + (unsigned)row) << 4) + (unsigned)clo;
            for (int s = 0; s < 4; ++s)
                for (int g = 0; g < (1 << s); ++g) out[Ntt16Layout::rowsB(row, (1 << s) - 1 + g, clo)] = entry((base << s) + (unsigned)g);
        }
}

// the compact last-round table of one prime below 2^44: w(k) = the twiddle of bit-reversed-table index k as a double
template <class F> inline void ntt16_fill_rows_b8(double *out, F w) {
    for (int row = 0; row < 256; ++row)
        for (int clo = 0; clo < 16; ++clo) {
            const unsigned base = ((256u + (unsigned)row) << 4) + (unsigned)clo;
            for (int s = 0; s < 4; ++s)
                for (int g = 0; g < (1 << s); ++g) out[(row * 15 + (1 << s) - 1 + g) * 16 + clo] = w((base << s) + (unsigned)g);
        }
}

// address of limb instance li: (li / period) * outer + (li % period) * N
struct LimbAddr16 {
    size_t outer;
    __device__ __forceinline__ size_t off(int li, int period) const { return (size_t)(li / period) * outer + (size_t)(li % period) * kN16; }
};

// The fifteen twiddles of a radix-16 round, j = (1 << s) - 1 + g of local stage s, group g.
struct TwiddlesA { // shared by many threads: (w, companion), consecutive
    const ulonglong2 *p;
    __device__ __forceinline__ explicit TwiddlesA(const ulonglong2 *q) : p(q) {}
    __device__ __forceinline__ ulonglong2 operator[](int j) const { return __ldg(p + j); }
};
// owned by one thread, 16 entries apart; EARLY: fetched when the object is made instead of when they are used
template <class T, bool EARLY> struct TwiddlesB;
template <class T> struct TwiddlesB<T, false> {
    const T *p;
    __device__ __forceinline__ explicit TwiddlesB(const T *q) : p(q) {}
    __device__ __forceinline__ T operator[](int j) const { return __ldg(p + j * 16); }
};
template <class T> struct TwiddlesB<T, true> {
    T w[15];
    __device__ __forceinline__ explicit TwiddlesB(const T *q) {
#pragma unroll
        for (int j = 0; j < 15; ++j) w[j] = __ldg(q + j * 16);
    }
    __device__ __forceinline__ T operator[](int j) const { return w[j]; }
};

// ---------------- Shoup butterflies on integers (primes of 45 bits and more) ----------------
// exact quotients, values in [0, 4q) and [0, 2q): the small-ring kernel
__device__ __forceinline__ void ct_bfly(u64 &x, u64 &y, u64 w, u64 ws, u64 q, u64 q2) {
    x = x >= q2 ? x - q2 : x;
    u64 t = mul_shoup_lazy(y, w, ws, q);
    y = x + q2 - t;
    x = x + t;
}
__device__ __forceinline__ void gs_bfly(u64 &x, u64 &y, u64 w, u64 ws, u64 q, u64 q2) {
    u64 s = x + y;
    u64 d = x + q2 - y;
    x = s >= q2 ? s - q2 : s;
    y = mul_shoup_lazy(d, w, ws, q);
}
// The arithmetic of the primes of 45 bits and more in these kernels, as a policy: LongPm where every such prime of the context lies within 2^26 below
// 2^60, as the first primes below it do, otherwise LongShoup.  Both keep values below 16 q in 64 bits and multiply by constants that come as two words.
struct LongShoup {
    struct Const { u64 q, nq, q4, q8; FoldQ f; };
    static __device__ __forceinline__ Const make(const PrimeConst &m) {
        Const c;
        c.q = m.q; c.nq = 0ull - m.q; c.q4 = m.q << 2; c.q8 = m.q << 3;
        c.f.shift = m.fold_shift; c.f.mask = (1u << m.fold_shift) - 1u; c.f.d = m.fold_d;
        return c;
    }
    static __device__ __forceinline__ u64 mul(u64 x, u64 w, u64 comp, const Const &c) { return mul_shoup4(x, w, comp, c.nq); } // any x -> below 4q
    static __device__ __forceinline__ u64 canon(u64 x, const Const &c) { return canon_q(x, c.q, c.f); }
    static __device__ __forceinline__ u64 above_fwd(const Const &c) { return c.q8; } // a multiple of q above what a forward transform leaves (5q)
    static __device__ __forceinline__ u64 above_inv(const Const &c) { return c.q8; } // and above what three stages of an inverse round leave (8q)
    // Four Cooley-Tukey stages on 16 register values; twiddles tp[j].
    // A stage adds 4q to the bound B of the values; x is folded below ~2^b before the additions of the stages named by the bit mask FOLD.
    // The words hold 16 q: in units of q the four rounds of a transform (masks 8, 4, 2, 9) run 3-7-11-15|5, 5-9-13|5-9, 9-13|5-9-13, 13|5-9-13|5 (| = a fold).
    // MADE: the upper half already carries the twiddle of the first stage (values below 4q)
    template <int ROUND, bool MADE = false, class TW> static __device__ __forceinline__ void fwd16(u64 (&v)[16], const TW &tp, const Const &c) {
        constexpr int FOLD = ROUND == 0 ? 8 : ROUND == 1 ? 4 : ROUND == 2 ? 2 : 9;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int half = 8 >> s;
#pragma unroll
            for (int g = 0; g < (1 << s); ++g) {
                const ulonglong2 tw = tp[(1 << s) - 1 + g];
#pragma unroll
                for (int j = 0; j < half; ++j) {
                    u64 &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                    const u64 t = MADE && s == 0 ? y : mul(y, tw.x, tw.y, c);
                    if ((FOLD >> s) & 1) x = fold_q(x, c.f);
                    y = x + c.q4 - t;
                    x = x + t;
                }
            }
        }
    }
    // Four Gentleman-Sande stages, the mirror image.  Values enter and leave below 4q: sums reach 8q, then 16q, and are folded at
    // every second stage.  LAST: the stage to end with
    template <int LAST = 0, class TW> static __device__ __forceinline__ void inv16(u64 (&v)[16], const TW &tp, const Const &c) {
#pragma unroll
        for (int s = 3; s >= LAST; --s) {
            const int half = 8 >> s;
#pragma unroll
            for (int g = 0; g < (1 << s); ++g) {
                const ulonglong2 tw = tp[(1 << s) - 1 + g];
#pragma unroll
                for (int j = 0; j < half; ++j) {
                    u64 &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                    const u64 d = x + ((s & 1) ? c.q4 : c.q8) - y, a = x + y;
                    x = (s & 1) ? a : fold_q(a, c.f);
                    y = mul(d, tw.x, tw.y, c);
                }
            }
        }
    }
};
// Primes q = 2^60 - d, d < 2^26.  A constant w comes as its two pieces and those of w' = w * 2^32 mod q (29 low and 31 high bits in the words of a u64), so
// that x * w = x0 w + x1 w' = A + B * 2^29 takes the words of x as they are, and B = Bl + Bh * 2^32 folds by 2^61 = 2d the same way: A + Bl * 2^29 + Bh * 2d.
// Five 32 x 32 products instead of the Shoup form's five and four low ones, and no carries in between.
// In units of 2^60, for x below X: A < 2 + X/8, Bl * 2^29 < 2, Bh * 2d < 1/2: below 4.5 + X/8, 6.5 for any x.
// A radix-16 round, cycles per warp butterfly and scheduler with eight warps: 27 against 38 (Cooley-Tukey), 30 against 39 (Gentleman-Sande); half of the
// warps in FP64 butterflies: 19 on average against 26, as products with 64-bit addends leave FP64 products few issue slots.  7q comes
// from memory: where the compiler sees seven times q, it multiplies (35 and 34 cycles).
struct LongPm {
    struct Const { u64 q, q7; u32 d, d2; };
    static __device__ __forceinline__ Const make(const PrimeConst &m) {
        Const c;
        c.q = m.q; c.q7 = m.q7; c.d = m.d60; c.d2 = 2 * m.d60;
        return c;
    }
    // separate instructions: the compiler would join most of them to products with 64-bit addends, which take longer than both
    static __device__ __forceinline__ u64 add(u64 a, u64 b) { u64 r; asm volatile("add.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
    static __device__ __forceinline__ u64 wide(u32 a, u32 b) { u64 r; asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b)); return r; }
    static __device__ __forceinline__ u64 shl29(u32 x) { u64 r; asm("{.reg .u32 l, h; shl.b32 l, %1, 29; shr.u32 h, %1, 3; mov.b64 %0, {l, h};}" : "=l"(r) : "r"(x)); return r; }
    static __device__ __forceinline__ u64 mul(u64 x, u64 w, u64 comp, const Const &c) {
        const u32 x0 = (u32)x, x1 = (u32)(x >> 32);
        const u64 a = add(wide(x1, (u32)comp), wide(x0, (u32)w)), b = add(wide(x1, (u32)(comp >> 32)), wide(x0, (u32)(w >> 32)));
        return add(add(a, shl29((u32)b)), wide((u32)(b >> 32), c.d2));
    }
    // x < 16 * 2^60 -> congruent value below 2^60 + 2^30
    static __device__ __forceinline__ u64 fold(u64 x, const Const &c) {
        const u32 hi = (u32)(x >> 32);
        return (((u64)(hi & 0x0FFFFFFFu) << 32) | (u32)x) + (hi >> 28) * c.d;
    }
    static __device__ __forceinline__ u64 canon(u64 x, const Const &c) {
        const u64 r = fold(x, c);
        return r >= c.q ? r - c.q : r;
    }
    static __device__ __forceinline__ u64 above_fwd(const Const &c) { return c.q7 << 1; } // a forward transform leaves 8.1
    static __device__ __forceinline__ u64 above_inv(const Const &c) { return c.q7; }      // an inverse round 6.3
    // x is folded before the additions of every second stage; differences are taken from 7q, above every product.  Bounds (units of 2^60) alternate: 8.1 behind
    // a stage with a fold, 15.1 behind one without, whose products are below 4.5 + 15.1 / 8 = 6.4.
    // MADE: the upper half already carries the twiddle of the first stage (both halves below 6.5, so sums and differences below 13.6)
    template <int ROUND, bool MADE = false, class TW> static __device__ __forceinline__ void fwd16(u64 (&v)[16], const TW &tp, const Const &c) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int half = 8 >> s;
#pragma unroll
            for (int g = 0; g < (1 << s); ++g) {
                const ulonglong2 tw = tp[(1 << s) - 1 + g];
#pragma unroll
                for (int j = 0; j < half; ++j) {
                    u64 &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                    const u64 t = MADE && s == 0 ? y : mul(y, tw.x, tw.y, c);
                    if (s & 1) x = fold(x, c);
                    y = x + c.q7 - t;
                    x = x + t;
                }
            }
        }
    }
    // Values enter and leave below 6.3: sums (below 12.6) are folded at every stage, products of differences (below 13.3) are below 4.5 + 13.3 / 8.
    template <int LAST = 0, class TW> static __device__ __forceinline__ void inv16(u64 (&v)[16], const TW &tp, const Const &c) {
#pragma unroll
        for (int s = 3; s >= LAST; --s) {
            const int half = 8 >> s;
#pragma unroll
            for (int g = 0; g < (1 << s); ++g) {
                const ulonglong2 tw = tp[(1 << s) - 1 + g];
#pragma unroll
                for (int j = 0; j < half; ++j) {
                    u64 &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                    const u64 d = x + c.q7 - y, a = x + y;
                    x = fold(a, c);
                    y = mul(d, tw.x, tw.y, c);
                }
            }
        }
    }
};
// The last stage of an inverse transform together with the multiplication by N^-1 (or another constant): its only twiddle goes into the
// constant of the differences, so that the stage costs no products of its own.  sw, sc: constant, constant * twiddle.  store(e, canonical).
template <class LONG, class STORE> __device__ __forceinline__ void inv16_int_last(const u64 (&v)[16], const u64 (&sw)[2], const u64 (&sc)[2], const typename LONG::Const &c, STORE &&store) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { // below 8q before, sums and differences below 16q
        const u64 a = v[j] + v[j + 8], d = v[j] + LONG::above_inv(c) - v[j + 8];
        store(j, LONG::canon(LONG::mul(a, sw[0], sc[0], c), c));
        store(j + 8, LONG::canon(LONG::mul(d, sw[1], sc[1], c), c));
    }
}

// ---------------- double-storage butterflies (primes below 2^44) ----------------
constexpr double kMagic = 6755399441055744.0; // 2^52 + 2^51: adding it leaves a signed integer |v| < 2^51 in the low mantissa bits
struct DsConst { double qd, qinv; };
__device__ __forceinline__ DsConst ds_const(const PrimeConst &m) {
    DsConst c;
    c.qd = (double)m.q; c.qinv = m.q_inv_f;
    return c;
}
// canonical residue -> double, exact for values below 2^52
__device__ __forceinline__ double ds_load(u64 a) { return u52_to_double(a); }
// t = y * w mod q as a signed double in (-0.52 q, 0.52 q); y integer-valued, |y| < 2^49; wf = w / q
// wbits = bits of the double w.  Six FP64 instructions, every one exact: p + e = y * w (product and its rounding error),
// qh = rint(y * w / q) up to 0.02, p - qh * q is an integer below 2^45 and so is its sum with e.
__device__ __forceinline__ double ds_mul(double y, u64 wbits, double wf, const DsConst &c) {
    const double wd = __longlong_as_double((long long)wbits);
    const double qh = __dadd_rn(__fma_rn(y, wf, kMagic), -kMagic);
    const double p = __dmul_rn(y, wd);
    const double e = __fma_rn(y, wd, -p);
    const double t1 = __fma_rn(-qh, c.qd, p);
    return __dadd_rn(t1, e);
}
// the same with the quotient estimated from the rounded product instead of from a precomputed w / q (one operand less to
// fetch; the estimate is off by less than 0.07, so the result lies within 0.57 q of zero)
__device__ __forceinline__ double ds_mul_w(double y, double wd, const DsConst &c) {
    const double p = __dmul_rn(y, wd);
    const double e = __fma_rn(y, wd, -p);
    const double qh = __dadd_rn(__fma_rn(p, c.qinv, kMagic), -kMagic);
    return __dadd_rn(__fma_rn(-qh, c.qd, p), e);
}
// the form of a twiddle w that ds_mul takes as its second operand
__host__ __device__ __forceinline__ u64 ds_twiddle_word(u64 w) {
    const double d = (double)w; // exact below 2^53
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(d);
#else
    u64 b; memcpy(&b, &d, 8); return b;
#endif
}
// x - rint(x / q) * q, |result| <= 0.52 q
__device__ __forceinline__ double ds_reduce(double x, const DsConst &c) {
    const double k = __fma_rn(x, c.qinv, kMagic) - kMagic;
    return __fma_rn(-k, c.qd, x);
}
// integer-valued double, |v| < 2^20 q  ->  canonical residue in [0, q)
__device__ __forceinline__ u64 ds_store(double v, const DsConst &c, double shift /* a multiple of q above |v| */, double qinv_up) {
    const double v2 = v + shift;                                         // positive
    const double k = __fma_rd(v2, qinv_up, kTwo52) - kTwo52;            // floor(v2 / q): qinv_up >= 1/q by less than 2^-49 relative
    const double rb = __fma_rn(-k, c.qd, v2 + kTwo52);                   // 2^52 + (v2 - k q), exact
    return (u64)__double_as_longlong(rb) & 0x000FFFFFFFFFFFFFull;
}
// MADE: as in LongShoup::fwd16
template <bool MADE = false, class TW> __device__ __forceinline__ void fwd16_ds(double (&v)[16], const TW &tp, const DsConst &c) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int half = 8 >> s;
#pragma unroll
        for (int g = 0; g < (1 << s); ++g) {
            const ulonglong2 tw = tp[(1 << s) - 1 + g];
            const double wf = __longlong_as_double((long long)tw.y);
#pragma unroll
            for (int j = 0; j < half; ++j) {
                double &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                const double t = MADE && s == 0 ? y : ds_mul(y, tw.x, wf, c);
                y = x - t;
                x = x + t;
            }
        }
    }
}
template <class TW> __device__ __forceinline__ void fwd16_ds8(double (&v)[16], const TW &tp, const DsConst &c) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int half = 8 >> s;
#pragma unroll
        for (int g = 0; g < (1 << s); ++g) {
            const double wd = tp[(1 << s) - 1 + g];
#pragma unroll
            for (int j = 0; j < half; ++j) {
                double &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                const double t = ds_mul_w(y, wd, c);
                y = x - t;
                x = x + t;
            }
        }
    }
}
template <class TW> __device__ __forceinline__ void inv16_ds8(double (&v)[16], const TW &tp, const DsConst &c) {
#pragma unroll
    for (int s = 3; s >= 0; --s) {
        const int half = 8 >> s;
#pragma unroll
        for (int g = 0; g < (1 << s); ++g) {
            const double wd = tp[(1 << s) - 1 + g];
#pragma unroll
            for (int j = 0; j < half; ++j) {
                double &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                const double d = x - y;
                x = x + y;
                y = ds_mul_w(d, wd, c);
            }
        }
    }
    v[0] = ds_reduce(v[0], c);
}
// Gentleman-Sande round.  The sum path doubles per stage; only v[0] takes the sum at all four stages (16 x its
// inputs), v[1] ends below 4.2 q whatever came in, the others lower: the caller reduces v[0] after each round, so
// every round starts from values below 4.2 q and stays below 68 q.
template <int LAST = 0, class TW> __device__ __forceinline__ void inv16_ds(double (&v)[16], const TW &tp, const DsConst &c) {
#pragma unroll
    for (int s = 3; s >= LAST; --s) {
        const int half = 8 >> s;
#pragma unroll
        for (int g = 0; g < (1 << s); ++g) {
            const ulonglong2 tw = tp[(1 << s) - 1 + g];
            const double wf = __longlong_as_double((long long)tw.y);
#pragma unroll
            for (int j = 0; j < half; ++j) {
                double &x = v[g * 2 * half + j], &y = v[g * 2 * half + j + half];
                const double d = x - y;
                x = x + y;
                y = ds_mul(d, tw.x, wf, c);
            }
        }
    }
    if (LAST == 0) v[0] = ds_reduce(v[0], c);
}
// as inv16_int_last; the values come from three stages without a reduction (below 34 q, sums below 68 q), the products lie within 0.7 q of zero
template <class STORE> __device__ __forceinline__ void inv16_ds_last(const double (&v)[16], const u64 (&sw)[2], const u64 (&sc)[2], const DsConst &c, STORE &&store) {
    const double s0 = __longlong_as_double((long long)sc[0]), s1 = __longlong_as_double((long long)sc[1]), qinv_up = c.qinv * (1.0 + 0x1p-50);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        store(j, ds_store(ds_mul(v[j] + v[j + 8], sw[0], s0, c), c, c.qd, qinv_up));
        store(j + 8, ds_store(ds_mul(v[j] - v[j + 8], sw[1], s1, c), c, c.qd, qinv_up));
    }
}

// ---- forward, column pass: stages 1..8 ----
template <int MINB, class LONG>
__global__ void __launch_bounds__(256, MINB) ntt16v2_fwd_cols(const u64 *src, LimbAddr16 sa, u64 *dst, LimbAddr16 da,
                                                        const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    __shared__ u64 sm[4096];
    const int li = blockIdx.y, pi = map.prime[li % map.n];
    const PrimeConst m = pc[pi];
    const ulonglong2 *tab = tb.fwd + (size_t)pi * Ntt16Layout::kEntries;
    const int tid = threadIdx.x, lane = tid & 15, sub = tid >> 4;
    const u64 *p = src + sa.off(li, map.n) + blockIdx.x * 16 + lane;
    u64 *o = dst + da.off(li, map.n) + blockIdx.x * 16 + lane;
    if (m.small) {
        const DsConst c = ds_const(m);
        double v[16];
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = ds_load(p[(e * 16 + sub) * 256]);
        fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
        double *smd = reinterpret_cast<double *>(sm);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[(e * 16 + sub) * 16 + lane] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smd[(sub * 16 + e) * 16 + lane];
        fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
        double *od = reinterpret_cast<double *>(o);
#pragma unroll
        for (int e = 0; e < 16; ++e) od[(sub * 16 + e) * 256] = v[e];
    } else {
        u64 v[16];
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = p[(e * 16 + sub) * 256];
        const typename LONG::Const c = LONG::make(m);
        LONG::template fwd16<0>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) sm[(e * 16 + sub) * 16 + lane] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sm[(sub * 16 + e) * 16 + lane];
        LONG::template fwd16<1>(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[(sub * 16 + e) * 256] = v[e];
    }
}

// ---- forward, row pass: stages 9..16; stores canonical residues ----
template <int MINB, class LONG>
__global__ void __launch_bounds__(256, MINB) ntt16v2_fwd_rows(const u64 *src, LimbAddr16 sa, u64 *dst, LimbAddr16 da,
                                                        const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    __shared__ u64 sm[16 * kRowStride];
    const int li = blockIdx.y, pi = map.prime[li % map.n];
    const PrimeConst m = pc[pi];
    const ulonglong2 *tab = tb.fwd + (size_t)pi * Ntt16Layout::kEntries;
    const int tid = threadIdx.x, clo = tid & 15, rl = tid >> 4;
    const int row = blockIdx.x * 16 + rl;
    const u64 *p = src + sa.off(li, map.n) + (size_t)row * 256 + clo;
    u64 *o = dst + da.off(li, map.n) + (size_t)row * 256 + clo;
    u64 *smr = sm + rl * kRowStride;
    if (m.small) {
        const DsConst c = ds_const(m);
        const double *pd = reinterpret_cast<const double *>(p);
        double *smd = reinterpret_cast<double *>(smr);
        double v[16];
        const TwiddlesB<double, MINB <= 2> tw(tb.fwdB8 + (size_t)pi * kRowsB8 + (row * 15) * 16 + clo);
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = pd[e * 16];
        fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[e * 17 + clo] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smd[clo * 17 + e];
        fwd16_ds8(v, tw, c);
        const double shift = 16.0 * c.qd, qinv_up = c.qinv * (1.0 + 0x1p-50);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = ds_store(v[e], c, shift, qinv_up); // the words this thread read itself
    } else {
        const typename LONG::Const c = LONG::make(m);
        u64 v[16];
        const TwiddlesB<ulonglong2, MINB <= 2> tw(tab + Ntt16Layout::rowsB(row, 0, clo));
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = p[e * 16];
        LONG::template fwd16<2>(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[e * 17 + clo] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smr[clo * 17 + e];
        LONG::template fwd16<3>(v, tw, c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = LONG::canon(v[e], c);
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e * 16] = smr[e * 17 + clo];
}

// ---- inverse, row pass: undoes stages 16..9 ----
template <int MINB, class LONG>
__global__ void __launch_bounds__(256, MINB) ntt16v2_inv_rows(const u64 *src, LimbAddr16 sa, u64 *dst, LimbAddr16 da,
                                                        const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    __shared__ u64 sm[16 * kRowStride];
    const int li = blockIdx.y, pi = map.prime[li % map.n];
    const PrimeConst m = pc[pi];
    const ulonglong2 *tab = tb.inv + (size_t)pi * Ntt16Layout::kEntries;
    const int tid = threadIdx.x, clo = tid & 15, rl = tid >> 4;
    const int row = blockIdx.x * 16 + rl;
    const u64 *p = src + sa.off(li, map.n) + (size_t)row * 256 + clo;
    u64 *o = dst + da.off(li, map.n) + (size_t)row * 256 + clo;
    u64 *smr = sm + rl * kRowStride;
    const auto exchange_in = [&] { // the coefficients, row-major into shared memory
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[e * 17 + clo] = p[e * 16];
        __syncwarp();
    };
    if (m.small) {
        const TwiddlesB<double, MINB <= 2> tw(tb.invB8 + (size_t)pi * kRowsB8 + (row * 15) * 16 + clo);
        exchange_in();
        const DsConst c = ds_const(m);
        double *smd = reinterpret_cast<double *>(smr);
        double v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = ds_load(smr[clo * 17 + e]);
        inv16_ds8(v, tw, c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[clo * 17 + e] = v[e]; // the words this thread read itself
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smd[e * 17 + clo];
        inv16_ds(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
        double *od = reinterpret_cast<double *>(o);
#pragma unroll
        for (int e = 0; e < 16; ++e) od[e * 16] = v[e];
    } else {
        const TwiddlesB<ulonglong2, MINB <= 2> tw(tab + Ntt16Layout::rowsB(row, 0, clo));
        exchange_in();
        u64 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smr[clo * 17 + e];
        const typename LONG::Const c = LONG::make(m);
        LONG::inv16(v, tw, c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smr[e * 17 + clo];
        LONG::inv16(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e * 16] = v[e];
    }
}

// ---- inverse, column pass: undoes stages 8..1, scales by N^-1, stores canonical residues ----
template <int MINB, class LONG>
__global__ void __launch_bounds__(256, MINB) ntt16v2_inv_cols(const u64 *src, LimbAddr16 sa, u64 *dst, LimbAddr16 da,
                                                        const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    __shared__ u64 sm[4096];
    const int li = blockIdx.y, pi = map.prime[li % map.n];
    const PrimeConst m = pc[pi];
    const ulonglong2 *tab = tb.inv + (size_t)pi * Ntt16Layout::kEntries;
    const int tid = threadIdx.x, lane = tid & 15, sub = tid >> 4;
    const u64 *p = src + sa.off(li, map.n) + blockIdx.x * 16 + lane;
    u64 *o = dst + da.off(li, map.n) + blockIdx.x * 16 + lane;
    if (m.small) {
        const DsConst c = ds_const(m);
        const double *pd = reinterpret_cast<const double *>(p);
        double *smd = reinterpret_cast<double *>(sm);
        double v[16];
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = pd[(sub * 16 + e) * 256];
        inv16_ds(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[(sub * 16 + e) * 16 + lane] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smd[(e * 16 + sub) * 16 + lane];
        inv16_ds<1>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
        inv16_ds_last(v, m.n_inv_w, m.n_inv_c, c, [&](int e, u64 w) { o[(e * 16 + sub) * 256] = w; });
    } else {
        u64 v[16];
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = p[(sub * 16 + e) * 256];
        const typename LONG::Const c = LONG::make(m);
        LONG::inv16(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) sm[(sub * 16 + e) * 16 + lane] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sm[(e * 16 + sub) * 16 + lane];
        LONG::template inv16<1>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
        inv16_int_last<LONG>(v, m.n_inv_w, m.n_inv_c, c, [&](int e, u64 w) { o[(e * 16 + sub) * 256] = w; });
    }
}

// the column pass of a forward transform alone
inline cudaError_t launch_fwd_cols16(cudaStream_t st, u64 *d, size_t outer, int count, const LimbMap &map, const PrimeConst *pc, const Ntt16Tables &tb) {
    auto go = [&](auto *kernel) { return launch_pdl(st, kernel, dim3(16, count), 256, 0, d, LimbAddr16{outer}, d, LimbAddr16{outer}, map, pc, tb); };
    return tb.pm ? go(ntt16v2_fwd_cols<4, LongPm>) : go(ntt16v2_fwd_cols<4, LongShoup>);
}
// Launch a batched transform of `count` limb instances of 2^16 coefficients.  src == dst gives an in-place transform;
// with distinct buffers `dst` also serves as the intermediate between the two passes.  MINB = CTAs per SM the kernels
// are compiled for (register budget 65536 / (256 * MINB)); four measured fastest with the FP64 butterflies.
template <int MINB = 4>
inline cudaError_t launch_ntt16(cudaStream_t st, const u64 *src, size_t src_outer, u64 *dst, size_t dst_outer, int count, const LimbMap &map,
                                const PrimeConst *pc, const Ntt16Tables &tb, bool inverse) {
    if (count == 0) return cudaSuccess;
    LimbAddr16 sa{src_outer}, da{dst_outer};
    dim3 grid(16, count);
    auto passes = [&](auto *first, auto *second) {
        const cudaError_t e = launch_pdl(st, first, grid, 256, 0, src, sa, dst, da, map, pc, tb);
        return e != cudaSuccess ? e : launch_pdl(st, second, grid, 256, 0, dst, da, dst, da, map, pc, tb);
    };
    if (tb.pm) return inverse ? passes(ntt16v2_inv_rows<MINB, LongPm>, ntt16v2_inv_cols<MINB, LongPm>) : passes(ntt16v2_fwd_cols<MINB, LongPm>, ntt16v2_fwd_rows<MINB, LongPm>);
    return inverse ? passes(ntt16v2_inv_rows<MINB, LongShoup>, ntt16v2_inv_cols<MINB, LongShoup>) : passes(ntt16v2_fwd_cols<MINB, LongShoup>, ntt16v2_fwd_rows<MINB, LongShoup>);
}

} // namespace hb
