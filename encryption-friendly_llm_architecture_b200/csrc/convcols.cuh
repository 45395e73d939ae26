// Base conversions fused between the two halves of the 2^16 transforms (sm_100a).
//
// A base conversion (the lift of a key-switch digit, ModDown, the division by P * q_l, a rescale) works coefficient by
// coefficient across limbs, and the column pass of a transform works column by column inside a limb.  So one CTA that owns
// a strip of columns can finish the inverse transforms of the source limbs (their column pass), convert, and begin the
// forward transforms of the target limbs, without the coefficients ever leaving shared memory:
//
//     inverse row pass (ntt16v2_inv_rows)  ->  conv_cols / lift_cols  ->  forward row pass (ntt16v2_fwd_rows*)
//
// replaces inverse columns, conversion and forward columns as three kernels: for a conversion of S limbs to T, S reads + T
// writes instead of 3 S + S + 3 T limb transfers, and one launch instead of three.  The constants of a conversion carry the scale of the
// inverse transforms, the twiddle of their last stage and that of the first forward stage, which so cost no products of their own.
//
// At S = 4, T = 6 (the division by P * q_level at level 6) 96 polynomials take 315 us (324 with the counters; 413 with Shoup butterflies, 363 before the
// targets next to 2^60 were converted by pieces): half of the issue slots, FP64 38 % of the cycles, the wide multiply pipe 37 %.  Four warps a scheduler,
// whose fixed latencies, shared-memory exchanges and bursts on one pipe are the rest.  FP64 and integer products do overlap on a scheduler, unless the
// latter carry 64-bit addends.  What did not help: six warps a scheduler (4 x 4 strips, three CTAs at 80 registers, spills of 8 bytes: 364 us), a
// persistent version in which some groups transform the next strip's sources while others convert targets, CTAs of an SM started half a turn apart.
//
// A CTA is G groups of COLS * 16 threads.  Sources are dealt to the groups, then (one CTA barrier later) targets; inside a
// group a radix-16 round exchanges through shared memory behind a named barrier of that group only, so one group's loads,
// barriers and exchanges overlap the other's arithmetic.  Source residues stay in shared memory as two 30-bit pieces per
// word: products with 26-bit (or 30-bit) pieces of the constants are single 32 x 32 multiply-adds into 64-bit sums, on the
// integer pipe, which the FP64 butterflies around them leave idle.
#pragma once
#include "modarith.cuh"
#include "pdl.cuh"
#include "kernels.cuh"
#include "ntt16.cuh"
#include "conv_shared.hpp"
#include <type_traits>

namespace hb {

// One conversion: sources [ns] -> targets [nt].  scale: N^-1 * (D / d_s)^-1 mod d_s, as the last multiplication of the inverse transform.
struct ConvPlan {
    int ns, nt;
    int src_limb, dst_limb;             // first limb of the sources / targets inside one instance of the arrays
    unsigned char src_prime[8], dst_prime[kMaxPrimes];
    unsigned char order[kMaxPrimes];    // targets in the order they are taken: those of the long primes, which take twice the time, first
    u64 scale_w[8][2], scale_c[8][2];   // as scale_words makes them; [1]: times psi^(-N/2), the twiddle of the last inverse stage
    unsigned char fp[kMaxPrimes];       // target t converts on the FP64 pipe (see ConvFp)
    // The constants as they lie in shared memory: conv_const_words(ns) * 2 * ns words of 16 bytes for each target, in them [half of the rows][source],
    // the second half times psi^(N/2), the twiddle of the first forward stage: C = D / d_s mod target.
    //   fp targets, two words each: doubles C = d1 + d0 with d1 a multiple of 2^21, |d0| <= 2^20, C taken within q/2 of zero; the same for C * 2^30.
    //               Set when every sum of the products is exact in a double
    //   others, one word each: below 2^44 the 26-bit pieces of C and of C * 2^30; long targets the 30-bit pieces of C, their sum, 0, or (kPieceSources)
    //               the pieces of 29 and 31 bits of C and of C * 2^30
    uint4 k[conv_const_bytes(8, kMaxPrimes) / 16];
    // conv_mma (up to four sources, primes of LongPm): the target at position p of `order` has the 512 bytes from 32 p on, in them [half of the rows][block of
    // sixteen k][byte j][k]: byte j of C_s * 2^(8 i) modulo the target, k = 8 s + i
    uint4 bytes[kMaxPrimes * 32];
};
static_assert(conv_const_bytes(kFpSources, kMaxPrimes) <= conv_const_bytes(8, kMaxPrimes), "room for the longer constants");

template <int COLS> struct StripIndex { // [256 rows][COLS] words in shared memory, COLS pad words per 16 rows: both access patterns are conflict-free
    static constexpr int kWords = strip_words(COLS);
    static __device__ __forceinline__ int a(int e, int sub, int lane) { return e * 17 * COLS + sub * COLS + lane; }  // row e * 16 + sub
    static __device__ __forceinline__ int b(int e, int sub, int lane) { return sub * 17 * COLS + e * COLS + lane; }  // row sub * 16 + e
};
template <int THREADS> __device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(THREADS) : "memory"); }

// The words of a limb strip on their way to sm (at I::b), 16 bytes a copy; r: thread of the group.
template <int COLS> __device__ __forceinline__ void strip_fetch(const u64 *p /* limb + first column */, u64 *sm, int r) {
    using I = StripIndex<COLS>;
    constexpr int kChunks = COLS / 2; // of a row
    const int chunk = r % kChunks, row0 = r / kChunks;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int row = row0 + 32 * k;
        cp_async16(smem_u32(sm + I::b(row % 16, row / 16, 2 * chunk)), p + row * 256 + 2 * chunk);
    }
    cp_async_commit();
}
// Inverse column pass of one limb strip, whose words of the rows sub * 16 + e are in(e): word(canonical value times the scale) goes to sm at I::a,
// where this thread has read its own words.  sw, sc: the scale, and the scale times the twiddle of the last stage.
template <int COLS, class LONG, class IN, class WORD>
__device__ __forceinline__ void strip_inverse(IN &&in, u64 *sm, const PrimeConst &m, const ulonglong2 *__restrict__ tab, const u64 (&sw)[2], const u64 (&sc)[2],
                                              int g, int sub, int lane, WORD &&word) {
    using I = StripIndex<COLS>;
    if (m.small) {
        const DsConst c = ds_const(m);
        double *smd = reinterpret_cast<double *>(sm);
        double d[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) d[e] = __longlong_as_double((long long)in(e));
        inv16_ds(d, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[I::b(e, sub, lane)] = d[e];
        group_sync<COLS * 16>(g);
#pragma unroll
        for (int e = 0; e < 16; ++e) d[e] = smd[I::a(e, sub, lane)];
        inv16_ds<1>(d, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
        inv16_ds_last(d, sw, sc, c, [&](int e, u64 w) { sm[I::a(e, sub, lane)] = word(w); });
    } else {
        const typename LONG::Const c = LONG::make(m);
        u64 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = in(e);
        LONG::inv16(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) sm[I::b(e, sub, lane)] = v[e];
        group_sync<COLS * 16>(g);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sm[I::a(e, sub, lane)];
        LONG::template inv16<1>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
        inv16_int_last<LONG>(v, sw, sc, c, [&](int e, u64 w) { sm[I::a(e, sub, lane)] = word(w); });
    }
}
// Forward column pass of one limb strip that lies in sm (words of this thread at I::a; double bits below 2^44, |v| < 2q; otherwise below 3q, below 6.5q next to 2^60).
// MADE: the rows from 128 on already carry the twiddle of the first stage.
// between(): done before the barrier between the rounds.
template <int COLS, class LONG, bool MADE, class BETWEEN>
__device__ __forceinline__ void strip_forward(u64 *o /* limb + column */, u64 *sm, const PrimeConst &m, const ulonglong2 *__restrict__ tab, int g, int sub, int lane, BETWEEN &&between) {
    using I = StripIndex<COLS>;
    if (m.small) {
        const DsConst c = ds_const(m);
        double *smd = reinterpret_cast<double *>(sm);
        double d[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) d[e] = smd[I::a(e, sub, lane)];
        fwd16_ds<MADE>(d, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[I::a(e, sub, lane)] = d[e];
        between();
        group_sync<COLS * 16>(g);
#pragma unroll
        for (int e = 0; e < 16; ++e) d[e] = smd[I::b(e, sub, lane)];
        fwd16_ds(d, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) reinterpret_cast<double *>(o)[(sub * 16 + e) * 256] = d[e];
    } else {
        const typename LONG::Const c = LONG::make(m);
        u64 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sm[I::a(e, sub, lane)];
        LONG::template fwd16<0, MADE>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) sm[I::a(e, sub, lane)] = v[e];
        between();
        group_sync<COLS * 16>(g);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sm[I::b(e, sub, lane)];
        LONG::template fwd16<1>(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[(sub * 16 + e) * 256] = v[e];
    }
}

// a0 + a1 * 2^26 modulo a prime below 2^44 (a1 < 2^52, a0 < 2^61) as an integer-valued double within 2q of zero.  The quotient
// comes from the FP64 pipe (both sums enter through the 2^52 exponent without a conversion, the offsets are folded into `base`),
// the remainder is exact in the low 64 bits.  The quotient is off by its two roundings, by the low word of a0 that it leaves out
// (up to 2^32 / q) and by the rounding of `base`, whose size is 2^84 / q: 1.7 in all from q = 2^34 on, but 50 at 27 bits.  The
// forward row pass adds 16 q to outputs that carry coefficient 0 unreduced, so below 2^34 the remainder is reduced once more (it
// is below 2^36 there, whatever q).
struct SmallFinish { double k1, k0, base; u32 n0, n1, hi0; bool again; };
__device__ __forceinline__ SmallFinish small_finish(const PrimeConst &m) {
    SmallFinish f;
    f.k1 = 0x1p26 * m.q_inv_f; f.k0 = 0x1p32 * m.q_inv_f;
    f.base = kMagic - kTwo52 * (f.k1 + f.k0);
    const u64 nq = 0ull - m.q;
    f.n0 = (u32)nq; f.n1 = (u32)(nq >> 32);
    f.hi0 = 0x43380000u - 0x43380000u * f.n0; // exponent word of the result, minus what the exponent word of the quotient contributes
    f.again = m.q < (1ull << 34);
    return f;
}
__device__ __forceinline__ double finish_small(u64 a0, u64 a1, const SmallFinish &f) {
    const double d1 = __hiloint2double((int)((u32)(a1 >> 32) | 0x43300000u), (int)(u32)a1), d0 = __hiloint2double(0x43300000, (int)(u32)(a0 >> 32));
    const double qh = __fma_rn(d1, f.k1, __fma_rn(d0, f.k0, f.base));
    const u64 l = a0 + (a1 << 26);
    const u32 q0 = (u32)__double2loint(qh), q1 = (u32)__double2hiint(qh);
    const u64 r = mad_wide(q0, f.n0, l);
    const u32 hi = q1 * f.n0 + (q0 * f.n1 + (u32)(r >> 32)) + f.hi0;
    return __hiloint2double((int)hi, (int)(u32)r) - kMagic;
}
// The conversions of one target for this thread's sixteen coefficients, into sm (at I::a).  Eight coefficients at a time in a rolled loop:
// the constants are fetched twice instead of held, and the straight-line code stays small (warps of a CTA work on
// different targets, so long code is fetched again and again).  NS: the number of sources, 0 for any; three (ModDown) and four (digits, the
// division by P * q_level) are unrolled.  Not in the narrow strips with Shoup products, whose transforms are the longest code: their short launches
// spend more on fetching it than the unrolled products save.  One ciphertext at level 8, its two conversions, us, unrolled / not: 38.3 / 36.4 and
// 31.6 / 29.7.  Next to 2^60 it goes both ways by 2 %: rotations of one ciphertext at level 8 106.1 / 103.5, of four at level 12 354 / 356.
//
// On the FP64 pipe: y = y0 + y1 * 2^30 as two doubles, sums a0 of y * d0 and a1 of y * d1 (both exact: below 2^53, and below 2^53
// units of 2^21), remainder of a1 + a0.  Sixteen products and eight conversions for four sources, 58 FP64 cycles per warp
// coefficient of the 79 that it takes with four warps a scheduler (four coefficients at a time and a loop over the sources: 88).
template <int COLS, int NS>
__device__ __forceinline__ void convert_target_fp(u64 *sm, const u64 *ysm, const uint4 *cst, int ns_, const PrimeConst &m, int sub, int lane) {
    using I = StripIndex<COLS>;
    const int ns = NS ? NS : ns_;
    const double qinv = m.q_inv_f, qd = (double)m.q;
#pragma unroll 1
    for (int e0 = 0; e0 < 16; e0 += 8) {
        double a0[8], a1[8];
        auto source = [&](int s, bool first) {
            const double2 *k = reinterpret_cast<const double2 *>(cst + ((e0 >> 3) * ns + s) * 2), k0 = k[0], k1 = k[1];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const u64 y = ysm[s * I::kWords + I::a(e0 + u, sub, lane)];
                const double y0 = __hiloint2double(0x43300000, (int)(u32)y) - kTwo52, y1 = __hiloint2double(0x43300000, (int)(u32)(y >> 32)) - kTwo52;
                a0[u] = first ? __dmul_rn(y0, k0.x) : __fma_rn(y0, k0.x, a0[u]); a1[u] = first ? __dmul_rn(y0, k0.y) : __fma_rn(y0, k0.y, a1[u]);
                a0[u] = __fma_rn(y1, k1.x, a0[u]); a1[u] = __fma_rn(y1, k1.y, a1[u]);
            }
        };
        source(0, true);
#pragma unroll (NS ? NS : 1)
        for (int s = 1; s < ns; ++s) source(s, false);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double qh = __fma_rn(a1[u], qinv, __fma_rn(a0[u], qinv, kMagic)) - kMagic;
            sm[I::a(e0 + u, sub, lane)] = (u64)__double_as_longlong(__fma_rn(-qh, qd, a1[u]) + a0[u]); // within 1.1 q of zero
        }
    }
}
template <int COLS>
__device__ __forceinline__ void convert_target_small(u64 *sm, const u64 *ysm, const uint4 *cst, int ns, const PrimeConst &m, int sub, int lane) {
    using I = StripIndex<COLS>;
    const SmallFinish f = small_finish(m);
    const DsConst ds = ds_const(m);
#pragma unroll 1
    for (int e0 = 0; e0 < 16; e0 += 4) {
        u64 a0[4], a1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { a0[u] = 0; a1[u] = 0; }
#pragma unroll 1
        for (int s = 0; s < ns; ++s) {
            const uint4 c = cst[(e0 >> 3) * ns + s];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u64 y = ysm[s * I::kWords + I::a(e0 + u, sub, lane)];
                a0[u] = mad_wide((u32)y, c.x, a0[u]); a1[u] = mad_wide((u32)y, c.y, a1[u]);
                a0[u] = mad_wide((u32)(y >> 32), c.z, a0[u]); a1[u] = mad_wide((u32)(y >> 32), c.w, a1[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            double v = finish_small(a0[u], a1[u], f);
            if (f.again) v = ds_reduce(v, ds);
            sm[I::a(e0 + u, sub, lane)] = (u64)__double_as_longlong(v);
        }
    }
}
template <int COLS>
__device__ __forceinline__ void convert_target_wide(u64 *sm, const u64 *ysm, const uint4 *cst, int ns, const PrimeConst &m, int sub, int lane) {
    using I = StripIndex<COLS>;
#pragma unroll 1
    for (int e0 = 0; e0 < 16; e0 += 4) {
        u64 a0[4], am[4], a2[4]; // as in PieceAcc
#pragma unroll
        for (int u = 0; u < 4; ++u) { a0[u] = 0; am[u] = 0; a2[u] = 0; }
#pragma unroll 2
        for (int s = 0; s < ns; ++s) {
            const uint4 c = cst[(e0 >> 3) * ns + s];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u64 y = ysm[s * I::kWords + I::a(e0 + u, sub, lane)];
                const u32 y0 = (u32)y, y1 = (u32)(y >> 32);
                a0[u] = mad_wide(y0, c.x, a0[u]); am[u] = mad_wide(y0 + y1, c.z, am[u]); a2[u] = mad_wide(y1, c.y, a2[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) sm[I::a(e0 + u, sub, lane)] = finish_wide(a0[u], am[u] - a0[u] - a2[u], a2[u], m);
    }
}

// The same to a prime next to 2^60 from at most four sources: C and C * 2^30 in pieces of 29 and 31 bits, sums A and B of weight 2^29 that stay below 2^63
// and 2^64, folded as in LongPm::mul: below 6.5 * 2^60.  Four sources take 85 cycles per warp coefficient with four warps a
// scheduler, three 72; three products a source (convert_target_wide) with their longer reduction 126 and 107.
template <int COLS, int NS>
__device__ __forceinline__ void convert_target_pm(u64 *sm, const u64 *ysm, const uint4 *cst, int ns_, const PrimeConst &m, int sub, int lane) {
    using I = StripIndex<COLS>;
    const int ns = NS ? NS : ns_;
    const u32 d2 = 2 * m.d60;
#pragma unroll 1
    for (int e0 = 0; e0 < 16; e0 += 4) {
        u64 a[4], b[4];
        auto source = [&](int s, bool first) {
            const uint4 c = cst[(e0 >> 3) * ns + s];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u64 y = ysm[s * I::kWords + I::a(e0 + u, sub, lane)];
                const u32 y0 = (u32)y, y1 = (u32)(y >> 32);
                const u64 p = LongPm::add(LongPm::wide(y0, c.x), LongPm::wide(y1, c.z)), r = LongPm::add(LongPm::wide(y0, c.y), LongPm::wide(y1, c.w));
                a[u] = first ? p : LongPm::add(a[u], p);
                b[u] = first ? r : LongPm::add(b[u], r);
            }
        };
        source(0, true);
#pragma unroll (NS ? NS : 1)
        for (int s = 1; s < ns; ++s) source(s, false);
#pragma unroll
        for (int u = 0; u < 4; ++u) sm[I::a(e0 + u, sub, lane)] = LongPm::add(LongPm::add(a[u], LongPm::shl29((u32)b[u])), LongPm::wide((u32)(b[u] >> 32), d2));
    }
}
template <class LONG> constexpr int kPieceSources = 0; // up to this many sources the constants of long targets are those of convert_target_pm
template <> inline constexpr int kPieceSources<LongPm> = 4;

// src: half-inverse limbs (after the inverse row pass), instance b at src + b * src_outer; dst: half-forward limbs.
// grid = (256 / COLS, plans, instances).  Dynamic shared memory: (largest ns + G) strips, then 2 * nt * ns constants: their loads stand in front of
// every few products, and what L1 is left beside the strips holds no more than the twiddles.  All sources are on their way
// from the start instead of behind one another.  The two together: 139 -> 129 ms
// of the layer's conversions, products of 256 members at level 8 5.69 -> 5.33 ms.
// The constants take no more room than they need: with eight sources the second CTA of an SM depends on it (conv_shared.hpp).  Divisions of 24 polynomials
// by P * q_22, eight sources, us: 32 bytes a constant and one CTA 518, 16 bytes and two 421.
// MAXNS: the most sources a conversion may have.  With no more of them than groups and Shoup products their words go straight to registers:
// the way through shared memory and the barrier behind it hide nothing then (one ciphertext at level 8, three digits and ModDown, us, through shared memory / straight: 36.8 / 35.7 and 29.8 /
// 28.9).  Next to 2^60 it is even: divisions of one ciphertext at level 12 78.3 / 79.1, rotations 135.9 / 135.5.  Six sources on four groups 59.0 /
// 62.2: there the second strip arrives behind the first one's work.
template <int COLS, int G, int MINB, int MAXNS, class LONG>
__global__ void __launch_bounds__(COLS * 16 * G, MINB) conv_cols(const u64 *src, size_t src_outer, u64 *dst, size_t dst_outer, const ConvPlan *__restrict__ plans,
                                                                         const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    extern __shared__ __align__(128) u64 strips[]; // rows of 32 bytes at an odd multiple of 16 take 2.4 % longer in all
    __shared__ int next, turn[2][G];
    using I = StripIndex<COLS>;
    constexpr bool kShoup = kPieceSources<LONG> == 0, kOne = MAXNS <= G && kShoup;
    if (threadIdx.x == 0) next = G <= 2 ? G : 0;
    const ConvPlan *pl = plans + blockIdx.y;
    const int ns = pl->ns, nt = pl->nt, words = MAXNS <= kFpSources ? 2 : conv_const_words(ns);
    const int g = threadIdx.x / (COLS * 16), r = threadIdx.x % (COLS * 16), lane = r % COLS, sub = r / COLS;
    const int col = blockIdx.x * COLS + lane;
    const u64 *sp = src + (size_t)blockIdx.z * src_outer + (size_t)pl->src_limb * kN16 + blockIdx.x * COLS;
    u64 *dp = dst + (size_t)blockIdx.z * dst_outer + (size_t)pl->dst_limb * kN16 + col;
    uint4 *consts = reinterpret_cast<uint4 *>(strips + (ns + G) * I::kWords);
    for (int i = threadIdx.x; i < 2 * nt * ns * words; i += COLS * 16 * G) consts[i] = pl->k[i];
    pdl_wait();
    if (!kOne) for (int s = g; s < ns; s += G) strip_fetch<COLS>(sp + (size_t)s * kN16, strips + s * I::kWords, r);
    for (int s = g; s < ns; s += G) {
        if (!kOne) {
            if (s + G < ns) cp_async_wait<1>(); else cp_async_wait<0>(); // at most one more strip of this group may be on its way
            group_sync<COLS * 16>(g);
        }
        const int pi = pl->src_prime[s];
        u64 *sm = strips + s * I::kWords;
        const u64 *gm = sp + (size_t)s * kN16 + lane;
        strip_inverse<COLS, LONG>([&](int e) { return kOne ? gm[(sub * 16 + e) * 256] : sm[I::b(e, sub, lane)]; }, sm, pc[pi], tb.inv + (size_t)pi * Ntt16Layout::kEntries, pl->scale_w[s], pl->scale_c[s], g, sub, lane,
                            [](u64 v) { return ((v >> 30) << 32) | ((u32)v & 0x3FFFFFFFu); });
    }
    __syncthreads();
    u64 *ex = strips + (ns + g) * I::kWords;
    // The groups take targets from a common counter.  Two groups take their next one in the middle of the present transform, whose barrier makes it known:
    // asked for at the end it costs a barrier and a round trip, 1000 cycles a target (conversions of 256 products at level 8 4.66 -> 4.50 ms).  More
    // groups keep the end: there one with a long target would take early what another could begin at once.
    auto target = [&](int k, auto &&between) {
        const int t = pl->order[k];
        const int pi = pl->dst_prime[t];
        const PrimeConst m = pc[pi];
        const uint4 *cst = consts + 2 * t * ns * words;
        const bool fp = pl->fp[t];
        constexpr bool kUnroll = COLS == 8 || !kShoup;
        if (fp) {
            if (kUnroll && ns == 4) convert_target_fp<COLS, kUnroll ? 4 : 0>(ex, strips, cst, ns, m, sub, lane);
            else if (kUnroll && ns == 3) convert_target_fp<COLS, kUnroll ? 3 : 0>(ex, strips, cst, ns, m, sub, lane);
            else convert_target_fp<COLS, 0>(ex, strips, cst, ns, m, sub, lane);
        } else if (!kShoup && !m.small && ns <= kPieceSources<LONG>) {
            if (kUnroll && ns == 4) convert_target_pm<COLS, kUnroll ? 4 : 0>(ex, strips, cst, ns, m, sub, lane);
            else if (kUnroll && ns == 3) convert_target_pm<COLS, kUnroll ? 3 : 0>(ex, strips, cst, ns, m, sub, lane);
            else convert_target_pm<COLS, 0>(ex, strips, cst, ns, m, sub, lane);
        } else if (m.small) convert_target_small<COLS>(ex, strips, cst, ns, m, sub, lane);
        else convert_target_wide<COLS>(ex, strips, cst, ns, m, sub, lane);
        strip_forward<COLS, LONG, true>(dp + (size_t)t * kN16, ex, m, tb.fwd + (size_t)pi * Ntt16Layout::kEntries, g, sub, lane, between);
    };
    if constexpr (G <= 2) {
        for (int k = g, odd = 0; k < nt; odd ^= 1) {
            target(k, [&] { if (r == 0) turn[odd][g] = atomicAdd(&next, 1); });
            k = turn[odd][g];
            group_sync<COLS * 16>(g); // the strip has been read
        }
    } else {
        while (true) {
            group_sync<COLS * 16>(g); // the strip of the previous target has been read
            if (r == 0) turn[0][g] = atomicAdd(&next, 1);
            group_sync<COLS * 16>(g);
            const int k = turn[0][g];
            if (k >= nt) break;
            target(k, [] {});
        }
    }
}

// Rescale: one source limb (prime index `level`), lifted centred to the limbs 0 .. level - 1.  One group per CTA where there are many
// instances: a second one would wait for the source.
// grid = (256 / COLS, instances); dynamic shared memory: 1 + G strips.
template <int COLS, int G, int MINB, class LONG>
__global__ void __launch_bounds__(COLS * 16 * G, MINB) lift_cols(const u64 *src, size_t src_outer, u64 *dst, size_t dst_outer, int level,
                                                                         const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    extern __shared__ __align__(128) u64 strips[];
    using I = StripIndex<COLS>;
    const int g = threadIdx.x / (COLS * 16), r = threadIdx.x % (COLS * 16), lane = r % COLS, sub = r / COLS;
    const int col = blockIdx.x * COLS + lane;
    const u64 ql = pc[level].q;
    const bool src_small = pc[level].small;
    pdl_wait();
    if (g == 0) {
        const PrimeConst m = pc[level];
        const u64 *sp = src + (size_t)blockIdx.y * src_outer + col;
        strip_inverse<COLS, LONG>([&](int e) { return sp[(sub * 16 + e) * 256]; }, strips, m, tb.inv + (size_t)level * Ntt16Layout::kEntries, m.n_inv_w, m.n_inv_c, g, sub, lane,
                            [&](u64 v) { return v > (ql >> 1) ? v - ql : v; }); // signed
    }
    __syncthreads();
    u64 *dp = dst + (size_t)blockIdx.y * dst_outer + col, *ex = strips + (1 + g) * I::kWords;
    for (int t = g; t < level; t += G) {
        const PrimeConst m = pc[t];
        group_sync<COLS * 16>(g); // the strip of the previous target has been read
#pragma unroll 4
        for (int e = 0; e < 16; ++e) {
            const i64 y = (i64)strips[I::a(e, sub, lane)];
            u64 &w = ex[I::a(e, sub, lane)];
            if (m.small && src_small && (ql >> 1) < 2 * m.q) w = (u64)__double_as_longlong(__longlong_as_double(y + 0x4338000000000000ll) - kMagic); // within 2q of zero
            else if (m.small) w = (u64)__double_as_longlong(u52_to_double(reduce_i64(y, m)));
            else if ((ql >> 1) < m.q) w = y < 0 ? (u64)(y + (i64)m.q) : (u64)y;
            else w = reduce_i64(y, m);
        }
        strip_forward<COLS, LONG, false>(dp + (size_t)t * kN16, ex, m, tb.fwd + (size_t)t * Ntt16Layout::kEntries, g, sub, lane, [] {});
    }
}

// ---- forward row pass with the last step of a division ----
//   out[b][p][l] = (x[b][p][l] - t[b][p][l]) * inv_l  (+ add_p[b][l] o perm_g, ADD: addends and g of the member's group)
// t arrives half-forward (conv_cols / lift_cols).  grid = (16, n, instances), instance bp = b * np + p.  The operands of the last
// step are read after the barrier of the final exchange, when the registers of the transform are free.  Without addends bound by DRAM
// and the FP64 pipe together: 128 polynomials of six limbs 226 us, 5.4 TB/s of DRAM traffic (0.83 of a copy), FP64 pipe 50 % busy; with
// addends 424 us for 96 of nine limbs, 4.5 TB/s.  64 registers for four CTAs per SM spill 4 to 16 bytes a thread.
struct RowsFin {
    const u64 *x; size_t x_outer;            // instance stride of x; limb l at l * N
    u64 *out; size_t out_outer;              // ciphertext stride; polynomial p at p * n * N
    int np, batch; size_t add_outer;         // ciphertexts per group, ciphertext stride of the addends
};
struct InvScale { u64 w[kMaxPrimes], c[kMaxPrimes]; }; // per limb, as scale_words makes them
struct NoAddends {};
template <int MINB, class ADD /* SwitchList or NoAddends */, class LONG>
__global__ void __launch_bounds__(256, MINB) ntt16v2_fwd_rows_fin(const u64 *t, size_t t_outer, const __grid_constant__ RowsFin f, const __grid_constant__ InvScale sc, const __grid_constant__ ADD add,
                                                            const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    __shared__ u64 sm[16 * kRowStride];
    const int l = blockIdx.y, bp = blockIdx.z, b = bp / f.np, p = bp % f.np, n = gridDim.y;
    const PrimeConst m = pc[l];
    const ulonglong2 *tab = tb.fwd + (size_t)l * Ntt16Layout::kEntries;
    const int tid = threadIdx.x, clo = tid & 15, rl = tid >> 4;
    const int row = blockIdx.x * 16 + rl;
    const size_t pos = (size_t)row * 256 + clo, limb = (size_t)l * kN16;
    const u64 *tp = t + (size_t)bp * t_outer + limb + pos;
    const u64 *xp = f.x + (size_t)bp * f.x_outer + limb + pos;
    const u64 *ap = nullptr;
    u32 g = 0;
    if constexpr (!std::is_same_v<ADD, NoAddends>) {
        const SwitchGroup &sg = add.s[b / f.batch];
        g = sg.g;
        if (sg.add[p]) ap = sg.add[p] + (size_t)(b % f.batch) * f.add_outer + limb;
    }
    u64 *o = f.out + (size_t)b * f.out_outer + ((size_t)p * n + l) * kN16 + pos;
    u64 *smr = sm + rl * kRowStride;
    if (tid == 0) { // what the last step reads is on its way while the transform runs
        const size_t first = (size_t)blockIdx.x * 4096;
        prefetch_l2(f.x + (size_t)bp * f.x_outer + limb + first, 4096 * 8);
        if (ap) prefetch_l2(ap + (g ? ntt_perm((u32)first, g, 16) & ~4095u : (u32)first), 4096 * 8);
    }
    if (m.small) {
        const DsConst c = ds_const(m);
        const double *td = reinterpret_cast<const double *>(tp);
        double *smd = reinterpret_cast<double *>(smr);
        double v[16];
        const TwiddlesB<double, MINB <= 2> tw(tb.fwdB8 + (size_t)l * kRowsB8 + (row * 15) * 16 + clo);
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = td[e * 16];
        fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[e * 17 + clo] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smd[clo * 17 + e];
        fwd16_ds8(v, tw, c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smd[clo * 17 + e] = v[e]; // the words this thread read itself
        u64 x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = xp[e * 16];
        __syncwarp();
        const double sf = __longlong_as_double((long long)sc.c[l]), qinv_up = c.qinv * (1.0 + 0x1p-50);
        const u64 sw = sc.w[l];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            double r = ds_mul(ds_load(x[e]) - smd[e * 17 + clo], sw, sf, c); // within 0.52 q of zero
            if (ap) r += ds_load(ap[g ? ntt_perm((u32)(pos + e * 16), g, 16) : (u32)(pos + e * 16)]);
            o[e * 16] = ds_store(r, c, c.qd, qinv_up);
        }
    } else {
        const typename LONG::Const c = LONG::make(m);
        u64 v[16];
        const TwiddlesB<ulonglong2, MINB <= 2> tw(tab + Ntt16Layout::rowsB(row, 0, clo));
        pdl_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = tp[e * 16];
        LONG::template fwd16<2>(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[e * 17 + clo] = v[e];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = smr[clo * 17 + e];
        LONG::template fwd16<3>(v, tw, c);
#pragma unroll
        for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = v[e];
        u64 x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = xp[e * 16];
        __syncwarp();
        const u64 sw = sc.w[l], ss = sc.c[l];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            u64 r = LONG::mul(x[e] + LONG::above_fwd(c) - smr[e * 17 + clo], sw, ss, c); // below 7q
            if (ap) r += ap[g ? ntt_perm((u32)(pos + e * 16), g, 16) : (u32)(pos + e * 16)];
            o[e * 16] = LONG::canon(r, c);
        }
    }
}

// Single passes, for the fused sequences.  A grid of one or two CTAs per SM takes the kernels that may use 128 registers and
// fetch the twiddles of the second round (which nobody shares) before anything else, under the tail of the predecessor.
constexpr int kSmallGrid = 2 * 148;
// From this many CTAs on, the passes that follow a conversion are launched the ordinary way: under programmatic dependence their CTAs would
// move onto SMs that the conversion still holds at its 208 KB of shared memory, and the SMs would keep that split, with the smallest L1, for
// all kernels of the sequence (forward row passes with the last step 255 -> 312 us, tensor products 201 -> 229, masked inner products 484 -> 537).
constexpr int kPlainGrid = 4 * 4 * 148;
template <class... P, class... A> inline cudaError_t launch_plain(cudaStream_t st, void (*kernel)(P...), dim3 grid, dim3 block, A &&...args) {
    kernel<<<grid, block, 0, st>>>(P(std::forward<A>(args))...);
    return cudaPeekAtLastError();
}
inline cudaError_t launch_inv_rows16(cudaStream_t st, const u64 *src, size_t src_outer, u64 *dst, size_t dst_outer, int count, const LimbMap &map, const PrimeConst *pc, const Ntt16Tables &tb) {
    auto go = [&](auto *small, auto *kernel) { return launch_pdl(st, 16 * count <= kSmallGrid ? small : kernel, dim3(16, count), 256, 0, src, LimbAddr16{src_outer}, dst, LimbAddr16{dst_outer}, map, pc, tb); };
    return tb.pm ? go(ntt16v2_inv_rows<2, LongPm>, ntt16v2_inv_rows<4, LongPm>) : go(ntt16v2_inv_rows<2, LongShoup>, ntt16v2_inv_rows<4, LongShoup>);
}
inline cudaError_t launch_fwd_rows16(cudaStream_t st, u64 *d, size_t outer, int count, const LimbMap &map, const PrimeConst *pc, const Ntt16Tables &tb) {
    auto go = [&](auto *small, auto *kernel) {
        if (16 * count >= kPlainGrid) return launch_plain(st, kernel, dim3(16, count), 256, d, LimbAddr16{outer}, d, LimbAddr16{outer}, map, pc, tb);
        return launch_pdl(st, 16 * count <= kSmallGrid ? small : kernel, dim3(16, count), 256, 0, d, LimbAddr16{outer}, d, LimbAddr16{outer}, map, pc, tb);
    };
    return tb.pm ? go(ntt16v2_fwd_rows<2, LongPm>, ntt16v2_fwd_rows<4, LongPm>) : go(ntt16v2_fwd_rows<2, LongShoup>, ntt16v2_fwd_rows<4, LongShoup>);
}
template <class ADD>
inline cudaError_t launch_fwd_rows_fin16(cudaStream_t st, const u64 *t, size_t t_outer, int n, int instances, const RowsFin &f, const InvScale &sc, const ADD &add, const PrimeConst *pc, const Ntt16Tables &tb) {
    auto go = [&](auto *small, auto *kernel) {
        if (16 * n * instances >= kPlainGrid) return launch_plain(st, kernel, dim3(16, n, instances), 256, t, t_outer, f, sc, add, pc, tb);
        return launch_pdl(st, 16 * n * instances <= kSmallGrid ? small : kernel, dim3(16, n, instances), 256, 0, t, t_outer, f, sc, add, pc, tb);
    };
    return tb.pm ? go(ntt16v2_fwd_rows_fin<2, ADD, LongPm>, ntt16v2_fwd_rows_fin<4, ADD, LongPm>) : go(ntt16v2_fwd_rows_fin<2, ADD, LongShoup>, ntt16v2_fwd_rows_fin<4, ADD, LongShoup>);
}

} // namespace hb
