// Base conversions between the two halves of the 2^16 transforms with their products on the tensor cores (sm_100a): what conv_cols does, for up to four
// sources and LongPm primes.
//
// A target residue is sum_s y_s * C_s modulo q.  With y_s in its eight bytes and the constants C_s * 2^(8 i) mod q in theirs, the eight sums
//     S_j = sum_(s, i) byte_i(y_s) * byte_j(C_s * 2^(8 i) mod q)         (at most 4 * 8 products of bytes, below 2^21)
// are the columns of a product of whole numbers, [coefficients x 32] * [32 x 8 per target], and sum_j S_j * 2^(8 j) is congruent to the residue.  tcgen05.mma
// of kind i8 forms them in tensor memory for 128 coefficients a piece; what is left for a thread is to put the eight columns of its
// coefficient together, with one small quotient, and it takes them in the very order in which it starts the forward transform, so
// that they go from tensor memory to the registers of its first round.
//
// Three digits of 48 polynomials at level 8: 513 us, conv_cols 548 (277 -> 239 million warp instructions; ModDown of 96 polynomials 370 -> 355, 198 -> 167);
// calls beside the other strips at the rule that chooses (conv_shape).  The tensor cores are busy in 2 % of the cycles; bound, as before, by four
// warps a scheduler that issue in 44 % of the slots: FP64 33 % of the cycles, the wide multiply pipe 30 %, tensor and shared
// memory leave no room for more warps.  Not better: twiddles asked for early or from one address (no change), targets of long and short primes side by
// side (0 to 1 % either way), one persistent CTA per place that fetches its next strips behind the last products (2 to 4 % slower; with
// four groups 2 % faster, still behind two).
#pragma once
#include "convcols.cuh"

namespace hb {

__device__ __forceinline__ u64 mma_desc(u32 smem, u32 k_bytes, u32 row_bytes) { // operand without swizzle: 8 x 16 byte blocks, strides along K and along the rows
    return (u64)(smem >> 4) | (u64)(k_bytes >> 4) << 16 | (u64)(row_bytes >> 4) << 32 | (u64)1 << 46;
}
__device__ __forceinline__ void mma_i8(u32 d, u64 a, u64 b, u32 idesc) { // d = a * b, 128 rows, unsigned bytes
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(0) : "memory");
}
__device__ __forceinline__ void mma_commit(u64 *bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// eight columns of this thread's row at a, at a + step, ... : four coefficients
__device__ __forceinline__ void tmem_load4x8(u32 (&s)[4][8], u32 a, u32 step) {
    asm volatile("{\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%33];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%34];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%35];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t}"
                 : "=r"(s[0][0]), "=r"(s[0][1]), "=r"(s[0][2]), "=r"(s[0][3]), "=r"(s[0][4]), "=r"(s[0][5]), "=r"(s[0][6]), "=r"(s[0][7]),
                   "=r"(s[1][0]), "=r"(s[1][1]), "=r"(s[1][2]), "=r"(s[1][3]), "=r"(s[1][4]), "=r"(s[1][5]), "=r"(s[1][6]), "=r"(s[1][7]),
                   "=r"(s[2][0]), "=r"(s[2][1]), "=r"(s[2][2]), "=r"(s[2][3]), "=r"(s[2][4]), "=r"(s[2][5]), "=r"(s[2][6]), "=r"(s[2][7]),
                   "=r"(s[3][0]), "=r"(s[3][1]), "=r"(s[3][2]), "=r"(s[3][3]), "=r"(s[3][4]), "=r"(s[3][5]), "=r"(s[3][6]), "=r"(s[3][7])
                 : "r"(a), "r"(a + step), "r"(a + 2 * step), "r"(a + 3 * step)
                 : "memory");
}
// sum of S_j * 2^(8 j), j < 6 (below 2^62), modulo a prime below 2^44: an integer-valued double within 1.1 q of zero.  The sums enter the FP64 pipe through
// exponents of 2^52, 2^68 and 2^84 without a conversion; every step but the quotient is exact.
__device__ __forceinline__ double join_small(const u32 (&s)[8], double qinv, double qd) {
    const u32 t0 = s[0] + (s[1] << 8), t1 = s[2] + (s[3] << 8), t2 = s[4] + (s[5] << 8); // below 2^30
    const double a0 = (__hiloint2double(0x44300000, (int)t1) - (0x1p68 + 0x1p52)) + __hiloint2double(0x43300000, (int)t0);
    const double a1 = __hiloint2double(0x45300000, (int)t2) - 0x1p84;
    const double qh = __fma_rn(a1, qinv, __fma_rn(a0, qinv, kMagic)) - kMagic;
    return __fma_rn(-qh, qd, a1) + a0;
}
// the same for all eight modulo 2^60 - d: below 2^60 + 2^46
__device__ __forceinline__ u64 join_long(const u32 (&s)[8], u32 d) {
    const u64 lo = mad_wide(s[2] + (s[3] << 8), 1u << 16, (u64)(s[0] + (s[1] << 8))), hi = mad_wide(s[6] + (s[7] << 8), 1u << 16, (u64)(s[4] + (s[5] << 8))); // below 2^46
    return mad_wide((u32)(hi >> 28), d, lo) + ((u64)((u32)hi & 0x0FFFFFFFu) << 32); // 2^60 = d
}

// Grid as conv_cols: (32, plans, instances), strips of eight columns, G groups of 128 threads, G sources and then G targets at a time.
// Shared memory: four source strips, an exchange strip per group, the constants.  A pair of source strips turns into one half of the operand
// tiles: tile e has the coefficients of rows 16 e .. 16 e + 15 (of the thread r of a group in row r), sources 2 h and 2 h + 1 in the 16 bytes of block column h.
// Tensor memory: 16 tiles x 8 columns a target, G targets; all of it for two CTAs of two groups or one of four.
constexpr size_t conv_mma_smem(int G, int nt) { return ((size_t)(4 + G) * strip_words(8)) * 8 + (size_t)((nt + G - 1) / G * G) * 512; }
template <int G, int MINB>
__global__ void __launch_bounds__(128 * G, MINB) conv_mma(const u64 *src, size_t src_outer, u64 *dst, size_t dst_outer, const ConvPlan *__restrict__ plans, const PrimeConst *__restrict__ pc,
                                                          Ntt16Tables tb, int *err) {
    using LONG = LongPm;
    using I = StripIndex<8>;
    constexpr u32 kPair = 2 * I::kWords * 8, kColumns = 128 * G, kIdesc = 2u << 4 | (u32)G << 17 | 8u << 24; // 32-bit sums, 8 G columns, 128 rows
    extern __shared__ __align__(128) u64 strips[];
    __shared__ __align__(8) u64 bar;
    __shared__ u32 tmem;
    const int tid = threadIdx.x, g = tid / 128, r = tid % 128, lane = r % 8, sub = r / 8;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem)), "n"(kColumns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    const ConvPlan *pl = plans + blockIdx.y;
    const int ns = pl->ns, nt = pl->nt;
    const u64 *sp = src + (size_t)blockIdx.z * src_outer + (size_t)pl->src_limb * kN16 + blockIdx.x * 8;
    u64 *dp = dst + (size_t)blockIdx.z * dst_outer + (size_t)pl->dst_limb * kN16 + blockIdx.x * 8 + lane;
    u64 *ex = strips + (4 + g) * I::kWords;
    uint4 *consts = reinterpret_cast<uint4 *>(strips + (4 + G) * I::kWords);
    for (int i = tid; i < (nt + G - 1) / G * G * 32; i += 128 * G) consts[i] = i < nt * 32 ? pl->bytes[i] : make_uint4(0, 0, 0, 0);
    pdl_wait();
    for (int s = g; s < ns; s += G) strip_fetch<8>(sp + (size_t)s * kN16, strips + s * I::kWords, r);
#pragma unroll 1
    for (int s0 = 0; s0 < ns; s0 += G) {
        const int s = s0 + g;
        const bool mine = s < ns;
        const int pi = mine ? pl->src_prime[s] : 0;
        const PrimeConst m = pc[pi];
        const ulonglong2 *tab = tb.inv + (size_t)pi * Ntt16Layout::kEntries;
        const u64 *sm = strips + s * I::kWords;
        if (mine) {
            if (s + G < ns) cp_async_wait<1>(); else cp_async_wait<0>(); // at most one more strip of this group may be on its way
            group_sync<128>(g);
            if (m.small) {
                const DsConst c = ds_const(m);
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = __longlong_as_double((long long)sm[I::b(e, sub, lane)]);
                inv16_ds(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) ex[I::b(e, sub, lane)] = (u64)__double_as_longlong(v[e]);
            } else {
                const typename LONG::Const c = LONG::make(m);
                u64 v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = sm[I::b(e, sub, lane)];
                LONG::inv16(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) ex[I::b(e, sub, lane)] = v[e];
            }
        }
        __syncthreads(); // both strips of a pair have been read
        if (mine) {
            u64 *a = strips + (s >> 1) * (2 * I::kWords) + r * 2 + (s & 1);
            auto put = [&](int e, u64 w) { a[e * 256] = w; };
            if (m.small) {
                const DsConst c = ds_const(m);
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = __longlong_as_double((long long)ex[I::a(e, sub, lane)]);
                inv16_ds<1>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
                inv16_ds_last(v, pl->scale_w[s], pl->scale_c[s], c, put);
            } else {
                const typename LONG::Const c = LONG::make(m);
                u64 v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = ex[I::a(e, sub, lane)];
                LONG::template inv16<1>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
                inv16_int_last<LONG>(v, pl->scale_w[s], pl->scale_c[s], c, put);
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the operands are read by the tensor cores
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const u32 tm = tmem;
    auto issue = [&](int k) { // the sums of the targets at k .. k + G - 1
        const u32 a = smem_u32(strips), b = smem_u32(consts) + k * 512;
#pragma unroll 4
        for (int e = 0; e < 16; ++e) mma_i8(tm + e * 8 * G, mma_desc(a + e * 2048, kPair, 128), mma_desc(b + (e >> 3) * 256, 128, 512), kIdesc);
        mma_commit(&bar);
    };
    if (tid == 0) issue(0);
    __syncwarp();
    const u32 row = tm + ((u32)(r >> 5) << 21) + g * 8; // this warp's lanes, this group's columns
#pragma unroll 1
    for (int k0 = 0, phase = 0; k0 < nt; k0 += G, phase ^= 1) {
        const int k = k0 + g;
        const bool mine = k < nt;
        const int t = mine ? pl->order[k] : 0, pi = mine ? pl->dst_prime[t] : 0;
        const PrimeConst m = pc[pi];
        const ulonglong2 *tab = tb.fwd + (size_t)pi * Ntt16Layout::kEntries;
        mbar_wait_bounded(&bar, phase, err);
        __syncwarp();
        tmem_fence_after();
        if (mine) {
            if (m.small) {
                const DsConst c = ds_const(m);
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    u32 s[4][8];
                    tmem_load4x8(s, row + e * 8 * G, 8 * G);
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[e + u] = join_small(s[u], c.qinv, c.qd);
                }
                fwd16_ds<true>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) ex[I::a(e, sub, lane)] = (u64)__double_as_longlong(v[e]);
            } else {
                const typename LONG::Const c = LONG::make(m);
                u64 v[16];
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    u32 s[4][8];
                    tmem_load4x8(s, row + e * 8 * G, 8 * G);
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[e + u] = join_long(s[u], m.d60);
                }
                LONG::template fwd16<0, true>(v, TwiddlesA(tab + Ntt16Layout::colsA(0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) ex[I::a(e, sub, lane)] = v[e];
            }
        }
        tmem_fence_before();
        __syncthreads(); // every group has its sums
        if (tid == 0 && k0 + G < nt) { tmem_fence_after(); issue(k0 + G); }
        __syncwarp();
        if (mine) {
            u64 *o = dp + (size_t)t * kN16;
            if (m.small) {
                const DsConst c = ds_const(m);
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = __longlong_as_double((long long)ex[I::b(e, sub, lane)]);
                fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) reinterpret_cast<double *>(o)[(sub * 16 + e) * 256] = v[e];
            } else {
                const typename LONG::Const c = LONG::make(m);
                u64 v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = ex[I::b(e, sub, lane)];
                LONG::template fwd16<1>(v, TwiddlesA(tab + Ntt16Layout::colsB(sub, 0)), c);
#pragma unroll
                for (int e = 0; e < 16; ++e) o[(sub * 16 + e) * 256] = v[e];
            }
            group_sync<128>(g); // the strip has been read
        }
    }
    if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "n"(kColumns)); // every warp has read its last sums before the last CTA barrier
}

} // namespace hb
