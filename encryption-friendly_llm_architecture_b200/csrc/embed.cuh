// The canonical embedding and the samplers on the device (sm_100a): slot values <-> coefficients, error polynomials, assembly of
// ciphertexts.
//
// The embedding is a transform of N / 2 complex doubles over the orbit of 5.  Its rounding is part of a ciphertext's bits, so every
// butterfly is the same sequence of IEEE operations whatever kernel carries it out: additions, subtractions and products rounded
// one by one (the _rn intrinsics are never contracted), with the twiddles taken from tables that the host fills.  Grouping the
// stages differently changes no result.
//
// 2^15 slots are a 256 x 128 matrix (index = row * 128 + column).  The inverse transform (encoding; decimation in frequency, natural
// order in) does the eight stages of distance >= 128 on columns, then seven on rows; the forward one (decoding) the mirror image.
// A thread keeps sixteen complex values in registers and takes four stages at a time, with one exchange through shared memory per
// pass.  A twiddle depends on the whole position inside its block, so the column pass reads as many twiddle bytes as it has data per
// two stages; the 512 KB table of a direction stays in L2.  The sides that face the coefficients are permuted by bit reversal: a CTA
// takes the sixteen rows that agree in their low four bits, whose images are runs of sixteen coefficients.
// Bound by latency (16 CTAs of 128 threads a member): for eight members 7 and 14 us to encode, 40 and 35 us to decode, where the
// host cores took 2.0 and 1.8 ms a member for the same transforms and 2.8 and 1.4 ms for sampling and CRT lift.  Thirteen messages
// of two tiles from host memory to ciphertexts 7.3 -> 0.82 -> 0.66 ms (0.82 before uniform parts and errors were drawn ahead of the messages), thirteen
// ciphertexts to host memory 5.5 -> 0.80 -> 0.65 ms (0.80 before their pages were asked for meanwhile), each pass through the Python call on other buffers; the library
// call on the same buffers again 0.53 and 0.35 ms.  The copies are most of all of these.
#pragma once
#include "modarith.cuh"
#include "kernels.cuh"
#include "pdl.cuh"

namespace hb {

constexpr int kSlots16 = 32768, kEmbRows = 256, kEmbCols = 128;
struct EmbedTables { const double2 *inv, *fwd; }; // twiddle of distance h, position j < h at [h + j]

__device__ __forceinline__ double2 c_add(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ double2 c_mul(double2 a, double2 w) {
    return make_double2(__dsub_rn(__dmul_rn(a.x, w.x), __dmul_rn(a.y, w.y)), __dadd_rn(__dmul_rn(a.x, w.y), __dmul_rn(a.y, w.x)));
}
__device__ __forceinline__ void inv_bfly(double2 &a, double2 &b, double2 w) { const double2 d = c_sub(a, b); a = c_add(a, b); b = c_mul(d, w); }
__device__ __forceinline__ void fwd_bfly(double2 &a, double2 &b, double2 w) { const double2 t = c_mul(b, w); b = c_sub(a, t); a = c_add(a, t); }
// Stages of in-register distance TOP, TOP / 2 .. 1 (inverse) or 1 .. TOP (forward) over v[16]; register e lies at position e * step + off
// of its block, one register apart is `step` positions.
template <int TOP> __device__ __forceinline__ void inv_round(double2 (&v)[16], const double2 *__restrict__ tw, int step, int off) {
#pragma unroll
    for (int half = TOP; half >= 1; half >>= 1)
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const double2 w = __ldg(tw + (half + j) * step + off);
#pragma unroll
            for (int g = 0; g < 16; g += 2 * half) inv_bfly(v[g + j], v[g + j + half], w);
        }
}
template <int TOP> __device__ __forceinline__ void fwd_round(double2 (&v)[16], const double2 *__restrict__ tw, int step, int off) {
#pragma unroll
    for (int half = 1; half <= TOP; half <<= 1)
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const double2 w = __ldg(tw + (half + j) * step + off);
#pragma unroll
            for (int g = 0; g < 16; g += 2 * half) fwd_bfly(v[g + j], v[g + j + half], w);
        }
}
// x86 semantics of a conversion to 64 bits: everything that does not fit becomes the most negative value
__device__ __forceinline__ i64 to_i64(double rounded) { return fabs(rounded) < 0x1p63 ? (i64)rounded : (i64)0x8000000000000000ull; }

constexpr int kEmbThreads = 128;
// messages re / im [count][n] (im may be null, slots from n on are zero) -> half-transformed slots v [count][2^15].  grid = (16, count)
__global__ void __launch_bounds__(kEmbThreads) k_embed_inv_cols(double2 *v, const double *re, const double *im, int n, EmbedTables tb) {
    __shared__ double2 sm[kEmbRows * 8];
    const int lane = threadIdx.x & 7, sub = threadIdx.x >> 3, col = blockIdx.x * 8 + lane;
    const size_t base = (size_t)blockIdx.y * n;
    double2 x[16];
    pdl_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const int i = (e * 16 + sub) * kEmbCols + col;
        x[e] = make_double2(i < n ? re[base + i] : 0.0, i < n && im ? im[base + i] : 0.0);
    }
    inv_round<8>(x, tb.inv, 16 * kEmbCols, sub * kEmbCols + col);
#pragma unroll
    for (int e = 0; e < 16; ++e) sm[(e * 16 + sub) * 8 + lane] = x[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = sm[(sub * 16 + e) * 8 + lane];
    inv_round<8>(x, tb.inv, kEmbCols, col);
    double2 *o = v + (size_t)blockIdx.y * kSlots16 + col;
#pragma unroll
    for (int e = 0; e < 16; ++e) o[(sub * 16 + e) * kEmbCols] = x[e];
}
// -> rounded coefficients at scale sc, coef [count][2^16]: real parts, then imaginary parts.  grid = (16, count)
__global__ void __launch_bounds__(kEmbThreads) k_embed_inv_rows(i64 *coef, const double2 *v, double sc, EmbedTables tb) {
    constexpr int kStride = kEmbCols + 8; // one pad word per sixteen
    __shared__ __align__(16) double2 sm[16 * kStride];
    static_assert(sizeof(sm) == 2 * kEmbCols * 17 * sizeof(i64), "the output exchange takes the same room");
    const int c = threadIdx.x & 7, r = threadIdx.x >> 3, f = blockIdx.x;
    const double2 *p = v + (size_t)blockIdx.y * kSlots16 + (r * 16 + f) * kEmbCols;
    double2 x[16];
    pdl_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = p[c + 8 * e];
    inv_round<8>(x, tb.inv, 8, c);
#pragma unroll
    for (int e = 0; e < 16; ++e) sm[r * kStride + c + 8 * e + (e >> 1)] = x[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = sm[r * kStride + c * 17 + e];
    inv_round<4>(x, tb.inv, 1, 0);
    __syncthreads();
    i64 *out = reinterpret_cast<i64 *>(sm);
    const int rr = (int)(__brev((u32)r) >> 28);
    constexpr double inv = 1.0 / kSlots16;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const int i = c * 16 + e;
        out[i * 17 + rr] = to_i64(rint(__dmul_rn(__dmul_rn(x[e].x, inv), sc)));
        out[(kEmbCols + i) * 17 + rr] = to_i64(rint(__dmul_rn(__dmul_rn(x[e].y, inv), sc)));
    }
    __syncthreads();
    i64 *o = coef + (size_t)blockIdx.y * 2 * kSlots16 + (int)(__brev((u32)f) >> 28) * 16;
#pragma unroll 4
    for (int w = threadIdx.x; w < 2 * kEmbCols * 16; w += kEmbThreads) {
        const int k = w & 15, i = (w >> 4) & (kEmbCols - 1), plane = w >> 11;
        o[(size_t)plane * kSlots16 + (__brev((u32)i) >> 25) * 256 + k] = out[(plane * kEmbCols + i) * 17 + k];
    }
}

// ---- centred lift of the residues modulo q_0 (and q_1) ----
struct CentreConst { u64 q0, half0, Q_hi, Q_lo, half_hi, half_lo, q0_inv; }; // Q = q0 * q1, half = Q / 2, q0_inv modulo q1
__device__ __forceinline__ double u128_to_double(u64 hi, u64 lo) { // rounded to nearest
    if (!hi) return __ull2double_rn(lo);
    const int s = __clzll((long long)hi);
    const u64 top = s ? (hi << s) | (lo >> (64 - s)) : hi, rest = lo << s;
    return __ull2double_rn(top | (rest ? 1ull : 0ull)) * __longlong_as_double((long long)(1023 + 64 - s) << 52); // the last bits of top only say on which side of a tie
}
__device__ __forceinline__ double centred(u64 r0, u64 r1, bool two, const CentreConst &k, const PrimeConst &m1) {
    if (!two) return r0 > k.half0 ? -__ull2double_rn(k.q0 - r0) : __ull2double_rn(r0);
    const u64 t = mul_mod(sub_mod(r1, reduce_u64(r0, m1), m1.q), k.q0_inv, m1);
    u64 lo = k.q0 * t, hi = mul_hi(k.q0, t);
    lo += r0; hi += lo < r0;
    if (hi > k.half_hi || (hi == k.half_hi && lo > k.half_lo)) {
        const u64 nl = k.Q_lo - lo, nh = k.Q_hi - hi - (k.Q_lo < lo);
        return -u128_to_double(nh, nl);
    }
    return u128_to_double(hi, lo);
}
// One member of a decryption: ciphertext [np][n][N], limbs used (1 or 2) and scale.  An encoded plaintext is a ciphertext of one polynomial.
struct DecItem { const u64 *ct; int n, np; double scale; };
// residues c [count][2][2^16] (coefficient form) -> half-transformed slots v [count][2^15].  grid = (16, count)
__global__ void __launch_bounds__(kEmbThreads) k_embed_fwd_rows(double2 *v, const u64 *c, const DecItem *items, const __grid_constant__ CentreConst k, const PrimeConst *__restrict__ pc, EmbedTables tb) {
    constexpr int kStride = kEmbCols + 8;
    __shared__ __align__(16) double2 sm[16 * kStride];
    const int lane = threadIdx.x & 7, r = threadIdx.x >> 3, f = blockIdx.x;
    const u64 *c0 = c + (size_t)blockIdx.y * 4 * kSlots16 + (int)(__brev((u32)f) >> 28) * 16, *c1 = c0 + 2 * kSlots16;
    double *in = reinterpret_cast<double *>(sm);
    const PrimeConst m1 = pc[1];
    pdl_wait();
    const bool two = items[blockIdx.y].n > 1;
    const double sc = items[blockIdx.y].scale;
#pragma unroll 4
    for (int w = threadIdx.x; w < 2 * kEmbCols * 16; w += kEmbThreads) {
        const int q = w & 15, i = (w >> 4) & (kEmbCols - 1), plane = w >> 11;
        const size_t pos = (size_t)plane * kSlots16 + (__brev((u32)i) >> 25) * 256 + q;
        in[(plane * kEmbCols + i) * 17 + q] = __ddiv_rn(centred(c0[pos], two ? c1[pos] : 0, two, k, m1), sc);
    }
    __syncthreads();
    const int rr = (int)(__brev((u32)r) >> 28);
    double2 x[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) { const int i = lane * 16 + e; x[e] = make_double2(in[i * 17 + rr], in[(kEmbCols + i) * 17 + rr]); }
    fwd_round<4>(x, tb.fwd, 1, 0);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) sm[r * kStride + lane * 17 + e] = x[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = sm[r * kStride + lane + 8 * e + (e >> 1)];
    fwd_round<8>(x, tb.fwd, 8, lane);
    double2 *o = v + (size_t)blockIdx.y * kSlots16 + (r * 16 + f) * kEmbCols;
#pragma unroll
    for (int e = 0; e < 16; ++e) o[lane + 8 * e] = x[e];
}
// -> slot values: member b, slot s at re[(b * 2^15 + s) * stride] (im likewise).  grid = (16, count)
__global__ void __launch_bounds__(kEmbThreads) k_embed_fwd_cols(double *re, double *im, int stride, const double2 *v, EmbedTables tb) {
    __shared__ double2 sm[kEmbRows * 8];
    const int lane = threadIdx.x & 7, sub = threadIdx.x >> 3, col = blockIdx.x * 8 + lane;
    const double2 *p = v + (size_t)blockIdx.y * kSlots16 + col;
    double2 x[16];
    pdl_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = p[(sub * 16 + e) * kEmbCols];
    fwd_round<8>(x, tb.fwd, kEmbCols, col);
#pragma unroll
    for (int e = 0; e < 16; ++e) sm[(sub * 16 + e) * 8 + lane] = x[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = sm[(e * 16 + sub) * 8 + lane];
    fwd_round<8>(x, tb.fwd, 16 * kEmbCols, sub * kEmbCols + col);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const size_t s = ((size_t)blockIdx.y * kSlots16 + (e * 16 + sub) * kEmbCols + col) * stride;
        re[s] = x[e].x; im[s] = x[e].y;
    }
}
// Rings up to 2^12: one CTA per member, the whole transform in shared memory (at most 2048 complex values), a barrier per stage.
constexpr int kEmbSmallMax = 2048;
__global__ void __launch_bounds__(256) k_embed_inv_small(i64 *coef, const double *re, const double *im, int n, int log_slots, double sc, EmbedTables tb) {
    __shared__ double2 sm[kEmbSmallMax];
    const int slots = 1 << log_slots;
    const size_t base = (size_t)blockIdx.x * n;
    pdl_wait();
    for (int i = threadIdx.x; i < slots; i += 256) sm[i] = make_double2(i < n ? re[base + i] : 0.0, i < n && im ? im[base + i] : 0.0);
    for (int h = slots >> 1; h >= 1; h >>= 1) {
        __syncthreads();
        for (int t = threadIdx.x; t < slots / 2; t += 256) {
            const int j = t & (h - 1), a = (t - j) * 2 + j;
            inv_bfly(sm[a], sm[a + h], __ldg(tb.inv + h + j));
        }
    }
    __syncthreads();
    const double inv = 1.0 / (double)slots;
    i64 *o = coef + (size_t)blockIdx.x * 2 * slots;
    for (int i = threadIdx.x; i < slots; i += 256) {
        const double2 x = sm[__brev((u32)i) >> (32 - log_slots)];
        o[i] = to_i64(rint(__dmul_rn(__dmul_rn(x.x, inv), sc)));
        o[i + slots] = to_i64(rint(__dmul_rn(__dmul_rn(x.y, inv), sc)));
    }
}
__global__ void __launch_bounds__(256) k_embed_fwd_small(double *re, double *im, int stride, const u64 *c, const DecItem *items, int log_slots, const __grid_constant__ CentreConst k,
                                                         const PrimeConst *__restrict__ pc, EmbedTables tb) {
    __shared__ double2 sm[kEmbSmallMax];
    const int slots = 1 << log_slots;
    const u64 *c0 = c + (size_t)blockIdx.x * 4 * slots, *c1 = c0 + 2 * slots;
    const PrimeConst m1 = pc[1];
    pdl_wait();
    const bool two = items[blockIdx.x].n > 1;
    const double sc = items[blockIdx.x].scale;
    for (int i = threadIdx.x; i < slots; i += 256)
        sm[__brev((u32)i) >> (32 - log_slots)] = make_double2(__ddiv_rn(centred(c0[i], two ? c1[i] : 0, two, k, m1), sc), __ddiv_rn(centred(c0[i + slots], two ? c1[i + slots] : 0, two, k, m1), sc));
    for (int h = 1; h < slots; h <<= 1) {
        __syncthreads();
        for (int t = threadIdx.x; t < slots / 2; t += 256) {
            const int j = t & (h - 1), a = (t - j) * 2 + j;
            fwd_bfly(sm[a], sm[a + h], __ldg(tb.fwd + h + j));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < slots; i += 256) {
        const size_t s = ((size_t)blockIdx.x * slots + i) * stride;
        re[s] = sm[i].x; im[s] = sm[i].y;
    }
}

// ---- ChaCha20 ----
__device__ __forceinline__ u32 rotl32(u32 v, int c) { return __funnelshift_l(v, v, c); }
#define HB_QR(a, b, c, d)                                   \
    a += b; d ^= a; d = rotl32(d, 16); c += d; b ^= c; b = rotl32(b, 12); \
    a += b; d ^= a; d = rotl32(d, 8);  c += d; b ^= c; b = rotl32(b, 7);
struct ChaChaKey { u32 k[8]; };
__device__ __forceinline__ void chacha_block(const ChaChaKey &key, u32 domain, u64 id, u32 counter, u32 (&o)[16]) {
    u32 in[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u, key.k[0], key.k[1], key.k[2], key.k[3], key.k[4], key.k[5], key.k[6], key.k[7],
                  counter, domain, (u32)id, (u32)(id >> 32)};
    u32 x0 = in[0], x1 = in[1], x2 = in[2], x3 = in[3], x4 = in[4], x5 = in[5], x6 = in[6], x7 = in[7];
    u32 x8 = in[8], x9 = in[9], x10 = in[10], x11 = in[11], x12 = in[12], x13 = in[13], x14 = in[14], x15 = in[15];
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        HB_QR(x0, x4, x8, x12) HB_QR(x1, x5, x9, x13) HB_QR(x2, x6, x10, x14) HB_QR(x3, x7, x11, x15)
        HB_QR(x0, x5, x10, x15) HB_QR(x1, x6, x11, x12) HB_QR(x2, x7, x8, x13) HB_QR(x3, x4, x9, x14)
    }
    o[0] = x0 + in[0]; o[1] = x1 + in[1]; o[2] = x2 + in[2]; o[3] = x3 + in[3]; o[4] = x4 + in[4]; o[5] = x5 + in[5]; o[6] = x6 + in[6]; o[7] = x7 + in[7];
    o[8] = x8 + in[8]; o[9] = x9 + in[9]; o[10] = x10 + in[10]; o[11] = x11 + in[11]; o[12] = x12 + in[12]; o[13] = x13 + in[13]; o[14] = x14 + in[14]; o[15] = x15 + in[15];
}
// Streams of a launch: member b draws from the stream ids[b] (ids null: from `first` + b) of the domain.
struct StreamIds { ChaChaKey key; u32 domain; const u64 *ids; u64 first; };
__device__ __forceinline__ u64 stream_id(const StreamIds &s, int b) { return s.ids ? s.ids[b] : s.first + (u64)b; }

// eight values of a discrete Gaussian from block t of a stream: magnitude = number of the `cdt_n` increasing table entries that are <= the upper 63 bits of
// the word, sign from its lowest bit
__device__ __forceinline__ void gauss8(int (&e)[8], const StreamIds &s, u64 id, int t, const u64 *__restrict__ cdt, int cdt_n) {
    u32 o[16];
    chacha_block(s.key, s.domain, id, (u32)t, o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const u64 r = (u64)o[2 * k] | ((u64)o[2 * k + 1] << 32), u = r >> 1;
        int lo = 0, hi = cdt_n; // entries [0, lo) are <= u, entries [hi, n) above
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(cdt + mid) <= u) lo = mid + 1; else hi = mid;
        }
        e[k] = (r & 1) ? -lo : lo;
    }
}
// Residues of integer polynomials: out[b][l][i] = (coef[b][i] + error[b][i]) mod prime l, coefficient form.  Either part may be missing.
// The error is a discrete Gaussian, from word i of the member's stream.  A thread makes the eight coefficients of one ChaCha block
// for every gridDim.z-th limb: for all limbs where it makes an error, for one otherwise (the limbs one after the other / side by side: key
// generation, which reduces the secret, 112 / 101 us, 52 / 40 at 2^10 points; one real message at level 12 to a plaintext 92 / 80).
// grid = (ceil(N/8/128), count, 1 or limbs)
template <bool MSG, bool ERR>
__global__ void __launch_bounds__(128) k_residues(u64 *out, const i64 *coef, const __grid_constant__ StreamIds ids, const u64 *__restrict__ cdt, int cdt_n, const __grid_constant__ LimbMap map,
                                                  const PrimeConst *__restrict__ pc, int N) {
    const int t = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
    pdl_wait();
    if (t * 8 >= N) return;
    int e[8];
    if constexpr (ERR) gauss8(e, ids, stream_id(ids, b), t, cdt, cdt_n);
    i64 m[8];
    if constexpr (MSG) {
        const longlong2 *p = reinterpret_cast<const longlong2 *>(coef + (size_t)b * N) + t * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k) { const longlong2 w = p[k]; m[2 * k] = w.x; m[2 * k + 1] = w.y; }
    }
    ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out + (size_t)b * map.n * N) + t * 4;
    for (int l = blockIdx.z; l < map.n; l += gridDim.z) {
        const PrimeConst *q = pc + map.prime[l];
        u64 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            u64 r = 0;
            if constexpr (MSG) r = reduce_i64_any(m[k], *q);
            if constexpr (ERR) r = add_mod(r, reduce_i64_any(e[k], *q), q->q);
            v[k] = r;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) o[(size_t)l * (N / 2) + k] = make_ulonglong2(v[2 * k], v[2 * k + 1]);
    }
}
// four uniform residues modulo prime pi from words 4 t .. of the stream (128-bit word pi * N + c of it modulo the prime)
__device__ __forceinline__ void uniform4(u64 (&a)[4], const StreamIds &s, u64 id, int pi, int t, const PrimeConst &m, int N) {
    u32 o[16];
    chacha_block(s.key, s.domain, id, (u32)(((u64)pi * N + (u64)t * 4) >> 2), o);
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = barrett128((u64)o[4 * k + 2] | ((u64)o[4 * k + 3] << 32), (u64)o[4 * k] | ((u64)o[4 * k + 1] << 32), m);
}
__device__ __forceinline__ void load4(u64 (&v)[4], const u64 *p) {
    const ulonglong2 x = reinterpret_cast<const ulonglong2 *>(p)[0], y = reinterpret_cast<const ulonglong2 *>(p)[1];
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void store4(u64 *p, const u64 (&v)[4]) {
    reinterpret_cast<ulonglong2 *>(p)[0] = make_ulonglong2(v[0], v[1]);
    reinterpret_cast<ulonglong2 *>(p)[1] = make_ulonglong2(v[2], v[3]);
}
// What an encryption draws, ahead of the messages (2^16 rings; sampling depends on none of them and so runs while the first ones are on their way):
// noise[b][i] = coefficient i of the member's error polynomial, below 128 in magnitude.  grid = (N/8/128, count)
__global__ void __launch_bounds__(128) k_noise(signed char *noise, const __grid_constant__ StreamIds ids, const u64 *__restrict__ cdt, int cdt_n, int N) {
    const int t = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
    pdl_wait();
    int e[8];
    gauss8(e, ids, stream_id(ids, b), t, cdt, cdt_n);
    u64 w = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) w |= (u64)(unsigned char)e[k] << (8 * k);
    reinterpret_cast<u64 *>(noise + (size_t)b * N)[t] = w;
}
// -(coef[b][i] + noise[b][i]) modulo prime l, coefficient form: the negative, so that the last step of a division (x - t) finishes an encryption.  A
// thread has four coefficients of one limb.  grid = (N/4/256, limbs, count)
__global__ void __launch_bounds__(256) k_noisy_residues(u64 *out, const i64 *coef, const signed char *noise, const PrimeConst *__restrict__ pc, int N) {
    const int t = blockIdx.x * 256 + threadIdx.x, l = blockIdx.y, b = blockIdx.z;
    const PrimeConst m = pc[l];
    pdl_wait();
    const longlong2 *p = reinterpret_cast<const longlong2 *>(coef + (size_t)b * N) + t * 2;
    const longlong2 p0 = p[0], p1 = p[1];
    const char4 e4 = reinterpret_cast<const char4 *>(noise + (size_t)b * N)[t];
    const i64 v[4] = {p0.x, p0.y, p1.x, p1.y};
    const int e[4] = {e4.x, e4.y, e4.z, e4.w};
    u64 r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const u64 s = add_mod(reduce_i64_any(v[k], m), e[k] < 0 ? m.q - (u64)-e[k] : (u64)e[k], m.q);
        r[k] = s ? m.q - s : 0;
    }
    store4(out + ((size_t)b * gridDim.y + l) * N + t * 4, r);
}
// ct [count][2][n][N]: a uniform (second polynomial) and -a s (first one).  One thread per ChaCha block of four coefficients.  grid = (N/4/256, n, count)
__global__ void __launch_bounds__(256) k_uniform(u64 *ct, const u64 *__restrict__ s, const __grid_constant__ StreamIds ids, const PrimeConst *__restrict__ pc, int N) {
    const int t = blockIdx.x * 256 + threadIdx.x, l = blockIdx.y, n = gridDim.y, b = blockIdx.z;
    const PrimeConst m = pc[l];
    u64 a[4], sv[4], r[4];
    load4(sv, s + (size_t)l * N + t * 4);
    pdl_wait();
    uniform4(a, ids, stream_id(ids, b), l, t, m, N);
#pragma unroll
    for (int k = 0; k < 4; ++k) { const u64 p = mul_mod_any(a[k], sv[k], m); r[k] = p ? m.q - p : 0; }
    u64 *o = ct + ((size_t)b * 2 * n + l) * N + t * 4;
    store4(o, r);
    store4(o + (size_t)n * N, a);
}
// Ciphertexts ct [count][2][n][N]: a uniform, b = e - a s (+ msg), e [count][n][N] (message included, or msg [n][N] apart), all NTT form.
// One thread per ChaCha block of four coefficients; the generator's additions, exclusive ors and rotations bound it.  grid = (ceil(N/4/256), n, count)
__global__ void __launch_bounds__(256) k_encrypt(u64 *ct, const u64 *e, const u64 *msg, const u64 *s, const __grid_constant__ StreamIds ids, const PrimeConst *__restrict__ pc, int N) {
    const int t = blockIdx.x * 256 + threadIdx.x, l = blockIdx.y, n = gridDim.y, b = blockIdx.z;
    pdl_wait();
    if (t * 4 >= N) return;
    const PrimeConst m = pc[l];
    u64 a[4], ev[4], sv[4], r[4];
    load4(ev, e + ((size_t)b * n + l) * N + t * 4);
    load4(sv, s + (size_t)l * N + t * 4);
    uniform4(a, ids, stream_id(ids, b), l, t, m, N);
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = sub_mod(ev[k], mul_mod_any(a[k], sv[k], m), m.q);
    if (msg) {
        u64 mv[4];
        load4(mv, msg + (size_t)l * N + t * 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = add_mod(r[k], mv[k], m.q);
    }
    u64 *o = ct + ((size_t)b * 2 * n + l) * N + t * 4;
    store4(o, r);
    store4(o + (size_t)n * N, a);
}
// Switching key [nd][2][primes][N]: a uniform, b = e - a s + [prime in digit] (P mod q) s',  s' = s^2 (g == 0) or s o perm_g.
// Digits are alpha limbs long, the first one limb less.  e [nd][primes][N], NTT form.  grid = (ceil(N/4/256), primes, nd)
__global__ void __launch_bounds__(256) k_keygen(u64 *key, const u64 *e, const u64 *s, const __grid_constant__ StreamIds ids, const PrimeConst *__restrict__ pc, int N, int logn, u32 g, int q_limbs,
                                                int alpha, const __grid_constant__ Scalars pmod) {
    const int t = blockIdx.x * 256 + threadIdx.x, pi = blockIdx.y, np = gridDim.y, dg = blockIdx.z;
    if (t * 4 >= N) return;
    const PrimeConst m = pc[pi];
    u64 a[4], ev[4], sv[4], r[4];
    load4(ev, e + ((size_t)dg * np + pi) * N + t * 4);
    load4(sv, s + (size_t)pi * N + t * 4);
    uniform4(a, ids, stream_id(ids, dg), pi, t, m, N);
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = sub_mod(ev[k], mul_mod(a[k], sv[k], m), m.q);
    if (pi < q_limbs && (pi + 1) / alpha == dg) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const u64 sp = g == 0 ? mul_mod(sv[k], sv[k], m) : s[(size_t)pi * N + ntt_perm((u32)(t * 4 + k), g, logn)];
            r[k] = add_mod(r[k], mul_mod(sp, pmod.v[pi], m), m.q);
        }
    }
    u64 *o = key + ((size_t)dg * 2 * np + pi) * N + t * 4;
    store4(o, r);
    store4(o + (size_t)np * N, a);
}
// out [count][2][N]: b + a s (+ d2 s^2) of the first one or two limbs of every member (one polynomial: b alone; a limb that the member does
// not have: 0).  grid = (gx, 1 or 2, count)
__global__ void k_decrypt(u64 *out, const DecItem *items, const u64 *s, const PrimeConst *__restrict__ pc, int N) {
    const int l = blockIdx.y;
    pdl_wait();
    const DecItem it = items[blockIdx.z];
    const int np = it.np;
    const size_t poly = (size_t)it.n * N;
    const PrimeConst m = pc[l];
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const size_t off = (size_t)l * N + i;
        if (l >= it.n) { out[(size_t)blockIdx.z * 2 * N + off] = 0; continue; }
        const u64 sv = s[off];
        u64 v = it.ct[off];
        if (np > 1) v = add_mod(v, mul_mod_any(it.ct[poly + off], sv, m), m.q);
        if (np > 2) v = add_mod(v, mul_mod_any(it.ct[2 * poly + off], mul_mod_any(sv, sv, m), m), m.q);
        out[(size_t)blockIdx.z * 2 * N + off] = v;
    }
}

} // namespace hb
