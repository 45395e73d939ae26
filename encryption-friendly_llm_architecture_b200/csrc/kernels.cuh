// Element-wise, base-conversion, automorphism and accumulate kernels (sm_100a).
// Arrays are dense [instances][N] uint64 unless a stride is named; instance li uses prime
// map.prime[li % map.n].  One thread handles one coefficient of one limb instance; a warp
// touches 256 contiguous bytes per array, so every stream is fully coalesced.  Gathers through
// ntt_perm stay inside an aligned 32-element block (the automorphism permutes aligned blocks
// of the bit-reversed index as units), so they cost no extra sectors.
#pragma once
#include "modarith.cuh"
#include "bulk.cuh"
#include "pdl.cuh"

namespace hb {

// Every thread handles kElems coefficients, blockDim apart (each access stays a 256-byte run per warp): four
// independent loads per array are in flight per thread and the grid has four times fewer, fatter CTAs --
// with one coefficient per thread these kernels were bound by CTA turnover at about 2 TB/s.
constexpr int kElems = 4;

// out = a + b  (mode 0) | a - b (mode 1) | -a (mode 2)
__global__ void k_addsub(u64 *__restrict__ out, const u64 *__restrict__ a, const u64 *__restrict__ b, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc,
                         int N, int mode) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[map.prime[li % map.n]];
        const size_t off = (size_t)li * N + i;
        u64 x = a[off];
        if (mode == 0) out[off] = add_mod(x, b[off], m.q);
        else if (mode == 1) out[off] = sub_mod(x, b[off], m.q);
        else out[off] = x ? m.q - x : 0;
    }
}

struct Scalars { u64 v[kMaxPrimes]; };
// out = a * s[prime]
__global__ void k_scalar_mul(u64 *__restrict__ out, const u64 *__restrict__ a, size_t a_outer, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N, const __grid_constant__ Scalars s) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const int pi = map.prime[li % map.n];
        const PrimeConst m = pc[pi];
        const size_t soff = (size_t)(li / map.n) * a_outer + (size_t)(li % map.n) * N + i;
        out[(size_t)li * N + i] = mul_mod_any(a[soff], s.v[pi], m);
    }
}
// multiplication by X^(N/2): +iu on the first half of an NTT-form limb, -iu on the second
__global__ void k_mult_imag(u64 *__restrict__ out, const u64 *__restrict__ a, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[map.prime[li % map.n]];
        const size_t off = (size_t)li * N + i;
        u64 r = mul_shoup(a[off], m.iu, m.iu_sh, m.q);
        if (i >= N / 2) r = r ? m.q - r : 0;
        out[off] = r;
    }
}
// out = a (.) pt, pt limb = li % map.n
__global__ void k_mul_pt(u64 *__restrict__ out, const u64 *__restrict__ a, const u64 *__restrict__ pt, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[map.prime[li % map.n]];
        const size_t off = (size_t)li * N + i;
        out[off] = mul_mod_any(a[off], pt[(size_t)(li % map.n) * N + i], m);
    }
}
// tensor product, optional accumulation.  grid.y = batch * n; x, y: [groups][batch][2][n][N]; d: [batch][3][n][N]
//   d[b] (+)= sum over the groups g of tensor(x[g][b], y[g][b])
// (groups = 1 is the plain tensor product; several groups are several iterations of a product loop in one launch).
// Two coefficients per thread, so that eight loads of a group are in flight, and one reduction per sum: 256 ciphertexts at level 8
// 1634 -> 1498 us (5.6 TB/s), a launch of the layer's product loop 620 -> 517 us.  48 ciphertexts at level 8: 253 us, DRAM 4.3 TB/s,
// 54 % of the issue slots.  grid.x = N/512
__global__ void __launch_bounds__(256) k_tensor(u64 *d, const u64 *x, const u64 *y, int n, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N,
                                                int accumulate, int groups, int batch) {
    constexpr int EL = 2;
    const int bl = blockIdx.y, b = bl / n, l = bl % n;
    const size_t gstride = (size_t)batch * 2 * n * N, poly = (size_t)n * N;
    const PrimeConst m = pc[map.prime[l]];
    const u32 i0 = blockIdx.x * (256 * EL) + threadIdx.x;
    const u64 *xp = x + ((size_t)(b * 2) * n + l) * N + i0, *yp = y + ((size_t)(b * 2) * n + l) * N + i0;
    u64 *dp = d + ((size_t)(b * 3) * n + l) * N + i0;
    u64 r[3][EL];
    pdl_wait();
    auto terms = [&](auto &&product) {
        for (int g = 0; g < groups; ++g, xp += gstride, yp += gstride) {
            u64 b1[EL], a1[EL], b2[EL], a2[EL];
#pragma unroll
            for (int u = 0; u < EL; ++u) { b1[u] = xp[u * 256]; a1[u] = xp[poly + u * 256]; b2[u] = yp[u * 256]; a2[u] = yp[poly + u * 256]; }
            product(g, b1, a1, b2, a2);
        }
    };
    if (m.fp) { // exact sums; the middle one takes two products per group: 64 groups below 2^42, four below 2^44, before it is reduced
        const double qd = (double)m.q;
        const int room = m.q < (1ull << 42) ? 64 : 4;
        FpAcc s[3][EL];
#pragma unroll
        for (int u = 0; u < EL; ++u) { s[0][u].zero(); s[1][u].zero(); s[2][u].zero(); }
        terms([&](int g, const u64 (&b1)[EL], const u64 (&a1)[EL], const u64 (&b2)[EL], const u64 (&a2)[EL]) {
            if (g && g % room == 0) {
#pragma unroll
                for (int u = 0; u < EL; ++u)
#pragma unroll
                    for (int k = 0; k < 3; ++k) s[k][u].relax(m.q_inv_f, qd);
            }
#pragma unroll
            for (int u = 0; u < EL; ++u) {
                const double b1d = u52_to_double(b1[u]), a1d = u52_to_double(a1[u]), b2d = u52_to_double(b2[u]), a2d = u52_to_double(a2[u]);
                s[0][u].mac(b1d, b2d); s[2][u].mac(a1d, a2d);
                s[1][u].mac(a1d, b2d); s[1][u].mac(a2d, b1d);
            }
        });
#pragma unroll
        for (int u = 0; u < EL; ++u)
#pragma unroll
            for (int k = 0; k < 3; ++k) r[k][u] = s[k][u].finish(m.q_inv_f, qd);
    } else {
        PieceAcc s[3][EL];
#pragma unroll
        for (int u = 0; u < EL; ++u) { s[0][u].zero(); s[1][u].zero(); s[2][u].zero(); }
        terms([&](int g, const u64 (&b1)[EL], const u64 (&a1)[EL], const u64 (&b2)[EL], const u64 (&a2)[EL]) {
            if (g && g % 4 == 0) {
#pragma unroll
                for (int u = 0; u < EL; ++u)
#pragma unroll
                    for (int k = 0; k < 3; ++k) s[k][u].relax(m);
            }
#pragma unroll
            for (int u = 0; u < EL; ++u) { s[0][u].mac(b1[u], b2[u]); s[2][u].mac(a1[u], a2[u]); s[1][u].mac(a1[u], b2[u]); s[1][u].mac(a2[u], b1[u]); }
        });
#pragma unroll
        for (int u = 0; u < EL; ++u)
#pragma unroll
            for (int k = 0; k < 3; ++k) r[k][u] = s[k][u].finish(m);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int u = 0; u < EL; ++u) {
            u64 *o = dp + k * poly + u * 256;
            *o = accumulate ? add_mod(r[k][u], *o, m.q) : r[k][u];
        }
}
// out[li][i] = in[li][perm_g(i)]
__global__ void k_permute(u64 *__restrict__ out, const u64 *__restrict__ in, u32 g, int logn, int N) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        out[(size_t)li * N + i] = in[(size_t)li * N + ntt_perm((u32)i, g, logn)];
    }
}
// x mod q for lazily summed residues
__global__ void k_mod_reduce(u64 *__restrict__ a, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[map.prime[li % map.n]];
        const size_t off = (size_t)li * N + i;
        a[off] = reduce_u64(a[off], m);
    }
}
// out = (x_0 + ... + x_{count-1}) mod q for canonical residues (count <= 16: the sum stays below 2^64)
struct SumList { const u64 *x[16]; int count; };
__global__ void k_sum_mod(u64 *__restrict__ out, const __grid_constant__ SumList sl, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int N) {
    const int li = blockIdx.y;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[map.prime[li % map.n]];
        const size_t off = (size_t)li * N + i;
        u64 v = 0;
        for (int t = 0; t < sl.count; ++t) v += sl.x[t][off];
        out[off] = reduce_u64(v, m);
    }
}

// ---------------- rescale ----------------
// t[bp][l][i] = centred(last[bp][i]) mod q_l, l < level.  grid.y = nbp * level
__global__ void k_rescale_prep(u64 *__restrict__ t, const u64 *__restrict__ last, int level, const PrimeConst *__restrict__ pc, int N) {
    const int w = blockIdx.y, bp = w / level, l = w % level;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[l];
        const u64 ql = pc[level].q;
        const u64 r = last[(size_t)bp * N + i];
        const i64 centred = r > (ql >> 1) ? (i64)r - (i64)ql : (i64)r;
        t[(size_t)w * N + i] = reduce_i64_any(centred, m);
    }
}
// out[bp][l] = (x[bp][l] - t[bp][l]) * q_level^-1 ; x has level+1 limbs per poly
__global__ void k_rescale_fin(u64 *__restrict__ out, const u64 *__restrict__ x, const u64 *__restrict__ t, int level, const PrimeConst *__restrict__ pc, int N,
                              const __grid_constant__ Scalars qlinv) {
    const int w = blockIdx.y, bp = w / level, l = w % level;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const PrimeConst m = pc[l];
        const u64 xv = x[((size_t)bp * (level + 1) + l) * N + i];
        out[(size_t)w * N + i] = mul_mod_any(sub_mod(xv, t[(size_t)w * N + i], m.q), qlinv.v[l], m);
    }
}

// ---------------- fused plaintext products with rescale ----------------
// out = sum_j rescale(a_j (.) p_j)          (separate == 1: every term is rescaled on its own, as
//                                             eval.mult(ct, mask) does, and the results are added)
// out = rescale(sum_j a_j (.) p_j)          (separate == 0: the "assemble" step)
// Rescale subtracts NTT_i(centred lift of the last limb) from limb i; NTT is linear modulo q_i, so the
// centred lifts of all terms are summed as integers first and ONE transform per limb serves the whole
// sum.  The stored residues equal those of the term-by-term sequence.
constexpr int kMaxTerms = 24;
struct TermList { const u64 *a[kMaxTerms]; const u64 *p[kMaxTerms]; int count; }; // `count` terms per sum; sum k takes terms k * count ...
// last[g][k * nbp + bp][x] = (the terms of group g of sum k) a_j[bp][level][x] * p_j[level][x] mod q_level
// grid = (N/256, sums * nbp, groups)   groups = count (separate) or 1
__global__ void k_last_prod(u64 *last, const __grid_constant__ TermList tl, int separate, int level, int nbp, const PrimeConst *__restrict__ pc, int N) {
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int x = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (u_ == 0) pdl_wait();
        if (x >= N) break;
        const int bp = blockIdx.y % nbp, first = (blockIdx.y / nbp) * tl.count, g = blockIdx.z;
        const PrimeConst m = pc[level];
        const size_t ao = ((size_t)bp * (level + 1) + level) * N + x, po = (size_t)level * N + x;
        const int j0 = first + (separate ? g : 0), j1 = separate ? j0 + 1 : first + tl.count;
        u64 r;
        if (m.fp) {
            u64 acc = 0;
            for (int j = j0; j < j1; ++j) acc += mul_small_lazy(tl.a[j][ao], tl.p[j][po], m.q_inv_f, m.q);
            r = reduce_fp(acc, m.q_inv_f, m.q);
        } else {
            PieceAcc s; s.zero();
            for (int j = j0; j < j1; ++j) {
                if (j > j0 && (j - j0) % 7 == 0) s.relax(m);
                s.mac(tl.a[j][ao], tl.p[j][po]);
            }
            r = s.finish(m);
        }
        last[((size_t)g * gridDim.y + blockIdx.y) * N + x] = r;
    }
}
// S[k * nbp + bp][x] = sum_g centred(last[(k * groups + g) * nbp + bp][x]) as a signed integer (|S| <= groups * q_level / 2)
// grid = (N/(256*kElems), sums * nbp)
__global__ void k_centre_sum(i64 *__restrict__ S, const u64 *__restrict__ last, int groups, int nbp, int level, const PrimeConst *__restrict__ pc, int N) {
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int x = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (x >= N) break;
        const int bp = blockIdx.y % nbp, k = blockIdx.y / nbp;
        const u64 ql = pc[level].q, half = ql >> 1;
        i64 acc = 0;
        for (int g = 0; g < groups; ++g) {
            const u64 r = last[((size_t)(k * groups + g) * nbp + bp) * N + x];
            acc += r > half ? (i64)r - (i64)ql : (i64)r;
        }
        S[(size_t)blockIdx.y * N + x] = acc;
    }
}
// t[bp][l][x] = S[bp][x] mod q_l.  grid.y = nbp * level
__global__ void k_lift_mod(u64 *__restrict__ t, const i64 *__restrict__ S, int level, const PrimeConst *__restrict__ pc, int N) {
    const int w = blockIdx.y, bp = w / level, l = w % level;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int x = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (x >= N) break;
        t[(size_t)w * N + x] = reduce_i64_any(S[(size_t)bp * N + x], pc[l]);
    }
}
// out[bp][l][x] = (sum_j a_j[bp][l][x] * p_j[l][x] - t[bp][l][x]) * q_level^-1.  grid = (N/(256*kElems), sums * nbp * level); instance k * nbp + bp.
// The four coefficients of a thread sit in the inner loop so that eight loads of one term (and, unrolled, of the
// next) are in flight together: the kernel streams `count` ciphertexts per output and lives on memory parallelism.
// Blocks are ordered limb-major (all batch members of limb 0, then of limb 1, ...): the plaintext limbs of a sum are
// shared by every member, and in this order they stay in L2 while the members stream past.
__global__ void k_prod_rescale_fin(u64 *out, const __grid_constant__ TermList tl, const u64 *t, int level, int nbp, const PrimeConst *__restrict__ pc, int N, const __grid_constant__ Scalars qlinv) {
    const int total = gridDim.y / level, l = blockIdx.y / total, inst = blockIdx.y % total, bp = inst % nbp, first = (inst / nbp) * tl.count, w = inst * level + l;
    const PrimeConst m = pc[l];
    pdl_wait();
    const u32 x0 = blockIdx.x * (blockDim.x * kElems) + threadIdx.x;
    const size_t ao = ((size_t)bp * (level + 1) + l) * N + x0, po = (size_t)l * N + x0;
    u64 v[kElems];
    if (m.fp) {
        u64 acc[kElems];
#pragma unroll
        for (int u = 0; u < kElems; ++u) acc[u] = 0;
#pragma unroll 2
        for (int j = first; j < first + tl.count; ++j) {
            const u64 *a = tl.a[j] + ao, *p = tl.p[j] + po;
#pragma unroll
            for (int u = 0; u < kElems; ++u) acc[u] += mul_small_lazy(a[u * blockDim.x], p[u * blockDim.x], m.q_inv_f, m.q);
        }
#pragma unroll
        for (int u = 0; u < kElems; ++u) v[u] = reduce_fp(acc[u], m.q_inv_f, m.q);
    } else {
        PieceAcc s[kElems];
#pragma unroll
        for (int u = 0; u < kElems; ++u) s[u].zero();
#pragma unroll 2
        for (int j = 0; j < tl.count; ++j) {
            const u64 *a = tl.a[first + j] + ao, *p = tl.p[first + j] + po;
            if (j && j % 7 == 0) {
#pragma unroll
                for (int u = 0; u < kElems; ++u) s[u].relax(m);
            }
#pragma unroll
            for (int u = 0; u < kElems; ++u) s[u].mac(a[u * blockDim.x], p[u * blockDim.x]);
        }
#pragma unroll
        for (int u = 0; u < kElems; ++u) v[u] = s[u].finish(m);
    }
    const u64 *tp = t + (size_t)w * N + x0;
    u64 *op = out + (size_t)w * N + x0;
#pragma unroll
    for (int u = 0; u < kElems; ++u) op[u * blockDim.x] = mul_mod_any(sub_mod(v[u], tp[u * blockDim.x], m.q), qlinv.v[l], m);
}

// out[inst][l][x] = sum_j a_j[bp][l][x] * p_j[l][x], canonical, for all limbs up to `level`; instance k * nbp + bp, terms and block order as above.  On 2^16
// rings the sums of a masked sum go from here through a rescale like any other ciphertext's: last limb to coefficients, lift, forward row pass that ends
// in the division (k_last_prod and a k_prod_rescale_fin behind whole transforms: five launches instead of four, and the division's product on its own).
// grid = (N/(256*kElems), instances * (level + 1))
__global__ void __launch_bounds__(256) k_prod_sums(u64 *out, const __grid_constant__ TermList tl, int level, int nbp, const PrimeConst *__restrict__ pc, int N) {
    const int total = gridDim.y / (level + 1), l = blockIdx.y / total, inst = blockIdx.y % total, bp = inst % nbp, first = inst / nbp * tl.count;
    const PrimeConst m = pc[l];
    pdl_wait();
    const u32 x0 = blockIdx.x * (256 * kElems) + threadIdx.x;
    const size_t ao = ((size_t)bp * (level + 1) + l) * N + x0, po = (size_t)l * N + x0;
    u64 v[kElems];
    auto sum = [&](auto &s, int room) {
#pragma unroll
        for (int u = 0; u < kElems; ++u) s[u].zero();
#pragma unroll 2
        for (int j = 0; j < tl.count; ++j) {
            const u64 *a = tl.a[first + j] + ao, *p = tl.p[first + j] + po;
            if (j && j % room == 0) {
#pragma unroll
                for (int u = 0; u < kElems; ++u) s[u].relax(m);
            }
#pragma unroll
            for (int u = 0; u < kElems; ++u) s[u].product(a[u * 256], p[u * 256]);
        }
#pragma unroll
        for (int u = 0; u < kElems; ++u) v[u] = s[u].canonical(m);
    };
    if (m.fp) { FpAcc s[kElems]; sum(s, m.q < (1ull << 42) ? 64 : 7); } // with what relax leaves: 128 products, eight (FpAcc, PieceAcc)
    else { PieceAcc s[kElems]; sum(s, 7); }
    u64 *op = out + ((size_t)inst * (level + 1) + l) * N + x0;
#pragma unroll
    for (int u = 0; u < kElems; ++u) op[u * 256] = v[u];
}

// Form of a factor that many products share (masks in shared memory, words of a masked key; nothing outside the kernels sees it): an integer-valued double for primes below 2^44, the two
// 30-bit pieces in the halves of the word otherwise.
__device__ __forceinline__ u64 key_word(u64 w, bool fp) { return fp ? (u64)__double_as_longlong(u52_to_double(w)) : ((w >> 30) << 32) | ((u32)w & 0x3FFFFFFFu); }
// ---- the same for all giant-step parts of a baby-step / giant-step transform at once ----
// A transform with bs baby rotations a_j and 2 gs parts computes  out_g = rescale(sum_j a_j (.) p_gj): every part reads
// the same a_j.  One pass per limb keeps a part accumulator per g in registers and reads every a_j once (and, for
// primes below 2^44, converts it once) instead of once per part; the masks p_gj are shared by all members and come
// from L2.  Absent terms of a part are null pointers.
constexpr int kMaxParts = 17, kMaxPartTerms = 17;
struct PartTerms { const u64 *a[kMaxPartTerms]; const u64 *p[kMaxParts][kMaxPartTerms]; int count, parts; };
// last[(g * count + j) * nbp + bp][x] = a_j[bp][level][x] * p_gj[level][x] mod q_level, zero for an absent term: every product is
// rescaled on its own (as eval.mult(ct, mask) does).  grid = (N/256, nbp, parts * count)
__global__ void k_last_prod_parts(u64 *last, const __grid_constant__ PartTerms pt, int level, int nbp, const PrimeConst *__restrict__ pc, int N) {
    const int bp = blockIdx.y, g = blockIdx.z / pt.count, j = blockIdx.z % pt.count;
    const PrimeConst m = pc[level];
    const u64 *p = pt.p[g][j];
    pdl_wait();
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int x = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (x >= N) break;
        last[((size_t)blockIdx.z * nbp + bp) * N + x] = p ? mul_mod_any(pt.a[j][((size_t)bp * (level + 1) + level) * N + x], p[(size_t)level * N + x], m) : 0;
    }
}
// A CTA of 512 threads keeps the mask chunks of G parts for its kPartLanes coefficients of one limb in shared memory (bulk copies, up to
// G * 17 chunks of 1 KB, one mbarrier, bounded wait) and walks over the polynomials, eight at a time (thread = coefficient +
// kPartLanes * pair of polynomials): the masks cross L2 once per CTA and shared memory once per two polynomials.  The words a_j, and the words of
// t that a sum is subtracted from, come through a ring of kPartRing stages in shared memory that runs on across terms and polynomials, each
// thread copying its own (cp.async, no barrier).  With two loads ahead in registers and t loaded when it was needed, 6.1 ms for 48
// polynomials, sixteen terms, twelve parts at level 7 (both launches); with the ring for the a_j 5.5, with t in it as well 4.1, with addresses
// from a table instead of branches and one instruction per wide multiply-add 3.7 ms.  Memory hardly shows any more (DRAM 16 %, half a
// warp waiting for loads): four warps a scheduler issue in 57 % of the slots, between fixed latencies and their turns at the math pipes (FP64 45 % of
// the time on a short limb, wide multiply-adds 37 % over all).
// t == nullptr: raw sums of the limbs from `from` on, out[((g * nbp + bp) * limbs + k) * N + x] for limb from + k    grid = (ceil(parts/G), N/kPartLanes, limbs)
// else: out[((g * nbp + bp) * level + l) * N + x] = (sum - t[same]) * q_level^-1 mod q_l      grid = (ceil(parts/G), N/kPartLanes, level)
// (parts first, so that the CTAs that read the same words run together)
constexpr int kPartLanes = 128, kPartRing = 8;
constexpr size_t part_smem(int g, int count) { return ((size_t)g * count * kPartLanes + (size_t)kPartRing * 2 * 512) * 8; }
template <int G>
__global__ void __launch_bounds__(512, 1) k_prod_parts(u64 *__restrict__ out, const __grid_constant__ PartTerms pt, const u64 *__restrict__ t, int level, int from, int nbp,
                                                       const PrimeConst *__restrict__ pc, int N, const __grid_constant__ Scalars qlinv, int *__restrict__ err) {
    constexpr int M = 2, kSlots = 512 / kPartLanes, kStage = M * 512; // members of a thread
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) u64 bar;
    const int count = pt.count;
    const u64 *ring = reinterpret_cast<u64 *>(smem_raw) + threadIdx.x;   // [kPartRing][2][512]
    u64 *ptile = reinterpret_cast<u64 *>(smem_raw) + kPartRing * kStage; // [count][G][kPartLanes]
    const u32 ring_at = smem_u32(ring);
    const int tid = threadIdx.x, lane = tid & (kPartLanes - 1), slot = tid / kPartLanes;
    const int l = from + (int)blockIdx.z, g0 = blockIdx.x * G;
    const int gn = min(G, pt.parts - g0);
    const u32 x0 = blockIdx.y * kPartLanes;
    // What a member needs, in order: its terms a_j, then the words of t that its parts are subtracted from.  (address at member 0, bytes per member)
    __shared__ ulonglong2 table[kMaxPartTerms + G];
    const u32 words = (u32)(count + (t ? gn : 0));
    const size_t member = (size_t)(level + 1) * N, t_member = (size_t)level * N, t_part = (size_t)nbp * t_member, first = (size_t)l * N + x0;
    if ((u32)tid < words)
        table[tid] = tid < count ? make_ulonglong2((u64)(size_t)(pt.a[tid] + first), member * 8) : make_ulonglong2((u64)(size_t)(t + (size_t)(g0 + tid - count) * t_part + first), t_member * 8);
    if (tid == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    __syncthreads();
    if (tid < 32) {
        if (tid == 0) {
            u32 present = 0;
            for (int ci = 0; ci < gn * count; ++ci) present += pt.p[g0 + ci / count][ci % count] != nullptr;
            mbar_arrive_expect_tx(&bar, present * (kPartLanes * 8u));
        }
        __syncwarp();
        for (int ci = tid; ci < gn * count; ci += 32) {
            const u64 *src = pt.p[g0 + ci / count][ci % count];
            if (src) bulk_load(ptile + (size_t)((ci % count) * G + ci / count) * kPartLanes, src + (size_t)l * N + x0, kPartLanes * 8u, &bar);
        }
    }
    // The words of this thread: members slot * M .., then kSlots * M further on, by the table's rows for each.  Past the last member the
    // last one is fetched again, and not used.
    const u32 lane_at = (u32)lane * 8u, last_member = (u32)nbp - 1u;
    u32 row = 0, fb = (u32)(M * slot), to = 0; // what is fetched next; byte offset of the stage that it goes to
    auto fetch = [&] {
        const ulonglong2 r = table[row];
        const u64 p = r.x + lane_at;
        cp_async8(ring_at + to, reinterpret_cast<const void *>(p + (u64)min(fb, last_member) * (u32)r.y));
        cp_async8(ring_at + to + 4096, reinterpret_cast<const void *>(p + (u64)min(fb + 1u, last_member) * (u32)r.y));
        cp_async_commit();
        const bool wrap = row + 1u == words;
        row = wrap ? 0u : row + 1u;
        fb += wrap ? (u32)(kSlots * M) : 0u;
        to = (to + kStage * 8) & (kPartRing * kStage * 8 - 1);
    };
#pragma unroll 1
    for (int k = 0; k < kPartRing - 1; ++k) fetch();
    u32 have[G]; // bit j: part g0 + g has term j
#pragma unroll
    for (int g = 0; g < G; ++g) {
        have[g] = 0;
        if (g < gn)
            for (int j = 0; j < count; ++j) have[g] |= (pt.p[g0 + g][j] != nullptr ? 1u : 0u) << j;
    }
    mbar_wait_bounded(&bar, 0, err);
    const PrimeConst m = pc[l];
    const u64 qli = t ? qlinv.v[l] : 0;
    const double qd = (double)m.q;
    // Absent terms get zero masks, so the product loop below is straight-line code (no test per part and term: the
    // independent chains of the G parts interleave); the masks become doubles or pairs of pieces once.
#pragma unroll
    for (int g = 0; g < G; ++g)
        for (int j = slot; j < count; j += kSlots) {
            u64 *w = ptile + (size_t)(j * G + g) * kPartLanes + lane;
            *w = ((have[g] >> j) & 1u) ? key_word(*w, m.fp) : 0;
        }
    __syncthreads();
    const bool eight = !(m.fp && m.q < (1ull << 42)); // at most eight products between two reductions of a sum, else 128 (FpAcc, PieceAcc)
    int use = 0; // word offset of the stage that is read next
    auto next = [&](u64 (&a)[M]) {
        cp_async_wait<kPartRing - 2>();
#pragma unroll
        for (int i = 0; i < M; ++i) a[i] = ring[use + i * 512];
        use = (use + kStage) & (kPartRing * kStage - 1);
        fetch();
    };
    for (int bp = M * slot; bp < nbp; bp += kSlots * M) {
        u64 v[M][G];
        const u64 *w = ptile + lane;
        auto term = [&](int j, auto &&product) {
            u64 a[M];
            next(a);
            product(a, w, eight && j && j % 8 == 0);
            w += G * kPartLanes;
        };
        if (m.fp) { // products and sums exactly on the FP64 pipe
            FpAcc s[M][G];
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int g = 0; g < G; ++g) s[i][g].zero();
            auto product = [&](const u64 (&a)[M], const u64 *w, bool full) {
                if (full) {
#pragma unroll
                    for (int i = 0; i < M; ++i)
#pragma unroll
                        for (int g = 0; g < G; ++g) s[i][g].relax(m.q_inv_f, qd);
                }
                double d[M];
#pragma unroll
                for (int i = 0; i < M; ++i) d[i] = u52_to_double(a[i]);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const double k = __longlong_as_double((long long)w[g * kPartLanes]);
#pragma unroll
                    for (int i = 0; i < M; ++i) s[i][g].mac(d[i], k);
                }
            };
#pragma unroll 2
            for (int j = 0; j < count; ++j) term(j, product);
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int g = 0; g < G; ++g) v[i][g] = s[i][g].finish(m.q_inv_f, qd);
        } else {
            PieceAcc s[M][G];
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int g = 0; g < G; ++g) s[i][g].zero();
            auto product = [&](const u64 (&a)[M], const u64 *w, bool full) {
                if (full) {
#pragma unroll
                    for (int i = 0; i < M; ++i)
#pragma unroll
                        for (int g = 0; g < G; ++g) s[i][g].relax(m);
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const u64 k = w[g * kPartLanes];
#pragma unroll
                    for (int i = 0; i < M; ++i) s[i][g].mac((u32)a[i] & 0x3FFFFFFFu, (u32)(a[i] >> 30), (u32)k, (u32)(k >> 32));
                }
            };
#pragma unroll 1
            for (int j = 0; j < count; ++j) term(j, product);
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int g = 0; g < G; ++g) v[i][g] = s[i][g].finish(m);
        }
        const size_t o_member = (size_t)gridDim.z * N, o_part = (size_t)nbp * o_member;
        u64 *o = out + (size_t)g0 * o_part + (size_t)bp * o_member + (size_t)blockIdx.z * N + x0 + lane;
#pragma unroll
        for (int g = 0; g < G; ++g, o += o_part)
            if (g < gn) {
                u64 a[M];
                if (t) next(a);
#pragma unroll
                for (int i = 0; i < M; ++i)
                    if (bp + i < nbp) o[i * o_member] = t ? mul_mod_any(sub_mod(v[i][g], a[i], m.q), qli, m) : v[i][g];
            }
    }
    cp_async_wait<0>(); // what was fetched past the end
}
// The same for a few polynomials or parts: the masks are then most of the bytes, so they are streamed instead of kept.  A thread holds the words
// a_j of its coefficient in two polynomials and walks over the parts, with the masks of a part in flight together.  A launch for one two-tile
// product 604 -> 215 us (2.5 TB/s of masks).  TERMS: the most terms there can be; all of them are multiplied, and what a call does not have is
// zero.  With seventeen for every call, one term and eight parts of eight polynomials took 871 us at level 7 (kept masks 739);
// with two 523.  grid = (N/256 * pairs of polynomials, limbs), arguments as above
template <int TERMS>
__global__ void __launch_bounds__(256, TERMS <= 4 ? 4 : TERMS <= 8 ? 3 : 2) k_prod_parts_few(u64 *__restrict__ out, const __grid_constant__ PartTerms pt, const u64 *__restrict__ t, int level, int from, int nbp,
                                                                                            const PrimeConst *__restrict__ pc, int N, const __grid_constant__ Scalars qlinv) {
    const int pairs = (nbp + 1) / 2, bp = blockIdx.x % pairs * 2; // the pairs that read the same masks run together
    const int limbs = gridDim.y, k = blockIdx.y, l = from + k, count = pt.count, x = blockIdx.x / pairs * 256 + threadIdx.x;
    const bool both = bp + 1 < nbp;
    const PrimeConst m = pc[l];
    const u64 qli = t ? qlinv.v[l] : 0;
    const double qd = (double)m.q;
    const size_t po = (size_t)l * N + x, ao = po + (size_t)bp * (level + 1) * N, ao1 = both ? ao + (size_t)(level + 1) * N : ao;
    u64 a[2][TERMS];
#pragma unroll
    for (int j = 0; j < TERMS; ++j) {
        a[0][j] = j < count ? key_word(pt.a[j][ao], m.fp) : 0;
        a[1][j] = j < count ? key_word(pt.a[j][ao1], m.fp) : 0;
    }
    const bool eight = !(m.fp && m.q < (1ull << 42));
#pragma unroll 1
    for (int g = 0; g < pt.parts; ++g) {
        u64 w[TERMS], v[2];
#pragma unroll
        for (int j = 0; j < TERMS; ++j) w[j] = j < count && pt.p[g][j] ? pt.p[g][j][po] : 0;
        if (m.fp) {
            FpAcc s[2]; s[0].zero(); s[1].zero();
#pragma unroll
            for (int j = 0; j < TERMS; ++j) {
                if (j && j % 8 == 0 && eight) { s[0].relax(m.q_inv_f, qd); s[1].relax(m.q_inv_f, qd); }
                const double wd = u52_to_double(w[j]);
                s[0].mac(__longlong_as_double((long long)a[0][j]), wd); s[1].mac(__longlong_as_double((long long)a[1][j]), wd);
            }
            v[0] = s[0].finish(m.q_inv_f, qd); v[1] = s[1].finish(m.q_inv_f, qd);
        } else {
            PieceAcc s[2]; s[0].zero(); s[1].zero();
#pragma unroll
            for (int j = 0; j < TERMS; ++j) {
                if (j && j % 8 == 0) { s[0].relax(m); s[1].relax(m); }
                const u32 k0 = (u32)w[j] & 0x3FFFFFFFu, k1 = (u32)(w[j] >> 30);
                s[0].mac((u32)a[0][j], (u32)(a[0][j] >> 32), k0, k1); s[1].mac((u32)a[1][j], (u32)(a[1][j] >> 32), k0, k1);
            }
            v[0] = s[0].finish(m); v[1] = s[1].finish(m);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (i == 0 || both) {
                const size_t o = (((size_t)g * nbp + bp + i) * limbs + k) * N + x;
                out[o] = t ? mul_mod_any(sub_mod(v[i], t[o], m.q), qli, m) : v[i];
            }
    }
}

// ---------------- key switching ----------------
// Per-level plan held in device memory.
struct KsPlan {
    int level, n, ne, nd, K;
    int dt_count;                               // lifted (non-own) limbs over all digits
    int dig_lo[8], dig_hi[8];                   // own limb range of each digit
    int dt_start[8];                            // first compact entry of each digit
    short dt_entry[8][kMaxPrimes];              // [digit][ext limb j] -> compact entry or -1 (own)
    unsigned char ext_prime[kMaxPrimes];        // ext limb j -> prime index
    u64 hat_inv[8][kMaxDigitLimbs], hat_inv_sh[8][kMaxDigitLimbs];
    u64 hat_mod[8][kMaxDigitLimbs][kMaxPrimes]; // [digit][source][ext limb j]
    u64 hat_mod_d0[8][kMaxDigitLimbs][kMaxPrimes]; // the same as a double (bit pattern), and times 2^30 mod the target: for
    u64 hat_mod_d1[8][kMaxDigitLimbs][kMaxPrimes]; // targets below 2^44 the conversion runs on the FP64 pipe
    u64 p_hat_inv[8], p_hat_inv_sh[8];          // ModDown: per special prime
    u64 p_hat_mod[8][kMaxPrimes];               // [special k][q limb l]
    u64 p_hat_mod_d0[8][kMaxPrimes], p_hat_mod_d1[8][kMaxPrimes]; // as doubles, and times 2^30 mod q_l
    u64 p_inv[kMaxPrimes];                      // P^-1 mod q_l
};

// ModUp: a_coef [batch][n][N] (coefficient form) -> dt [batch][dt_count][N] (coefficient form).
// grid = (N/256, nd, batch).  The source count of a digit is a template parameter so that the per-target
// contraction is fully unrolled with no predicated-off iterations.
template <int NS>
__device__ __forceinline__ void modup_body(u64 *__restrict__ dt, const u64 *__restrict__ a_coef, const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int N,
                                           int i, int dg, int b) {
    const int lo = pl->dig_lo[dg], hi = lo + NS, n = pl->n, ne = pl->ne;
    u64 y[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) y[s] = mul_shoup(a_coef[((size_t)b * n + lo + s) * N + i], pl->hat_inv[dg][s], pl->hat_inv_sh[dg][s], pc[lo + s].q);
    u64 *o = dt + ((size_t)b * pl->dt_count + pl->dt_start[dg]) * N + i;
    double y0[NS], y1[NS]; // 30-bit pieces of the sources as doubles, for the targets below 2^44
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        y0[k] = __hiloint2double(0x43300000, (int)((u32)y[k] & 0x3FFFFFFFu)) - kTwo52;
        y1[k] = __hiloint2double(0x43300000, (int)(u32)(y[k] >> 30)) - kTwo52;
    }
    for (int j = 0; j < ne; ++j) {
        if (j >= lo && j < hi) continue;
        const PrimeConst *m = pc + pl->ext_prime[j];
        if (m->fp) {
            const double qinv = m->q_inv_f, qd = (double)m->q;
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                acc = __dadd_rn(acc, mul_fp64_lazy(y0[k], __longlong_as_double((long long)pl->hat_mod_d0[dg][k][j]), qinv, qd));
                acc = __dadd_rn(acc, mul_fp64_lazy(y1[k], __longlong_as_double((long long)pl->hat_mod_d1[dg][k][j]), qinv, qd));
            }
            *o = canon_fp64(acc, qinv, qd);
        } else {
            PieceAcc s; s.zero(); // at most 8 sources
#pragma unroll
            for (int k = 0; k < NS; ++k) s.mac(y[k], pl->hat_mod[dg][k][j]);
            *o = s.finish(*m);
        }
        o += N;
    }
}
__global__ void k_modup(u64 *__restrict__ dt, const u64 *__restrict__ a_coef, const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int N) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int dg = blockIdx.y, b = blockIdx.z;
    switch (pl->dig_hi[dg] - pl->dig_lo[dg]) {
    case 1: modup_body<1>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 2: modup_body<2>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 3: modup_body<3>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 4: modup_body<4>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 5: modup_body<5>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 6: modup_body<6>(dt, a_coef, pl, pc, N, i, dg, b); break;
    case 7: modup_body<7>(dt, a_coef, pl, pc, N, i, dg, b); break;
    default: modup_body<8>(dt, a_coef, pl, pc, N, i, dg, b); break;
    }
}

// What the inner products of many waves of CTAs need of a level's plan before their first loads, as an argument: read from memory it stood in front of them
// in every CTA (wrapped copies of one member 185 -> 178 us a launch, inner products of fifteen rotations of one member 195 -> 189).  ks_rows, whose
// launches are short, reads it from memory: arguments come through a cache that every launch finds cold (rotation of one ciphertext 113 -> 117 us).
struct DigitPlan { int n, ne, dt_count; short entry[8][kMaxPrimes]; unsigned char prime[kMaxPrimes]; }; // as in KsPlan
// Up to 16 groups of `batch` members, each group with its own key switch: operand (limbs of the switched polynomial in NTT form and
// its lifted digits), key, Galois element (0: no automorphism) and addends (null: none).
struct SwitchGroup { const u64 *a_ntt, *dt, *key, *add[2]; u32 g, pad; };
constexpr int kMaxSwitchGroups = 16;
struct SwitchList { SwitchGroup s[kMaxSwitchGroups]; int count; };
// Inner product with the switching key over Q_level u P.
//   acc[ob][p][j][i] = sum_dg digit_dg[j][perm_g(i)] * key[dg][p][prime(j)][i],   member ob = group * batch + b
// digit_dg[j] is a_ntt[j] for own limbs and dt[...] otherwise.  A CTA owns 256 * EL coefficients of one limb for `per` members of a group:
// a thread keeps the key words of its EL coefficients in registers (as doubles, or cut into pieces) and walks over the
// members with the next member's digits in flight, so the keys -- two thirds of the words a member needs -- are read once.
// One member per CTA read and converted them every time: 517 us for 64 members at level 6.  Bound by DRAM: 48 members at level 8 take
// 285 us at 5.3 TB/s (0.82 of a copy), 43 % of the issue slots.  Eight digits spill (160 bytes a thread), seven 32, fewer none.
// grid = (N/(256*EL), groups * ceil(batch/per), ne); ND = digits in use
template <int ND, int EL>
__global__ void __launch_bounds__(256, EL == 1 ? 4 : ND <= 2 ? 3 : 2) k_ks_inner(u64 *acc, const __grid_constant__ SwitchList sl, int batch, int per, size_t a_outer, int key_primes, const __grid_constant__ DigitPlan pl,
                                                                   const PrimeConst *__restrict__ pc, int logn, int N) {
    const int chunks = (batch + per - 1) / per, grp = blockIdx.y / chunks, b0 = (blockIdx.y % chunks) * per, b1 = min(batch, b0 + per);
    const int j = blockIdx.z; // limb-major block order
    const SwitchGroup &sg = sl.s[grp];
    const u32 g = sg.g;
    const int pj = pl.prime[j], ne = pl.ne;
    const PrimeConst m = pc[pj];
    const u32 x0 = blockIdx.x * (256 * EL) + threadIdx.x;
    u32 src[EL];
#pragma unroll
    for (int u = 0; u < EL; ++u) { const u32 i = x0 + u * 256; src[u] = g ? ntt_perm(i, g, logn) : i; }
    const u64 *sp[ND];
    size_t stride[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int en = pl.entry[d][j];
        stride[d] = en < 0 ? a_outer : (size_t)pl.dt_count * N;
        sp[d] = (en < 0 ? sg.a_ntt + (size_t)j * N : sg.dt + (size_t)en * N) + (size_t)b0 * stride[d];
    }
    const u64 *kbase = sg.key + (size_t)pj * N + x0;
    const size_t kpoly = (size_t)key_primes * N;
    u64 *o = acc + (((size_t)(grp * batch + b0) * 2) * ne + j) * N + x0;
    const size_t opoly = (size_t)ne * N;
    pdl_wait();
    u64 cur[ND][EL];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int u = 0; u < EL; ++u) cur[d][u] = sp[d][src[u]];
    if (m.fp) {
        const double qd = (double)m.q;
        double k[ND][2][EL];
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int u = 0; u < EL; ++u) k[d][p][u] = u52_to_double(kbase[(size_t)(d * 2 + p) * kpoly + u * 256]);
        for (int b = b0; b < b1; ++b) {
            double v[ND][EL];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                sp[d] += stride[d];
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    v[d][u] = u52_to_double(cur[d][u]);
                    if (b + 1 < b1) cur[d][u] = sp[d][src[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < EL; ++u)
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    FpAcc s;
                    s.first(v[0][u], k[0][p][u]);
#pragma unroll
                    for (int d = 1; d < ND; ++d) s.mac(v[d][u], k[d][p][u]);
                    o[(size_t)p * opoly + u * 256] = s.finish(m.q_inv_f, qd);
                }
            o += 2 * opoly;
        }
    } else {
        u32 k0[ND][2][EL], k1[ND][2][EL];
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    const u64 w = kbase[(size_t)(d * 2 + p) * kpoly + u * 256];
                    k0[d][p][u] = (u32)w & 0x3FFFFFFFu; k1[d][p][u] = (u32)(w >> 30);
                }
        for (int b = b0; b < b1; ++b) {
            u32 v0[ND][EL], v1[ND][EL];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                sp[d] += stride[d];
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    v0[d][u] = (u32)cur[d][u] & 0x3FFFFFFFu; v1[d][u] = (u32)(cur[d][u] >> 30);
                    if (b + 1 < b1) cur[d][u] = sp[d][src[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < EL; ++u)
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    PieceAccT<true> s; s.zero(); // at most eight digits
#pragma unroll
                    for (int d = 0; d < ND; ++d) s.mac(v0[d][u], v1[d][u], k0[d][p][u], k1[d][p][u]);
                    o[(size_t)p * opoly + u * 256] = s.finish(m);
                }
            o += 2 * opoly;
        }
    }
}

// ModDown conversion: pcoef [bp][K][N] (special limbs, coefficient form) -> t [bp][n][N] (coefficient form)
// grid = (N/256, 1, nbp)
template <int K>
__device__ __forceinline__ void moddown_conv_body(u64 *__restrict__ t, const u64 *__restrict__ pcoef, const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int Lp1,
                                                  int N, int i, int bp) {
    const int n = pl->n;
    u64 y[K];
#pragma unroll
    for (int k = 0; k < K; ++k) y[k] = mul_shoup(pcoef[((size_t)bp * K + k) * N + i], pl->p_hat_inv[k], pl->p_hat_inv_sh[k], pc[Lp1 + k].q);
    u64 *o = t + (size_t)bp * n * N + i;
    double y0[K], y1[K]; // 30-bit pieces of the sources as doubles, for the targets below 2^44
#pragma unroll
    for (int k = 0; k < K; ++k) {
        y0[k] = __hiloint2double(0x43300000, (int)((u32)y[k] & 0x3FFFFFFFu)) - kTwo52;
        y1[k] = __hiloint2double(0x43300000, (int)(u32)(y[k] >> 30)) - kTwo52;
    }
    for (int l = 0; l < n; ++l) {
        if (pc[l].fp) {
            const double qinv = pc[l].q_inv_f, qd = (double)pc[l].q;
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                acc = __dadd_rn(acc, mul_fp64_lazy(y0[k], __longlong_as_double((long long)pl->p_hat_mod_d0[k][l]), qinv, qd));
                acc = __dadd_rn(acc, mul_fp64_lazy(y1[k], __longlong_as_double((long long)pl->p_hat_mod_d1[k][l]), qinv, qd));
            }
            *o = canon_fp64(acc, qinv, qd);
        } else {
            PieceAcc s; s.zero();
#pragma unroll
            for (int k = 0; k < K; ++k) s.mac(y[k], pl->p_hat_mod[k][l]);
            *o = s.finish(pc[l]);
        }
        o += N;
    }
}
__global__ void k_moddown_conv(u64 *__restrict__ t, const u64 *__restrict__ pcoef, const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int Lp1, int N) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int bp = blockIdx.z;
    switch (pl->K) {
    case 1: moddown_conv_body<1>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 2: moddown_conv_body<2>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 3: moddown_conv_body<3>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 4: moddown_conv_body<4>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 5: moddown_conv_body<5>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 6: moddown_conv_body<6>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    case 7: moddown_conv_body<7>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    default: moddown_conv_body<8>(t, pcoef, pl, pc, Lp1, N, i, bp); break;
    }
}
// out[ob][p][l][i] = (acc[ob][p][l][i] - t[ob][p][l][i]) * P^-1 + add_p[b][l][perm_g(i)],  addends and g of ob's group
// grid = (N/256, n, groups*batch*2)
__global__ void k_moddown_fin(u64 *out, size_t out_outer, const u64 *acc, const u64 *t, const __grid_constant__ SwitchList sl, int batch, size_t add_outer, const KsPlan *__restrict__ pl,
                              const PrimeConst *__restrict__ pc, int logn, int N) {
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const int l = blockIdx.y, bp = blockIdx.z, ob = bp >> 1, b = ob % batch, p = bp & 1;
        const SwitchGroup &sg = sl.s[ob / batch];
        const int n = pl->n, ne = pl->ne;
        const PrimeConst m = pc[l];
        u64 v = sub_mod(acc[((size_t)bp * ne + l) * N + i], t[((size_t)bp * n + l) * N + i], m.q);
        v = mul_mod_any(v, pl->p_inv[l], m);
        const u64 *ad = sg.add[p];
        if (ad) {
            const u32 s = sg.g ? ntt_perm((u32)i, sg.g, logn) : (u32)i;
            v = add_mod(v, ad[(size_t)b * add_outer + (size_t)l * N + s], m.q);
        }
        out[(size_t)ob * out_outer + ((size_t)p * n + l) * N + i] = v;
    }
}

// ---------------- sum of rotations with one ModDown ----------------
// Up to 16 terms (ciphertext batch x_t rotated by g_t): the inner products of all terms are added up in Q_level u P.
struct RotTerm { const u64 *a_ntt; const u64 *dt; const u64 *key; u32 g; u32 pad; };
struct RotTermList { RotTerm t[16]; int count; };
//   acc[b][p][j][i] = sum_t sum_dg digit_t,dg[j][perm_t(i)] * key_t[dg][p][prime(j)][i]
// A thread works on EL coefficients of M members: a key word is read (and converted or cut) once for M products, and the sums take
// one reduction each.  One member per thread, every product reduced: 1068 us a launch in the layer pass, now 907 us (four members);
// a single ciphertext 107 -> 100 us.  Bound by instruction issue, half of it on the 60-bit limbs.
// grid = (N/(256*EL), ceil(batch/M), ne); members beyond the batch repeat the last one and are not stored
template <int EL, int M>
__global__ void __launch_bounds__(256, 2) k_ks_inner_sum(u64 *acc, const __grid_constant__ RotTermList tl, int batch, size_t a_outer, int key_primes, const KsPlan *__restrict__ pl,
                                                         const PrimeConst *__restrict__ pc, int logn, int N) {
    const int j = blockIdx.z, b0 = blockIdx.y * M;
    const int pj = pl->ext_prime[j], nd = pl->nd, ne = pl->ne;
    const PrimeConst m = pc[pj];
    const u32 x0 = blockIdx.x * (256 * EL) + threadIdx.x;
    const size_t kpoly = (size_t)key_primes * N, d_outer = (size_t)pl->dt_count * N;
    u64 r[2][M][EL];
    // every term meets EL * (M digit words + 2 key words) per digit
    auto terms = [&](auto &&product) {
        for (int t = 0; t < tl.count; ++t) {
            const RotTerm &rt = tl.t[t];
            u32 src[EL];
#pragma unroll
            for (int u = 0; u < EL; ++u) src[u] = ntt_perm(x0 + u * 256, rt.g, logn);
            const u64 *kbase = rt.key + (size_t)pj * N + x0;
#pragma unroll 2
            for (int dg = 0; dg < nd; ++dg) {
                const int en = pl->dt_entry[dg][j];
                const u64 *sp = en < 0 ? rt.a_ntt + (size_t)j * N : rt.dt + (size_t)en * N;
                const size_t outer = en < 0 ? a_outer : d_outer;
                u64 v[M][EL], k[2][EL];
#pragma unroll
                for (int u = 0; u < EL; ++u) {
#pragma unroll
                    for (int i = 0; i < M; ++i) v[i][u] = sp[(size_t)min(b0 + i, batch - 1) * outer + src[u]];
                    k[0][u] = kbase[(size_t)(dg * 2) * kpoly + u * 256];
                    k[1][u] = kbase[(size_t)(dg * 2 + 1) * kpoly + u * 256];
                }
                product(v, k);
            }
        }
    };
    if (m.fp) { // exact sums (see FpAcc): 128 products of primes below 2^42, eight below 2^44, before they are reduced
        const double qd = (double)m.q;
        const int room = m.q < (1ull << 42) ? 128 : 8;
        FpAcc s[2][M][EL];
        int held = 0;
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int u = 0; u < EL; ++u) s[p][i][u].zero();
        terms([&](const u64 (&v)[M][EL], const u64 (&k)[2][EL]) {
            if (++held > room) {
                held = 1;
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int i = 0; i < M; ++i)
#pragma unroll
                        for (int u = 0; u < EL; ++u) s[p][i][u].relax(m.q_inv_f, qd);
            }
#pragma unroll
            for (int u = 0; u < EL; ++u) {
                const double k0 = u52_to_double(k[0][u]), k1 = u52_to_double(k[1][u]);
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    const double vd = u52_to_double(v[i][u]);
                    s[0][i][u].mac(vd, k0);
                    s[1][i][u].mac(vd, k1);
                }
            }
        });
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int u = 0; u < EL; ++u) r[p][i][u] = s[p][i][u].finish(m.q_inv_f, qd);
    } else {
        PieceAcc s[2][M][EL];
        int held = 0; // products in the accumulators
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int u = 0; u < EL; ++u) s[p][i][u].zero();
        terms([&](const u64 (&v)[M][EL], const u64 (&k)[2][EL]) {
            if (++held > 8) {
                held = 1;
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int i = 0; i < M; ++i)
#pragma unroll
                        for (int u = 0; u < EL; ++u) s[p][i][u].relax(m);
            }
#pragma unroll
            for (int u = 0; u < EL; ++u)
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    s[0][i][u].mac(v[i][u], k[0][u]);
                    s[1][i][u].mac(v[i][u], k[1][u]);
                }
        });
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int i = 0; i < M; ++i)
#pragma unroll
                for (int u = 0; u < EL; ++u) r[p][i][u] = s[p][i][u].finish(m);
    }
#pragma unroll
    for (int i = 0; i < M; ++i)
        if (b0 + i < batch) {
            u64 *o = acc + (((size_t)(b0 + i) * 2) * ne + j) * N + x0;
#pragma unroll
            for (int u = 0; u < EL; ++u) { o[u * 256] = r[0][i][u]; o[(size_t)ne * N + u * 256] = r[1][i][u]; }
        }
}
// add[b][p][l][i] = sum over the rotated terms of (p == 0) c0_t[b][l][perm_t(i)]  +  sum over the unrotated terms of x_t[b][p][l][i]
// rot: terms with g != 1 (a_ntt - n limbs = c0); plain: terms added as they are.  grid = (N/(256*kElems), n, batch*2)
struct PlainTermList { const u64 *x[16]; int count; };
__global__ void k_rot_sum_addend(u64 *__restrict__ add, const __grid_constant__ RotTermList rot, const __grid_constant__ PlainTermList plain, int n, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int logn, int N) {
    const int l = blockIdx.y, bp = blockIdx.z, b = bp >> 1, p = bp & 1;
    const u64 q = pc[map.prime[l]].q;
    const size_t ct_outer = (size_t)2 * n * N;
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        u64 v = 0;
        if (p == 0)
            for (int t = 0; t < rot.count; ++t) // a_ntt points at the second polynomial; the first sits n limbs before it
                v = add_mod(v, (rot.t[t].a_ntt - (size_t)n * N)[(size_t)b * ct_outer + (size_t)l * N + ntt_perm((u32)i, rot.t[t].g, logn)], q);
        for (int t = 0; t < plain.count; ++t) v = add_mod(v, plain.x[t][(size_t)b * ct_outer + ((size_t)p * n + l) * N + i], q);
        add[((size_t)bp * n + l) * N + i] = v;
    }
}

// ---------------- masked pair of rotations with one division by P * q_level ----------------
// Constants of the division of a Q_level u P polynomial by D = P * q_level (sources: q_level, p_1 .. p_K).
struct DivPlan {
    int level, ns;                     // ns = K + 1 source limbs
    unsigned char src_prime[8];
    u64 hat_inv[8], hat_inv_sh[8];     // (D / d_s)^-1 mod d_s
    u64 hat_mod[8][kMaxPrimes];        // (D / d_s) mod q_i, i < level
    u64 hat_mod_d0[8][kMaxPrimes];     // the same as a double (bit pattern), for targets below 2^44
    u64 hat_mod_d1[8][kMaxPrimes];     // (D / d_s) * 2^30 mod q_i as a double (bit pattern)
    u64 d_inv[kMaxPrimes];             // D^-1 mod q_i
    u64 p_mod[kMaxPrimes];             // P mod q_j, j <= level
};
struct RotPair {                       // the two rotations of one call
    const u64 *key[2];                 // switching keys
    const u64 *mask[2];                // extended plaintexts [ne][N]
    u32 g[2];
};
// E[b][p][j][i] = sum_r mask_r[j][i] * (sum_dg digit_dg[j][perm_r(i)] * key_r[dg][p][prime(j)][i])
//               + (p == 0 and j < n)  P * sum_r mask_r[j][i] * c0[b][j][perm_r(i)]
// Every term is reduced to its canonical residue before the next operation uses it.  grid = (N/(256*kElems), ne, batch)
__global__ void k_ks_inner_pair(u64 *__restrict__ E, const u64 *__restrict__ c0, const u64 *__restrict__ a_ntt, size_t a_outer, const u64 *__restrict__ dt, const __grid_constant__ RotPair rp,
                                int key_primes, const KsPlan *__restrict__ pl, const DivPlan *__restrict__ dv, const PrimeConst *__restrict__ pc, int logn, int N) {
    const int j = blockIdx.y, b = blockIdx.z;
    const int pj = pl->ext_prime[j], nd = pl->nd, ne = pl->ne, n = pl->n;
    const PrimeConst m = pc[pj];
    const u32 x0 = blockIdx.x * (blockDim.x * kElems) + threadIdx.x;
    const u64 *abase = a_ntt + (size_t)b * a_outer + (size_t)j * N;
    const u64 *cbase = c0 + (size_t)b * a_outer + (size_t)j * N;
    const u64 *dbase = dt + (size_t)b * pl->dt_count * N;
    const size_t kpoly = (size_t)key_primes * N;
    u64 e0[kElems], e1[kElems], f[kElems];
#pragma unroll
    for (int u = 0; u < kElems; ++u) { e0[u] = 0; e1[u] = 0; f[u] = 0; }
    // When both steps are the same rotation (a row shift by a whole tile height on a full slot grid) the two inner
    // products are the same polynomial: it is computed once and multiplied by mask_0 + mask_1, which gives the same
    // residues as the two-term sum.
    const int nrot = rp.g[0] == rp.g[1] ? 1 : 2;
    for (int r = 0; r < nrot; ++r) {
        u32 src[kElems];
#pragma unroll
        for (int u = 0; u < kElems; ++u) src[u] = ntt_perm(x0 + u * blockDim.x, rp.g[r], logn);
        const u64 *kbase = rp.key[r] + (size_t)pj * N + x0;
        u64 r0[kElems], r1[kElems];
        if (m.fp) {
#pragma unroll
            for (int u = 0; u < kElems; ++u) { r0[u] = 0; r1[u] = 0; }
            for (int dg = 0; dg < nd; ++dg) {
                const int en = pl->dt_entry[dg][j];
                const u64 *sp = en < 0 ? abase : dbase + (size_t)en * N;
                const u64 *k0 = kbase + (size_t)dg * 2 * kpoly;
#pragma unroll
                for (int u = 0; u < kElems; ++u) {
                    const u64 v = sp[src[u]], ka = k0[u * blockDim.x], kb = k0[kpoly + u * blockDim.x];
                    const double vd = u52_to_double(v);
                    r0[u] += mul_small_lazy_d(v, vd, ka, u52_to_double(ka), m.q_inv_f, m.q);
                    r1[u] += mul_small_lazy_d(v, vd, kb, u52_to_double(kb), m.q_inv_f, m.q);
                }
            }
#pragma unroll
            for (int u = 0; u < kElems; ++u) { r0[u] = reduce_fp(r0[u], m.q_inv_f, m.q); r1[u] = reduce_fp(r1[u], m.q_inv_f, m.q); }
        } else {
            PieceAcc s0[kElems], s1[kElems];
#pragma unroll
            for (int u = 0; u < kElems; ++u) { s0[u].zero(); s1[u].zero(); }
            for (int dg = 0; dg < nd; ++dg) {
                const int en = pl->dt_entry[dg][j];
                const u64 *sp = en < 0 ? abase : dbase + (size_t)en * N;
                const u64 *k0 = kbase + (size_t)dg * 2 * kpoly;
#pragma unroll
                for (int u = 0; u < kElems; ++u) {
                    const u64 v = sp[src[u]];
                    s0[u].mac(v, k0[u * blockDim.x]);
                    s1[u].mac(v, k0[kpoly + u * blockDim.x]);
                }
            }
#pragma unroll
            for (int u = 0; u < kElems; ++u) { r0[u] = s0[u].finish(m); r1[u] = s1[u].finish(m); }
        }
        const u64 *mk = rp.mask[r] + (size_t)j * N + x0, *mk2 = rp.mask[1] + (size_t)j * N + x0;
#pragma unroll
        for (int u = 0; u < kElems; ++u) {
            u64 w = mk[u * blockDim.x];
            if (nrot == 1) w = add_mod(w, mk2[u * blockDim.x], m.q);
            e0[u] = add_mod(e0[u], mul_mod_any(w, r0[u], m), m.q);
            e1[u] = add_mod(e1[u], mul_mod_any(w, r1[u], m), m.q);
            if (j < n) f[u] = add_mod(f[u], mul_mod_any(w, cbase[src[u]], m), m.q);
        }
    }
    if (j < n) {
        const u64 pm = dv->p_mod[j];
#pragma unroll
        for (int u = 0; u < kElems; ++u) e0[u] = add_mod(e0[u], mul_mod_any(pm, f[u], m), m.q);
    }
    u64 *o0 = E + (((size_t)b * 2) * ne + j) * N + x0, *o1 = o0 + (size_t)ne * N;
#pragma unroll
    for (int u = 0; u < kElems; ++u) { o0[u * blockDim.x] = e0[u]; o1[u * blockDim.x] = e1[u]; }
}
// ---- the same sum with the masks folded into the switching keys ----
// sum_dg digit_dg * (mask * key_dg) = mask * sum_dg digit_dg * key_dg modulo q, so a key multiplied by the mask once
// (k_mask_key) turns the masked pair of rotations into ONE lazy inner product with ONE reduction per output residue;
// the residues are those of k_ks_inner_pair.
// mkey[dg][p][j][i] = (mask[j][i] + mask2[j][i]) * key[dg][p][prime(j)][i];  grid = (N/(256*kElems), ne, nd*2)
__global__ void k_mask_key(u64 *__restrict__ mkey, const u64 *__restrict__ key, int key_primes, const u64 *__restrict__ mask, const u64 *__restrict__ mask2,
                           const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int N) {
    const int j = blockIdx.y, dgp = blockIdx.z, ne = pl->ne;
    const int pj = pl->ext_prime[j];
    const PrimeConst m = pc[pj];
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        u64 w = mask[(size_t)j * N + i];
        if (mask2) w = add_mod(w, mask2[(size_t)j * N + i], m.q);
        mkey[((size_t)dgp * ne + j) * N + i] = key_word(mul_mod_any(w, key[((size_t)dgp * key_primes + pj) * N + i], m), m.fp);
    }
}
// pm[j][i] = P * (mask[j][i] + mask2[j][i]) mod q_j for the Q limbs;  grid = (N/(256*kElems), n)
__global__ void k_mask_p(u64 *__restrict__ pm, const u64 *__restrict__ mask, const u64 *__restrict__ mask2, const DivPlan *__restrict__ dv, const PrimeConst *__restrict__ pc, int N) {
    const int j = blockIdx.y;
    const PrimeConst m = pc[j];
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        u64 w = mask[(size_t)j * N + i];
        if (mask2) w = add_mod(w, mask2[(size_t)j * N + i], m.q);
        pm[(size_t)j * N + i] = key_word(mul_mod_any(w, dv->p_mod[j], m), m.fp);
    }
}
struct MaskedRot {
    const u64 *mkey[2];   // [nd][2][ne][N]
    const u64 *pm[2];     // [n][N]
    u32 g[2];
    int count;            // 1 or 2 rotations
};
constexpr int kMaxRotGroups = 16;
struct MaskedRotList { MaskedRot r[kMaxRotGroups]; }; // one entry per wrapped copy made by the same launch
// E[b][p][j][i] = sum_r sum_dg digit_dg[j][perm_r(i)] * mkey_r[dg][p][j][i]  +  (p == 0, j < n) sum_r c0[b][j][perm_r(i)] * pm_r[j][i]
// Output member g * batch + b is wrapped copy number g (its own one or two masked keys) of input member b: several iterations
// of a shift loop in one launch.
//
// Any number of digits: one member and four coefficients per thread.  grid = (N/1024, groups * batch, ne)
__global__ void __launch_bounds__(256, 2) k_ks_inner_mk(u64 *E, const u64 *c0, const u64 *a_ntt, size_t a_outer, const u64 *dt, const __grid_constant__ MaskedRotList mrl, int batch,
                                                        const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, int logn, int N) {
    constexpr int EL = 4;
    const int j = blockIdx.z, ob = blockIdx.y, b = ob % batch; // limb-major block order: the key limbs stay in L2 across the members
    const MaskedRot &mr = mrl.r[ob / batch];
    const int pj = pl->ext_prime[j], nd = pl->nd, ne = pl->ne, n = pl->n;
    const PrimeConst m = pc[pj];
    const u32 x0 = blockIdx.x * (blockDim.x * EL) + threadIdx.x;
    const u64 *abase = a_ntt + (size_t)b * a_outer + (size_t)j * N;
    const u64 *cbase = c0 + (size_t)b * a_outer + (size_t)j * N;
    const u64 *dbase = dt + (size_t)b * pl->dt_count * N;
    const size_t kpoly = (size_t)ne * N;
    u64 r0[EL], r1[EL];
    pdl_wait();
    if (m.fp) { // products reduced one by one, signed double sums (up to 18 of them)
        const double qd = (double)m.q;
        double d0[EL], d1[EL];
#pragma unroll
        for (int u = 0; u < EL; ++u) { d0[u] = 0.0; d1[u] = 0.0; }
        for (int r = 0; r < mr.count; ++r) {
            u32 src[EL];
#pragma unroll
            for (int u = 0; u < EL; ++u) src[u] = ntt_perm(x0 + u * blockDim.x, mr.g[r], logn);
            const double *kbase = reinterpret_cast<const double *>(mr.mkey[r]) + (size_t)j * N + x0;
            for (int dg = 0; dg < nd; ++dg) {
                const int en = pl->dt_entry[dg][j];
                const u64 *sp = en < 0 ? abase : dbase + (size_t)en * N;
                const double *k0 = kbase + (size_t)dg * 2 * kpoly;
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    const double vd = u52_to_double(sp[src[u]]);
                    d0[u] = __dadd_rn(d0[u], mul_fp64_lazy(vd, k0[u * blockDim.x], m.q_inv_f, qd));
                    d1[u] = __dadd_rn(d1[u], mul_fp64_lazy(vd, k0[kpoly + u * blockDim.x], m.q_inv_f, qd));
                }
            }
            if (j < n) {
                const double *pmb = reinterpret_cast<const double *>(mr.pm[r]) + (size_t)j * N + x0;
#pragma unroll
                for (int u = 0; u < EL; ++u) d0[u] = __dadd_rn(d0[u], mul_fp64_lazy(u52_to_double(cbase[src[u]]), pmb[u * blockDim.x], m.q_inv_f, qd));
            }
        }
#pragma unroll
        for (int u = 0; u < EL; ++u) { r0[u] = canon_fp64(d0[u], m.q_inv_f, qd); r1[u] = canon_fp64(d1[u], m.q_inv_f, qd); }
    } else {
        PieceAcc s0[EL], s1[EL];
#pragma unroll
        for (int u = 0; u < EL; ++u) { s0[u].zero(); s1[u].zero(); }
        int held = 0; // products in the accumulators
        for (int r = 0; r < mr.count; ++r) {
            u32 src[EL];
#pragma unroll
            for (int u = 0; u < EL; ++u) src[u] = ntt_perm(x0 + u * blockDim.x, mr.g[r], logn);
            const u64 *kbase = mr.mkey[r] + (size_t)j * N + x0;
            for (int dg = 0; dg < nd; ++dg) {
                if (++held >= 8) {
                    held = 1;
#pragma unroll
                    for (int u = 0; u < EL; ++u) { s0[u].relax(m); s1[u].relax(m); }
                }
                const int en = pl->dt_entry[dg][j];
                const u64 *sp = en < 0 ? abase : dbase + (size_t)en * N;
                const u64 *k0 = kbase + (size_t)dg * 2 * kpoly;
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    const u64 v = sp[src[u]], ka = k0[u * blockDim.x], kb = k0[kpoly + u * blockDim.x];
                    const u32 v0 = (u32)v & 0x3FFFFFFFu, v1 = (u32)(v >> 30);
                    s0[u].mac(v0, v1, (u32)ka, (u32)(ka >> 32));
                    s1[u].mac(v0, v1, (u32)kb, (u32)(kb >> 32));
                }
            }
            if (j < n) {
                const u64 *pmb = mr.pm[r] + (size_t)j * N + x0;
#pragma unroll
                for (int u = 0; u < EL; ++u) {
                    const u64 v = cbase[src[u]], k = pmb[u * blockDim.x];
                    s0[u].mac((u32)v & 0x3FFFFFFFu, (u32)(v >> 30), (u32)k, (u32)(k >> 32));
                }
                ++held;
            }
        }
#pragma unroll
        for (int u = 0; u < EL; ++u) { r0[u] = s0[u].finish(m); r1[u] = s1[u].finish(m); }
    }
    u64 *o0 = E + (((size_t)ob * 2) * ne + j) * N + x0, *o1 = o0 + (size_t)ne * N;
#pragma unroll
    for (int u = 0; u < EL; ++u) { o0[u * blockDim.x] = r0[u]; o1[u * blockDim.x] = r1[u]; }
}
// At most two digits: a thread keeps the words of the one or two masked keys for its coefficient in registers and walks over `per`
// input members with the next member's words in flight.  Up to eleven masked-key words meet six words per member and coefficient;
// staging both in shared memory by bulk copies for three members at a time took 1.6 times as long (they crossed L2 for every
// third member, and a CTA's copies, sums and stores did not overlap).  Two coefficients per thread and two CTAs per SM: 869 us a launch
// for 168 outputs at level 6; one coefficient and three CTAs 837 us, four CTAs 776 us (64 registers), 712 with the
// products and additions of the 60-bit limbs apart: their integer chains want warps more than they want independent work in a thread (each of these with the program
// of its day; now, with two rotations an output, 824, with one 703).  With joined products
// 65 % of the issue slots and 52 % of the wide multiply-adds for 64 outputs (367 us), DRAM 3.1 TB/s; in a third of the cycles it waits for loads.
// grid = (N/256, groups * ceil(batch/per), ne)
template <int ND, int CNT>
__device__ __forceinline__ void ks_inner_mkr_body(u64 *o, const u64 *c0, const u64 *a_ntt, size_t a_outer, const u64 *dt, const MaskedRot &mr, int b0, int b1, const DigitPlan &pl,
                                                  const PrimeConst &m, int j, u32 x0, int logn, int N) {
    constexpr int EL = 1;
    const int ne = pl.ne;
    const bool has_c0 = j < pl.n;
    const size_t kpoly = (size_t)ne * N;
    u32 src[CNT][EL];
#pragma unroll
    for (int r = 0; r < CNT; ++r)
#pragma unroll
        for (int u = 0; u < EL; ++u) src[r][u] = ntt_perm(x0 + u * 256, mr.g[r], logn);
    const u64 *sp[ND];
    size_t stride[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int en = pl.entry[d][j];
        stride[d] = en < 0 ? a_outer : (size_t)pl.dt_count * N;
        sp[d] = (en < 0 ? a_ntt + (size_t)j * N : dt + (size_t)en * N) + (size_t)b0 * stride[d];
    }
    const u64 *cp = c0 + (size_t)b0 * a_outer + (size_t)j * N;
    u64 cur[CNT][ND][EL], cc[CNT][EL], k[CNT][ND][2][EL], pm[CNT][EL];
#pragma unroll
    for (int r = 0; r < CNT; ++r)
#pragma unroll
        for (int u = 0; u < EL; ++u) {
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                cur[r][d][u] = sp[d][src[r][u]];
                k[r][d][0][u] = mr.mkey[r][(size_t)(d * 2) * kpoly + (size_t)j * N + x0 + u * 256];
                k[r][d][1][u] = mr.mkey[r][(size_t)(d * 2 + 1) * kpoly + (size_t)j * N + x0 + u * 256];
            }
            cc[r][u] = has_c0 ? cp[src[r][u]] : 0;
            pm[r][u] = has_c0 ? mr.pm[r][(size_t)j * N + x0 + u * 256] : 0;
        }
    const double qd = (double)m.q;
    for (int b = b0; b < b1; ++b) {
        u64 v[CNT][ND][EL], w[CNT][EL];
        cp += a_outer;
#pragma unroll
        for (int d = 0; d < ND; ++d) sp[d] += stride[d];
#pragma unroll
        for (int r = 0; r < CNT; ++r)
#pragma unroll
            for (int u = 0; u < EL; ++u) {
#pragma unroll
                for (int d = 0; d < ND; ++d) { v[r][d][u] = cur[r][d][u]; if (b + 1 < b1) cur[r][d][u] = sp[d][src[r][u]]; }
                w[r][u] = cc[r][u];
                if (has_c0 && b + 1 < b1) cc[r][u] = cp[src[r][u]];
            }
        if (m.fp) {
#pragma unroll
            for (int u = 0; u < EL; ++u) {
                FpAcc s0, s1;
#pragma unroll
                for (int r = 0; r < CNT; ++r) {
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const double x = u52_to_double(v[r][d][u]), k0 = __longlong_as_double((long long)k[r][d][0][u]), k1 = __longlong_as_double((long long)k[r][d][1][u]);
                        if (r == 0 && d == 0) { s0.first(x, k0); s1.first(x, k1); }
                        else { s0.mac(x, k0); s1.mac(x, k1); }
                    }
                    if (has_c0) s0.mac(u52_to_double(w[r][u]), __longlong_as_double((long long)pm[r][u]));
                }
                o[u * 256] = s0.finish(m.q_inv_f, qd);
                o[kpoly + u * 256] = s1.finish(m.q_inv_f, qd);
            }
        } else {
#pragma unroll
            for (int u = 0; u < EL; ++u) {
                PieceAccT<true> s0, s1; s0.zero(); s1.zero(); // at most six products
#pragma unroll
                for (int r = 0; r < CNT; ++r) {
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const u32 v0 = (u32)v[r][d][u] & 0x3FFFFFFFu, v1 = (u32)(v[r][d][u] >> 30);
                        s0.mac(v0, v1, (u32)k[r][d][0][u], (u32)(k[r][d][0][u] >> 32));
                        s1.mac(v0, v1, (u32)k[r][d][1][u], (u32)(k[r][d][1][u] >> 32));
                    }
                    if (has_c0) s0.mac((u32)w[r][u] & 0x3FFFFFFFu, (u32)(w[r][u] >> 30), (u32)pm[r][u], (u32)(pm[r][u] >> 32));
                }
                o[u * 256] = s0.finish(m);
                o[kpoly + u * 256] = s1.finish(m);
            }
        }
        o += 2 * kpoly;
    }
}
template <int ND>
__global__ void __launch_bounds__(256, 4) k_ks_inner_mkr(u64 *E, const u64 *c0, const u64 *a_ntt, size_t a_outer, const u64 *dt, const __grid_constant__ MaskedRotList mrl, int batch, int per,
                                                         const __grid_constant__ DigitPlan pl, const PrimeConst *__restrict__ pc, int logn, int N) {
    const int chunks = (batch + per - 1) / per, grp = blockIdx.y / chunks, b0 = (blockIdx.y % chunks) * per, b1 = min(batch, b0 + per);
    const int j = blockIdx.z; // limb-major block order: the digits of one limb stay in L2 across the copies
    const MaskedRot &mr = mrl.r[grp];
    const PrimeConst m = pc[pl.prime[j]];
    const u32 x0 = blockIdx.x * (256 * 1) + threadIdx.x;
    u64 *o = E + (((size_t)(grp * batch + b0) * 2) * pl.ne + j) * N + x0;
    pdl_wait();
    if (mr.count == 1) ks_inner_mkr_body<ND, 1>(o, c0, a_ntt, a_outer, dt, mr, b0, b1, pl, m, j, x0, logn, N);
    else ks_inner_mkr_body<ND, 2>(o, c0, a_ntt, a_outer, dt, mr, b0, b1, pl, m, j, x0, logn, N);
}
// Base conversion of the division: src [bp][ns][N] (limbs q_level, P; coefficient form) -> t [bp][level][N]
// grid = (N/256, 1, nbp)
template <int NS>
__device__ __forceinline__ void div_conv_body(u64 *__restrict__ t, const u64 *__restrict__ src, const DivPlan *__restrict__ dv, const PrimeConst *__restrict__ pc, int N, int i, int bp) {
    const int nl = dv->level;
    u64 y[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const u64 v = src[((size_t)bp * NS + k) * N + i];
        y[k] = mul_shoup(v, dv->hat_inv[k], dv->hat_inv_sh[k], pc[dv->src_prime[k]].q);
    }
    u64 *o = t + (size_t)bp * nl * N + i;
    // targets below 2^44: y = y1 * 2^30 + y0 with both pieces as doubles, products on the FP64 pipe against the constants
    // (D / d_s) and (D / d_s) * 2^30 mod q: sixteen exact products of at most 0.51 q each, one canonicalisation
    double y0[NS], y1[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        y0[k] = __hiloint2double(0x43300000, (int)((u32)y[k] & 0x3FFFFFFFu)) - kTwo52;
        y1[k] = __hiloint2double(0x43300000, (int)(u32)(y[k] >> 30)) - kTwo52;
    }
    for (int l = 0; l < nl; ++l) {
        if (pc[l].fp) {
            const double qinv = pc[l].q_inv_f, qd = (double)pc[l].q;
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                acc = __dadd_rn(acc, mul_fp64_lazy(y0[k], __longlong_as_double((long long)dv->hat_mod_d0[k][l]), qinv, qd));
                acc = __dadd_rn(acc, mul_fp64_lazy(y1[k], __longlong_as_double((long long)dv->hat_mod_d1[k][l]), qinv, qd));
            }
            *o = canon_fp64(acc, qinv, qd);
        } else {
            PieceAcc s; s.zero();
#pragma unroll
            for (int k = 0; k < NS; ++k) s.mac(y[k], dv->hat_mod[k][l]);
            *o = s.finish(pc[l]);
        }
        o += N;
    }
}
__global__ void k_div_conv(u64 *__restrict__ t, const u64 *__restrict__ src, const DivPlan *__restrict__ dv, const PrimeConst *__restrict__ pc, int N) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int bp = blockIdx.z;
    switch (dv->ns) {
    case 2: div_conv_body<2>(t, src, dv, pc, N, i, bp); break;
    case 3: div_conv_body<3>(t, src, dv, pc, N, i, bp); break;
    case 4: div_conv_body<4>(t, src, dv, pc, N, i, bp); break;
    case 5: div_conv_body<5>(t, src, dv, pc, N, i, bp); break;
    case 6: div_conv_body<6>(t, src, dv, pc, N, i, bp); break;
    case 7: div_conv_body<7>(t, src, dv, pc, N, i, bp); break;
    default: div_conv_body<8>(t, src, dv, pc, N, i, bp); break;
    }
}
// out[bp][l][i] = (E[bp][l][i] - t[bp][l][i]) * D^-1 for l < level.  grid = (N/(256*kElems), level, batch*2)
__global__ void k_div_fin(u64 *__restrict__ out, const u64 *__restrict__ E, const u64 *__restrict__ t, int ne, const DivPlan *__restrict__ dv,
                          const PrimeConst *__restrict__ pc, int N) {
    const int l = blockIdx.y, bp = blockIdx.z, nl = dv->level;
    const PrimeConst m = pc[l];
    const u64 dinv = dv->d_inv[l];
#pragma unroll
    for (int u_ = 0; u_ < kElems; ++u_) {
        const int i = (blockIdx.x * kElems + u_) * blockDim.x + threadIdx.x;
        if (i >= N) break;
        const u64 v = sub_mod(E[((size_t)bp * ne + l) * N + i], t[((size_t)bp * nl + l) * N + i], m.q);
        out[((size_t)bp * nl + l) * N + i] = mul_mod_any(v, dinv, m);
    }
}

// ---------------- fused plaintext-matmul accumulate ----------------
// out_t[p][l][i] = sum_{b < bcount} sum_{k < kcount} pre[k * btotal + b0 + b][p][l][i] * pt_tb[l][perm_{g_k}(i)]
// (scale Delta^2, no rescale) for T output tiles t that share the shifted copies, which are stored k-major; the sum over b adds the
// partial products of several K-groups in the same pass.  A thread works on one coefficient of both polynomials: a copy word is
// read once for T tiles and a weight word once (and converted or cut once) for two polynomials.  Both come through a ring of kAccRing stages
// in shared memory that every thread fills for itself (cp.async), so a dozen loads of each of its 16 warps per SM are in flight without
// registers for them.  Four tiles, words loaded to registers one or two terms ahead: 675 us a launch in the layer pass, 611 in the Q/K/V
// projections; then 380 and 305.  Nothing is fetched past the last term, in a loop of its own: with the last word fetched again into every
// stage one copy and one tile took 15.7 us (12.1 before there was a ring), now 12.3; 128 copies of two inputs and four tiles 580, now 566.
// These issue in 66 % of the slots with sixteen warps per SM, DRAM 35 %, FP64 34 %.
// grid = (N/256, n)
template <int T> struct TilePts { const u64 *p[T][16]; u64 *out[T]; };
constexpr int kAccRing = 8;
constexpr size_t acc_smem(int T) { return (size_t)kAccRing * (2 + T) * 256 * 8; }
template <int T>
__global__ void __launch_bounds__(256, 2) k_matmul_acc(const __grid_constant__ TilePts<T> tp, const u64 *__restrict__ pre, int kcount, int btotal, int b0, int bcount, const u32 *__restrict__ gal,
                                                       int n, const __grid_constant__ LimbMap map, const PrimeConst *__restrict__ pc, int logn, int N) {
    extern __shared__ __align__(16) u64 words[]; // [kAccRing][2 + T][256]
    constexpr int kStage = (2 + T) * 256;
    const int l = blockIdx.y;
    const PrimeConst m = pc[map.prime[l]];
    const size_t poly = (size_t)n * N, limb = (size_t)l * N;
    const u32 x0 = blockIdx.x * 256 + threadIdx.x;
    const u64 *ring = words + threadIdx.x;
    const u32 ring_at = smem_u32(ring);
    // what is fetched next: copy fk of input fb, and the weights' words that meet it (nothing past the end, where the stages stay empty)
    const int total = kcount * bcount;
    int fk = 0, fb = 0;
    u32 to = 0, g = __ldg(gal), src = g == 1 ? x0 : ntt_perm(x0, g, logn);
    const u64 *fa = pre + (size_t)b0 * 2 * poly + limb + x0;
    const size_t to_next_copy = (size_t)(btotal - bcount + 1) * 2 * poly;
    auto fetch = [&] {
        const u32 r = ring_at + to;
        cp_async8(r, fa); cp_async8(r + 2048, fa + poly);
#pragma unroll
        for (int t = 0; t < T; ++t) cp_async8(r + (2 + t) * 2048, tp.p[t][fb] + limb + src);
        cp_async_commit();
        if (++fb < bcount) fa += 2 * poly;
        else if (fk + 1 < kcount) {
            fb = 0; ++fk; fa += to_next_copy;
            g = __ldg(gal + fk);
            src = g == 1 ? x0 : ntt_perm(x0, g, logn);
        }
        to += kStage * 8;
        if (to == kAccRing * kStage * 8) to = 0; // a stage is no power of two
    };
#pragma unroll 1
    for (int k = 0; k < kAccRing - 1; ++k) {
        if (k < total) fetch();
        else cp_async_commit();
    }
    u64 r[T][2];
    auto terms = [&](auto &&product) {
        int from = 0;
        auto term = [&](auto &&then) {
            cp_async_wait<kAccRing - 2>();
            const u64 *q = ring + from;
            u64 v[2] = {q[0], q[256]}, w[T];
#pragma unroll
            for (int t = 0; t < T; ++t) w[t] = q[(2 + t) * 256];
            from += kStage;
            if (from == kAccRing * kStage) from = 0;
            then();
            product(v, w);
        };
        const int fetching = max(0, total - (kAccRing - 1));
#pragma unroll 2
        for (int k = 0; k < fetching; ++k) term(fetch);
#pragma unroll 1
        for (int k = fetching; k < total; ++k) term([] { cp_async_commit(); });
    };
    if (m.fp) { // exact sums (see FpAcc): 128 products of primes below 2^42, eight below 2^44, before they are reduced
        const double qd = (double)m.q;
        const int room = m.q < (1ull << 42) ? 128 : 8;
        FpAcc s[T][2];
        int held = 0;
#pragma unroll
        for (int t = 0; t < T; ++t) { s[t][0].zero(); s[t][1].zero(); }
        terms([&](const u64 (&v)[2], const u64 (&w)[T]) {
            if (++held > room) {
                held = 1;
#pragma unroll
                for (int t = 0; t < T; ++t) { s[t][0].relax(m.q_inv_f, qd); s[t][1].relax(m.q_inv_f, qd); }
            }
            const double v0 = u52_to_double(v[0]), v1 = u52_to_double(v[1]);
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const double wd = u52_to_double(w[t]);
                s[t][0].mac(v0, wd);
                s[t][1].mac(v1, wd);
            }
        });
#pragma unroll
        for (int t = 0; t < T; ++t) { r[t][0] = s[t][0].finish(m.q_inv_f, qd); r[t][1] = s[t][1].finish(m.q_inv_f, qd); }
    } else {
        PieceAcc s[T][2];
        int held = 0; // products in the accumulators
#pragma unroll
        for (int t = 0; t < T; ++t) { s[t][0].zero(); s[t][1].zero(); }
        terms([&](const u64 (&v)[2], const u64 (&w)[T]) {
            if (++held > 8) {
                held = 1;
#pragma unroll
                for (int t = 0; t < T; ++t) { s[t][0].relax(m); s[t][1].relax(m); }
            }
#pragma unroll
            for (int t = 0; t < T; ++t) {
                s[t][0].mac(v[0], w[t]);
                s[t][1].mac(v[1], w[t]);
            }
        });
#pragma unroll
        for (int t = 0; t < T; ++t) { r[t][0] = s[t][0].finish(m); r[t][1] = s[t][1].finish(m); }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
        u64 *o = tp.out[t] + limb + x0;
        o[0] = r[t][0]; o[poly] = r[t][1];
    }
}

} // namespace hb
