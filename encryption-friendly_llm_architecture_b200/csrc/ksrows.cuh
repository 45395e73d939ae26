// The middle of a key switch whose digits serve one rotation only, on 2^16 rings with LongPm primes (sm_100a): forward row pass of the lifted
// digits, inner products with the switching key and inverse row pass of the special limbs in one kernel.
//
//     inverse row pass -> conv_cols (lift) -> ks_rows -> conv_cols (ModDown) -> forward row pass with the last step
//
// An automorphism maps aligned blocks of the transformed order onto aligned blocks, so a CTA that owns two rows of outputs finds what it needs in
// two rows of every digit.  A warp per digit and member transforms them (or fetches them, where the limb is the digit's own) into shared
// memory; then all threads form the sums of their coefficients, gathering the digits' words from there.  The lifted limbs are read
// once and never written back, the special limbs of the result leave half transformed.
//
// Bound by instruction issue (48 members at level 8: 640 us, 56 % of the slots, DRAM 2.3 TB/s; the three kernels it replaces 310 + 286 + 86 at 3.5 to 5.3
// TB/s).  At 64 registers a thread spills 4 to 12 bytes.  Blocks of few warps, because their loads, transforms and sums alternate behind barriers: eight rows a CTA 4 to 7 % of a whole rotation
// slower, four 1 to 2 %.  Two members a CTA share the key words that each coefficient meets: 64 members at level 8 2671 -> 2603 us.  Limbs in the inner order,
// so that integer and FP64 work meet on an SM: 2729 us, twiddles and keys then come from L2 every time.
// Rotations with three kernels and with this one stand at the rule that chooses (one_kernel_switch).  256 products at level 8 14.2 / 13.9 ms.
#pragma once
#include "convcols.cuh"

namespace hb {

constexpr int kKsRows = 2;
constexpr size_t ks_rows_smem(int nd, int members) { return (size_t)members * nd * kKsRows * kRowStride * 8; }

// acc[ob][p][j] = sum_dg perm_g(digit_dg[j]) * key[dg][p][prime(j)], member ob = group * batch + b: canonical for the limbs of Q, half inverse for the
// special ones.  dt: half-forward digits as conv_cols leaves them.  ND digits (at least two), M members a CTA; grid = (256 / kKsRows, groups * ceil(batch / M), ne).
template <int ND, int M>
__global__ void __launch_bounds__(16 * kKsRows * ND * M, 1024 / (16 * kKsRows * ND * M)) ks_rows(u64 *acc, const __grid_constant__ SwitchList sl, int batch, size_t a_outer, int key_primes,
                                                                                              const KsPlan *__restrict__ pl, const PrimeConst *__restrict__ pc, Ntt16Tables tb) {
    using LONG = LongPm;
    static_assert(ND >= 2, "the two polynomials of the result take the places of two digits");
    constexpr int R = kKsRows, TM = ND; // tiles of a member
    constexpr int kTile = R * 256, kTileWords = R * kRowStride, kThreads = 16 * R * ND * M;
    extern __shared__ __align__(128) u64 tiles[];
    const int j = blockIdx.z, chunks = (batch + M - 1) / M, grp = blockIdx.y / chunks, b0 = blockIdx.y % chunks * M, tid = threadIdx.x;
    const SwitchGroup &sg = sl.s[grp];
    const u32 g = sg.g, i0 = blockIdx.x * kTile;
    const int pj = pl->ext_prime[j], ne = pl->ne;
    const PrimeConst m = pc[pj];
    const bool small = tb.small(pj);
    const u64 *key = sg.key + (size_t)pj * kN16 + i0;
    const size_t kpoly = (size_t)key_primes * kN16;
    if (b0 == 0 && tid < 2 * ND) prefetch_l2(key + tid * kpoly, kTile * 8);
    auto source = [&](u32 i) { return g ? ntt_perm(i, g, 16) : i; };
    const u32 s0 = source(i0) & ~(u32)(kTile - 1);
    const int clo = tid & 15, rl = (tid >> 4) & (R - 1), gr = tid / (16 * R); // group gr: digit gr % ND of member gr / ND
    {
        const int dg = gr % ND, mb = gr / ND, b = min(b0 + mb, batch - 1), en = pl->dt_entry[dg][j], row = s0 / 256 + rl;
        const u64 *p = (en < 0 ? sg.a_ntt + (size_t)b * a_outer + (size_t)j * kN16 : sg.dt + ((size_t)b * pl->dt_count + en) * kN16) + s0 + rl * 256 + clo;
        u64 *smr = tiles + (mb * TM + dg) * kTileWords + rl * kRowStride;
        const ulonglong2 *tab = tb.fwd + (size_t)pj * Ntt16Layout::kEntries;
        pdl_wait();
        if (en < 0) {
#pragma unroll
            for (int e = 0; e < 16; ++e) smr[e * 17 + clo] = key_word(p[e * 16], small);
        } else if (small) {
            const DsConst c = ds_const(m);
            double *smd = reinterpret_cast<double *>(smr);
            double v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = __longlong_as_double((long long)p[e * 16]);
            fwd16_ds(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smd[e * 17 + clo] = v[e];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = smd[clo * 17 + e];
            fwd16_ds8(v, TwiddlesB<double, false>(tb.fwdB8 + (size_t)pj * kRowsB8 + (row * 15) * 16 + clo), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smd[clo * 17 + e] = ds_reduce(v[e], c); // within 0.52 q of zero
        } else {
            const typename LONG::Const c = LONG::make(m);
            u64 v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = p[e * 16];
            LONG::template fwd16<2>(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smr[e * 17 + clo] = v[e];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = smr[clo * 17 + e];
            LONG::template fwd16<3>(v, TwiddlesB<ulonglong2, false>(tab + Ntt16Layout::rowsB(row, 0, clo)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = key_word(LONG::canon(v[e], c), false);
        }
    }
    auto at = [](u32 s) { return (s >> 8 & (R - 1)) * kRowStride + (s >> 4 & 15) * 17 + (s & 15); }; // where a tile holds coefficient s
    const bool special = j >= pl->n;
    u64 *o = acc + ((size_t)(grp * batch + b0) * 2 * ne + j) * kN16 + i0;
    constexpr int kAll = (kTile + kThreads - 1) / kThreads, EL = kAll <= 4 && ND * kAll <= 8 ? kAll : ND <= 2 ? 4 : ND == 3 ? 3 : 2;
    u64 k[ND][2][EL];
    auto keys = [&](int x0) {
#pragma unroll
        for (int u = 0; u < EL; ++u)
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
                for (int q = 0; q < 2; ++q) k[d][q][u] = __ldg(key + (size_t)(2 * d + q) * kpoly + min(x0 + u * kThreads, kTile - 1));
    };
    keys(tid);
    __syncthreads();
#pragma unroll 1
    for (int x0 = tid; x0 < kTile; x0 += EL * kThreads) {
        if (x0 >= kThreads) keys(x0);
#pragma unroll
        for (int u = 0; u < EL; ++u) {
            const int x = x0 + u * kThreads;
            if (x >= kTile) break;
            const u32 w = at(source(i0 + x));
#pragma unroll
            for (int mb = 0; mb < M; ++mb) {
                u64 r[2], *tile = tiles + mb * TM * kTileWords + w;
                if (small) {
                    const double qd = (double)m.q;
                    FpAcc s[2];
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const double v = __longlong_as_double((long long)tile[d * kTileWords]);
#pragma unroll
                        for (int q = 0; q < 2; ++q) { const double kd = u52_to_double(k[d][q][u]); if (d == 0) s[q].first(v, kd); else s[q].mac(v, kd); }
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) r[q] = s[q].finish(m.q_inv_f, qd);
                } else {
                    PieceAccT<true> s[2]; s[0].zero(); s[1].zero();
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const u64 v = tile[d * kTileWords];
#pragma unroll
                        for (int q = 0; q < 2; ++q) s[q].mac((u32)v, (u32)(v >> 32), (u32)k[d][q][u] & 0x3FFFFFFFu, (u32)(k[d][q][u] >> 30));
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) r[q] = s[q].finish(m);
                }
                if (special) { // where this thread alone has read
                    tile[0] = r[0];
                    tile[kTileWords] = r[1];
                } else if (b0 + mb < batch) {
                    o[(size_t)(2 * mb) * ne * kN16 + x] = r[0];
                    o[(size_t)(2 * mb + 1) * ne * kN16 + x] = r[1];
                }
            }
        }
    }
    if (!special) return;
    __syncthreads();
    // Inverse row pass, a group for each polynomial.  A row of outputs lies in one row of the tile, which its sixteen threads also exchange through.
    const ulonglong2 *tab = tb.inv + (size_t)pj * Ntt16Layout::kEntries;
    const int row = i0 / 256 + rl;
    const u32 first = i0 + rl * 256 + clo * 16;
#pragma unroll 1
    for (int q = gr; q < 2 * M; q += ND * M) {
        if (b0 + q / 2 >= batch) break;
        u64 *tile = tiles + (q / 2 * TM + q % 2) * kTileWords, *smr = tile + (source(i0 + rl * 256) >> 8 & (R - 1)) * kRowStride;
        u64 *op = o + (size_t)q * ne * kN16 + rl * 256 + clo;
        if (small) {
            const DsConst c = ds_const(m);
            double *smd = reinterpret_cast<double *>(smr);
            double v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = ds_load(tile[at(source(first + e))]);
            __syncwarp();
            inv16_ds8(v, TwiddlesB<double, false>(tb.invB8 + (size_t)pj * kRowsB8 + (row * 15) * 16 + clo), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smd[clo * 17 + e] = v[e];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = smd[e * 17 + clo];
            inv16_ds(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) reinterpret_cast<double *>(op)[e * 16] = v[e];
        } else {
            const typename LONG::Const c = LONG::make(m);
            u64 v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = tile[at(source(first + e))];
            __syncwarp();
            LONG::inv16(v, TwiddlesB<ulonglong2, false>(tab + Ntt16Layout::rowsB(row, 0, clo)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) smr[clo * 17 + e] = v[e];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = smr[e * 17 + clo];
            LONG::inv16(v, TwiddlesA(tab + Ntt16Layout::rowsA(row, 0)), c);
#pragma unroll
            for (int e = 0; e < 16; ++e) op[e * 16] = v[e];
        }
    }
}

} // namespace hb
