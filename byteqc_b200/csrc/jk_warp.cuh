// One thread per quartet: J/K kernel of the shell-quartet classes of at most
// SMALL_NF Cartesian components, and, as launches over ranges of the
// components of shell k, of the classes that split into a few such ranges.
//
// A warp takes a 16 x 16 tile: a lane holds one ket pair and steps over the
// bra pairs, two a step (one per half warp).  What a lane needs of its ket
// pair is read once a tile, what belongs to a bra pair is the same address for
// 16 lanes, and only D_jl, its bound and the atomic on K_jl are per quartet;
// the 128-thread half tiles that this replaces read all of it per quartet
// (77 % of the L1 wavefront peak for (ps|ss)) and met at block barriers.
// Measured on B200 against those: one build of (H2O)_32 / cc-pVDZ, (ps|ss) 18.7 ->
// 13.7 ms, (ss|ss) 10.3 -> 6.6 ms, (ps|ps) 11.6 -> 8.6 ms, (ds|ds) 1.10 -> 0.71 ms, (dp|ps)
// 4.1 -> 3.7 ms, (ds|pp) 2.3 -> 2.1 ms; C60H122 / 6-31G**, FP32 band, (ps|ss) 37.7 -> 30.3
// ms, (dp|pp) 8.4 -> 7.3 ms, but (ds|pp) 5.8 -> 5.9 ms and (dp|ps) 10.7 -> 11.0 ms.  What
// bounds it now is latency: 0.43 instructions a cycle and scheduler at 16 warps an SM.
#pragma once
#include "jk_common.cuh"

namespace bqc {

constexpr int WARP_CTA = 128;              // threads of a CTA: four independent warps
constexpr int WARPS = WARP_CTA / 32;
constexpr int ROW_STEPS = TILE / 2;        // steps of a warp over a tile, two bra pairs each

// Sum v over the 16 lanes of each half warp.  Step BIT exchanges half of the
// vector with the lane at distance BIT, so a lane ends up with the sums of
// the elements [off, off + cnt) only (cnt <= ceil(V / 16)): V exchanges in
// all instead of four per element.
template <int V, int BIT>
__device__ __forceinline__ void halve(double *v, int lane, int &off, int &cnt) {
    if constexpr (BIT > 0) {
        const bool up = lane & BIT;
        if constexpr (V == 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], BIT);
            if (up) cnt = 0;
            halve<1, BIT / 2>(v, lane, off, cnt);
        } else {
            constexpr int H = (V + 1) / 2;
#pragma unroll
            for (int n = 0; n < H; n++) {
                const double hi = n + H < V ? v[n + H < V ? n + H : 0] : 0.;
                const double x = __shfl_xor_sync(0xffffffffu, up ? v[n] : hi, BIT);
                v[n] = (up ? hi : v[n]) + x;
            }
            off += up ? H : 0;
            cnt = up ? max(cnt - H, 0) : min(cnt, H);
            halve<H, BIT / 2>(v, lane, off, cnt);
        }
    }
}

// of two numbers that are not NaN (the density maxima never are)
__device__ __forceinline__ double larger(double a, double b) { return a > b ? a : b; }

template <int V, typename Emit>
__device__ __forceinline__ void half_warp_sum(double (&v)[V], int lane, Emit emit) {
    int off = 0, cnt = V;
    halve<V, 8>(v, lane, off, cnt);
#pragma unroll
    for (int n = 0; n < cdiv(V, 16); n++)
        if (n < cnt && v[n] != 0) emit(off + n, v[n]);
}

constexpr int LARGE_NF = 54;   // blocks of so many components fill the registers

template <int LI, int LJ, int LK, int LL, int KN>
struct WarpCfg {
    static constexpr int NFI = ncart(LI), NFJ = ncart(LJ), NFK = KN, NFL = ncart(LL);
    static constexpr int NF = NFI * NFJ * NFK * NFL;
    // sums carried over the bra pairs of a tile: J_kl, K_il, K_ik
    static constexpr int PERS = NFK * NFL + NFI * NFL + NFI * NFK;
    // sums over a half warp: J_ij, K_jk
    static constexpr int RED = NFI * NFJ + NFJ * NFK;
    // in registers beside the quartet block where both fit (64 doubles are half
    // of the largest register budget), else in shared memory, one column per
    // lane, which no other lane touches
    static constexpr bool SMEM_SUMS = NF + PERS > 64;
    static constexpr int SMEM = SMEM_SUMS ? PERS * WARP_CTA * (int)sizeof(double) : 0;
    // CTAs per SM of the register budget: 64, 128, 168 and 255 registers.  One
    // build of (H2O)_32 / cc-pVDZ and of C60H122 / 6-31G** on B200: (ss|ss), whose
    // block is one double, 8.0 and 9.2 ms at 96 registers, 6.7 and 7.3 ms at 64
    // in spite of some spills; (ps|ss) 14.2 and 17.6 ms at 128, 16.5 and 21.7
    // ms at 80; (ps|ps) 8.8 and 11.2 ms at 168, 9.3 and 11.5 ms at 128; (dp|ps)
    // 4.2 and 7.2 ms at 255, 6.3 and 11.3 ms at 168.
    static constexpr int MINB = NF == 1 ? 8 : (NF <= 3 ? 4 : (NF <= 9 ? 3 : 2));
};

template <int LI, int LJ, int LK, int LL, typename F, int K0 = 0, int KN = ncart(LK)>
__global__ void __launch_bounds__(WARP_CTA, WarpCfg<LI, LJ, LK, LL, KN>::MINB)
jk_warp(JKArgs A, JKTask T) {
    static_assert(K0 >= 0 && KN >= 1 && K0 + KN <= ncart(LK), "ket component range");
    using C = WarpCfg<LI, LJ, LK, LL, KN>;
    constexpr int NFI = C::NFI, NFJ = C::NFJ, NFK = C::NFK, NFL = C::NFL;
    constexpr int NIJ = NFI * NFJ, NKL = NFK * NFL, NF = NIJ * NKL;
    constexpr int NR = (LI + LJ + LK + LL) / 2 + 1;
    constexpr int GSZ = (LI + 1) * (LJ + 1) * (LK + 1) * (LL + 1);
    // roots one after another where unrolling them would make the code long
    constexpr int UNROLL_ROOTS = NR * NF <= 60 ? NR : 1;
    // A large FP32 block is digested one fi at a time, so that few converted
    // components (9 of the 54) are live beside it: 36 bytes of spill stores instead of 612 for
    // (dp|ps); C60H122 / 6-31G**, FP32 band, (dp|pp) 8.2 -> 7.4 ms, (dp|ds) 5.2 -> 4.6
    // ms.  In FP64, where nothing is converted, and for smaller blocks the other
    // order is the better one: (dp|ps) 4.0 against 4.8 ms, (ds|ps) 4.3 against 4.8 ms
    // of a build of (H2O)_32 / cc-pVDZ.
    constexpr bool SLICES = sizeof(F) == 4 && NF >= LARGE_NF && NFJ * NKL <= 9;
    constexpr int S_KL = 0, S_IL = NKL, S_IK = NKL + NFI * NFL;   // slots of the carried sums
    extern __shared__ double s_sum[];
    const int lane = threadIdx.x & 31, half = lane >> 4, col = lane & 15;
    const int nao = A.nao;
    const size_t nn = (size_t)nao * nao;
    const int kr = T.k_transposed ? 1 : nao, kc = T.k_transposed ? nao : 1;   // K strides: bra, ket

    double r_sum[C::SMEM_SUMS ? 1 : C::PERS] = {};
    auto sum_add = [&](int n, double v) {
        if constexpr (C::SMEM_SUMS) s_sum[n * WARP_CTA + threadIdx.x] += v; else r_sum[n] += v;
    };
    auto sum_clear = [&](int n) {
        if constexpr (C::SMEM_SUMS) s_sum[n * WARP_CTA + threadIdx.x] = 0.; else r_sum[n] = 0.;
    };
    auto sum_take = [&](int n) -> double {   // and clear
        double v;
        if constexpr (C::SMEM_SUMS) v = s_sum[n * WARP_CTA + threadIdx.x]; else v = r_sum[n];
        sum_clear(n);
        return v;
    };

    auto tile = [&](const long long x, int part, int nparts) {
        JKSub s;
        int r, c, kpart;
        tile_of_block(T, x, s, r, c, part, nparts, kpart);
        const int ta = s.rows_are_b ? c : r, tb = s.rows_are_b ? r : c;
        const int a_begin = s.a0 + ta * TILE, b_begin = s.b0 + tb * TILE;
        const int a_end = min(s.a0 + s.na, a_begin + TILE), b_end = min(s.b0 + s.nb, b_begin + TILE);
        if (s.diag && b_begin > a_end - 1) return;

        // the ket pair of this lane (the tile's first pair where it has none)
        const bool col_ok = b_begin + col < b_end;
        const int b = col_ok ? b_begin + col : b_begin;
        Pair ket;
        load_pair(A, b, ket);
        const int ksh = ket.i, lsh = ket.j, k0 = ket.i0 + K0, l0 = ket.j0;
        const bool ket_uni = __all_sync(0xffffffffu, ksh == __shfl_sync(0xffffffffu, ksh, 0));
        const double qb = A.pair_q != nullptr ? __ldg(A.pair_q + b) : 0.;
        const double ckl = A.dm_cond != nullptr ? __ldg(A.dm_cond + (size_t)ksh * A.nbas + lsh) : 0.;
        const int pb = s.pb0 + (b - s.b0) * s.nprim_b;
        const F CD[3] = {F(ket.AB[0]), F(ket.AB[1]), F(ket.AB[2])};

#pragma unroll
        for (int n = 0; n < C::PERS; n++) sum_clear(n);
        const bool one = A.n_dm == 1;

        // row steps of this part
        const int steps = max(ROW_STEPS / nparts, 1);
        const int it_end = min((part + 1) * steps, ROW_STEPS);
        // primitive quartets of this part, bra pairs innermost
        const PrimRange pr = prim_range(s, kpart);
        bool pending = false;                // the carried sums hold contributions
        auto bra_pair = [&](int it) { return min(a_begin + 2 * it + half, a_end - 1); };
        int a = bra_pair(part * steps);
        Pair bra;
        load_pair(A, a, bra);
        bool new_i = true;                   // shell i differs from the last step's
        double ci_max = 0.;                  // max |D| over (kl), (ik), (il)
        for (int it = part * steps; it < it_end; it++) {
            const bool row_ok = a_begin + 2 * it + half < a_end;
            const int ish = bra.i, jsh = bra.j, i0 = bra.i0, j0 = bra.j0;
            if (new_i && A.dm_cond != nullptr) {
                const double *ci = A.dm_cond + (size_t)ish * A.nbas;
                ci_max = larger(ckl, larger(__ldg(ci + ksh), __ldg(ci + lsh)));
            }
            bool active = row_ok && col_ok && (!s.diag || a >= b);
            if (A.pair_q != nullptr) {
                double bound = __ldg(A.pair_q + a) * qb;
                if (A.dm_cond != nullptr) {
                    const double *cj = A.dm_cond + (size_t)jsh * A.nbas;
                    bound *= larger(larger(ci_max, __ldg(A.dm_cond + (size_t)ish * A.nbas + jsh)),
                                    larger(__ldg(cj + ksh), __ldg(cj + lsh)));
                }
                active = active && bound >= A.tol && (A.tol_hi <= 0. || bound < A.tol_hi);
            }
            const bool any = __any_sync(0xffffffffu, active);

            // every lane evaluates its quartet, one that is screened out with a
            // factor of zero: no divergent region around the integrals
            F acc[NF];
            if (any) {
#pragma unroll
                for (int n = 0; n < NF; n++) acc[n] = F(0);
                const F AB[3] = {F(bra.AB[0]), F(bra.AB[1]), F(bra.AB[2])};
                const double fac = !active ? 0. : (a == b && A.eri == nullptr) ? 0.5 * TWO_PI_2P5 : TWO_PI_2P5;
                const int pa = s.pa0 + (a - s.a0) * s.nprim_a;
                int kp = pr.k, ip = pr.i;
                PrimPair pk;
                load_prim(A, pb + kp, pk);
                for (int left = pr.num; left > 0; left--) {
                    PrimPair pi;
                    load_prim(A, pa + ip, pi);
                    PrimQuartet P;
                    prim_quartet(pi, pk, bra.A, ket.A, fac, P);
                    if (++ip == s.nprim_a) {
                        ip = 0;
                        if (left > 1) load_prim(A, pb + ++kp, pk);
                    }
                    double rt[NR], wt[NR];
                    rys_roots<NR>(A.rys_lm, P.x, rt, wt);
#pragma unroll UNROLL_ROOTS
                    for (int rr = 0; rr < NR; rr++) {
                        RootCoef cf = root_coef(rt[rr], P);
                        F g[3][GSZ];
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            F seed = (d == 2) ? F(wt[rr] * P.pref) : F(1);
                            gen_2d<LI, LJ, LK, LL, F>(seed, F(P.PA[d] - cf.qs * P.PQ[d]),
                                                      F(P.QC[d] + cf.ps * P.PQ[d]), F(cf.b00),
                                                      F(cf.b10), F(cf.b01), AB[d], CD[d], g[d]);
                        }
#pragma unroll
                        for (int fi = 0; fi < NFI; fi++)
#pragma unroll
                        for (int fj = 0; fj < NFJ; fj++)
#pragma unroll
                        for (int fk = 0; fk < NFK; fk++)
#pragma unroll
                        for (int fl = 0; fl < NFL; fl++) {
                            constexpr int SJ = (LK + 1) * (LL + 1), SI = (LJ + 1) * SJ;
                            const int ix = cart_pow(LI, fi, 0) * SI + cart_pow(LJ, fj, 0) * SJ +
                                           cart_pow(LK, K0 + fk, 0) * (LL + 1) + cart_pow(LL, fl, 0);
                            const int iy = cart_pow(LI, fi, 1) * SI + cart_pow(LJ, fj, 1) * SJ +
                                           cart_pow(LK, K0 + fk, 1) * (LL + 1) + cart_pow(LL, fl, 1);
                            const int iz = cart_pow(LI, fi, 2) * SI + cart_pow(LJ, fj, 2) * SJ +
                                           cart_pow(LK, K0 + fk, 2) * (LL + 1) + cart_pow(LL, fl, 2);
                            acc[((fi * NFJ + fj) * NFK + fk) * NFL + fl] += g[0][ix] * g[1][iy] * g[2][iz];
                        }
                    }
                }
            }

            if (A.eri != nullptr) {
                // ERI output mode: add the block, no digestion
                if (active) {
                    const long long s0 = A.eri_stride[0], s1 = A.eri_stride[1], s2 = A.eri_stride[2],
                                    s3 = A.eri_stride[3];
                    double *base = A.eri + (i0 - A.eri_off[0]) * s0 + (j0 - A.eri_off[1]) * s1 +
                                   (k0 - A.eri_off[2]) * s2 + (l0 - A.eri_off[3]) * s3;
#pragma unroll
                    for (int n = 0; n < NF; n++)
                        atomicAdd(base + n / (NFJ * NKL) * s0 + n / NKL % NFJ * s1 + n / NFL % NFK * s2 +
                                      n % NFL * s3, (double)acc[n]);
                }
                a = bra_pair(it + 1);
                load_pair(A, a, bra);
                new_i = true;
                continue;
            }

            // the next bra pair: the sums over pairs that share shell i end
            // where i changes, all sums with the last step
            a = bra_pair(it + 1);
            load_pair(A, a, bra);
            const bool last = it + 1 == it_end;
            const bool end_i = last || __any_sync(0xffffffffu, ish != bra.i);
            pending |= any;

            // ---- digestion ----
#define ACC(fi, fj, fk, fl) ((double)acc[(((fi) * NFJ + (fj)) * NFK + (fk)) * NFL + (fl)])
            for (int id = 0; pending && id < A.n_dm; id++) {
                const double *__restrict__ D = A.dm + id * nn;
                double *VJ = A.vj + id * nn, *VK = A.vk + id * nn;
                if (any) {
                    // J_ij and K_jk: summed over the lanes of a half warp
                    double v[NIJ + NFJ * NFK];
#pragma unroll
                    for (int n = 0; n < NIJ + NFJ * NFK; n++) v[n] = 0.;
                    // a lane that is screened out touches no density: it may hold anything
                    if (active) {
                        // rows of the density: an element is one address step from its row
                        const double *Di[NFI], *Dj[NFJ], *Dk[NFK];
#pragma unroll
                        for (int n = 0; n < NFI; n++) Di[n] = D + (long long)(i0 + n) * nao;
#pragma unroll
                        for (int n = 0; n < NFJ; n++) Dj[n] = D + (long long)(j0 + n) * nao;
#pragma unroll
                        for (int n = 0; n < NFK; n++) Dk[n] = D + (long long)(k0 + n) * nao;
                        if constexpr (SLICES) {
                            double d_kl[NKL], d_jl[NFJ * NFL], d_jk[NFJ * NFK];
                            double jkl[NKL], pjl[NFJ * NFL];
#pragma unroll
                            for (int n = 0; n < NKL; n++) {
                                d_kl[n] = A.vj != nullptr ? __ldg(Dk[n / NFL] + l0 + n % NFL) : 0.;
                                jkl[n] = 0.;
                            }
#pragma unroll
                            for (int n = 0; n < NFJ * NFL; n++) {
                                d_jl[n] = A.vk != nullptr ? __ldg(Dj[n / NFL] + l0 + n % NFL) : 0.;
                                pjl[n] = 0.;
                            }
#pragma unroll
                            for (int n = 0; n < NFJ * NFK; n++)
                                d_jk[n] = A.vk != nullptr ? __ldg(Dj[n / NFK] + k0 + n % NFK) : 0.;
                            // one fi at a time
#pragma unroll
                            for (int fi = 0; fi < NFI; fi++) {
                                double e[NFJ * NKL];
#pragma unroll
                                for (int n = 0; n < NFJ * NKL; n++) e[n] = (double)acc[fi * NFJ * NKL + n];
                                if (A.vj != nullptr) {
#pragma unroll
                                    for (int fj = 0; fj < NFJ; fj++) {
                                        const double d_ij = __ldg(Di[fi] + j0 + fj);
#pragma unroll
                                        for (int kl = 0; kl < NKL; kl++) {
                                            v[fi * NFJ + fj] += e[fj * NKL + kl] * d_kl[kl];
                                            jkl[kl] += e[fj * NKL + kl] * d_ij;
                                        }
                                    }
                                }
                                if (A.vk != nullptr) {
#pragma unroll
                                    for (int fl = 0; fl < NFL; fl++) {
                                        const double d_il = __ldg(Di[fi] + l0 + fl);
                                        double t = 0.;   // K_il
#pragma unroll
                                        for (int fj = 0; fj < NFJ; fj++)
#pragma unroll
                                            for (int fk = 0; fk < NFK; fk++) {
                                                v[NIJ + fj * NFK + fk] += e[(fj * NFK + fk) * NFL + fl] * d_il;
                                                t += e[(fj * NFK + fk) * NFL + fl] * d_jk[fj * NFK + fk];
                                            }
                                        sum_add(S_IL + fi * NFL + fl, t);
                                    }
#pragma unroll
                                    for (int fk = 0; fk < NFK; fk++) {
                                        const double d_ik = __ldg(Di[fi] + k0 + fk);
                                        double t = 0.;   // K_ik
#pragma unroll
                                        for (int fj = 0; fj < NFJ; fj++)
#pragma unroll
                                            for (int fl = 0; fl < NFL; fl++) {
                                                pjl[fj * NFL + fl] += e[(fj * NFK + fk) * NFL + fl] * d_ik;
                                                t += e[(fj * NFK + fk) * NFL + fl] * d_jl[fj * NFL + fl];
                                            }
                                        sum_add(S_IK + fi * NFK + fk, t);
                                    }
                                }
                            }
                            if (A.vj != nullptr) {
#pragma unroll
                                for (int n = 0; n < NKL; n++) sum_add(S_KL + n, jkl[n]);
                            }
                            if (A.vk != nullptr) {
                                // K_jl: one target per quartet
#pragma unroll
                                for (int n = 0; n < NFJ * NFL; n++)
                                    atomicAdd(VK + (long long)(j0 + n / NFL) * kr + (long long)(l0 + n % NFL) * kc, pjl[n]);
                            }
                        } else {
                            if (A.vj != nullptr) {
#pragma unroll
                                for (int kl = 0; kl < NKL; kl++) {
                                    const double d = __ldg(Dk[kl / NFL] + l0 + kl % NFL);
#pragma unroll
                                    for (int ij = 0; ij < NIJ; ij++) v[ij] += (double)acc[ij * NKL + kl] * d;
                                }
                                // J_kl
                                double d_ij[NIJ];
#pragma unroll
                                for (int n = 0; n < NIJ; n++) d_ij[n] = __ldg(Di[n / NFJ] + j0 + n % NFJ);
#pragma unroll
                                for (int kl = 0; kl < NKL; kl++) {
                                    double t = 0.;
#pragma unroll
                                    for (int ij = 0; ij < NIJ; ij++) t += (double)acc[ij * NKL + kl] * d_ij[ij];
                                    sum_add(S_KL + kl, t);
                                }
                            }
                            if (A.vk != nullptr) {
                                // K_jk
#pragma unroll
                                for (int fi = 0; fi < NFI; fi++)
#pragma unroll
                                    for (int fl = 0; fl < NFL; fl++) {
                                        const double d = __ldg(Di[fi] + l0 + fl);
#pragma unroll
                                        for (int fj = 0; fj < NFJ; fj++)
#pragma unroll
                                            for (int fk = 0; fk < NFK; fk++)
                                                v[NIJ + fj * NFK + fk] += ACC(fi, fj, fk, fl) * d;
                                    }
                                // K_jl: one target per quartet
                                double pjl[NFJ * NFL];
#pragma unroll
                                for (int n = 0; n < NFJ * NFL; n++) pjl[n] = 0.;
#pragma unroll
                                for (int fi = 0; fi < NFI; fi++)
#pragma unroll
                                    for (int fk = 0; fk < NFK; fk++) {
                                        const double d = __ldg(Di[fi] + k0 + fk);
#pragma unroll
                                        for (int fj = 0; fj < NFJ; fj++)
#pragma unroll
                                            for (int fl = 0; fl < NFL; fl++) pjl[fj * NFL + fl] += ACC(fi, fj, fk, fl) * d;
                                    }
#pragma unroll
                                for (int n = 0; n < NFJ * NFL; n++)
                                    atomicAdd(VK + (long long)(j0 + n / NFL) * kr + (long long)(l0 + n % NFL) * kc, pjl[n]);
                                // K_ik
                                double d_jl[NFJ * NFL];
#pragma unroll
                                for (int n = 0; n < NFJ * NFL; n++) d_jl[n] = __ldg(Dj[n / NFL] + l0 + n % NFL);
#pragma unroll
                                for (int fi = 0; fi < NFI; fi++)
#pragma unroll
                                    for (int fk = 0; fk < NFK; fk++) {
                                        double t = 0.;
#pragma unroll
                                        for (int n = 0; n < NFJ * NFL; n++) t += ACC(fi, n / NFL, fk, n % NFL) * d_jl[n];
                                        sum_add(S_IK + fi * NFK + fk, t);
                                    }
                                // K_il
                                double d_jk[NFJ * NFK];
#pragma unroll
                                for (int n = 0; n < NFJ * NFK; n++) d_jk[n] = __ldg(Dj[n / NFK] + k0 + n % NFK);
#pragma unroll
                                for (int fi = 0; fi < NFI; fi++)
#pragma unroll
                                    for (int fl = 0; fl < NFL; fl++) {
                                        double t = 0.;
#pragma unroll
                                        for (int n = 0; n < NFJ * NFK; n++) t += ACC(fi, n / NFK, n % NFK, fl) * d_jk[n];
                                        sum_add(S_IL + fi * NFL + fl, t);
                                    }
                                }
                        }
                        if (A.vk != nullptr && !ket_uni) {
                            // no shell k shared by the lanes: K_jk one by one
#pragma unroll
                            for (int n = 0; n < NFJ * NFK; n++) {
                                atomicAdd(VK + (long long)(j0 + n / NFK) * kr + (long long)(k0 + n % NFK) * kc, v[NIJ + n]);
                                v[NIJ + n] = 0.;
                            }
                        }
                    }
                    half_warp_sum(v, lane, [&](int n, double y) {
                        double *dst = n < NIJ ? VJ + (size_t)(i0 + n / NFJ) * nao + j0 + n % NFJ
                                              : VK + (long long)(j0 + (n - NIJ) / NFK) * kr + (long long)(k0 + (n - NIJ) % NFK) * kc;
                        atomicAdd(dst, y);
                    });
                }
                if (one && !end_i) continue;
                if (A.vj != nullptr && (last || !one)) {
#pragma unroll
                    for (int n = 0; n < NKL; n++) {
                        double v = sum_take(S_KL + n);
                        v += __shfl_xor_sync(0xffffffffu, v, 16);
                        if (half == 0 && col_ok && v != 0)
                            atomicAdd(VJ + (size_t)(k0 + n / NFL) * nao + l0 + n % NFL, v);
                    }
                }
                if (A.vk != nullptr) {
                    // both halves of the warp at the same shell i: their sums together
                    const bool same = __all_sync(0xffffffffu, ish == __shfl_sync(0xffffffffu, ish, 0));
                    const bool mine = half == 0 || !same;
#pragma unroll
                    for (int n = 0; n < NFI * NFL; n++) {
                        double v = sum_take(S_IL + n);
                        if (same) v += __shfl_xor_sync(0xffffffffu, v, 16);
                        if (mine && v != 0) atomicAdd(VK + (long long)(i0 + n / NFL) * kr + (long long)(l0 + n % NFL) * kc, v);
                    }
                    double v[NFI * NFK];
#pragma unroll
                    for (int n = 0; n < NFI * NFK; n++) {
                        v[n] = sum_take(S_IK + n);
                        if (same) v[n] += __shfl_xor_sync(0xffffffffu, v[n], 16);
                        if (!ket_uni) {
                            if (mine && v[n] != 0) atomicAdd(VK + (long long)(i0 + n / NFK) * kr + (long long)(k0 + n % NFK) * kc, v[n]);
                            v[n] = 0.;
                        }
                    }
                    half_warp_sum(v, lane, [&](int n, double y) {
                        if (mine) atomicAdd(VK + (long long)(i0 + n / NFK) * kr + (long long)(k0 + n % NFK) * kc, y);
                    });
                }
            }
            if (end_i) pending = pending && !last && A.vj != nullptr;
#undef ACC
            new_i = end_i;
        }
    };

    // virtual tile vb = part vb % S of tile vb / S, one per warp
    long long nt;
    int S;
    if (T.ntiles_dev == nullptr) {
        nt = T.ntiles;
        S = T.split;
    } else {
        nt = __ldg(T.ntiles_dev);
        S = warp_split(nt, T.nsm);
    }
    const long long nvb = nt * S;
    const int lg = __ffs(S) - 1;
    for (long long vb = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5); vb < nvb;
         vb += (long long)gridDim.x * WARPS)
        tile(vb >> lg, (int)vb & (S - 1), S);   // S is a power of two
}

template <int LI, int LJ, int LK, int LL, typename F, int K0, int KN>
static int launch_warp_range(const JKArgs &args, const JKTask &task, cudaStream_t stream) {
    constexpr int cap = 4 * WarpCfg<LI, LJ, LK, LL, KN>::MINB;   // persistent CTAs per SM
    const int grid = task.ntiles_dev == nullptr
                         ? bqc_grid(task, (task.ntiles * task.split + WARPS - 1) / WARPS, 1, 0)
                         : bqc_grid(task, task.ntiles, ROW_STEPS / WARPS, cap);
    constexpr int smem = WarpCfg<LI, LJ, LK, LL, KN>::SMEM;
    if (smem > 48 * 1024 && smem_attr<jk_warp<LI, LJ, LK, LL, F, K0, KN>>(smem)) return 1;
    launch_at(jk_warp<LI, LJ, LK, LL, F, K0, KN>, grid, WARP_CTA, smem, stream, args, task);
    return 0;
}

// Launches over fk in [K0, K0 + CK), [K0 + CK, ...) until shell k is covered:
// every J/K target is linear in the quartet block, so they add up to the
// whole class.
template <int LI, int LJ, int LK, int LL, typename F, int K0, int CK>
static int launch_warp_f(const JKArgs &args, const JKTask &task, cudaStream_t stream) {
    constexpr int KN = imin(CK, ncart(LK) - K0);
    if (launch_warp_range<LI, LJ, LK, LL, F, K0, KN>(args, task, stream)) return 1;
    if constexpr (K0 + CK < ncart(LK))
        return launch_warp_f<LI, LJ, LK, LL, F, K0 + CK, CK>(args, task, stream);
    return 0;
}

template <int LI, int LJ, int LK, int LL, int CK, typename F>
static int launch_warp_t(const JKArgs &args, const JKTask &task, cudaStream_t stream) {
    JKTask t = task;
    t.ntiles = task_tiles(task);
    if (t.ntiles == 0) return 0;
    if (t.nsm <= 0 && (t.nsm = device_sms()) <= 0) return 1;
    if (t.ntiles_dev == nullptr) t.split = warp_split(t.ntiles, t.nsm);
    bqc_count_launch(cdiv(ncart(LK), CK) - 1);   // the dispatcher counted one
    return launch_warp_f<LI, LJ, LK, LL, F, 0, CK>(args, t, stream);
}

template <int LI, int LJ, int LK, int LL, int CK>
static int launch_warp(const JKArgs &args, const JKTask &task, int fp32, cudaStream_t stream) {
    if (fp32) return launch_warp_t<LI, LJ, LK, LL, CK, float>(args, task, stream);
    return launch_warp_t<LI, LJ, LK, LL, CK, double>(args, task, stream);
}

// A class of at most SMALL_NF components, in one of its two orientations.  The
// lanes hold the ket pairs and carry J_kl, K_il and K_ik over the bra pairs:
// the orientation that carries fewer sums.  From LARGE_NF components on the
// registers decide.  FP64: the one with fewer sums over the half warp, whose
// vector is live with the block: one build of (H2O)_32 / cc-pVDZ, (dp|ps) with 9 of
// them 3.6 ms, with 27 3.9 ms, (ds|pp) 2.2 and 2.4 ms.  Below, the carried sums
// cost more: (pp|ss) 5.1 ms with 4 of them and 15 carried, 4.6 ms with 12 and 7,
// (pp|ps) 6.1 and 5.6 ms.  FP32: the one with the smaller slices (jk_warp), 9
// components against 18: C60H122 / 6-31G**, FP32 band, with the whole block and with
// slices, (dp|ps) 12.1 -> 11.0 ms, (ds|pp) 6.6 -> 5.9 ms.
template <int L1, int L2, int L3, int L4, typename F>
static int launch_small_t(const JKArgs &args, const JKTask &task, cudaStream_t stream) {
    using C = WarpCfg<L1, L2, L3, L4, ncart(L3)>;
    using S = WarpCfg<L3, L4, L1, L2, ncart(L1)>;
    constexpr bool swap = C::NF < LARGE_NF      ? S::PERS < C::PERS
                          : sizeof(F) == 8      ? S::RED < C::RED
                                                : S::NFI > C::NFI;
    if constexpr (swap) {
        JKTask sw = jk_swap_task(task);
        sw.k_transposed = !sw.k_transposed;
        return launch_warp_t<L3, L4, L1, L2, ncart(L1), F>(jk_args_swap_eri(args), sw, stream);
    } else {
        return launch_warp_t<L1, L2, L3, L4, ncart(L3), F>(args, task, stream);
    }
}

template <int L1, int L2, int L3, int L4>
static int launch_small(const JKArgs &args, const JKTask &task, int fp32, cudaStream_t stream) {
    if (fp32) return launch_small_t<L1, L2, L3, L4, float>(args, task, stream);
    return launch_small_t<L1, L2, L3, L4, double>(args, task, stream);
}

}  // namespace bqc
