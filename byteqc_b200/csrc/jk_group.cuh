// Group-per-quartet J/K kernel of the larger shell-quartet classes.
#pragma once
#include "jk_common.cuh"

namespace bqc {

// Shared-memory traffic bounds it: the table loads of the products, the
// density blocks and the reductions.  A thread therefore owns as many
// components as its registers hold (at most ACC_MAX = 60): the rows of the 2D
// tables and the density values it loads serve TJ fj at once, and fewer
// threads meet in the reductions.  Against one (fi, fj) and at most 36
// components a thread, one build of (H2O)_11 / cc-pVTZ on B200: (fd|dp)
// 2.67 -> 1.70 ms, (fd|fp) 1.30 -> 0.72 ms, (ff|fp) 1.05 -> 0.38 ms, (fp|pp)
// 2.41 -> 1.71 ms, (dp|dp) 3.30 -> 2.71 ms, (fp|dp) 2.66 -> 2.34 ms; the (fd|
// and (ff| classes gain most, whose ket components had been dealt to two or
// three threads that loaded all three factors of every product.
//
// A quartet (LI LJ | LK LL) runs on TPQ threads; thread (fi, jc, chunk) owns
// the components (fi, fj, fk, fl) with fj in [jc TJ, (jc + 1) TJ), fk in its
// chunk and every fl.
template <int LI, int LJ, int LK, int LL, int TJ, int NSPLIT>
struct GroupCfg {
    static constexpr int NFI = ncart(LI), NFJ = ncart(LJ), NFK = ncart(LK), NFL = ncart(LL);
    static constexpr int NIJ = NFI * NFJ, NKL = NFK * NFL;
    static constexpr int NR = (LI + LJ + LK + LL) / 2 + 1;
    static constexpr int NJC = NFJ / TJ;
    static constexpr int TPQ = NFI * NJC * NSPLIT;
    static constexpr int GSZ = (LI + 1) * (LJ + 1) * (LK + 1) * (LL + 1);
    static constexpr int KLS = (LK + 1) * (LL + 1);
    // row stride of the 2D tables in shared memory, odd so that the rows
    // the threads of a group read start in different banks
    static constexpr int KLP = KLS | 1;
    static constexpr int GSZP = (LI + 1) * (LJ + 1) * KLP;
    static constexpr int CK = cdiv(NFK, NSPLIT);
    static constexpr int NCKL = CK * NFL;          // ket components of a thread
    static constexpr int NACC = TJ * NCKL;
    static constexpr int GBUF = 3 * NR * GSZP;
    // K_ik and K_il: complete in one thread when it owns every fj and fk
    static constexpr bool OWN_I = NJC == 1 && NSPLIT == 1;
    // reduction slots: K_jk, K_jl over fi (odd stride for the reads), K_ik and
    // K_il over jc and chunk, J_kl over the threads of one chunk
    static constexpr int FIP = NFI | 1;
    static constexpr int S_JK = 0, S_JL = S_JK + NFJ * NFK * FIP, S_IK = S_JL + NFJ * NFL * NSPLIT * FIP;
    static constexpr int S_IL = S_IK + (OWN_I ? 0 : NFI * NFK * NJC);
    static constexpr int KSLOTS = S_IL + (OWN_I ? 0 : NFI * NFL * NJC * NSPLIT);
    static constexpr int NTH = NFI * NJC, THP = NTH | 1;
    static constexpr int JSLOTS = NKL * THP;
    // J_kl in the same pass as K where its slots fit behind, else in
    // blocks of FKB rows fk
    static constexpr bool ONE_PASS = KSLOTS + JSLOTS <= GBUF;
    static constexpr int RB = imax(GBUF, imax(KSLOTS, NFL * THP));
    static constexpr int FKB = ONE_PASS ? NFK : imin(NFK, RB / (NFL * THP));
    static constexpr int DBUF = NIJ + NKL + NFI * NFK + NFI * NFL + NFJ * NFK + NFJ * NFL;
    static constexpr int RW = 2 * NR;
    // doubles per group, odd so that neighbouring groups start in different banks
    static constexpr int PER_GROUP = (RB + DBUF + RW) | 1;
    // groups per CTA: up to 128 threads and a third of an SM's shared memory
    // (small CTAs let the barrier-separated phases of different CTAs overlap
    // on an SM), the count that fills its warps best
    static constexpr int NT_CAP = 128;
    static constexpr int SMEM_BUDGET = 72 * 1024;
    static constexpr int NG_CAP = imax(1, imin(NT_CAP / TPQ, SMEM_BUDGET / (PER_GROUP * 8)));
    static constexpr int pick_ng() {
        int best = 1;
        for (int n = 1; n <= NG_CAP; n++)
            if ((long long)n * TPQ * (cdiv(best * TPQ, 32)) >= (long long)best * TPQ * cdiv(n * TPQ, 32)) best = n;
        return best;
    }
    static constexpr int NG = pick_ng();
    static constexpr int NT = cdiv(NG * TPQ, 32) * 32;
    static constexpr size_t SMEM = (size_t)NG * PER_GROUP * sizeof(double);
    // CTAs per SM the register budget is sized for
    static constexpr int REGS = NACC <= 20 ? 128 : (NACC <= 36 ? 168 : 240);
    static constexpr int MB_SMEM = (int)(227 * 1024 / (SMEM + 2304));
    static constexpr int MB_REGS = 65536 / (NT * REGS);
    static constexpr int MINB = imax(1, imin(MB_SMEM, MB_REGS));
};

template <int LI, int LJ, int LK, int LL, int TJ, int NSPLIT, typename F>
__global__ void __launch_bounds__(GroupCfg<LI, LJ, LK, LL, TJ, NSPLIT>::NT,
                                  GroupCfg<LI, LJ, LK, LL, TJ, NSPLIT>::MINB)
jk_group(JKArgs A, JKTask T) {
    using C = GroupCfg<LI, LJ, LK, LL, TJ, NSPLIT>;
    constexpr int NFI = C::NFI, NFJ = C::NFJ, NFK = C::NFK, NFL = C::NFL;
    constexpr int NR = C::NR, TPQ = C::TPQ, NG = C::NG, CK = C::CK, NJC = C::NJC;
    constexpr int NCKL = C::NCKL, GSZP = C::GSZP, KLP = C::KLP, KLS = C::KLS;
    extern __shared__ double smem[];
    __shared__ int s_list[TILE * TILE];
    __shared__ int s_count;

    const int g = threadIdx.x / TPQ;
    const int lane = threadIdx.x % TPQ;
    const bool in_group = g < NG;
    double *gbuf = smem + (in_group ? g : 0) * C::PER_GROUP;   // RB: 2D tables / reduction slots
    double *dbuf = gbuf + C::RB;                                // density blocks
    double *rw = dbuf + C::DBUF;                                // roots, weights
    F *gtab = reinterpret_cast<F *>(gbuf);
    double *Dij = dbuf, *Dkl = Dij + C::NIJ, *Dik = Dkl + C::NKL, *Dil = Dik + NFI * NFK;
    double *Djk = Dil + NFI * NFL, *Djl = Djk + NFJ * NFK;

    const int chunk = lane % NSPLIT, jc = lane / NSPLIT % NJC, fi = lane / (NSPLIT * NJC);
    const int fj0 = jc * TJ, fk0 = chunk * CK;
    int pw[3] = {0, 0, 0};
#pragma unroll
    for (int c = 0; c < NFI; c++)
        if (c == fi) { pw[0] = cart_pow(LI, c, 0); pw[1] = cart_pow(LI, c, 1); pw[2] = cart_pow(LI, c, 2); }
    // table rows of (fi, fj): the first direction's offset of fj is a constant
    // when the thread owns every fj
    int row[3][TJ];
#pragma unroll
    for (int t = 0; t < TJ; t++) {
        int pj[3] = {cart_pow(LJ, t, 0), cart_pow(LJ, t, 1), cart_pow(LJ, t, 2)};
        if constexpr (NJC > 1) {
#pragma unroll
            for (int c = 0; c < NFJ; c++)
                if (c == fj0 + t) { pj[0] = cart_pow(LJ, c, 0); pj[1] = cart_pow(LJ, c, 1); pj[2] = cart_pow(LJ, c, 2); }
        }
#pragma unroll
        for (int d = 0; d < 3; d++) row[d][t] = (d * NR * (LI + 1) * (LJ + 1) + pw[d] * (LJ + 1) + pj[d]) * KLP;
    }

    auto tile = [&](const long long x, const int part, const int nparts) {
    JKSub s;
    int a_begin, b_begin, count, kpart;
    if (!tile_screen(A, T, x, s, s_list, &s_count, a_begin, b_begin, count, kpart, part, nparts)) return;
    // primitive quartets of this part
    const PrimRange pr = prim_range(s, kpart);

    const int nrounds = (count + NG - 1) / NG;
    for (int round = 0; round < nrounds; round++) {
        const int item = round * NG + g;
        const bool active = in_group && item < count;
        Pair bra, ket;
        int pa = 0, pb = 0;
        double fac = TWO_PI_2P5;
        if (active) {
            const int e = s_list[item], a = a_begin + (e >> 16), b = b_begin + (e & 0xffff);
            load_pair(A, a, bra);
            load_pair(A, b, ket);
            if (a == b && A.eri == nullptr) fac *= 0.5;
            pa = s.pa0 + (a - s.a0) * s.nprim_a;
            pb = s.pb0 + (b - s.b0) * s.nprim_b;
        }
        F acc[TJ][NCKL];
#pragma unroll
        for (int t = 0; t < TJ; t++)
#pragma unroll
            for (int n = 0; n < NCKL; n++) acc[t][n] = F(0);
        // The six density blocks of this quartet, lane-strided over the group
        // into dbuf (which the 2D tables do not touch); the first density's
        // copies run while the integrals are evaluated.
        auto stage = [&](const double *__restrict__ D) {
            for (int e = lane; e < C::DBUF; e += TPQ) {
                int r0 = 0, c0 = 0, nc = 1, o = e;
                if (o < C::NIJ) { r0 = bra.i0; c0 = bra.j0; nc = NFJ; }
                else if ((o -= C::NIJ) < C::NKL) { r0 = ket.i0; c0 = ket.j0; nc = NFL; }
                else if ((o -= C::NKL) < NFI * NFK) { r0 = bra.i0; c0 = ket.i0; nc = NFK; }
                else if ((o -= NFI * NFK) < NFI * NFL) { r0 = bra.i0; c0 = ket.j0; nc = NFL; }
                else if ((o -= NFI * NFL) < NFJ * NFK) { r0 = bra.j0; c0 = ket.i0; nc = NFK; }
                else { o -= NFJ * NFK; r0 = bra.j0; c0 = ket.j0; nc = NFL; }
                cp_async8(dbuf + e, D + (size_t)(r0 + o / nc) * A.nao + c0 + o % nc);
            }
            cp_async_commit();
        };
        if (active && A.eri == nullptr) stage(A.dm);

        int kp = pr.k, ip = pr.i;
        for (int left = pr.num; left > 0; left--) {
            PrimQuartet P;
            if (active) {
                PrimPair pi, pk;
                load_prim(A, pa + ip, pi);
                load_prim(A, pb + kp, pk);
                if (++ip == s.nprim_a) { ip = 0; kp++; }
                prim_quartet(pi, pk, bra.A, ket.A, fac, P);
                for (int f = lane; f < 2 * NR; f += TPQ) rw[f] = rys_one<NR>(A.rys, P.x, f);
            }
            __syncthreads();
            if (active) {
                for (int task = lane; task < 3 * NR; task += TPQ) {
                    int r = task / 3, d = task % 3;
                    RootCoef c = root_coef(rw[r], P);
                    double seed = (d == 2) ? rw[NR + r] * P.pref : 1.0;
                    // d is a runtime index, so P and the centres sit in local memory
                    // (L1): measured faster than selecting from registers
                    gen_2d<LI, LJ, LK, LL, F, KLP>(
                        F(seed), F(P.PA[d] - c.qs * P.PQ[d]), F(P.QC[d] + c.ps * P.PQ[d]),
                        F(c.b00), F(c.b10), F(c.b01), F(bra.AB[d]), F(ket.AB[d]),
                        gtab + (d * NR + r) * GSZP);
                }
            }
            __syncthreads();
            if (active) {
#pragma unroll 1
                for (int r = 0; r < NR; r++) {
                    const F *gr = gtab + r * GSZP;
#pragma unroll
                    for (int t = 0; t < TJ; t++) {
                        const F *gx = gr + row[0][t], *gy = gr + row[1][t], *gz = gr + row[2][t];
                        if constexpr (NSPLIT == 1) {
                            F xs[KLS], ys[KLS], zs[KLS];
#pragma unroll
                            for (int u = 0; u < KLS; u++) {
                                xs[u] = gx[u];
                                ys[u] = gy[u];
                                zs[u] = gz[u];
                            }
#pragma unroll
                            for (int fk = 0; fk < NFK; fk++)
#pragma unroll
                            for (int fl = 0; fl < NFL; fl++) {
                                int ux = cart_pow(LK, fk, 0) * (LL + 1) + cart_pow(LL, fl, 0);
                                int uy = cart_pow(LK, fk, 1) * (LL + 1) + cart_pow(LL, fl, 1);
                                int uz = cart_pow(LK, fk, 2) * (LL + 1) + cart_pow(LL, fl, 2);
                                acc[t][fk * NFL + fl] = fma(xs[ux] * ys[uy], zs[uz], acc[t][fk * NFL + fl]);
                            }
                        } else {
#pragma unroll
                            for (int ck = 0; ck < CK; ck++) {
                                const int fk = fk0 + ck;
                                if (fk < NFK) {
                                    int kx = 0, ky = 0, kz = 0;
#pragma unroll
                                    for (int c = 0; c < NFK; c++)
                                        if (c == fk) { kx = cart_pow(LK, c, 0); ky = cart_pow(LK, c, 1); kz = cart_pow(LK, c, 2); }
                                    const F *rx = gx + kx * (LL + 1);
                                    const F *ry = gy + ky * (LL + 1);
                                    const F *rz = gz + kz * (LL + 1);
#pragma unroll
                                    for (int fl = 0; fl < NFL; fl++)
                                        acc[t][ck * NFL + fl] = fma(rx[cart_pow(LL, fl, 0)] * ry[cart_pow(LL, fl, 1)],
                                                                    rz[cart_pow(LL, fl, 2)], acc[t][ck * NFL + fl]);
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();
        }

        if (A.eri != nullptr) {
            // ERI output mode: add this thread's components, no digestion
            if (active) {
                const long long s0 = A.eri_stride[0], s1 = A.eri_stride[1], s2 = A.eri_stride[2],
                                s3 = A.eri_stride[3];
                double *base = A.eri + (bra.i0 + fi - A.eri_off[0]) * s0 + (bra.j0 + fj0 - A.eri_off[1]) * s1 +
                               (ket.i0 + fk0 - A.eri_off[2]) * s2 + (ket.j0 - A.eri_off[3]) * s3;
#pragma unroll
                for (int t = 0; t < TJ; t++)
#pragma unroll
                    for (int n = 0; n < NCKL; n++)
                        if (NSPLIT == 1 || fk0 + n / NFL < NFK)
                            atomicAdd(base + t * s1 + n / NFL * s2 + n % NFL * s3, (double)acc[t][n]);
            }
            continue;
        }

        // ---- digestion ----
        const int nao = A.nao;
        const size_t nn = (size_t)nao * nao;
        const size_t kr = T.k_transposed ? 1 : nao, kc = T.k_transposed ? nao : 1;   // K strides: bra, ket
        auto have = [&](int ck) { return NSPLIT == 1 || fk0 + ck < NFK; };
        double *Sj = gbuf + (C::ONE_PASS ? C::KSLOTS : 0);   // J_kl: [fk - first][fl][thread]
        const int th = fi * NJC + jc;
        for (int id = 0; id < A.n_dm; id++) {
            double *VJ = A.vj + id * nn, *VK = A.vk + id * nn;
            if (id > 0 && active) stage(A.dm + id * nn);
            cp_async_wait_all();
            __syncthreads();
            // this thread's J_kl contributions of rows fk in [first, first + FKB)
            auto put_j = [&](int first) {
                double d[TJ];
#pragma unroll
                for (int t = 0; t < TJ; t++) d[t] = Dij[fi * NFJ + fj0 + t];
#pragma unroll
                for (int n = 0; n < NCKL; n++) {
                    const int fk = fk0 + n / NFL;
                    if (have(n / NFL) && (C::FKB >= NFK || (fk >= first && fk < first + C::FKB))) {
                        double v = 0;
#pragma unroll
                        for (int t = 0; t < TJ; t++) v = fma((double)acc[t][n], d[t], v);
                        Sj[((fk - first) * NFL + n % NFL) * C::THP + th] = v;
                    }
                }
            };
            auto take_j = [&](int first) {
                const int nk = min(C::FKB, NFK - first);
                for (int o = lane; o < nk * NFL; o += TPQ) {
                    double v = 0;
#pragma unroll
                    for (int t = 0; t < C::NTH; t++) v += Sj[o * C::THP + t];
                    atomicAdd(VJ + (size_t)(ket.i0 + first + o / NFL) * nao + ket.j0 + o % NFL, v);
                }
            };
            if (active) {
                if (A.vj != nullptr) {
                    double v[TJ];
#pragma unroll
                    for (int t = 0; t < TJ; t++) v[t] = 0;
#pragma unroll
                    for (int n = 0; n < NCKL; n++) {
                        if (have(n / NFL)) {
                            const double d = Dkl[fk0 * NFL + n];
#pragma unroll
                            for (int t = 0; t < TJ; t++) v[t] = fma((double)acc[t][n], d, v[t]);
                        }
                    }
#pragma unroll
                    for (int t = 0; t < TJ; t++)
                        atomicAdd(VJ + (size_t)(bra.i0 + fi) * nao + bra.j0 + fj0 + t, v[t]);
                    if constexpr (C::ONE_PASS) put_j(0);
                }
                if (A.vk != nullptr) {
                    // K_ik and K_jk, one fk at a time
#pragma unroll
                    for (int ck = 0; ck < CK; ck++) {
                        if (have(ck)) {
                            const int fk = fk0 + ck;
                            double sik = 0;
#pragma unroll
                            for (int t = 0; t < TJ; t++) {
                                double sjk = 0;
#pragma unroll
                                for (int fl = 0; fl < NFL; fl++) {
                                    sik = fma((double)acc[t][ck * NFL + fl], Djl[(fj0 + t) * NFL + fl], sik);
                                    sjk = fma((double)acc[t][ck * NFL + fl], Dil[fi * NFL + fl], sjk);
                                }
                                gbuf[C::S_JK + ((fj0 + t) * NFK + fk) * C::FIP + fi] = sjk;
                            }
                            if constexpr (C::OWN_I)
                                atomicAdd(VK + (bra.i0 + fi) * kr + (ket.i0 + fk) * kc, sik);
                            else
                                gbuf[C::S_IK + (fi * NFK + fk) * NJC + jc] = sik;
                        }
                    }
                    // K_il and K_jl
                    double sil[NFL];
#pragma unroll
                    for (int fl = 0; fl < NFL; fl++) sil[fl] = 0;
#pragma unroll
                    for (int t = 0; t < TJ; t++) {
                        double sjl[NFL];
#pragma unroll
                        for (int fl = 0; fl < NFL; fl++) sjl[fl] = 0;
#pragma unroll
                        for (int ck = 0; ck < CK; ck++) {
                            if (have(ck)) {
                                const double djk = Djk[(fj0 + t) * NFK + fk0 + ck], dik = Dik[fi * NFK + fk0 + ck];
#pragma unroll
                                for (int fl = 0; fl < NFL; fl++) {
                                    sil[fl] = fma((double)acc[t][ck * NFL + fl], djk, sil[fl]);
                                    sjl[fl] = fma((double)acc[t][ck * NFL + fl], dik, sjl[fl]);
                                }
                            }
                        }
#pragma unroll
                        for (int fl = 0; fl < NFL; fl++)
                            gbuf[C::S_JL + (((fj0 + t) * NFL + fl) * NSPLIT + chunk) * C::FIP + fi] = sjl[fl];
                    }
#pragma unroll
                    for (int fl = 0; fl < NFL; fl++) {
                        if constexpr (C::OWN_I)
                            atomicAdd(VK + (bra.i0 + fi) * kr + (ket.j0 + fl) * kc, sil[fl]);
                        else
                            gbuf[C::S_IL + (fi * NFL + fl) * NJC * NSPLIT + jc * NSPLIT + chunk] = sil[fl];
                    }
                }
            }
            __syncthreads();
            if (active) {
                if (A.vk != nullptr) {
                    constexpr int O1 = NFJ * NFK, O2 = O1 + NFJ * NFL, O3 = O2 + (C::OWN_I ? 0 : NFI * NFK),
                                  O4 = O3 + (C::OWN_I ? 0 : NFI * NFL);
                    for (int o = lane; o < O4; o += TPQ) {
                        double v = 0;
                        size_t dst;
                        if (o < O1) {
#pragma unroll
                            for (int i = 0; i < NFI; i++) v += gbuf[C::S_JK + o * C::FIP + i];
                            dst = (bra.j0 + o / NFK) * kr + (ket.i0 + o % NFK) * kc;
                        } else if (o < O2) {
                            const int e = o - O1;
#pragma unroll
                            for (int h = 0; h < NSPLIT; h++)
#pragma unroll
                                for (int i = 0; i < NFI; i++) v += gbuf[C::S_JL + (e * NSPLIT + h) * C::FIP + i];
                            dst = (bra.j0 + e / NFL) * kr + (ket.j0 + e % NFL) * kc;
                        } else if (o < O3) {
                            const int e = o - O2;
#pragma unroll
                            for (int j = 0; j < NJC; j++) v += gbuf[C::S_IK + e * NJC + j];
                            dst = (bra.i0 + e / NFK) * kr + (ket.i0 + e % NFK) * kc;
                        } else {
                            const int e = o - O3;
#pragma unroll
                            for (int j = 0; j < NJC * NSPLIT; j++) v += gbuf[C::S_IL + e * NJC * NSPLIT + j];
                            dst = (bra.i0 + e / NFL) * kr + (ket.j0 + e % NFL) * kc;
                        }
                        atomicAdd(VK + dst, v);
                    }
                }
                if constexpr (C::ONE_PASS) {
                    if (A.vj != nullptr) take_j(0);
                }
            }
            __syncthreads();
            if constexpr (!C::ONE_PASS) {
                if (A.vj != nullptr) {
                    for (int first = 0; first < NFK; first += C::FKB) {
                        if (active) put_j(first);
                        __syncthreads();
                        if (active) take_j(first);
                        __syncthreads();
                    }
                }
            }
        }
    }
    };
    // virtual block vb = part vb % S of tile vb / S
    int S;
    long long nvb;
    if (T.ntiles_dev == nullptr) {
        S = T.split;
        nvb = T.ntiles * S;
    } else {
        const long long n = __ldg(T.ntiles_dev);
        S = group_split(n, T.nsm);
        nvb = n * S;
    }
    for (long long vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
        tile(vb / S, (int)(vb % S), S);
        __syncthreads();
    }
}

template <int LI, int LJ, int LK, int LL, int TJ, int NSPLIT, typename F>
static int launch_group_f(const JKArgs &args, const JKTask &task, cudaStream_t stream) {
    using C = GroupCfg<LI, LJ, LK, LL, TJ, NSPLIT>;
    static_assert(C::SMEM + 2304 <= 227 * 1024, "shared memory per CTA");
    static_assert(C::NT <= 1024, "threads per CTA");
    static_assert(C::NJC * TJ == C::NFJ, "bra components per thread");
    JKTask t = task;
    t.ntiles = task_tiles(task);
    if (t.ntiles == 0) return 0;
    if (smem_attr<jk_group<LI, LJ, LK, LL, TJ, NSPLIT, F>>((int)C::SMEM)) return 1;
    if (t.nsm <= 0 && (t.nsm = device_sms()) <= 0) return 1;
    if (t.ntiles_dev == nullptr) t.split = group_split(t.ntiles, t.nsm);
    // with a device tile count the kernel cuts tiles into at most 8 parts
    const int grid = t.ntiles_dev == nullptr ? bqc_grid(t, t.ntiles, t.split, 0) : bqc_grid(t, t.ntiles, 8, 8);
    launch_at(jk_group<LI, LJ, LK, LL, TJ, NSPLIT, F>, grid, C::NT, C::SMEM, stream, args, t);
    return 0;
}

template <int LI, int LJ, int LK, int LL, int TJ, int NSPLIT>
static int launch_group(const JKArgs &args, const JKTask &task, int fp32, cudaStream_t stream) {
    if (fp32) return launch_group_f<LI, LJ, LK, LL, TJ, NSPLIT, float>(args, task, stream);
    return launch_group_f<LI, LJ, LK, LL, TJ, NSPLIT, double>(args, task, stream);
}

// Components of one thread, for the bra (LI LJ) on the thread side: as many
// fj as keep the accumulators within ACC_MAX, a divisor of NFJ; a ket above
// that is cut into chunks of fk.
constexpr int ACC_MAX = 60;
struct GroupShape {
    int tj, nsplit, cost;
};
constexpr GroupShape group_shape(int li, int lj, int lk, int ll) {
    const int nfj = ncart(lj), nkl = ncart(lk) * ncart(ll), kls = (lk + 1) * (ll + 1);
    GroupShape g = {1, 1, 0};
    if (nkl > ACC_MAX) {
        g.nsplit = imin(cdiv(nkl, ACC_MAX), ncart(lk));
        g.cost = 3000;   // every product loads its three factors
        return g;
    }
    for (int t = 1; t <= nfj; t++)
        if (nfj % t == 0 && t * nkl <= ACC_MAX) g.tj = t;
    // table loads per 1000 components: all rows of j when the thread owns every
    // fj, else three rows per fj
    const int rows = g.tj == nfj && lj > 0 ? 3 * (lj + 1) : 3 * g.tj;
    g.cost = 1000 * rows * kls / (g.tj * nkl);
    return g;
}

}  // namespace bqc
