// Schwarz factors q_ij = sqrt(max over Cartesian components |(ij|ij)|) of
// every shell pair of one class, on the device.  The reference takes them
// from libcint on the CPU (cuobc/scf/hf.py:341, pyscf CVHFsetnr_direct_scf).
// One thread per pair; the loops over roots and directions are kept rolled
// (this is a one-time setup kernel, compact code matters more than speed).
//
// The factors order the pairs of every class, pairs that are equal by symmetry
// by their last bits, and the order of the pairs of one class decides which
// half of V holds a contribution (a >= b).  So this kernel evaluates its own
// primitive quantities and the Chebyshev series of the Rys rule, and a change of the J/K
// kernels' arithmetic does not reorder a molecule's pairs.
#include "jk_common.cuh"

namespace bqc {

struct Quartet {
    int a, b, ish, jsh, ksh, lsh, i0, j0, k0, l0;
    double A[3], B[3], C[3], D[3];
    double fac;
};

__device__ __forceinline__ void load_quartet(const JKArgs &A, int a, int b, Quartet &q) {
    q.a = a;
    q.b = b;
    q.ish = __ldg(A.pair_bra + a);
    q.jsh = __ldg(A.pair_ket + a);
    q.ksh = __ldg(A.pair_bra + b);
    q.lsh = __ldg(A.pair_ket + b);
    q.i0 = __ldg(A.ao_loc + q.ish);
    q.j0 = __ldg(A.ao_loc + q.jsh);
    q.k0 = __ldg(A.ao_loc + q.ksh);
    q.l0 = __ldg(A.ao_loc + q.lsh);
    const int sh[4] = {q.ish, q.jsh, q.ksh, q.lsh};
    double *dst[4] = {q.A, q.B, q.C, q.D};
#pragma unroll
    for (int s = 0; s < 4; s++) {
        dst[s][0] = __ldg(A.bas_x + sh[s]);
        dst[s][1] = __ldg(A.bas_y + sh[s]);
        dst[s][2] = __ldg(A.bas_z + sh[s]);
    }
    q.fac = (a == b && A.eri == nullptr) ? 0.5 * TWO_PI_2P5 : TWO_PI_2P5;
}

__device__ __forceinline__ void load_prim(const JKArgs &A, const Quartet &Q, int pi, int pk,
                                          PrimQuartet &P) {
    double aij = __ldg(A.a12 + pi), eij = __ldg(A.e12 + pi);
    double akl = __ldg(A.a12 + pk), ekl = __ldg(A.e12 + pk);
    double Pc[3] = {__ldg(A.x12 + pi), __ldg(A.y12 + pi), __ldg(A.z12 + pi)};
    double Qc[3] = {__ldg(A.x12 + pk), __ldg(A.y12 + pk), __ldg(A.z12 + pk)};
    P.p = aij;
    P.q = akl;
    const double s = aij + akl, pq = aij * akl;
    // 1/(p+q), 1/p and 1/q from one division
    const double t = 1.0 / (pq * s);
    P.inv_pq = pq * t;
    P.inv_p = akl * s * t;
    P.inv_q = aij * s * t;
    double rr = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        P.PA[d] = Pc[d] - Q.A[d];
        P.QC[d] = Qc[d] - Q.C[d];
        P.PQ[d] = Pc[d] - Qc[d];
        rr += P.PQ[d] * P.PQ[d];
    }
    P.x = pq * P.inv_pq * rr;
    P.pref = Q.fac * eij * ekl * (P.inv_p * P.inv_q) * rsqrt(s);
}

// One function of the order-N rule (q < N: node q, q >= N: weight q - N),
// by Clenshaw's recurrence.
template <int N>
__device__ __forceinline__ double cheb_one(const double *__restrict__ table, double x, int q) {
    constexpr int nint = kRysXmax[N];
    if (x < (double)nint) {
        int k = (int)x;
        double t = 2.0 * (x - k) - 1.0;
        double t2 = t + t;
        const double *c = table + RYS_TABLE_OFFSET[N] + k * (RYS_NCOEF * 2 * N) + q;
        double b1 = __ldg(c + (RYS_NCOEF - 1) * 2 * N), b2 = 0.0;
#pragma unroll
        for (int kk = RYS_NCOEF - 2; kk >= 1; kk--) {
            double n0 = fma(t2, b1, __ldg(c + kk * 2 * N) - b2);
            b2 = b1;
            b1 = n0;
        }
        return fma(t, b1, __ldg(c) - b2);
    }
    if (q < N) return RYS_HERM_R2[RYS_HERM_OFFSET[N] + q] / x;
    return RYS_HERM_W[RYS_HERM_OFFSET[N] + q - N] * sqrt(1.0 / x);
}


template <int LI, int LJ>
__global__ void schwarz_kernel(JKArgs A, int p0, int np, int pa0, int nprim, double diag_fac,
                               double *q_out) {
    constexpr int NFI = ncart(LI), NFJ = ncart(LJ);
    constexpr int NR = LI + LJ + 1;
    constexpr int GSZ = (LI + 1) * (LJ + 1) * (LI + 1) * (LJ + 1);
    constexpr int SJ = (LI + 1) * (LJ + 1), SI = (LJ + 1) * SJ;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= np) return;
    Quartet Q;
    load_quartet(A, p0 + t, p0 + t, Q);
    Q.fac = TWO_PI_2P5;
    double acc[NFI * NFJ], prod[NFI * NFJ];
#pragma unroll
    for (int n = 0; n < NFI * NFJ; n++) acc[n] = 0;
    int pa = pa0 + t * nprim;
    for (int ip = 0; ip < nprim; ip++) {
        for (int kp = 0; kp < nprim; kp++) {
            PrimQuartet P;
            load_prim(A, Q, pa + ip, pa + kp, P);
#pragma unroll 1
            for (int r = 0; r < NR; r++) {
                double s = cheb_one<NR>(A.rys, P.x, r);
                double w = cheb_one<NR>(A.rys, P.x, NR + r);
                RootCoef c = root_coef(s, P.p, P.q, P.inv_pq);
#pragma unroll 1
                for (int d = 0; d < 3; d++) {
                    double g[GSZ];
                    double ab = Q.A[d] - Q.B[d];
                    gen_2d<LI, LJ, LI, LJ, double>(d == 2 ? w * P.pref : 1.0,
                                                   P.PA[d] - c.qs * P.PQ[d],
                                                   P.QC[d] + c.ps * P.PQ[d], c.b00, c.b10,
                                                   c.b01, ab, ab, g);
#define BQC_DIAG(D)                                                                   \
    _Pragma("unroll") for (int fi = 0; fi < NFI; fi++)                                \
    _Pragma("unroll") for (int fj = 0; fj < NFJ; fj++) {                              \
        int ix = cart_pow(LI, fi, D), jx = cart_pow(LJ, fj, D);                       \
        double v = g[ix * SI + jx * SJ + ix * (LJ + 1) + jx];                        \
        if (D == 0) prod[fi * NFJ + fj] = v;                                          \
        else if (D == 1) prod[fi * NFJ + fj] *= v;                                    \
        else acc[fi * NFJ + fj] += prod[fi * NFJ + fj] * v;                           \
    }
                    if (d == 0) { BQC_DIAG(0) }
                    else if (d == 1) { BQC_DIAG(1) }
                    else { BQC_DIAG(2) }
#undef BQC_DIAG
                }
            }
        }
    }
    double m = 0;
#pragma unroll
    for (int n = 0; n < NFI * NFJ; n++) m = fmax(m, fabs(acc[n]));
    if (Q.ish == Q.jsh) m /= diag_fac * diag_fac;
    q_out[t] = sqrt(m);
}

}  // namespace bqc

using namespace bqc;

int bqc_launch_schwarz(int li, int lj, const JKArgs &args, int p0, int np, int pa0, int nprim,
                       double diag_fac, double *q_out, cudaStream_t stream) {
    if (np <= 0) return 0;
    int nb = (np + 127) / 128;
    JKArgs a_ = args;   // (not "a": the name is a parameter of BQC_SCASE)
    a_.rys = bqc_rys_cheb();
    bqc_count_launch(1);
    switch (li * 4 + lj) {
#define BQC_SCASE(a, b)                                                                        \
    case a * 4 + b:                                                                            \
        schwarz_kernel<a, b><<<nb, 128, 0, stream>>>(a_, p0, np, pa0, nprim, diag_fac, q_out); \
        break;
        BQC_SCASE(0, 0) BQC_SCASE(1, 0) BQC_SCASE(1, 1) BQC_SCASE(2, 0) BQC_SCASE(2, 1)
        BQC_SCASE(2, 2) BQC_SCASE(3, 0) BQC_SCASE(3, 1) BQC_SCASE(3, 2) BQC_SCASE(3, 3)
#undef BQC_SCASE
    default:
        return 2;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
