// What the J/K kernels share: the tile lookup and screening, the per-quartet
// and per-primitive quantities, and launch helpers.
#pragma once
#include <stdio.h>
#include <atomic>
#include "jk_device.cuh"

namespace bqc {

constexpr int TILE = 16;
constexpr int SMALL_NF = 54;   // largest quartet block one thread holds
constexpr double TWO_PI_2P5 = 34.986836655249725693;  // 2 pi^(5/2)

// 8-byte asynchronous global -> shared copies (cp.async, completed by the
// issuing thread's wait): the density blocks a quartet digests are fetched
// while its integrals are evaluated.
__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
__device__ __forceinline__ double dmax6(const double *__restrict__ dmc, int nbas, int i, int j,
                                        int k, int l) {
    double m = fmax(__ldg(dmc + i * nbas + j), __ldg(dmc + k * nbas + l));
    m = fmax(m, __ldg(dmc + i * nbas + k));
    m = fmax(m, __ldg(dmc + i * nbas + l));
    m = fmax(m, __ldg(dmc + j * nbas + k));
    return fmax(m, __ldg(dmc + j * nbas + l));
}

// The sub-task s, tile row r and tile column c of block x.  With tile_prefix
// (tile_prefix[r] = first block of tile row r over the rows of every sub-task
// of the launch, non-decreasing) the row is the largest r with
// tile_prefix[r] <= x, found by a 32-way search: each round every
// lane of the warp tests one of 32 evenly spaced candidates and a ballot
// keeps the last one that qualifies, so a row index of up to 2^20 takes four
// rounds of loads instead of twenty dependent ones.  All 32 lanes of every
// warp must call it.
// Every tile of a launch over several blocks runs as rparts * kparts parts: kpart
// of kparts ranges of the primitive quartets, and one of rparts parts of its
// quartets; the caller's (part, nparts) of the whole tile is refined by the latter.
__device__ __forceinline__ void tile_of_block(const JKTask &T, long long x, JKSub &s, int &r, int &c,
                                              int &part, int &nparts, int &kpart) {
    if (T.tile_prefix != nullptr) {
        const int lane = threadIdx.x & 31;
        int lo = 0, hi = T.nrows;   // tile_prefix[lo] <= x; answer in [lo, hi)
        while (hi - lo > 1) {
            const int step = (hi - lo + 31) >> 5;
            const int idx = lo + lane * step;
            const bool le = idx < hi && __ldg(T.tile_prefix + idx) <= x;
            const unsigned m = __ballot_sync(0xffffffffu, le);   // bit 0 always set
            lo += (31 - __clz(m)) * step;
            hi = min(hi, lo + step);
        }
        r = lo;
        const int y = (int)(x - __ldg(T.tile_prefix + r));   // a row's parts fit 32 bits
        const int col0 = T.tile_col0 != nullptr ? __ldg(T.tile_col0 + r) : 0;
        s = T.sub;
        c = col0 + y;
        kpart = s.kfirst;
        if (T.subs != nullptr) {
            s = T.subs[__ldg(T.row_sub + r)];
            r -= s.row0;
            if (T.swapped) s = jk_swap_sub(s);
            const int parts = s.rparts * s.kparts;
            c = col0 + y / parts;
            const int p = y % parts;
            kpart = p % s.kparts;
            part = part * s.rparts + p / s.kparts;
            nparts *= s.rparts;
        }
    } else {
        s = T.sub;
        const int ncols = ((s.rows_are_b ? s.na : s.nb) + TILE - 1) / TILE;
        r = (int)(x / ncols);
        c = (int)(x % ncols);
        kpart = s.kfirst;
    }
}

// Surviving quartets of tile x into s_list (order unspecified).  With
// nparts > 1 (a power of two up to 64) only the quartets e = part (mod
// nparts) of the tile's 256 are screened, e = 16 * row + column: part p takes
// every nparts-th column of every row, so the parts are disjoint, cover the
// tile and get similar shares of a q-sorted tile.
__device__ __forceinline__ bool tile_screen(const JKArgs &A, const JKTask &T, long long x, JKSub &s,
                                            int *s_list, int *s_count, int &a_begin, int &b_begin,
                                            int &count, int &kpart, int part = 0, int nparts = 1) {
    int r, c;
    tile_of_block(T, x, s, r, c, part, nparts, kpart);
    int ta = s.rows_are_b ? c : r, tb = s.rows_are_b ? r : c;
    a_begin = s.a0 + ta * TILE;
    b_begin = s.b0 + tb * TILE;
    int a_end = min(s.a0 + s.na, a_begin + TILE);
    int b_end = min(s.b0 + s.nb, b_begin + TILE);
    if (s.diag && b_begin > a_end - 1) return false;
    if (threadIdx.x == 0) *s_count = 0;
    __syncthreads();
    for (int e0 = threadIdx.x; e0 < TILE * TILE / nparts; e0 += blockDim.x) {
        const int e = e0 * nparts + part;
        int a = a_begin + e / TILE, b = b_begin + e % TILE;
        bool keep = a < a_end && b < b_end && (!s.diag || a >= b);
        if (keep && A.pair_q != nullptr) {
            double bound = __ldg(A.pair_q + a) * __ldg(A.pair_q + b);
            if (A.dm_cond != nullptr) {
                int i = __ldg(A.pair_bra + a), j = __ldg(A.pair_ket + a);
                int k = __ldg(A.pair_bra + b), l = __ldg(A.pair_ket + b);
                bound *= dmax6(A.dm_cond, A.nbas, i, j, k, l);
            }
            keep = bound >= A.tol && (A.tol_hi <= 0. || bound < A.tol_hi);
        }
        if (keep) {
            int idx = atomicAdd(s_count, 1);
            s_list[idx] = ((a - a_begin) << 16) | (b - b_begin);
        }
    }
    __syncthreads();
    count = *s_count;
    return count > 0;
}

// Shells, first AOs and centres of a pair, and of a primitive pair the
// exponent p, its inverse, the factor e and the centre P.  As records they are
// four and three 16-byte loads from one address each; from the separate arrays
// twelve and six loads and, per array, the address arithmetic that
// outnumbered the floating-point instructions of the small classes (five to
// one for (ps|ss)).
struct Pair {
    int i, j, i0, j0;
    double A[3], AB[3];
};

__device__ __forceinline__ void load_pair(const JKArgs &A, int n, Pair &p) {
    if (A.pair_rec != nullptr) {
        const int4 *rec = A.pair_rec + (size_t)n * PAIR_REC;
        const int4 s = __ldg(rec);
        const double2 *c = reinterpret_cast<const double2 *>(rec + 1);
        const double2 u = __ldg(c), v = __ldg(c + 1), w = __ldg(c + 2);
        p.i = s.x; p.j = s.y; p.i0 = s.z; p.j0 = s.w;
        p.A[0] = u.x; p.A[1] = u.y; p.A[2] = v.x;
        p.AB[0] = v.y; p.AB[1] = w.x; p.AB[2] = w.y;
    } else {
        p.i = __ldg(A.pair_bra + n);
        p.j = __ldg(A.pair_ket + n);
        p.i0 = __ldg(A.ao_loc + p.i);
        p.j0 = __ldg(A.ao_loc + p.j);
        p.A[0] = __ldg(A.bas_x + p.i); p.A[1] = __ldg(A.bas_y + p.i); p.A[2] = __ldg(A.bas_z + p.i);
        p.AB[0] = p.A[0] - __ldg(A.bas_x + p.j);
        p.AB[1] = p.A[1] - __ldg(A.bas_y + p.j);
        p.AB[2] = p.A[2] - __ldg(A.bas_z + p.j);
    }
}

struct PrimPair {
    double p, inv_p, e, P[3];
};

__device__ __forceinline__ void load_prim(const JKArgs &A, int n, PrimPair &k) {
    if (A.prim_rec != nullptr) {
        const double2 *rec = A.prim_rec + (size_t)n * PRIM_REC;
        const double2 u = __ldg(rec), v = __ldg(rec + 1), w = __ldg(rec + 2);
        k.p = u.x; k.inv_p = u.y; k.e = v.x;
        k.P[0] = v.y; k.P[1] = w.x; k.P[2] = w.y;
    } else {
        k.p = __ldg(A.a12 + n);
        k.inv_p = 1.0 / k.p;
        k.e = __ldg(A.e12 + n);
        k.P[0] = __ldg(A.x12 + n);
        k.P[1] = __ldg(A.y12 + n);
        k.P[2] = __ldg(A.z12 + n);
    }
}

// quantities of one primitive quartet
struct PrimQuartet {
    double p, q, inv_pq, inv_p, inv_q, x, pref;
    double PA[3], QC[3], PQ[3];
};

__device__ __forceinline__ void prim_quartet(const PrimPair &i, const PrimPair &k, const double *Ax,
                                             const double *Cx, double fac, PrimQuartet &P) {
    P.p = i.p;
    P.q = k.p;
    const double rs = rsqrt_pos(i.p + k.p);
    P.inv_pq = rs * rs;
    P.inv_p = i.inv_p;
    P.inv_q = k.inv_p;
    double rr = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        P.PA[d] = i.P[d] - Ax[d];
        P.QC[d] = k.P[d] - Cx[d];
        P.PQ[d] = i.P[d] - k.P[d];
        rr += P.PQ[d] * P.PQ[d];
    }
    P.x = i.p * k.p * P.inv_pq * rr;
    P.pref = fac * i.e * k.e * (i.inv_p * k.inv_p) * rs;
}

// recursion coefficients of root s, without a division
__device__ __forceinline__ RootCoef root_coef(double s, const PrimQuartet &P) {
    RootCoef c;
    c.b00 = 0.5 * s * P.inv_pq;
    c.qs = P.q * s * P.inv_pq;
    c.ps = P.p * s * P.inv_pq;
    c.b10 = 0.5 * (1.0 - c.qs) * P.inv_p;
    c.b01 = 0.5 * (1.0 - c.ps) * P.inv_q;
    return c;
}

// tiles of a launch: the caller's count, or the full rectangle of its block
static inline long long task_tiles(const JKTask &task) {
    if (task.tile_prefix) return task.ntiles;
    return (long long)((task.sub.na + TILE - 1) / TILE) * ((task.sub.nb + TILE - 1) / TILE);
}

// Raise the dynamic shared-memory limit of kernel K to `bytes`, once per
// device: the attribute belongs to the (kernel, device) pair, so a process
// that drives several GPUs sets it on each (flags per device, race-free).
constexpr int MAX_DEVICES = 64;
template <auto K>
static int smem_attr(int bytes) {
    static std::atomic<unsigned char> done[MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return 1;
    if (!done[dev].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
            return 1;
        done[dev].store(1, std::memory_order_release);
    }
    return 0;
}

// One launch, at the task's priority if it has one; errors are left to
// cudaGetLastError().
static inline void launch_at(void (*kernel)(JKArgs, JKTask), int grid, int block, size_t smem, cudaStream_t stream,
                             const JKArgs &args, const JKTask &task) {
    if (task.ntiles_dev == nullptr || task.priority == 0) {
        kernel<<<grid, block, smem, stream>>>(args, task);
        return;
    }
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributePriority;
    attr.val.priority = task.priority;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args, task);
}

// SM count of the current device (cached per device; 0 on error)
static inline int device_sms() {
    static std::atomic<int> sms[MAX_DEVICES];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return 0;
    int n = sms[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

}  // namespace bqc
