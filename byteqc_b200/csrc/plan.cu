// J/K builds scheduled on the device (no reference counterpart; the
// reference prunes on the host, cuobc/scf/hf.py:111-166, and launches one
// kernel per kl bin, cuobc/lib/gvhf/nr_jk_driver.cu:252-280).
//
// A plan holds, per basis-product cache, everything of a J/K build that does
// not depend on the density: the class-pair task list, the Schwarz factor of
// the first (largest) pair of every 16-pair tile, and device scratch for the
// schedule.  A build then runs entirely on the stream without a host
// round trip or an allocation:
//
//   inputs   : dm_max = max over the density-block table, and the pair and
//              primitive-pair records from the cache's arrays (one kernel);
//   counts   : per tile row r of every task, the number of leading column
//              tiles c with q_row[r] q_col[c] dm_max >= tol (the tiles are
//              sorted by their first q, so a binary search), at most r + 1 on
//              a diagonal task; for batched molecules only the row's own
//              molecule's columns count;
//   prefix   : per class shape (li lj | lk ll), the exclusive scan of the row
//              counts of all its class pairs and the shape's tile total;
//   launches : one per shape and precision band, a fixed grid of CTAs that
//              strides over the shape's [0, total) tiles (JKTask::ntiles_dev),
//              dealt out costly first over side streams of the plan that fork
//              from and join the caller's stream.  The launches only add to
//              the outputs, so their order is free.  A small build's launches
//              are each too small to fill the GPU and as long as one quartet's
//              chain of loads and roots: get_jk of one water (cc-pVDZ shape)
//              took 3.17 ms with its 120 class pairs one after another, 0.88
//              ms over eight streams, 0.41 ms with its 21 shapes (two waters,
//              cc-pVTZ shape: 10.2, 2.4 and 1.03 ms).
//
// Every launch of a build has the same shape each time, so a build can be
// captured in a CUDA graph and replayed.
#include <algorithm>
#include <array>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <utility>
#include <map>
#include <mutex>
#include <vector>
#include "bqc.h"

namespace {

constexpr int TILE = 16;

// Side streams of a plan: as many as a process has hardware queues by default.
constexpr int SIDE_STREAMS = 8;

// What a plan takes from the device beside its caller's streams: side streams with
// their events, and one allocation for all its arrays.
struct Resources {
    cudaStream_t side[SIDE_STREAMS];
    cudaEvent_t fork, join[SIDE_STREAMS];
    char *slab;
    size_t bytes;
};

// Creating the streams and events takes 0.5 ms, an allocation of a few MB 1.4
// ms, as long as the rest of a small molecule's set-up: what a destroyed plan
// had is kept for the next plan on its device, at most SETS_KEPT sets of at most
// SLAB_KEPT bytes.  A set belongs to one plan at a time.  _VHFOpt.build() of
// geometries after one another, with an allocation for each array and none kept
// and now: four waters / cc-pVDZ 4.1 -> 3.75 ms, a 20-carbon chain / 6-31G** 17.0 ->
// 15.2 ms.
constexpr size_t SETS_KEPT = 4, SLAB_KEPT = 64 << 20;
std::mutex g_sets_lock;
std::vector<std::pair<int, Resources *>> g_sets;   // (device, idle set)

void free_set(Resources *s) {
    for (int n = 0; n < SIDE_STREAMS; n++) {
        if (s->side[n]) cudaStreamDestroy(s->side[n]);
        if (s->join[n]) cudaEventDestroy(s->join[n]);
    }
    if (s->fork) cudaEventDestroy(s->fork);
    cudaFree(s->slab);
    delete s;
}

// an idle set of the device, the smallest that holds `bytes` if one does, or a new one
Resources *take_set(int device, size_t bytes) {
    Resources *s = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_sets_lock);
        auto best = g_sets.end();
        for (auto it = g_sets.begin(); it != g_sets.end(); ++it) {
            if (it->first != device) continue;
            const size_t have = it->second->bytes, most = best == g_sets.end() ? 0 : best->second->bytes;
            if (best == g_sets.end() || (have >= bytes ? most < bytes || have < most : have > most)) best = it;
        }
        if (best != g_sets.end()) {
            s = best->second;
            g_sets.erase(best);
        }
    }
    bool ok = true;
    if (s == nullptr) {
        s = new Resources();   // value-initialised: every handle NULL
        ok = cudaEventCreateWithFlags(&s->fork, cudaEventDisableTiming) == cudaSuccess;
        for (int n = 0; ok && n < SIDE_STREAMS; n++)
            ok = cudaStreamCreateWithFlags(&s->side[n], cudaStreamNonBlocking) == cudaSuccess &&
                 cudaEventCreateWithFlags(&s->join[n], cudaEventDisableTiming) == cudaSuccess;
    }
    if (ok && s->bytes < bytes) {
        cudaFree(s->slab);
        s->slab = nullptr;
        s->bytes = 0;
        ok = cudaMalloc(&s->slab, bytes) == cudaSuccess;
        if (ok) s->bytes = bytes;
    }
    if (!ok) {
        free_set(s);
        return nullptr;
    }
    return s;
}

// back from a plan, nothing of which may be in flight any more
void give_set(int device, Resources *s) {
    if (s->bytes > SLAB_KEPT) {
        cudaFree(s->slab);
        s->slab = nullptr;
        s->bytes = 0;
    }
    {
        std::lock_guard<std::mutex> lock(g_sets_lock);
        if (g_sets.size() < SETS_KEPT) {
            g_sets.push_back({device, s});
            return;
        }
    }
    free_set(s);
}

// density-independent description of one class pair for the schedule kernels
struct SchedTask {
    int row_off;   // first global row of the class pair
    int ncols;
    int a_tile0;   // first tile of the row list in the tile arrays
    int b_tile0;   // of the column list
    int diag;
    int parts;     // parts every tile runs as
};

// rows [row0, row0 + nrows) of one class shape; its prefix entries start at
// row0 + (index of the shape)
struct SchedShape {
    int row0, nrows;
};

struct ShapeHost {
    int li, lj, lk, ll;
    int row0, nrows;
    int index;         // in the device arrays
    long long max_tiles;
    double cost;
};

// Largest n in [lo, hi] such that q[c] * qr >= tol for all c < n (q
// descending): the number of leading columns that reach tol.
__device__ __forceinline__ int leading_cols(const double *__restrict__ q, int lo, int hi, double qr,
                                            double tol) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(q + mid) * qr >= tol) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// first index in [lo, hi) whose molecule is >= m (molecules ascending)
__device__ __forceinline__ int first_mol(const int *__restrict__ mol, int lo, int hi, int m) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(mol + mid) < m) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// What a build derives from its inputs first.  Blocks [0, max_blocks): the
// maximum of the non-negative entries of x (as ordered 64-bit patterns).  The
// others: the records of JKArgs::pair_rec and prim_rec from the cache's arrays as
// they are at this point of the caller's stream.  Made by every build and not
// once per plan: 112 bytes per pair and primitive pair are microseconds beside
// its quartets, and the arrays may change between builds.
__global__ void inputs_kernel(const double *__restrict__ x, size_t n, unsigned long long *out, int max_blocks,
                              BasisProdCache bp, int npair, int nprim, int4 *__restrict__ pair_rec,
                              double2 *__restrict__ prim_rec) {
    if ((int)blockIdx.x < max_blocks) {
        double m = 0.;
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)max_blocks * blockDim.x)
            m = fmax(m, __ldg(x + i));
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
        return;
    }
    const long long first = (blockIdx.x - max_blocks) * (long long)blockDim.x + threadIdx.x;
    const long long step = (gridDim.x - max_blocks) * (long long)blockDim.x;
    const double *cx = bp.bas_coords, *cy = cx + bp.nbas, *cz = cy + bp.nbas;
    for (long long t = first; t < (long long)npair + nprim; t += step) {
        if (t < npair) {
            const int i = bp.bas_pair2bra[t], j = bp.bas_pair2ket[t];
            int4 *r = pair_rec + t * PAIR_REC;
            double2 *c = reinterpret_cast<double2 *>(r + 1);
            r[0] = make_int4(i, j, bp.ao_loc[i], bp.ao_loc[j]);
            c[0] = make_double2(cx[i], cy[i]);
            c[1] = make_double2(cz[i], cx[i] - cx[j]);
            c[2] = make_double2(cy[i] - cy[j], cz[i] - cz[j]);
        } else {
            const long long u = t - npair;
            double2 *r = prim_rec + u * PRIM_REC;
            r[0] = make_double2(bp.a12[u], 1.0 / bp.a12[u]);
            r[1] = make_double2(bp.e12[u], bp.x12[u]);
            r[2] = make_double2(bp.y12[u], bp.z12[u]);
        }
    }
}

// per global row: the column counts of the two precision bands (band 1 only
// when tol1 > 0) and, for batched molecules, the row's first column
__global__ void count_rows_kernel(const SchedTask *__restrict__ tasks, const int *__restrict__ row_task,
                                  int nrows_all, const double *__restrict__ tile_q,
                                  const int *__restrict__ tile_mol, const unsigned long long *dm_max_bits,
                                  double tol0, double tol1, int *__restrict__ cnt0,
                                  int *__restrict__ cnt1, int *__restrict__ col0) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nrows_all) return;
    const SchedTask t = tasks[__ldg(row_task + g)];
    const int r = g - t.row_off;
    const double dm_max = __longlong_as_double((long long)*dm_max_bits);
    const double qr = __ldg(tile_q + t.a_tile0 + r) * dm_max;
    const double *qb = tile_q + t.b_tile0;
    int c0 = 0, c1 = t.ncols;
    if (tile_mol != nullptr) {
        const int m = __ldg(tile_mol + t.a_tile0 + r);
        const int *mb = tile_mol + t.b_tile0;
        c0 = first_mol(mb, 0, t.ncols, m);
        c1 = first_mol(mb, c0, t.ncols, m + 1);
        col0[g] = c0;
    }
    const int lim = t.diag ? r - c0 + 1 : c1 - c0;
    int n0 = leading_cols(qb, c0, c1, qr, tol0) - c0;
    cnt0[g] = max(0, min(n0, lim)) * t.parts;
    if (tol1 > 0.) {
        int n1 = leading_cols(qb, c0, c1, qr, tol1) - c0;
        cnt1[g] = max(0, min(n1, lim)) * t.parts;
    }
}

// one CTA per shape and band: exclusive scan of its row counts into the prefix
// and the shape's total
__global__ void scan_rows_kernel(const SchedShape *__restrict__ shapes, const int *__restrict__ cnt_all,
                                 int cnt_stride, long long *__restrict__ prefix_all, int prefix_stride,
                                 long long *__restrict__ ntiles_all) {
    const SchedShape t = shapes[blockIdx.x];
    const int *cnt = cnt_all + (size_t)blockIdx.y * cnt_stride + t.row0;
    long long *prefix = prefix_all + (size_t)blockIdx.y * prefix_stride + t.row0 + blockIdx.x;
    __shared__ long long s_warp[32];
    __shared__ long long s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int base = 0; base < t.nrows; base += blockDim.x) {
        const int r = base + threadIdx.x;
        long long x = r < t.nrows ? __ldg(cnt + r) : 0;
        // inclusive scan within the warp
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            long long w = lane < nw ? s_warp[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const long long y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            if (lane < nw) s_warp[lane] = w;
        }
        __syncthreads();
        const long long incl = x + (warp > 0 ? s_warp[warp - 1] : 0) + s_carry;
        if (r < t.nrows) prefix[r + 1] = incl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_carry = incl;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        prefix[0] = 0;
        ntiles_all[blockIdx.y * gridDim.x + blockIdx.x] = s_carry;
    }
}

}  // namespace

struct BQCPlan {
    const BasisProdCache *bp;
    int device;
    int nsm;
    std::vector<ShapeHost> shapes;   // costly first
    int nshapes, nrows_all, npfx, npair, nprim;
    Resources *res;
    // device: parts of the set's allocation
    SchedTask *d_tasks;
    SchedShape *d_shapes;
    JKSub *d_subs;
    int *d_row_task;
    double *d_tile_q;
    int *d_tile_mol;   // NULL unless batched molecules
    int *d_cnt;        // 2 x nrows_all
    int *d_col0;       // nrows_all (batched molecules)
    long long *d_prefix;   // 2 x npfx
    long long *d_ntiles;   // 2 x nshapes
    unsigned long long *d_dm_max;
    int4 *d_pair_rec;      // JKArgs::pair_rec, prim_rec
    double2 *d_prim_rec;
};

namespace {

// cost of one quartet of a class shape per primitive quartet (flops of the
// Rys quadrature), to launch the costly shapes first
double prim_cost(int li, int lj, int lk, int ll) {
    const int n = (li + lj + lk + ll) / 2 + 1;
    const double nf = (li + 1) * (li + 2) / 2 * ((lj + 1) * (lj + 2) / 2) * ((lk + 1) * (lk + 2) / 2) *
                      ((ll + 1) * (ll + 2) / 2);
    return n * (15. * (li + lj + 1) * (lk + ll + 1) + 3. * nf) + 30.;
}

}  // namespace

extern "C" {

int BQCplan_create(const BasisProdCache *bp, const double *pair_q_host, const int *pair_mol_host,
                   BQCPlan **out) {
    if (bp == nullptr || pair_q_host == nullptr || out == nullptr) return 3;
    *out = nullptr;
    BQCPlan *p = new BQCPlan();   // value-initialised: every pointer NULL
    p->bp = bp;
    if (cudaGetDevice(&p->device) != cudaSuccess) { delete p; return 1; }
    int nsm = 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, p->device) != cudaSuccess) {
        delete p;
        return 1;
    }
    p->nsm = nsm;
    // tiles of every class: q of the first pair (the tile's largest)
    std::vector<int> class_tile0(bp->ncptype + 1, 0);
    for (int c = 0; c < bp->ncptype; c++)
        class_tile0[c + 1] = class_tile0[c] + (bp->cptype[c].npairs + TILE - 1) / TILE;
    const int ntile_all = class_tile0[bp->ncptype];
    std::vector<double> tile_q(std::max(ntile_all, 1));
    std::vector<int> tile_mol(pair_mol_host ? std::max(ntile_all, 1) : 0);
    for (int c = 0; c < bp->ncptype; c++) {
        const int p0 = bp->bas_pairs_locs[c], np = bp->cptype[c].npairs;
        for (int t = 0; t * TILE < np; t++) {
            tile_q[class_tile0[c] + t] = pair_q_host[p0 + t * TILE];
            if (pair_mol_host) tile_mol[class_tile0[c] + t] = pair_mol_host[p0 + t * TILE];
        }
    }
    // the class pairs by shape
    struct Pair {
        int cij, ckl;
        JKSub sub;
        double cost;
    };
    std::map<std::array<int, 4>, std::vector<Pair>> by_shape;
    for (int cij = 0; cij < bp->ncptype; cij++) {
        const ContractionProdType *tij = bp->cptype + cij;
        if (tij->npairs == 0) continue;
        for (int ckl = 0; ckl <= cij; ckl++) {
            const ContractionProdType *tkl = bp->cptype + ckl;
            if (tkl->npairs == 0) continue;
            if (tij->l_bra > BQC_LMAX || tkl->l_bra > BQC_LMAX) { delete p; return 2; }
            Pair x;
            memset(&x.sub, 0, sizeof(x.sub));
            x.cij = cij;
            x.ckl = ckl;
            x.sub.a0 = bp->bas_pairs_locs[cij];
            x.sub.na = tij->npairs;
            x.sub.b0 = bp->bas_pairs_locs[ckl];
            x.sub.nb = tkl->npairs;
            x.sub.pa0 = bp->primitive_pairs_locs[cij];
            x.sub.pb0 = bp->primitive_pairs_locs[ckl];
            x.sub.nprim_a = tij->nprim_12;
            x.sub.nprim_b = tkl->nprim_12;
            x.sub.diag = cij == ckl;
            x.cost = (double)tij->nprim_12 * tkl->nprim_12;
            split_prims(x.sub);
            std::array<int, 4> key = {tij->l_bra, tij->l_ket, tkl->l_bra, tkl->l_ket};
            // canonical order: pair index of the bra >= that of the ket
            if (key[0] * (key[0] + 1) / 2 + key[1] < key[2] * (key[2] + 1) / 2 + key[3]) {
                key = {key[2], key[3], key[0], key[1]};
                x.sub = jk_swap_sub(x.sub);
            }
            by_shape[key].push_back(x);
        }
    }
    std::vector<SchedTask> st;
    std::vector<SchedShape> ss;
    std::vector<JKSub> subs;
    std::vector<int> row_task;
    for (auto &entry : by_shape) {
        const std::array<int, 4> &l = entry.first;
        // the longest quartets first: they would be the tail otherwise
        std::stable_sort(entry.second.begin(), entry.second.end(),
                         [](const Pair &x, const Pair &y) { return x.cost > y.cost; });
        ShapeHost h;
        h.li = l[0]; h.lj = l[1]; h.lk = l[2]; h.ll = l[3];
        h.row0 = (int)row_task.size();
        h.max_tiles = 0;
        h.cost = 0.;
        for (Pair &x : entry.second) {
            const int nrows = (bp->cptype[x.cij].npairs + TILE - 1) / TILE;
            const int ncols = (bp->cptype[x.ckl].npairs + TILE - 1) / TILE;
            const long long tiles = x.sub.diag ? (long long)nrows * (nrows + 1) / 2 : (long long)nrows * ncols;
            x.sub.row0 = (int)row_task.size() - h.row0;
            SchedTask s;
            s.row_off = (int)row_task.size();
            s.ncols = ncols;
            s.a_tile0 = class_tile0[x.cij];
            s.b_tile0 = class_tile0[x.ckl];
            s.diag = x.sub.diag;
            s.parts = x.sub.rparts * x.sub.kparts;
            row_task.insert(row_task.end(), nrows, (int)st.size());
            st.push_back(s);
            subs.push_back(x.sub);
            h.max_tiles += tiles * s.parts;
            h.cost += (double)tiles * x.cost * prim_cost(l[0], l[1], l[2], l[3]);
        }
        h.nrows = (int)row_task.size() - h.row0;
        ss.push_back({h.row0, h.nrows});
        p->shapes.push_back(h);
    }
    p->nshapes = (int)ss.size();
    p->nrows_all = (int)row_task.size();
    p->npfx = p->nrows_all + p->nshapes;
    const size_t nt = std::max<size_t>(st.size(), 1), nr = std::max(p->nrows_all, 1),
                 np_ = std::max(p->npfx, 1), ns = std::max(p->nshapes, 1);
    p->npair = bp->bas_pairs_locs[bp->ncptype];
    p->nprim = bp->primitive_pairs_locs[bp->ncptype];
    // One allocation: what the schedule reads, uploaded in one copy, then the scratch
    size_t bytes = 0;
    auto part = [&bytes](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t tasks = part(sizeof(SchedTask) * nt), shapes = part(sizeof(SchedShape) * ns),
                 subs_at = part(sizeof(JKSub) * nt), rows = part(sizeof(int) * nr),
                 tq = part(sizeof(double) * tile_q.size()), tm = part(sizeof(int) * tile_mol.size()),
                 upload = bytes;
    const size_t cnt = part(sizeof(int) * 2 * nr), col0 = part(sizeof(int) * nr),
                 prefix = part(sizeof(long long) * 2 * np_), ntiles = part(sizeof(long long) * 2 * ns),
                 dm_max = part(sizeof(unsigned long long)),
                 pair_rec = part(sizeof(int4) * PAIR_REC * std::max(p->npair, 1)),
                 prim_rec = part(sizeof(double2) * PRIM_REC * std::max(p->nprim, 1));
    std::vector<char> host(upload);
    auto fill = [&host](size_t at, const auto &v) {
        if (!v.empty()) memcpy(host.data() + at, v.data(), sizeof(v[0]) * v.size());
    };
    fill(tasks, st);
    fill(shapes, ss);
    fill(subs_at, subs);
    fill(rows, row_task);
    fill(tq, tile_q);
    fill(tm, tile_mol);
    p->res = take_set(p->device, bytes);
    if (p->res == nullptr || cudaMemcpy(p->res->slab, host.data(), upload, cudaMemcpyHostToDevice) != cudaSuccess) {
        BQCplan_destroy(p);
        return 1;
    }
    char *slab = p->res->slab;
    p->d_tasks = (SchedTask *)(slab + tasks);
    p->d_shapes = (SchedShape *)(slab + shapes);
    p->d_subs = (JKSub *)(slab + subs_at);
    p->d_row_task = (int *)(slab + rows);
    p->d_tile_q = (double *)(slab + tq);
    p->d_tile_mol = pair_mol_host ? (int *)(slab + tm) : nullptr;
    p->d_cnt = (int *)(slab + cnt);
    p->d_col0 = (int *)(slab + col0);
    p->d_prefix = (long long *)(slab + prefix);
    p->d_ntiles = (long long *)(slab + ntiles);
    p->d_dm_max = (unsigned long long *)(slab + dm_max);
    p->d_pair_rec = (int4 *)(slab + pair_rec);
    p->d_prim_rec = (double2 *)(slab + prim_rec);
    // costly shapes first, so that the cheap ones fill the tail
    // (the rows and prefixes stay in the order of the device arrays)
    for (int n = 0; n < p->nshapes; n++) p->shapes[n].index = n;
    std::stable_sort(p->shapes.begin(), p->shapes.end(),
                     [](const ShapeHost &x, const ShapeHost &y) { return x.cost > y.cost; });
    *out = p;
    return 0;
}

void BQCplan_destroy(BQCPlan *p) {
    if (p == nullptr) return;
    if (p->res != nullptr) {
        // the plan's launches end before its set serves another plan
        int dev = p->device;
        cudaGetDevice(&dev);
        if (dev != p->device) cudaSetDevice(p->device);
        cudaDeviceSynchronize();
        if (dev != p->device) cudaSetDevice(dev);
        give_set(p->device, p->res);
    }
    delete p;
}

int BQCbuild_jk_plan(const BQCPlan *p, const double *pair_q, const double *dm_cond, double *vj,
                     double *vk, const double *dm, int nao, int n_dm, double tol, double fp32_below,
                     cudaStream_t stream) {
    if (p == nullptr || pair_q == nullptr || dm_cond == nullptr || dm == nullptr) return 3;
    if (p->nshapes == 0) return 0;
    const BasisProdCache *bp = p->bp;
    const bool two = fp32_below > tol;
    // 1. dm_max and the records on the device
    if (cudaMemsetAsync(p->d_dm_max, 0, sizeof(unsigned long long), stream) != cudaSuccess) return 1;
    const size_t nn = (size_t)bp->nbas * bp->nbas;
    bqc_count_launch(3);
    const int max_blocks = (int)std::min<size_t>(1024, (nn + 255) / 256);
    const int rec_blocks = (int)std::min(8LL * p->nsm, ((long long)p->npair + p->nprim) / 256 + 1);
    inputs_kernel<<<max_blocks + rec_blocks, 256, 0, stream>>>(dm_cond, nn, p->d_dm_max, max_blocks, *bp,
                                                               p->npair, p->nprim, p->d_pair_rec, p->d_prim_rec);
    // 2. column counts per row (band 0: FP64, bound >= fp32_below when two
    //    bands, else >= tol; band 1: FP32, bound >= tol) and their scans
    int *cnt0 = p->d_cnt, *cnt1 = p->d_cnt + std::max(p->nrows_all, 1);
    count_rows_kernel<<<(p->nrows_all + 255) / 256, 256, 0, stream>>>(
        p->d_tasks, p->d_row_task, p->nrows_all, p->d_tile_q, p->d_tile_mol, p->d_dm_max,
        two ? fp32_below : tol, two ? tol : 0., cnt0, cnt1, p->d_col0);
    const int nr = std::max(p->nrows_all, 1), np_ = std::max(p->npfx, 1);
    scan_rows_kernel<<<dim3(p->nshapes, two ? 2 : 1), 1024, 0, stream>>>(p->d_shapes, p->d_cnt, nr,
                                                                         p->d_prefix, np_, p->d_ntiles);
    if (cudaGetLastError() != cudaSuccess) return 1;
    // 3. the class kernels, persistent over the device tile counts
    JKArgs args;
    memset(&args, 0, sizeof(args));
    args.pair_bra = bp->bas_pair2bra;
    args.pair_ket = bp->bas_pair2ket;
    args.a12 = bp->a12;
    args.e12 = bp->e12;
    args.pair_rec = p->d_pair_rec;
    args.prim_rec = p->d_prim_rec;
    args.x12 = bp->x12;
    args.y12 = bp->y12;
    args.z12 = bp->z12;
    args.bas_x = bp->bas_coords;
    args.bas_y = bp->bas_coords + bp->nbas;
    args.bas_z = bp->bas_coords + 2 * bp->nbas;
    args.ao_loc = bp->ao_loc;
    args.pair_q = pair_q;
    args.dm_cond = dm_cond;
    args.dm = dm;
    args.vj = vj;
    args.vk = vk;
    args.nao = nao;
    args.nbas = bp->nbas;
    args.n_dm = n_dm;
    args.rys = bqc_rys_table();
    args.rys_lm = bqc_rys_table_lm();
    int priority = 0;
    if (cudaStreamGetPriority(stream, &priority) != cudaSuccess) return 1;
    // fork: the shapes are independent (the outputs are accumulated by atomics)
    const Resources &ss = *p->res;
    if (cudaEventRecord(ss.fork, stream) != cudaSuccess) return 1;
    for (int n = 0; n < SIDE_STREAMS; n++)
        if (cudaStreamWaitEvent(ss.side[n], ss.fork, 0) != cudaSuccess) return 1;
    int err = 0, turn = 0;
    for (int i = 0; i < p->nshapes && !err; i++) {
        const ShapeHost &h = p->shapes[i];
        for (int band = 0; band < (two ? 2 : 1) && !err; band++) {
            JKArgs a = args;
            a.tol = band == 0 ? (two ? fp32_below : tol) : tol;
            a.tol_hi = band == 0 ? 0. : fp32_below;
            JKTask t;
            memset(&t, 0, sizeof(t));
            t.tile_prefix = p->d_prefix + (size_t)band * np_ + h.row0 + h.index;
            t.tile_col0 = p->d_tile_mol ? p->d_col0 + h.row0 : nullptr;
            t.nrows = h.nrows;
            t.ntiles = h.max_tiles;
            t.subs = p->d_subs;
            t.row_sub = p->d_row_task + h.row0;
            t.ntiles_dev = p->d_ntiles + (size_t)band * p->nshapes + h.index;
            t.nsm = p->nsm;
            t.priority = priority;
            err = bqc_launch_jk(h.li, h.lj, h.lk, h.ll, a, t, band == 1, ss.side[turn++ % SIDE_STREAMS]);
        }
    }
    // join, also after a failed launch: the caller's stream waits for all
    for (int n = 0; n < SIDE_STREAMS; n++)
        if (cudaEventRecord(ss.join[n], ss.side[n]) != cudaSuccess ||
            cudaStreamWaitEvent(stream, ss.join[n], 0) != cudaSuccess)
            err = err ? err : 1;
    return err;
}

}  // extern "C"
