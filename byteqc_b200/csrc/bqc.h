// Internal declarations shared by the CUDA translation units of libbyteqc_b200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "byteqc_b200.h"

#define BQC_LMAX 3          // s, p, d, f
#define BQC_NCART_MAX 10
#define PAIR_REC 4
#define PRIM_REC 3

// Everything a J/K kernel launch reads.  Device pointers unless noted.
struct JKArgs {
    const int *pair_bra;      // shell i of each pair        (bas_pair2bra)
    const int *pair_ket;      // shell j of each pair        (bas_pair2ket)
    const double *a12, *e12, *x12, *y12, *z12;  // primitive-pair data
    // the same data as records (made by the builds of a plan; NULL otherwise): per pair
    // PAIR_REC 16-byte words {shell i, shell j, ao_loc i, ao_loc j | A, A - B},
    // per primitive pair PRIM_REC words {a12, 1 / a12 | e12, x12 | y12, z12}
    const int4 *pair_rec;
    const double2 *prim_rec;
    const double *bas_x, *bas_y, *bas_z;        // shell centres
    const int *ao_loc;        // Cartesian AO offsets of the sorted, decontracted basis
    const double *pair_q;     // Schwarz factor of each pair, or NULL (no screening)
    const double *dm_cond;    // [nbas*nbas] max |D| over each shell block, or NULL
    const double *dm;         // [n_dm][nao][nao]
    double *vj, *vk;          // [n_dm][nao][nao] accumulated (NULL disables)
    int nao, nbas, n_dm;
    double tol;               // drop quartets with q_ij q_kl max|D| < tol
    double tol_hi;            // and, when > 0, those with a bound >= tol_hi (FP32 band)
    int *status;              // device error word (0 = ok), may be NULL
    const double *rys;        // Rys coefficient table, interval-major (bqc_rys_table())
    const double *rys_lm;     // the same, level-major (bqc_rys_table_lm())
    // ERI output mode (GINTfill_int2e) when eri != NULL: no density screen,
    // no 1/2 for a == b, and instead of the J/K digestion every quartet adds
    // its block (ij|kl) at eri[sum_n (ao_n - eri_off[n]) * eri_stride[n]]
    double *eri;
    long long eri_stride[4];
    int eri_off[4];
};

// the same launch arguments with the bra and ket roles of the ERI output
// exchanged (a kernel that evaluates (kl|ij) for (ij|kl))
static inline JKArgs jk_args_swap_eri(const JKArgs &a) {
    JKArgs s = a;
    s.eri_stride[0] = a.eri_stride[2];
    s.eri_stride[1] = a.eri_stride[3];
    s.eri_stride[2] = a.eri_stride[0];
    s.eri_stride[3] = a.eri_stride[1];
    s.eri_off[0] = a.eri_off[2];
    s.eri_off[1] = a.eri_off[3];
    s.eri_off[2] = a.eri_off[0];
    s.eri_off[3] = a.eri_off[1];
    return s;
}

// One rectangular (or triangular, when diag) block of the quartet space: one
// class pair.
struct JKSub {
    int a0, na;        // bra pairs [a0, a0 + na) (global pair indices)
    int b0, nb;        // ket pairs
    int pa0, pb0;      // primitive-pair offset of the first bra / ket pair
    int nprim_a, nprim_b;  // primitive pairs per bra / ket pair
    int diag;          // bra and ket lists are the same: keep a >= b only
    int rows_are_b;    // tile rows run over the b list instead of the a list
    int row0;          // first tile row of the block among the launch's rows
    // parts a tile runs as (at least 1 each): ranges of its quartets (a power
    // of two up to 8) and of the primitive quartets
    int rparts, kparts;
    int kfirst;        // the range of the primitive quartets of a launch of one block
};

// A launch of one block runs whole tiles, or as many ranges of the primitive
// quartets, one after another, as keep their length within 32 bits (four shells
// of 216 primitives and more).
inline void whole_prims(JKSub &s) {
    s.rparts = 1;
    s.kparts = (int)(((long long)s.nprim_a * s.nprim_b >> 31) + 1);
}

// Parts of the tiles of a class pair with many primitive quartets: a part
// holds about PART_PRIMS primitive quartets per lane, first by fewer bra pairs
// and then by a range of the primitives (the integrals are linear in it).  A
// whole tile of two 6-primitive s pairs is 8 x 1296 primitive quartets in a
// row, which no other work of a build hides: C60H122 / 6-31G**, (ss|ss) of both
// precision bands, 32.9 -> 24.1 ms.  The schedule counts the parts of a tile row
// in 32 bits, so the rows of a long pair list get fewer and longer parts.
constexpr int PART_PRIMS = 64;

inline void split_prims(JKSub &s) {
    const long long n = (long long)s.nprim_a * s.nprim_b;
    const long long cols = ((s.na > s.nb ? s.na : s.nb) + 15LL) / 16;
    whole_prims(s);
    while (s.rparts < 8 && 8 / s.rparts * n > PART_PRIMS && 2 * s.rparts * s.kparts * cols <= 0x7fffffffLL)
        s.rparts *= 2;
    const long long parts = n / PART_PRIMS + (n % PART_PRIMS != 0), most = 0x7fffffffLL / (cols * s.rparts);
    if (parts > s.kparts) s.kparts = (int)(parts < most ? parts : most);
}

// Primitive quartets of range kpart of the kparts, bra pairs innermost: num from
// the ket pair k and bra pair i on.  The product n * kpart passes 32 bits from
// shells of 25 primitives on; undivided tiles take no division.
struct PrimRange {
    int k, i, num;
};

__host__ __device__ inline PrimRange prim_range(const JKSub &s, int kpart) {
    if (s.kparts == 1) return {0, 0, s.nprim_a * s.nprim_b};
    const long long n = (long long)s.nprim_a * s.nprim_b;
    const long long begin = n * kpart / s.kparts, k = begin / s.nprim_a;
    return {(int)k, (int)(begin - k * s.nprim_a), (int)(n * (kpart + 1) / s.kparts - begin)};
}

// the same block with bra and ket exchanged (a diagonal block has identical
// lists on both sides; the a >= b rule stays)
__host__ __device__ inline JKSub jk_swap_sub(const JKSub &s) {
    JKSub t = s;
    t.a0 = s.b0; t.na = s.nb; t.b0 = s.a0; t.nb = s.na;
    t.pa0 = s.pb0; t.pb0 = s.pa0; t.nprim_a = s.nprim_b; t.nprim_b = s.nprim_a;
    t.rows_are_b = !s.rows_are_b;
    return t;
}

// What one launch covers: one block, or all blocks of one class shape.
struct JKTask {
    JKSub sub;         // the block, when subs is NULL
    // Tile pruning.  Tiles are rows x columns of 16 x 16 quartets,
    // rows over the a list (or the b list when rows_are_b).  With
    // tile_prefix (device, nrows + 1 entries) row r holds the columns
    // [0, tile_prefix[r+1] - tile_prefix[r]) and block x maps to the tile
    // with tile_prefix[r] <= x < tile_prefix[r+1]; without it the grid is
    // the full rectangle.
    const long long *tile_prefix;
    const int *tile_col0;   // optional first column of each row (batched molecules)
    int nrows;
    long long ntiles;  // number of tiles when tile_prefix is set
    // All class pairs of one shape in one launch (device arrays): the rows of
    // the blocks follow one another, row_sub is the block of every row.
    const JKSub *subs;
    const int *row_sub;
    int swapped;       // read the blocks with bra and ket exchanged
    // K block (row shell, column shell): 0 bra shell x ket shell of the launched
    // orientation, 1 ket x bra.  Callers add the transpose, so either is right;
    // the flag keeps the stored halves of a class the same whichever
    // orientation its kernel runs in.
    int k_transposed;
    // Persistent launch: when set, the tile count lives on the device (a
    // schedule computed there) and a fixed grid of CTAs strides over the
    // tiles [0, *ntiles_dev); ntiles is then only an upper bound, and the
    // grid holds at most a few CTAs per SM of the nsm SMs.
    const long long *ntiles_dev;
    int nsm;
    union {
        // without ntiles_dev: parts per tile (set by the launcher; with
        // ntiles_dev the kernel derives it from the device count)
        int split;
        // with ntiles_dev: priority of the launch (0: that of its stream), for the
        // host alone.  Side streams have the default priority, their launches
        // that of the caller's stream.  In the same word because a larger argument
        // costs: with four more bytes (ss|ss) took 6.85 instead of 6.52 ms, (ps|ss)
        // 14.15 instead of 13.72 ms of a build of (H2O)_32 / cc-pVDZ, by the
        // register allocation they got.
        int priority;
    };
};

static inline JKTask jk_swap_task(const JKTask &t) {
    JKTask s = t;
    s.sub = jk_swap_sub(t.sub);
    s.swapped = !t.swapped;
    return s;
}

// Parts a group-kernel tile is cut into: a launch with fewer than 16 tiles
// per SM cuts each tile into 2, 4 or 8 interleaved parts (one CTA each), so
// that small builds still fill every SM; larger ones keep one CTA per tile.
__host__ __device__ inline int group_split(long long ntiles, int nsm) {
    int s = 1;
    while (s < 8 && ntiles * s < 16LL * nsm) s *= 2;
    return s;
}

// The same for the kernel that gives each warp a tile: parts until every SM
// has 32 warps, at most one per step over the tile's bra pairs.
__host__ __device__ inline int warp_split(long long ntiles, int nsm) {
    int s = 1;
    while (s < 8 && ntiles * s < 32LL * nsm) s *= 2;
    return s;
}

// grid of a launch over ntiles tiles of per_tile CTAs each; persistent
// launches cap it at ctas_per_sm CTAs on each SM
static inline int bqc_grid(const JKTask &t, long long ntiles, int per_tile, int ctas_per_sm) {
    const long long n = ntiles * per_tile;
    const long long cap = t.ntiles_dev == nullptr ? 0x7fffffffLL : (long long)t.nsm * ctas_per_sm;
    return (int)(n < cap ? n : cap);
}

// number of kernel launches issued by the library so far (all threads)
unsigned long long bqc_count_launch(int n);

// launch variant of a class (canonical order), see launch_class
#define BQC_VARIANT_AUTO 0
#define BQC_VARIANT_GROUP 1
#define BQC_VARIANT_SPLIT 2
int bqc_class_variant(int li, int lj, int lk, int ll);

// device addresses of the Rys coefficient tables on the current device
// (rys_table.cu): RYS_POLY, RYS_POLY_LM, and the Chebyshev series RYS_TABLE
const double *bqc_rys_table();
const double *bqc_rys_table_lm();
const double *bqc_rys_cheb();

// launchers (jk_dispatch.cu, schwarz.cu)
int bqc_launch_jk(int li, int lj, int lk, int ll, const JKArgs &args, const JKTask &task,
                  int fp32, cudaStream_t stream);
int bqc_launch_count(const JKArgs &args, const JKTask &task, unsigned long long *count,
                     cudaStream_t stream);
int bqc_launch_dm_cond(const double *dm, int n_dm, int nao, const int *ao_loc, int nbas,
                       double *dm_cond, cudaStream_t stream);
int bqc_launch_schwarz(int li, int lj, const JKArgs &args, int p0, int np, int pa0, int nprim,
                       double diag_fac, double *q_out, cudaStream_t stream);
