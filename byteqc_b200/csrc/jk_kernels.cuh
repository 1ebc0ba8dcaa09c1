// Kernel choice of a shell-quartet class (LI LJ | LK LL).  A launch covers
// blocks of the quartet space, bra pairs [a0, a0 + na) x ket pairs
// [b0, b0 + nb), cut into 16 x 16 tiles; every tile screens its 256 quartets
// on the device against q_ij q_kl max|D| >= tol (the six density blocks a
// quartet touches) and evaluates the survivors:
//
// * jk_warp: one thread per quartet, a tile per warp: the lanes hold ket pairs
//   and step over the bra pairs; the 2D integrals and the contracted quartet
//   block live in registers.
// * jk_group: the survivors are packed into a shared-memory list and each
//   takes a group of threads; a thread owns one bra component fi, a few fj
//   and the ket components.  Per primitive quartet the group evaluates the Rys
//   roots and the per-root 2D tables (VRR + HRR) cooperatively into shared
//   memory, then every thread accumulates its components.  Digestion: sums over
//   a thread's own components in registers, the rest through shared memory,
//   one FP64 atomic per output element.
//
// The per-quartet factors follow the reference (cuobc/lib/gvhf/g2e.cu:1021-1028,
// cuobc/lib/gint/pair_data.c:135-139): 1/2 when the bra and ket pairs are the
// same pair (a == b), and the 1/2 of a diagonal shell pair carried in e12.
#pragma once
#include "jk_group.cuh"
#include "jk_warp.cuh"

namespace bqc {

// Kernel choice per class (canonical order, bra pair index >= ket's):
// at most SMALL_NF Cartesian components: jk_warp; otherwise, when shell k
// splits into at most MAX_SPLIT ranges of fk whose blocks fit SMALL_NF,
// ket-split jk_warp launches or jk_group as bqc_class_variant()
// says (BQCset_class_variant; by default the split for classes of up to
// SPLIT_AUTO ranges); else jk_group.
constexpr int MAX_SPLIT = 3;
constexpr int SPLIT_AUTO = 3;

template <int L1, int L2, int L3, int L4>
static int launch_class(const JKArgs &args, const JKTask &task, int fp32, cudaStream_t stream) {
    constexpr int N12 = ncart(L1) * ncart(L2), N34 = ncart(L3) * ncart(L4);
    if constexpr (N12 * N34 <= SMALL_NF) {
        return launch_small<L1, L2, L3, L4>(args, task, fp32, stream);
    } else {
        constexpr int CK = SMALL_NF / (N12 * ncart(L4));
        constexpr int NCH = CK >= 1 ? cdiv(ncart(L3), CK) : 0;
        if constexpr (NCH >= 1 && NCH <= MAX_SPLIT) {
            const int v = bqc_class_variant(L1, L2, L3, L4);
            if (v == BQC_VARIANT_SPLIT || (v == BQC_VARIANT_AUTO && NCH <= SPLIT_AUTO))
                return launch_warp<L1, L2, L3, L4, CK>(args, task, fp32, stream);
        }
        // the task with bra and ket exchanged
        const JKTask sw = jk_swap_task(task);
        // an s-s ket pair against a large bra pair ((fd|ss), (ff|ss)): split
        // the bra's first shell instead, with bra and ket exchanged
        constexpr int CKS = SMALL_NF / (N34 * ncart(L2));
        constexpr int NCHS = (NCH == 0 && N34 == 1 && CKS >= 1) ? cdiv(ncart(L1), CKS) : 0;
        if constexpr (NCHS >= 1 && NCHS <= MAX_SPLIT) {
            const int v = bqc_class_variant(L1, L2, L3, L4);
            if (v == BQC_VARIANT_SPLIT || v == BQC_VARIANT_AUTO)
                return launch_warp<L3, L4, L1, L2, CKS>(jk_args_swap_eri(args), sw, fp32, stream);
        }
        // the orientation with fewer table loads per component on the thread side
        constexpr GroupShape G1 = group_shape(L1, L2, L3, L4), G2 = group_shape(L3, L4, L1, L2);
        // K blocks are stored for the smaller pair as the bra (k_transposed)
        if constexpr (G1.cost <= G2.cost) {
            JKTask t = task;
            t.k_transposed = N12 > N34;
            return launch_group<L1, L2, L3, L4, G1.tj, G1.nsplit>(args, t, fp32, stream);
        } else {
            JKTask t = sw;
            t.k_transposed = N12 <= N34;
            return launch_group<L3, L4, L1, L2, G2.tj, G2.nsplit>(jk_args_swap_eri(args), t, fp32, stream);
        }
    }
}

}  // namespace bqc
