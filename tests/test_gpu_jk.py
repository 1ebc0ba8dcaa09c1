"""Parity of the device J/K engine with the CPU oracle (needs a B200).

Tolerances: J and K max-abs error <= 1e-10 in plain FP64 (the bar of the
drop-in), SCF total energy within 1e-9 Eh.
"""
import numpy as np
import pytest

from byteqc_b200.gto.mole import Mole
from byteqc_b200.gto.basis import synthetic_basis, sto3g_like
from byteqc_b200.gto.geom import water_cluster, linear_alkane
from oracle import oracle

pytestmark = pytest.mark.gpu

TOL_JK = 1e-10


def _rand_dm(nao, seed=2341):
    # the density recipe of the reference's timing script: rand + rand^T
    rng = np.random.default_rng(seed)
    dm = rng.random((nao, nao))
    return dm + dm.T


def _mol(kind, nw=1, seed=3):
    atoms = water_cluster(nw, seed=seed)
    return Mole(atoms, synthetic_basis(kind, ['O', 'H']))


@pytest.mark.parametrize('kind', ['cc-pvdz', 'cc-pvtz'])
def test_jk_water(cuda, kind):
    from byteqc_b200.scf import hf
    mol = _mol(kind)
    dm = _rand_dm(mol.nao)
    vj, vk = hf.get_jk(mol, dm)
    rj, rk = oracle.get_jk(mol, dm)
    ej, ek = abs(vj - rj).max(), abs(vk - rk).max()
    print('water %s: max|J| %.3g max|dJ| %.3e max|dK| %.3e' % (kind, abs(rj).max(), ej, ek))
    assert ej < TOL_JK and ek < TOL_JK


@pytest.mark.parametrize('variant', [1, 2])
def test_jk_class_variants(cuda, variant):
    """Every class in the group kernel (1) or, where it splits, in ket-split
    tile launches (2): the same J/K as the oracle."""
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    lib = L.load_library()
    shapes = [(a, b, c, d) for a in range(4) for b in range(a + 1)
              for c in range(4) for d in range(c + 1)]
    try:
        for sh in shapes:
            assert lib.BQCset_class_variant(*sh, variant) == 0
        mol = _mol('cc-pvtz', nw=2, seed=4)
        dm = _rand_dm(mol.nao) * 0.1
        vj, vk = hf.get_jk(mol, dm)
    finally:
        for sh in shapes:
            lib.BQCset_class_variant(*sh, 0)
    rj, rk = oracle.get_jk(mol, dm)
    print('variant %d: max|dJ| %.3e max|dK| %.3e' % (variant, abs(vj - rj).max(), abs(vk - rk).max()))
    assert abs(vj - rj).max() < TOL_JK
    assert abs(vk - rk).max() < TOL_JK
    assert lib.BQCset_class_variant(0, 0, 0, 0, 7) == 3
    assert lib.BQCset_class_variant(4, 0, 0, 0, 1) == 2


def test_jk_batch_and_flags(cuda):
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz')
    dms = np.stack([_rand_dm(mol.nao, s) for s in (1, 2)])
    opt = hf._VHFOpt(mol).build()
    vj, vk = hf.get_jk(mol, dms, vhfopt=opt)
    assert vj.shape == dms.shape and vk.shape == dms.shape
    for i in range(2):
        rj, rk = oracle.get_jk(mol, dms[i])
        assert abs(vj[i] - rj).max() < TOL_JK
        assert abs(vk[i] - rk).max() < TOL_JK
    vj_only, vk_none = hf.get_jk(mol, dms[0], vhfopt=opt, with_k=False)
    assert vk_none is None and abs(vj_only - vj[0]).max() < 1e-12
    vj_none, vk_only = hf.get_jk(mol, dms[0], vhfopt=opt, with_j=False)
    assert vj_none is None and abs(vk_only - vk[0]).max() < 1e-12
    with pytest.raises(NotImplementedError):
        hf.get_jk(mol, dms[0], hermi=0, vhfopt=opt)
    with pytest.raises(NotImplementedError):
        hf.get_jk(mol, dms[0], vhfopt=opt, omega=0.3)


def test_jk_two_waters_tz(cuda):
    """Every s-f class pair of the TZ-shaped basis, inter-molecular pairs included."""
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvtz', nw=2, seed=5)
    dm = _rand_dm(mol.nao, 7)
    vj, vk = hf.get_jk(mol, dm)
    rj, rk = oracle.get_jk(mol, dm)
    ej, ek = abs(vj - rj).max(), abs(vk - rk).max()
    print('TZ dimer: max|J| %.3g max|dJ| %.3e max|dK| %.3e' % (abs(rj).max(), ej, ek))
    assert ej < TOL_JK and ek < TOL_JK


def test_schwarz_and_int1e(cuda):
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvtz')
    opt = hf._VHFOpt(mol).build()
    S, T, V = [x.cpu().numpy() for x in opt.int1e()]
    rS, rT, rV = oracle.int1e(mol)
    assert abs(S - rS).max() < 1e-12
    assert abs(T - rT).max() < 1e-10
    assert abs(V - rV).max() < 1e-10
    # Schwarz factors of the kept pairs against the oracle's (ij|ij)
    q = oracle.q_cond(opt.mol)
    real = ~opt.pair_dummy          # padding pairs of the tile layout carry q = 0
    p2s = opt.bas_pair2shls[:, real]
    dev_q = opt.pair_q.cpu().numpy()[real]
    ref = q[p2s[0], p2s[1]]
    assert np.allclose(dev_q, ref, rtol=1e-10, atol=1e-14)
    assert (opt.pair_q.cpu().numpy()[~real] == 0).all()


def test_gint_abi_matches_native(cuda):
    """The reference-ABI entry point GINTbuild_jk, driven the way
    cuobc/scf/hf.py drives it (class pairs x bins), equals the native build."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=2, seed=11)
    opt = hf._VHFOpt(mol).build()
    lib = L.load_library()
    dm = _rand_dm(mol.nao, 3)
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(dm, device=cuda) @ C.T)[None].contiguous()
    nao = dmc.shape[-1]
    vj = torch.zeros_like(dmc)
    vk = torch.zeros_like(dmc)
    # the native pair lists are laid out in shell-grouped tiles (q is not
    # globally sorted, padding pairs are interleaved), so drive GINTbuild_jk
    # with one bin that spans each whole class
    nbins = 1
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for cij in range(opt.ncptype):
        for ckl in range(cij + 1):
            if len(opt.log_qs[cij]) == 0 or len(opt.log_qs[ckl]) == 0:
                continue
            bi = np.array([0, len(opt.log_qs[cij])], dtype=np.int32)
            bk = np.array([0, len(opt.log_qs[ckl])], dtype=np.int32)
            err = lib.GINTbuild_jk(opt.bpcache, ctypes.c_void_p(vj.data_ptr()),
                                   ctypes.c_void_p(vk.data_ptr()), ctypes.c_void_p(dmc.data_ptr()),
                                   ctypes.c_int(nao), ctypes.c_int(1),
                                   bi.ctypes.data_as(ctypes.c_void_p),
                                   bk.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(nbins),
                                   ctypes.c_int(cij), ctypes.c_int(ckl), stream)
            assert err == 0
    J = 2 * (vj + vj.transpose(-1, -2))
    K = vk + vk.transpose(-1, -2)
    J = (C.T @ J[0] @ C).cpu().numpy()
    K = (C.T @ K[0] @ C).cpu().numpy()
    rj, rk = oracle.get_jk(mol, dm)
    print('GINT ABI: max|J| %.3g max|dJ| %.3e max|dK| %.3e' % (abs(rj).max(), abs(J - rj).max(),
                                                             abs(K - rk).max()))
    assert abs(J - rj).max() < TOL_JK
    assert abs(K - rk).max() < TOL_JK


def test_rhf_energy(cuda):
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=2, seed=1)
    mf = hf.RHF(mol)
    mf.conv_tol = 1e-10
    e = mf.kernel()
    assert mf.converged
    e_ref, _, _ = oracle.rhf(mol, conv_tol=1e-11)
    assert abs(e - e_ref) < 1e-9


def test_host_loop_matches_device_loop(cuda):
    """The drop-in arrangement (host numpy SCF loop, get_jk with host
    densities, host DIIS) converges to the device loop's energy, in plain
    FP64 and in the fast form."""
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=2, seed=1)
    for fast in (False, True):
        ms = []
        for host in (False, True):
            mf = hf.RHF(mol)
            mf.conv_tol = 1e-10
            if fast:
                mf.fp32_threshold = 1e-4
                mf.early_tol = 1e-10
            e = mf.kernel_hostloop() if host else mf.kernel()
            assert mf.converged
            ms.append(e)
        assert abs(ms[0] - ms[1]) < 1e-9, (fast, ms)


def test_uhf_closed_shell_equals_rhf(cuda):
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=1, seed=2)
    e_r = hf.RHF(mol).kernel()
    mf = hf.UHF(mol)
    e_u = mf.kernel()
    assert abs(e_r - e_u) < 1e-8


def test_alkane_631gss(cuda):
    from byteqc_b200.scf import hf
    mol = Mole(linear_alkane(2), synthetic_basis('6-31g**', ['C', 'H']))
    dm = _rand_dm(mol.nao, 5) * 0.1
    vj, vk = hf.get_jk(mol, dm)
    rj, rk = oracle.get_jk(mol, dm)
    print('ethane: max|J| %.3g max|dJ| %.3e max|dK| %.3e' % (abs(rj).max(), abs(vj - rj).max(),
                                                           abs(vk - rk).max()))
    assert abs(vj - rj).max() < TOL_JK
    assert abs(vk - rk).max() < TOL_JK


def test_mixed_precision_jk_error(cuda):
    """FP32 band below 1e-6: J/K error against the FP64 build stays small."""
    import torch
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvtz', nw=2, seed=5)
    opt = hf._VHFOpt(mol).build()
    rng = np.random.default_rng(8)
    dm = rng.random((mol.nao, mol.nao)) * 1e-3
    dm = torch.as_tensor(dm + dm.T, device=cuda)[None]
    vj0, vk0 = opt.jk_ao(dm)
    vj1, vk1 = opt.jk_ao(dm, fp32_below=1e-6)
    ej = float((vj1 - vj0).abs().max())
    ek = float((vk1 - vk0).abs().max())
    assert ej < 1e-9 and ek < 1e-9, (ej, ek)
    # every quartet is in the FP32 band: still within FP32 accuracy of FP64
    vj2, vk2 = opt.jk_ao(dm, fp32_below=1e30)
    assert float((vj2 - vj0).abs().max()) < 1e-5 * float(vj0.abs().max())
    assert float((vk2 - vk0).abs().max()) < 1e-5 * float(vk0.abs().max())


def test_mixed_precision_scf_energy(cuda):
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=3, seed=4)
    mf0 = hf.RHF(mol)
    mf0.conv_tol = 1e-10
    e0 = mf0.kernel()
    mf1 = hf.RHF(mol)
    mf1.conv_tol = 1e-10
    mf1.fp32_threshold = 1e-6
    e1 = mf1.kernel()
    mf2 = hf.RHF(mol)
    mf2.conv_tol = 1e-10
    mf2.fp32_threshold = 1e-6
    mf2.early_tol = 1e-10
    e2 = mf2.kernel()
    assert mf0.converged and mf1.converged and mf2.converged
    assert abs(e1 - e0) < 1e-9
    assert abs(e2 - e0) < 1e-9
    assert any(rec[1] > 0 for rec in mf1.build_log)


def test_autotune_keeps_results(cuda):
    """The autotuner picks kernels per class; J/K stay the same."""
    import torch
    from byteqc_b200 import autotune
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvtz', nw=2, seed=6)
    opt = hf._VHFOpt(mol).build()
    dm = torch.as_tensor(_rand_dm(mol.nao) * 0.1, device=cuda)[None]
    vj0, vk0 = opt.jk_ao(dm)
    try:
        choice = autotune.tune(opt, reps=1)
        assert choice and set(choice.values()) <= {1, 2}
        vj1, vk1 = opt.jk_ao(dm)
    finally:
        lib = L.load_library()
        for key in choice:
            lib.BQCset_class_variant(*key, 0)
    assert float((vj1 - vj0).abs().max()) < 1e-11
    assert float((vk1 - vk0).abs().max()) < 1e-11


@pytest.mark.parametrize('kind', ['cc-pvdz', 'cc-pvtz'])
def test_fill_int2e_matches_oracle(cuda, kind):
    """GINTfill_int2e (the ERI writer) over every ordered class pair writes
    the Cartesian (ij|kl) blocks of the listed pairs; they equal the oracle's
    integrals of the same decontracted, sorted basis."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _stream
    lib = L.load_library()
    mol = _mol(kind)
    opt = hf._VHFOpt(mol).build(diag_block_with_triu=True)
    pmol = opt.mol
    n = int(pmol.ao_loc_nr(cart=True)[-1])
    eri = torch.zeros((n, n, n, n), dtype=torch.float64, device=cuda)
    strides = np.array([n ** 3, n ** 2, n, 1], dtype=np.int32)
    offs = np.zeros(4, dtype=np.int32)
    locs = opt.bas_pairs_locs
    vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    for cij in range(opt.ncptype):
        for ckl in range(opt.ncptype):
            nij, nkl = locs[cij + 1] - locs[cij], locs[ckl + 1] - locs[ckl]
            if nij == 0 or nkl == 0:
                continue
            bi = np.array([0, nij], dtype=np.int32)
            bk = np.array([0, nkl], dtype=np.int32)
            err = lib.GINTfill_int2e(ctypes.cast(opt.bpcache, ctypes.c_void_p),
                                     ctypes.c_void_p(eri.data_ptr()), n, vp(strides), vp(offs),
                                     vp(bi), vp(bk), 1, cij, ckl, _stream())
            assert err == 0
    torch.cuda.synchronize()
    got = eri.cpu().numpy()
    ref = oracle.eri_full_cart(pmol)
    ao = pmol.ao_loc_nr(cart=True)
    keep = ~opt.pair_dummy
    pairs = [(int(i), int(j)) for i, j, kp in zip(*opt.bas_pair2shls, keep) if kp]
    mask = np.zeros((n, n), bool)
    for i, j in pairs:
        mask[ao[i]:ao[i + 1], ao[j]:ao[j + 1]] = True
    sel = mask[:, :, None, None] & mask[None, None, :, :]
    assert sel.sum() > 0
    err = abs(got[sel] - ref[sel]).max()
    assert err < 1e-10 * max(1., abs(ref).max()), err
    # nothing is written outside the listed pairs
    assert abs(got[~sel]).max() == 0
    # a missing output buffer is an argument error
    assert lib.GINTfill_int2e(ctypes.cast(opt.bpcache, ctypes.c_void_p), None, n, vp(strides),
                              vp(offs), vp(bi), vp(bk), 1, 0, 0, _stream()) == 3


@pytest.mark.parametrize('fp32_below', [0., 1e-6])
def test_device_schedule_matches_host_pruning(cuda, fp32_below):
    """BQCbuild_jk_plan (tiles pruned and counted on the device, persistent
    launches) gives the J/K of BQCbuild_jk (tiles pruned on the host) for
    two densities at once, with and without the FP32 band."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr, _stream
    lib = L.load_library()
    mol = _mol('cc-pvtz', nw=3, seed=12)
    opt = hf._VHFOpt(mol).build()
    rng = np.random.default_rng(3)
    d = rng.random((2, mol.nao, mol.nao)) * 1e-2
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(d + d.transpose(0, 2, 1), device=cuda) @ C.T).contiguous()
    nao = dmc.shape[-1]
    dm_cond = torch.empty((opt.mol.nbas, opt.mol.nbas), dtype=torch.float64, device=cuda)
    assert lib.BQCdm_cond(_ptr(dmc), 2, nao, _ptr(opt._mem['ao_loc']), opt.mol.nbas, _ptr(dm_cond),
                          _stream()) == 0
    out = []
    for plan in (False, True):
        vj = torch.zeros_like(dmc)
        vk = torch.zeros_like(dmc)
        if plan:
            err = lib.BQCbuild_jk_plan(opt._plan, _ptr(opt.pair_q), _ptr(dm_cond), _ptr(vj), _ptr(vk),
                                       _ptr(dmc), nao, 2, opt.direct_scf_tol, fp32_below, _stream())
        else:
            err = lib.BQCbuild_jk(ctypes.cast(opt.bpcache, ctypes.c_void_p), _ptr(opt.pair_q),
                                  opt.pair_q_host.ctypes.data_as(ctypes.c_void_p), _ptr(dm_cond),
                                  float(dm_cond.max()), _ptr(vj), _ptr(vk), _ptr(dmc), nao, 2,
                                  opt.direct_scf_tol, fp32_below, None, _stream())
        assert err == 0
        out.append((vj, vk))
    torch.cuda.synchronize()
    (j0, k0), (j1, k1) = out
    assert float((j1 - j0).abs().max()) < 1e-12 * max(1., float(j0.abs().max()))
    assert float((k1 - k0).abs().max()) < 1e-12 * max(1., float(k0.abs().max()))
    assert float(j0.abs().max()) > 0


def test_repeated_builds_agree(cuda):
    """Two builds of the same density differ only by the order of the FP64
    atomic additions: at most a few units in the last place of the largest
    element (bound 1e-13 relative)."""
    import torch
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvtz', nw=3, seed=13)
    opt = hf._VHFOpt(mol).build()
    dm = torch.as_tensor(_rand_dm(mol.nao, 17) * 0.1, device=cuda)[None]
    vj0, vk0 = opt.jk_ao(dm)
    vj1, vk1 = opt.jk_ao(dm)
    dj = float((vj1 - vj0).abs().max()) / float(vj0.abs().max())
    dk = float((vk1 - vk0).abs().max()) / float(vk0.abs().max())
    print('repeat: relative max|dJ| %.2e max|dK| %.2e' % (dj, dk))
    assert dj < 1e-13 and dk < 1e-13


@pytest.mark.parametrize('fp32_below', [0., 1e-6])
def test_build_is_ordered_on_the_callers_stream(cuda, fp32_below):
    """The build's launches run on side streams: they start after what the
    caller's stream holds before the call (here the late arrival of the
    density) and what follows on it sees every contribution.  Bound as in
    test_repeated_builds_agree, for two builds."""
    import torch
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=2, seed=21)
    opt = hf._VHFOpt(mol).build()
    dm = torch.as_tensor(_rand_dm(mol.nao, 5) * 0.1, device=cuda)[None]
    ref = opt.jk_ao(dm, fp32_below=fp32_below)
    torch.cuda.synchronize()
    big = torch.ones((4096, 4096), dtype=torch.float64, device=cuda)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        late = torch.zeros_like(dm)
        for _ in range(3):
            big = big @ big * 1e-4           # some milliseconds of work ahead of the copy
        late.copy_(dm)
        vj, vk = opt.jk_ao(late, fp32_below=fp32_below)
        late.zero_()
        vj, vk = vj.clone(), vk.clone()
    s.synchronize()
    for a, b in zip((vj, vk), ref):
        assert float((a - b).abs().max()) < 1e-13 * float(b.abs().max())


@pytest.mark.parametrize('nc,n_dm,fp32_below', [(1, 1, 0.), (3, 1, 0.), (3, 2, 0.), (3, 1, 1e-6)])
def test_primitive_parts_match_whole_tiles(cuda, nc, n_dm, fp32_below):
    """A plan cuts the tiles of strongly contracted class pairs into ranges of
    their primitive quartets (up to 1296 for two pairs of 6-primitive s
    shells); the host-scheduled build runs whole tiles.  Same sums in another
    order: the bound of test_device_schedule_matches_host_pruning."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr, _stream
    lib = L.load_library()
    mol = Mole(linear_alkane(nc), synthetic_basis('6-31g**', ['C', 'H']))
    opt = hf._VHFOpt(mol).build()
    d = np.stack([_rand_dm(mol.nao, s) for s in range(n_dm)]) * 0.1
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(d, device=cuda) @ C.T).contiguous()
    nao = dmc.shape[-1]
    cond = torch.empty((opt.mol.nbas, opt.mol.nbas), dtype=torch.float64, device=cuda)
    assert lib.BQCdm_cond(_ptr(dmc), n_dm, nao, _ptr(opt._mem['ao_loc']), opt.mol.nbas, _ptr(cond),
                          _stream()) == 0
    out = []
    for plan in (False, True):
        vj, vk = torch.zeros_like(dmc), torch.zeros_like(dmc)
        if plan:
            err = lib.BQCbuild_jk_plan(opt._plan, _ptr(opt.pair_q), _ptr(cond), _ptr(vj), _ptr(vk),
                                       _ptr(dmc), nao, n_dm, opt.direct_scf_tol, fp32_below, _stream())
        else:
            err = lib.BQCbuild_jk(ctypes.cast(opt.bpcache, ctypes.c_void_p), _ptr(opt.pair_q),
                                  opt.pair_q_host.ctypes.data_as(ctypes.c_void_p), _ptr(cond),
                                  float(cond.max()), _ptr(vj), _ptr(vk), _ptr(dmc), nao, n_dm,
                                  opt.direct_scf_tol, fp32_below, None, _stream())
        assert err == 0
        out.append((vj, vk))
    torch.cuda.synchronize()
    for a, b in zip(*out):
        assert float(a.abs().max()) > 0
        # FP32 integrals are summed over the primitives in FP32: their order
        # changes them by their rounding, 1e-7 of quartets below 1e-6
        tol = 1e-12 * max(1., float(a.abs().max())) if fp32_below == 0. else 1e-10
        assert float((a - b).abs().max()) < tol


def _contracted(shells, n):
    """H2 with contracted shells [(l, number of primitives)] on each atom,
    the second atom's exponents shifted."""
    rng = np.random.default_rng(n)
    basis = {}
    for sym, shift in (('H', 1.), ('He', 1.3)):
        basis[sym] = [[l] + [[shift * .08 * 400. ** (i / max(k - 1, 1)), float(rng.uniform(.2, 1.))]
                             for i in range(k)] for l, k in shells]
    return Mole([('H', (0., 0., 0.)), ('He', (.3, -.2, .7))], basis)


@pytest.mark.parametrize('shells', [[(0, 25), (1, 1)], [(0, 3), (1, 3), (2, 3), (3, 3)], [(1, 2), (2, 7)]])
def test_deep_contractions(cuda, shells):
    """Ranges of the primitive quartets: 25^4 = 390,625 primitive quartets, the
    first number whose products with the range index pass 32 bits, and the
    contracted d and f classes of the group kernel.  J/K against the oracle and
    the plan against the host-scheduled whole tiles, the latter as in
    test_primitive_parts_match_whole_tiles."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr, _stream
    lib = L.load_library()
    mol = _contracted(shells, 11)
    opt = hf._VHFOpt(mol).build()
    dm = _rand_dm(mol.nao, 9) * .1
    vj, vk = hf.get_jk(mol, dm, vhfopt=opt)
    rj, rk = oracle.get_jk(mol, dm)
    scale = max(1., abs(rj).max() / 100)
    print('deep %s: max|J| %.3g max|dJ| %.3e max|dK| %.3e' % (shells, abs(rj).max(), abs(vj - rj).max(), abs(vk - rk).max()))
    assert abs(vj - rj).max() < TOL_JK * scale and abs(vk - rk).max() < TOL_JK * scale
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(dm, device=cuda) @ C.T)[None].contiguous()
    cond = torch.empty((opt.mol.nbas, opt.mol.nbas), dtype=torch.float64, device=cuda)
    assert lib.BQCdm_cond(_ptr(dmc), 1, dmc.shape[-1], _ptr(opt._mem['ao_loc']), opt.mol.nbas, _ptr(cond),
                          _stream()) == 0
    wj, wk = torch.zeros_like(dmc), torch.zeros_like(dmc)
    assert lib.BQCbuild_jk(ctypes.cast(opt.bpcache, ctypes.c_void_p), _ptr(opt.pair_q),
                           opt.pair_q_host.ctypes.data_as(ctypes.c_void_p), _ptr(cond), float(cond.max()),
                           _ptr(wj), _ptr(wk), _ptr(dmc), dmc.shape[-1], 1, opt.direct_scf_tol, 0., None,
                           _stream()) == 0
    pj, pk = torch.zeros_like(dmc), torch.zeros_like(dmc)
    assert lib.BQCbuild_jk_plan(opt._plan, _ptr(opt.pair_q), _ptr(cond), _ptr(pj), _ptr(pk), _ptr(dmc),
                                dmc.shape[-1], 1, opt.direct_scf_tol, 0., _stream()) == 0
    torch.cuda.synchronize()
    for a, b in ((wj, pj), (wk, pk)):
        assert float(a.abs().max()) > 0
        assert float((a - b).abs().max()) < 1e-12 * max(1., float(a.abs().max()))


@pytest.mark.parametrize('kind,bra,ket', [('cc-pvdz', (2, 0), (1, 1)), ('cc-pvdz', (2, 1), (1, 0)),
                                          ('cc-pvdz', (1, 1), (2, 2)),
                                          ('cc-pvdz', (1, 0), (2, 2)), ('cc-pvtz', (3, 0), (1, 1)),
                                          ('cc-pvtz', (1, 1), (3, 3)), ('cc-pvtz', (2, 0), (3, 3))])
def test_stored_half_of_k(cuda, kind, bra, ket):
    """V holds a class's exchange contributions with the rows at the shells of
    its bra pair, whichever orientation the kernel runs in: (2, 2) and (3, 3)
    pairs with a larger component count are the ket of the smaller pair in
    the group kernel, (2, 2) pairs the bra of (1, 0) in the split launches."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr, _stream
    lib = L.load_library()
    mol = _mol(kind, nw=2, seed=8)
    opt = hf._VHFOpt(mol).build()
    if bra == (1, 0) and ket == (2, 2):
        bra, ket = ket, bra
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(_rand_dm(mol.nao, 3), device=cuda) @ C.T)[None].contiguous()
    nao = dmc.shape[-1]
    l_of = np.repeat(opt.mol._bas[:, 1], (opt.mol._bas[:, 1] + 1) * (opt.mol._bas[:, 1] + 2) // 2)
    vk = torch.zeros_like(dmc)
    n = 0
    for ci in range(opt.ncptype):
        for ck in range(ci + 1):
            a, b = opt.cptype[ci][:2], opt.cptype[ck][:2]
            if sorted([a, b]) != sorted([bra, ket]) or not (opt.cptype[ci][3] and opt.cptype[ck][3]):
                continue
            assert lib.BQCbuild_jk_class(ctypes.cast(opt.bpcache, ctypes.c_void_p), ci, ck, _ptr(opt.pair_q),
                                         opt.pair_q_host.ctypes.data_as(ctypes.c_void_p), None, 1., None,
                                         _ptr(vk), _ptr(dmc), nao, 1, opt.direct_scf_tol ** 2, 0., None,
                                         _stream()) == 0
            n += 1
    torch.cuda.synchronize()
    K = vk[0].cpu().numpy()
    rows = np.isin(l_of, bra)
    cols = np.isin(l_of, ket)
    assert n > 0 and abs(K[np.ix_(rows, cols)]).max() > 0
    assert abs(K[~rows]).max() == 0 and abs(K[:, ~cols]).max() == 0


@pytest.mark.parametrize('n_dm,fp32_below', [(1, 0.), (2, 0.), (1, 1e-6)])
def test_screened_quartets_touch_no_density(cuda, n_dm, fp32_below):
    """A quartet that is screened out contributes nothing, whatever the density
    holds: with q = 0 for every pair of two shells (an s and a p shell, so that
    every other quartet survives) NaN in their rows and columns leaves the
    result as zeros there do.  Bound as in test_repeated_builds_agree."""
    import ctypes
    import torch
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr, _stream
    lib = L.load_library()
    mol = _mol('cc-pvdz', nw=2, seed=31)
    opt = hf._VHFOpt(mol).build()
    C = opt.coeff_dev
    dm = np.stack([_rand_dm(mol.nao, s) for s in range(n_dm)]) * .1
    dmc = (C @ torch.as_tensor(dm, device=cuda) @ C.T).contiguous()
    nao, loc = dmc.shape[-1], opt.mol.ao_loc_nr(cart=True)
    l_of = opt.mol._bas[:, 1]
    shells = [int(np.flatnonzero(l_of == 0)[2]), int(np.flatnonzero(l_of == 1)[1])]
    rows = np.concatenate([np.arange(loc[s], loc[s + 1]) for s in shells])
    q = opt.pair_q.clone()
    q[torch.as_tensor(np.isin(opt.bas_pair2shls, shells).any(0), device=cuda)] = 0.
    dmc[:, rows] = 0.
    dmc[:, :, rows] = 0.
    cond = torch.empty((opt.mol.nbas, opt.mol.nbas), dtype=torch.float64, device=cuda)
    assert lib.BQCdm_cond(_ptr(dmc), n_dm, nao, _ptr(opt._mem['ao_loc']), opt.mol.nbas, _ptr(cond),
                          _stream()) == 0
    bad = dmc.clone()
    bad[:, rows] = float('nan')
    bad[:, :, rows] = float('nan')
    for plan in (False, True):
        out = []
        for d in (dmc, bad):
            vj, vk = torch.zeros_like(d), torch.zeros_like(d)
            if plan:
                err = lib.BQCbuild_jk_plan(opt._plan, _ptr(q), _ptr(cond), _ptr(vj), _ptr(vk), _ptr(d), nao,
                                           n_dm, opt.direct_scf_tol, fp32_below, _stream())
            else:
                err = lib.BQCbuild_jk(ctypes.cast(opt.bpcache, ctypes.c_void_p), _ptr(q),
                                      opt.pair_q_host.ctypes.data_as(ctypes.c_void_p), _ptr(cond),
                                      float(cond.max()), _ptr(vj), _ptr(vk), _ptr(d), nao, n_dm,
                                      opt.direct_scf_tol, fp32_below, None, _stream())
            assert err == 0
            out.append((vj, vk))
        torch.cuda.synchronize()
        for a, b in zip(*out):
            assert float(a.abs().max()) > 0 and bool(torch.isfinite(b).all())
            assert float((a - b).abs().max()) < 1e-13 * float(a.abs().max())


def test_plan_reads_the_cache_at_the_build(cuda):
    """A build takes the cache's device arrays as they are on the caller's
    stream, as BQCbuild_jk does, not as they were when the plan was made: twice
    the pair factors e12, written behind some milliseconds of other work, give
    four times the integrals.  Bound as in test_repeated_builds_agree."""
    import torch
    from byteqc_b200.scf import hf
    mol = _mol('cc-pvdz', nw=2, seed=41)
    opt = hf._VHFOpt(mol).build()
    dm = torch.as_tensor(_rand_dm(mol.nao, 5) * 0.1, device=cuda)[None]
    ref = opt.jk_ao(dm)
    torch.cuda.synchronize()
    big = torch.ones((4096, 4096), dtype=torch.float64, device=cuda)
    e12 = opt._mem['aexyz'].view(5, -1)[1]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(3):
            big = big @ big * 1e-4
        e12 *= 2.
        got = opt.jk_ao(dm)
        e12 *= .5
        again = opt.jk_ao(dm)
    s.synchronize()
    for a, b, c in zip(ref, got, again):
        assert float((4. * a - b).abs().max()) < 1e-13 * float(b.abs().max())
        assert float((a - c).abs().max()) < 1e-13 * float(a.abs().max())


def test_plans_at_once_and_after_one_another(cuda):
    """Two plans' builds in flight on two streams, one plan destroyed and its
    streams and memory taken by a larger and by a smaller molecule's, more plans
    alive than sets are kept: each gives its own result.  Bound as in
    test_repeated_builds_agree."""
    import torch
    from byteqc_b200.scf import hf
    mols = [_mol('cc-pvdz', nw=n, seed=50 + n) for n in (1, 3, 2)]
    dms = [torch.as_tensor(_rand_dm(m.nao, n) * .1, device=cuda)[None] for n, m in enumerate(mols)]
    refs = [hf._VHFOpt(m).build().jk_ao(d) for m, d in zip(mols, dms)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in mols]

    def start(n, opt):
        with torch.cuda.stream(streams[n]):
            return opt.jk_ao(dms[n])

    def check(n, out):
        streams[n].synchronize()
        for a, b in zip(refs[n], out):
            assert float((a - b).abs().max()) < 1e-13 * float(a.abs().max())
    for first, second, third in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        a, b = hf._VHFOpt(mols[first]).build(), hf._VHFOpt(mols[second]).build()
        out_a, out_b = start(first, a), start(second, b)
        a.clear()
        c = hf._VHFOpt(mols[third]).build()
        out_c, again_b = start(third, c), start(second, b)
        check(first, out_a)
        check(second, out_b)
        check(second, again_b)
        check(third, out_c)
    many = [hf._VHFOpt(mols[n % 3]).build() for n in range(6)]
    outs = [start(n % 3, opt) for n, opt in enumerate(many)]
    for n, out in enumerate(outs):
        check(n % 3, out)


def test_build_keeps_the_priority_of_the_callers_stream(cuda):
    """The launches on the side streams run at the priority of the caller's
    stream: read off the kernel nodes of a captured build."""
    import torch
    from cuda.bindings import runtime as rt
    from byteqc_b200 import lib as L
    from byteqc_b200.scf import hf
    from byteqc_b200.scf.hf import _ptr
    import ctypes
    lib = L.load_library()
    mol = _mol('cc-pvdz', nw=1, seed=2)
    opt = hf._VHFOpt(mol).build()
    C = opt.coeff_dev
    dmc = (C @ torch.as_tensor(_rand_dm(mol.nao), device=cuda) @ C.T)[None].contiguous()
    cond = torch.ones((opt.mol.nbas, opt.mol.nbas), dtype=torch.float64, device=cuda)
    vj, vk = torch.zeros_like(dmc), torch.zeros_like(dmc)
    def build(s):
        assert lib.BQCbuild_jk_plan(opt._plan, _ptr(opt.pair_q), _ptr(cond), _ptr(vj), _ptr(vk), _ptr(dmc),
                                    dmc.shape[-1], 1, opt.direct_scf_tol, 1e-6, ctypes.c_void_p(s.cuda_stream)) == 0
    for priority in (0, -1):
        s = torch.cuda.Stream(priority=priority)
        s.wait_stream(torch.cuda.current_stream())
        build(s)
        s.synchronize()
        mode = rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal
        assert rt.cudaStreamBeginCapture(s.cuda_stream, mode)[0] == 0
        build(s)
        err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
        assert err == 0
        _, _, n = rt.cudaGraphGetNodes(graph)
        _, nodes, n = rt.cudaGraphGetNodes(graph, n)
        kernels = [x for x in nodes[:n]
                   if rt.cudaGraphNodeGetType(x)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel]
        got = [rt.cudaGraphKernelNodeGetAttribute(x, rt.cudaLaunchAttributeID.cudaLaunchAttributePriority)[1].priority
               for x in kernels]
        assert rt.cudaGraphDestroy(graph)[0] == 0
        assert len(got) > 20 and set(got) == {priority}
