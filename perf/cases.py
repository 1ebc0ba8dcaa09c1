"""Measured workloads of the direct-SCF engine.

Every case is one call, or one short sequence of calls, that a program built on
this package makes: a J/K build through ``get_jk`` (host arrays in and out, as a
host SCF loop calls it) or through ``_VHFOpt.jk_ao`` (device tensors, as the
device SCF loop calls it), the batched build of many molecules, the 3-centre
integrals of density fitting, and a complete small SCF.  Systems are the ones
of the repository's own benchmark and tests: water clusters in the cc-pVDZ and
cc-pVTZ shapes and all-trans alkanes in the 6-31G** shape.

The pair lists, Schwarz factors and plans (``_VHFOpt.build``) belong to the
molecule and are kept over all cycles of an SCF, so they are made in
``prepare``; the complete SCF contains that set-up, the one-electron integrals
and the guess too.

``exact`` evaluates every quartet in 64 bits with the McMurchie-Davidson scheme
over the primitive Cartesian functions in torch, independently of the package's
Rys kernels, without any screening.
"""
import math

import numpy as np
import torch

from byteqc_b200.gto.basis import synthetic_aux_basis, synthetic_basis
from byteqc_b200.gto.geom import linear_alkane, water_cluster
from byteqc_b200.gto.mole import Mole
from byteqc_b200.scf import hf

BASES = {'dz': 'cc-pvdz', 'tz': 'cc-pvtz', 'pople': '6-31g**'}


def _case(name, kind, system, k, basis, **opts):
    # distance: lattice spacing of the waters or C-C bond of the chain, Angstrom
    c = {'kind': kind, 'system': system, 'k': k, 'basis': basis, 'ndm': 1, 'density': 'full',
         'with_j': True, 'with_k': True, 'fp32_below': 0., 'tol': 0.,
         'distance': 3.1 if system == 'water' else 1.54}
    c.update(opts)
    if name is not None:
        c['name'] = name
    return c


def listed():
    return [
        # one molecule: the smallest call, an atom-count scan or a dissociation
        # curve; launches and host round trips
        _case('get_jk water1 dz', 'get_jk', 'water', 1, 'dz'),
        # the four-water reference system (96 AO) of the host-driven SCF
        _case('get_jk water4 dz', 'get_jk', 'water', 4, 'dz'),
        # a dimer with every class from s to f, one cycle of a host SCF loop
        _case('get_jk water2 tz', 'get_jk', 'water', 2, 'tz'),
        # difference spin densities of one unrestricted cycle (two densities)
        _case('jk uhf water7 dz', 'jk_ao', 'water', 7, 'dz', ndm=2, density='diff'),
        # a medium cluster, full first build
        _case('jk water32 dz', 'jk_ao', 'water', 32, 'dz'),
        # s-f classes at a size where the tiles fill the chip: full FP64 build
        _case('jk water11 tz', 'jk_ao', 'water', 11, 'tz'),
        # incremental build of the mixed-precision SCF: difference density,
        # FP32 band below 1e-4, early screen at 1e-10
        _case('jk mixed water24 tz', 'jk_ao', 'water', 24, 'tz', density='diff', fp32_below=1e-4,
              tol=1e-10),
        # contracted shells (up to 6 primitives) of a long chain, FP32 band 1e-6
        _case('jk mixed C60H122 pople', 'jk_ao', 'alkane', 60, 'pople', fp32_below=1e-6),
        # Coulomb matrix alone: functionals without exact exchange
        _case('j alkane20 pople', 'jk_ao', 'alkane', 20, 'pople', with_k=False),
        # many independent small molecules in one build
        _case('batched 16 waters dz', 'batched', 'water', 8, 'dz', nmol=16),
        # 3-centre integrals of density fitting over all class blocks
        _case('df int3c water3 dz', 'df', 'water', 3, 'dz'),
        # a complete restricted SCF, set-up and guess included
        _case('rhf water4 dz', 'rhf', 'water', 4, 'dz'),
    ]


def draw(rng):
    c = _draw(rng)
    c['distance'] = round(rng.uniform(3., 3.5) if c['system'] == 'water' else rng.uniform(1.5, 1.58), 3)
    return c


def _draw(rng):
    def size(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + .49))))))
    kind = rng.choice(['get_jk', 'get_jk', 'jk_ao', 'jk_ao', 'jk_ao', 'jk_ao', 'batched', 'df', 'rhf'])
    if kind == 'get_jk':
        basis = rng.choice(['dz', 'tz', 'pople'])
        system = 'alkane' if basis == 'pople' else 'water'
        k = size(1, {'dz': 12, 'tz': 5, 'pople': 12}[basis])
        return _case(None, kind, system, k, basis, density=rng.choice(['full', 'diff']))
    if kind == 'jk_ao':
        basis = rng.choice(['dz', 'tz', 'pople'])
        system = 'alkane' if basis == 'pople' else 'water'
        k = size(*{'dz': (3, 32), 'tz': (2, 12), 'pople': (4, 40)}[basis])
        c = _case(None, kind, system, k, basis, density=rng.choice(['full', 'diff']))
        form = rng.choice(['plain', 'plain', 'mixed', 'early', 'uhf', 'j', 'k'])
        if form == 'mixed':
            c['fp32_below'] = 1e-6
        elif form == 'early':
            c['fp32_below'], c['tol'] = 1e-4, 1e-10
        elif form == 'uhf':
            c['ndm'] = 2
        elif form == 'j':
            c['with_k'] = False
        elif form == 'k':
            c['with_j'] = False
        return c
    if kind == 'batched':
        return _case(None, kind, 'water', size(2, 10), 'dz', nmol=size(3, 24))
    system, basis = rng.choice([('water', 'dz'), ('alkane', 'pople')])
    if kind == 'df':
        return _case(None, kind, system, size(1, 4), basis)
    return _case(None, kind, system, size(1, 7), basis)


# ---------------------------------------------------------------------------
# inputs

_BASIS = {}


def _basis(name, elements):
    key = (name, elements)
    if key not in _BASIS:
        _BASIS[key] = synthetic_basis(BASES[name], list(elements))
    return _BASIS[key]


def _mol(case, seed):
    if case['system'] == 'water':
        return Mole(water_cluster(case['k'], seed=seed, spacing=case['distance']),
                    _basis(case['basis'], ('O', 'H')))
    # the ideal chain, its atoms moved by up to 0.02 Angstrom as in a relaxed or
    # sampled geometry
    rng = np.random.default_rng(seed)
    chain = linear_alkane(case['k'], rcc=case['distance'])
    atoms = [(s, tuple(np.add(xyz, rng.uniform(-.02, .02, 3)))) for s, xyz in chain]
    return Mole(atoms, _basis(case['basis'], ('C', 'H')))


def _aux(mol):
    return Mole(mol.atom, synthetic_aux_basis(sorted({s for s, _ in mol.atom})))


def _density(mol, seed, kind, ndm):
    """Symmetric densities whose blocks fall off with the distance of the atoms
    as those of an insulator do: 'full' as a whole density, 'diff' as the
    difference of two successive ones (smaller, longer ranged)."""
    rng = np.random.default_rng(seed + 1)
    amp, reach = (.1, 1.5) if kind == 'full' else (.02, 2.5)
    sl = mol.aoslice_by_atom()
    at = np.repeat(np.arange(mol.natm), sl[:, 3] - sl[:, 2])
    r = mol.atom_coords()
    decay = np.exp(-np.linalg.norm(r[:, None] - r[None], axis=-1) / reach)[at][:, at]
    dms = []
    for _ in range(ndm):
        d = rng.standard_normal((mol.nao, mol.nao))
        d = amp * (d + d.T) * decay
        if kind == 'full':
            d[np.arange(mol.nao), np.arange(mol.nao)] += .5
        dms.append(d)
    return np.stack(dms)


def _batch(case, seed):
    ks = np.round(np.linspace(1, case['k'], case['nmol']))
    return [Mole(water_cluster(int(k), seed=seed * 64 + i, spacing=case['distance']), _basis(case['basis'], ('O', 'H')))
            for i, k in enumerate(ks)]


def prepare(case, seed):
    dev = torch.device('cuda')
    if case['kind'] == 'batched':
        from byteqc_b200.scf.batched import BatchedVHFOpt
        mols = _batch(case, seed)
        opt = BatchedVHFOpt(mols).build()
        dmc = torch.zeros((1, opt.nao_cart, opt.nao_cart), dtype=torch.float64, device=dev)
        for b, m in enumerate(mols):
            c = opt.coeffs[b]
            d = c @ _density(m, seed + b, case['density'], 1)[0] @ c.T
            sl = slice(opt.ao_off[b], opt.ao_off[b + 1])
            dmc[0, sl, sl] = torch.as_tensor(d, device=dev)
        return {'kind': 'batched', 'opt': opt, 'dm': dmc}
    mol = _mol(case, seed)
    if case['kind'] == 'rhf':
        return {'kind': 'rhf', 'mol': mol}
    if case['kind'] == 'df':
        from byteqc_b200.df import int3c
        return {'kind': 'df', 'opt': int3c.VHFOpt3c(mol, _aux(mol)).build()}
    dm = _density(mol, seed, case['density'], case['ndm'])
    state = {'kind': case['kind'], 'mol': mol, 'opt': hf._VHFOpt(mol).build(),
             'flags': {'with_j': case['with_j'], 'with_k': case['with_k'],
                       'fp32_below': case['fp32_below'], 'tol': case['tol'] or None}}
    state['dm'] = dm[0] if case['kind'] == 'get_jk' else torch.as_tensor(dm, device=dev)
    return state


def run(state):
    kind = state['kind']
    if kind == 'get_jk':
        vj, vk = hf.get_jk(state['mol'], state['dm'], vhfopt=state['opt'], **state['flags'])
        return {'j': vj, 'k': vk}
    if kind == 'jk_ao':
        vj, vk = state['opt'].jk_ao(state['dm'], **state['flags'])
        return {n: v for n, v in (('j', vj), ('k', vk)) if v is not None}
    if kind == 'batched':
        vj, vk = state['opt'].jk_cart(state['dm'])
        return {'j': vj, 'k': vk}
    if kind == 'df':
        from byteqc_b200.df import int3c
        return {'int3c': int3c.int3c_ao(state['opt'])}
    mf = hf.RHF(state['mol'])
    e = mf.kernel()
    return {'e': np.array(e), 'mo_energy': mf.mo_energy, 'dm': mf.dm}


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _pair_groups(mol):
    """(l, nprim) of every shell as a J/K build sees it: contracted shells of
    several contractions split into their primitives."""
    out = []
    for l, nprim, nctr in mol._bas[:, [1, 2, 3]]:
        out += [(int(l), int(nprim))] if nctr == 1 else [(int(l), 1)] * int(nprim)
    return out


def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _quartet_flops(a, b, c, d, ndm):
    """Rys quadrature with roots and recurrences counted once, then the
    contraction with the densities, for one quartet of (l, nprim) shells."""
    (la, pa), (lb, pb), (lc, pc), (ld, pd) = a, b, c, d
    lij, lkl = la + lb, lc + ld
    n = (lij + lkl) // 2 + 1
    nf = _ncart(la) * _ncart(lb) * _ncart(lc) * _ncart(ld)
    prim = n * (15 * (lij + 1) * (lkl + 1) + 3 * nf) + 30
    return pa * pb * pc * pd * prim + 12 * nf * ndm


def _jk_flops(mol, ndm, part):
    """Shell quartets whose bra and ket pairs both overlap (atoms within 12
    Bohr of each other), times their average cost; a third of the contraction
    for J alone."""
    groups = _pair_groups(mol)
    atoms = np.repeat(mol._bas[:, 0], [1 if c == 1 else p for p, c in mol._bas[:, [2, 3]]])
    r = mol.atom_coords()[atoms]
    near = np.linalg.norm(r[:, None] - r[None], axis=-1) < 12.
    kinds = sorted(set(groups))
    gid = np.array([kinds.index(g) for g in groups])
    npair = {}
    for p in range(len(kinds)):
        for q in range(p + 1):
            n = near[np.ix_(gid == p, gid == q)].sum()
            npair[p, q] = n / 2. if p == q else float(n)
    keys, f = list(npair), 0.
    for x, (p, q) in enumerate(keys):
        for y in range(x + 1):
            u, v = keys[y]
            n = npair[p, q] * npair[u, v] * (.5 if x == y else 1.)
            # pairs, and then quartets, that survive the Schwarz and density
            # screening: about one in four of the overlapping ones per pair list
            f += n * _quartet_flops(kinds[p], kinds[q], kinds[u], kinds[v], ndm * part)
    many = min(1., (24. / max(mol.natm, 1)) ** .5)
    return f * .25 * many


def work(case):
    if case['kind'] == 'batched':
        mols = _batch(case, 0)
        f = sum(_jk_flops(m, 1, 1.) for m in mols)
        n = sum(m.nao_cart() ** 2 for m in mols)
        return {'bytes': 3 * 8 * n, 'flops': f}
    mol = _mol(case, 0)
    n = mol.nao
    if case['kind'] == 'df':
        aux = _aux(mol)
        na = aux.nao_cart()
        nc = sum(_ncart(l) for l, _ in _pair_groups(mol))
        return {'bytes': 8 * n * n * aux.nao, 'flops': 9. * nc * nc / 2 * na}
    if case['kind'] == 'rhf':
        # some ten cycles of a build, an eigensolve and a dozen products
        return {'bytes': 10 * 8 * 6 * n * n,
                'flops': 10 * (_jk_flops(mol, 1, 1.) + 12 * 2. * n ** 3 + 10. * n ** 3)}
    out = int(case['with_j']) + int(case['with_k'])
    part = (case['with_j'] + 2 * case['with_k']) / 3.
    return {'bytes': 8 * n * n * case['ndm'] * (1 + out), 'flops': _jk_flops(mol, case['ndm'], part)}


def tolerance(case):
    """About four times what was measured.  FP64 against a build with the
    thresholds at 1e-15 instead of 1e-13: up to 5e-12 (the quartets dropped);
    the FP32 band below 1e-6 adds less than that.  FP32 band below 1e-4 with
    the early screen at 1e-10 against plain FP64: 1.3e-8.  An SCF that stops
    at |dE| < 1e-9 against one cycle more: 2.3e-6 in the density."""
    if case['kind'] == 'rhf':
        return {'rel': 1e-5, 'max': 2e-4}
    if case['tol']:
        return {'rel': 5e-8, 'max': 2e-6}
    return {'rel': 2e-11, 'max': 3e-10}


# ---------------------------------------------------------------------------
# 64-bit reference: McMurchie-Davidson over primitive Cartesian functions

PRIM_MAX = 180     # n^4 primitive integrals: 180 takes some seconds


def _cart(l):
    return [(a, b, l - a - b) for a in range(l, -1, -1) for b in range(l - a, -1, -1)]


def _primitives(mol):
    """Primitive Cartesian shells of mol by l: {l: (centres, exponents, first
    function)} and C (nprim functions x nao) with AO = primitive @ C."""
    by_l, blocks, rows = {}, [], 0
    coords = mol.atom_coords()
    for ia, l, nprim, nctr, _, pe, pc, _ in mol._bas:
        exps = mol._env[pe:pe + nprim]
        c = mol._env[pc:pc + nprim * nctr].reshape(nctr, nprim)
        if l < 2:
            c = c * (math.sqrt(.25 / math.pi) if l == 0 else math.sqrt(.75 / math.pi))
        sph = _solid(l)
        blocks.append(np.einsum('ip,fs->pfis', c, sph).reshape(nprim * _ncart(l), -1))
        for p in range(nprim):
            by_l.setdefault(int(l), []).append((coords[ia], exps[p], rows))
            rows += _ncart(l)
    C = np.zeros((rows, sum(b.shape[1] for b in blocks)))
    r = c = 0
    for b in blocks:
        C[r:r + b.shape[0], c:c + b.shape[1]] = b
        r, c = r + b.shape[0], c + b.shape[1]
    return by_l, C


def _solid(l):
    """Real solid harmonics over Cartesian monomials, from the Laplacian-free
    polynomials r^(l-m) P_l^m(z/r) Re/Im (x+iy)^m (p in the order x, y, z)."""
    if l < 2:
        return np.eye(_ncart(l))
    idx = {p: n for n, p in enumerate(_cart(l))}
    out = np.zeros((_ncart(l), 2 * l + 1))
    for m in range(-l, l + 1):
        am = abs(m)
        norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - am) / math.factorial(l + am)
                         * (2 if m else 1))
        for k in range((l - am) // 2 + 1):
            # coefficient of z^(l-2k-am) r^(2k) in the am-th derivative of P_l
            n = l - 2 * k
            leg = (-1) ** k * math.comb(l, k) * math.comb(2 * l - 2 * k, l) / 2 ** l
            leg *= math.factorial(n) / math.factorial(n - am)
            for a in range(k + 1):
                for b in range(k - a + 1):
                    multi = math.factorial(k) / (math.factorial(a) * math.factorial(b)
                                                 * math.factorial(k - a - b))
                    for t in range(am + 1):
                        # (x + iy)^am: C(am, t) x^(am-t) y^t i^t
                        if (t % 2 == 1) != (m < 0):
                            continue
                        sign = -1. if t % 4 in (2, 3) else 1.
                        p = (2 * a + am - t, 2 * b + t, n - am + 2 * (k - a - b))
                        out[idx[p], m + l] += norm * leg * multi * sign * math.comb(am, t)
    return out


def _boys(m_max, x):
    """F_0..F_m_max(x): the series of the highest order and the downward
    recursion below x = 36, the error function and the upward one above."""
    ex = torch.exp(-x)
    xs = torch.clamp(x, max=36.)
    term = torch.full_like(x, 1. / (2 * m_max + 1))
    s = term.clone()
    for k in range(1, 170):
        term = term * (2 * xs / (2 * m_max + 2 * k + 1))
        s += term
    low = [None] * (m_max + 1)
    low[m_max] = torch.exp(-xs) * s
    for m in range(m_max, 0, -1):
        low[m - 1] = (2 * xs * low[m] + torch.exp(-xs)) / (2 * m - 1)
    xl = torch.clamp(x, min=36.)
    high = [.5 * torch.sqrt(math.pi / xl) * torch.erf(torch.sqrt(xl))]
    for m in range(m_max):
        high.append(((2 * m + 1) * high[m] - ex) / (2 * xl))
    return [torch.where(x < 36., a, b) for a, b in zip(low, high)]


def _hermite(L):
    return [(t, u, v) for n in range(L + 1) for t in range(n + 1) for u in range(n - t + 1)
            for v in [n - t - u]]


def _pairs(A, a, la, B, b, lb):
    """All pairs of two primitive shell lists: exponent p, centre P and the
    Hermite expansion E (pairs, components of a x components of b, Hermites)."""
    n, m = len(a), len(b)
    A, a = A.repeat_interleave(m, 0), a.repeat_interleave(m)
    B, b = B.repeat(n, 1), b.repeat(n)
    p = a + b
    P = (a[:, None] * A + b[:, None] * B) / p[:, None]
    E1 = []
    for d in range(3):
        pa, pb = P[:, d] - A[:, d], P[:, d] - B[:, d]
        e = {(0, 0, 0): torch.exp(-a * b / p * (A[:, d] - B[:, d]) ** 2)}
        get = lambda i, j, t: e.get((i, j, t), 0.) if 0 <= t <= i + j else 0.
        for i in range(la + 1):
            for j in range(lb + 1):
                if i == j == 0:
                    continue
                for t in range(i + j + 1):
                    if i > 0:
                        v = get(i - 1, j, t - 1) / (2 * p) + pa * get(i - 1, j, t) \
                            + (t + 1) * get(i - 1, j, t + 1)
                    else:
                        v = get(i, j - 1, t - 1) / (2 * p) + pb * get(i, j - 1, t) \
                            + (t + 1) * get(i, j - 1, t + 1)
                    e[i, j, t] = v
        E1.append(e)
    herm = _hermite(la + lb)
    E = torch.zeros((n * m, _ncart(la) * _ncart(lb), len(herm)), dtype=p.dtype, device=p.device)
    for x, pi in enumerate(_cart(la)):
        for y, pj in enumerate(_cart(lb)):
            for h, tuv in enumerate(herm):
                if all(tuv[d] <= pi[d] + pj[d] for d in range(3)):
                    v = 1.
                    for d in range(3):
                        v = v * E1[d][pi[d], pj[d], tuv[d]]
                    E[:, x * _ncart(lb) + y, h] = v
    return p, P, E


def _coulomb(L, alpha, R):
    """Hermite Coulomb integrals R_tuv, t + u + v <= L, as a dict."""
    F = _boys(L, alpha * (R * R).sum(-1))
    cur = {}
    for m in range(L, -1, -1):
        nxt = {(0, 0, 0): (-2 * alpha) ** m * F[m]}
        for t, u, v in _hermite(L - m)[1:]:
            d = 0 if t else (1 if u else 2)
            k = (t, u, v)[d]
            low = [t, u, v]
            low[d] -= 1
            val = R[..., d] * cur[tuple(low)]
            if k > 1:
                low[d] -= 1
                val = val + (k - 1) * cur[tuple(low)]
            nxt[t, u, v] = val
        cur = nxt
    return cur


def _eri_block(bra, lab, ket, lcd):
    p, P, Ea = bra
    q, Q, Ec = ket
    hb, hk = _hermite(lab), _hermite(lcd)
    sign = torch.tensor([(-1.) ** sum(h) for h in hk], dtype=p.dtype, device=p.device)
    Ec = Ec * sign
    out = []
    step = max(1, int(6e6 / (len(q) * max(1, len(hb) * len(hk) / 8))))
    for s in range(0, len(p), step):
        pp, PP = p[s:s + step, None], P[s:s + step, None]
        R = _coulomb(lab + lcd, pp * q / (pp + q), PP - Q)
        pre = 2 * math.pi ** 2.5 / (pp * q * torch.sqrt(pp + q))
        M = torch.stack([torch.stack([R[tuple(np.add(x, y))] for y in hk], -1) for x in hb], -2)
        M = M * pre[..., None, None]
        out.append(torch.einsum('pah,pqhk,qck->paqc', Ea[s:s + step], M, Ec))
    return torch.cat(out)


def _shell_lists(by_l, dev):
    out = {}
    for l, shells in by_l.items():
        out[l] = (torch.tensor(np.array([s[0] for s in shells]), device=dev),
                  torch.tensor(np.array([s[1] for s in shells]), device=dev),
                  torch.tensor(np.array([np.arange(s[2], s[2] + _ncart(l)) for s in shells]).ravel(),
                               device=dev))
    return out


def _exact_jk(mol, dms, dev='cuda'):
    by_l, C = _primitives(mol)
    C = torch.tensor(C, device=dev)
    lists = _shell_lists(by_l, dev)
    D = C @ torch.as_tensor(dms, device=dev) @ C.T
    J, K = torch.zeros_like(D), torch.zeros_like(D)
    pairs = {(la, lb): _pairs(*lists[la][:2], la, *lists[lb][:2], lb) for la in lists for lb in lists}
    for (la, lb), bra in pairs.items():
        for (lc, ld), ket in pairs.items():
            if (la, lb) < (lc, ld):
                continue
            blk = _eri_block(bra, la + lb, ket, lc + ld)
            na, nb, nc, nd = (len(lists[l][1]) for l in (la, lb, lc, ld))
            blk = blk.reshape(na, nb, _ncart(la), _ncart(lb), nc, nd, _ncart(lc), _ncart(ld))
            blk = blk.permute(0, 2, 1, 3, 4, 6, 5, 7).reshape(
                na * _ncart(la), nb * _ncart(lb), nc * _ncart(lc), nd * _ncart(ld))
            ia, ib, ic, id_ = (lists[l][2] for l in (la, lb, lc, ld))
            swap = (la, lb) != (lc, ld)
            for n in range(len(D)):
                d = D[n]
                J[n][ia[:, None], ib] += torch.einsum('abcd,cd->ab', blk, d[ic[:, None], id_])
                K[n][ia[:, None], ic] += torch.einsum('abcd,bd->ac', blk, d[ib[:, None], id_])
                if swap:
                    J[n][ic[:, None], id_] += torch.einsum('abcd,ab->cd', blk, d[ia[:, None], ib])
                    K[n][ic[:, None], ia] += torch.einsum('abcd,bd->ca', blk, d[ib[:, None], id_])
    return (C.T @ J @ C).cpu().numpy(), (C.T @ K @ C).cpu().numpy()


def _exact_int3c(mol, aux, dev='cuda'):
    by_l, C = _primitives(mol)
    aux_l, Ca = _primitives(aux)
    lists, alists = _shell_lists(by_l, dev), _shell_lists(aux_l, dev)
    one = (torch.zeros((1, 3), dtype=torch.float64, device=dev),
           torch.zeros(1, dtype=torch.float64, device=dev))
    out = torch.zeros((len(C), len(C), len(Ca)), dtype=torch.float64, device=dev)
    for la in lists:
        for lb in lists:
            bra = _pairs(*lists[la][:2], la, *lists[lb][:2], lb)
            for lc in alists:
                ket = _pairs(*alists[lc][:2], lc, *one, 0)
                blk = _eri_block(bra, la + lb, ket, lc)
                na, nb, nc = len(lists[la][1]), len(lists[lb][1]), len(alists[lc][1])
                blk = blk.reshape(na, nb, _ncart(la), _ncart(lb), nc, _ncart(lc))
                blk = blk.permute(0, 2, 1, 3, 4, 5).reshape(na * _ncart(la), nb * _ncart(lb),
                                                           nc * _ncart(lc))
                out[lists[la][2][:, None, None], lists[lb][2][:, None], alists[lc][2]] = blk
    C, Ca = torch.tensor(C, device=dev), torch.tensor(Ca, device=dev)
    out = torch.einsum('pqr,rk->pqk', out, Ca)
    out = torch.einsum('pqk,qj->pjk', out, C)
    return torch.einsum('pjk,pi->ijk', out, C).cpu().numpy()


def exact(case, seed):
    if case['kind'] in ('rhf', 'batched'):
        return None
    mol = _mol(case, seed)
    if sum(_ncart(l) * n for l, n in mol._bas[:, [1, 2]]) > PRIM_MAX:
        return None
    if case['kind'] == 'df':
        return {'int3c': _exact_int3c(mol, _aux(mol))}
    vj, vk = _exact_jk(mol, _density(mol, seed, case['density'], case['ndm']))
    if case['kind'] == 'get_jk':
        return {'j': vj[0], 'k': vk[0]}
    return {n: v for n, v, on in (('j', vj, case['with_j']), ('k', vk, case['with_k'])) if on}
