"""Measured cases of the J/K engine, through its public entry points.

Each case is one call a user's program makes over and over with its
per-geometry set-up in hand: a direct-SCF J/K build (``get_jk``), a batched
build of many molecules (``JKBatch.get_jk``), the dense ERI tensor
(``get_int4c``) or the density-fitting integrals (``get_int3c``,
``get_int2c``).  Molecules are seeded water clusters and random-walk
molecules of the benchmark's kinds; the seed draws both the geometry (the random-walk
molecules keep their elements and are displaced) and the density.  ``exact`` evaluates the same quantities by the McMurchie-Davidson
scheme in float64 torch on uncontracted Cartesian Gaussians, without the
engine.
"""
import math

import numpy as np
import torch

from byteqc_b200.cuobc import lib as jklib
from byteqc_b200.cuobc.lib import int3c, int4c
from byteqc_b200.cuobc.scf import hf
from byteqc_b200.cuobc.scf.batch import JKBatch
from byteqc_b200.gto import Mole, basis, geom

DZ, TZ, PO = 'standin-cc-pvdz', 'standin-def2-tzvp', 'standin-6-31g*'
QZ = 'tzvp+g'  # the TZVP stand-in with one g function on the heavy atoms

# even-tempered auxiliary basis of the benchmark's density-fitting section
DF_AUX = {'O': [[0, [8.0, 1.0]], [0, [2.0, 1.0]], [0, [0.5, 1.0]],
                [1, [3.0, 1.0]], [1, [0.8, 1.0]], [2, [1.5, 1.0]],
                [3, [1.1, 1.0]]],
          'H': [[0, [3.0, 1.0]], [0, [0.6, 1.0]], [1, [1.0, 1.0]]]}


def _jk(name, shape, n, bas, n_dm=1, j=True, k=True, fp32_cutoff=0.):
    return {'name': name, 'kind': 'jk', 'shape': shape, 'n': n, 'basis': bas,
            'n_dm': n_dm, 'with_j': j, 'with_k': k, 'fp32_cutoff': fp32_cutoff}


def listed():
    return [
        # one water: the smallest call, bound by launches and latency
        _jk('jk-h2o1-dz', 'water', 1, DZ),
        # an ordinary cluster; every class up to (dd|dd), all primitives split
        _jk('jk-h2o8-dz', 'water', 8, DZ),
        # an organic molecule in a contracted Pople basis, odd atom count
        _jk('jk-walk37-631gs', 'walk', 37, PO),
        # alpha and beta densities of an open-shell calculation
        _jk('jk-walk13-tzvp-2dm', 'walk', 13, TZ, n_dm=2),
        # J only: a pure density functional
        _jk('j-walk29-dz', 'walk', 29, DZ, k=False),
        # the headline build: s to f shells, 1376 functions
        _jk('jk-h2o32-tzvp', 'water', 32, TZ),
        # the largest cluster: many small quartets, digestion-heavy
        _jk('jk-h2o64-dz', 'water', 64, DZ),
        # mixed precision: FP32 recursion below the cutoff
        _jk('jk-h2o20-tzvp-mixed', 'water', 20, TZ, fp32_cutoff=1e-6),
        # shells above f, served by the generic kernels
        _jk('jk-h2o2-tzvpg', 'water', 2, QZ),
        # many molecules of 3 to 30 atoms in one batched pass
        {'name': 'batch-24-631gs', 'kind': 'batch', 'nmol': 24, 'atoms': 30,
         'basis': PO, 'fp32_cutoff': 0.},
        # the dense tensor for a correlated method on a small system
        {'name': 'eri-h2o2-dz', 'kind': 'eri', 'shape': 'water', 'n': 2,
         'basis': DZ},
        # three-centre blocks and metric factor of density fitting
        {'name': 'df-h2o8-dz', 'kind': 'df', 'n': 8, 'basis': DZ},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges that is not a listed one."""
    while True:
        c = _drawn(rng)
        if c not in [{k: v for k, v in x.items() if k != 'name'}
                     for x in listed()]:
            return c


def _drawn(rng):
    u = rng.random()
    if u < 0.12:
        return {'kind': 'batch', 'nmol': rng.randint(3, 28),
                'atoms': rng.randint(5, 30), 'basis': rng.choice([PO, PO, DZ]),
                'fp32_cutoff': rng.choice([0., 1e-6])}
    if u < 0.20:
        shape, bas, top = rng.choice([('walk', PO, 6), ('walk', DZ, 4),
                                      ('water', DZ, 2), ('water', PO, 3)])
        return {'kind': 'eri', 'shape': shape, 'n': rng.randint(1, top),
                'basis': bas}
    if u < 0.27:
        return {'kind': 'df', 'n': rng.randint(1, 9), 'basis': DZ}
    shape = rng.choice(['water', 'walk'])
    bas = rng.choice([DZ, TZ, PO, DZ, TZ, PO, QZ])
    top = {('water', DZ): 64, ('water', TZ): 30, ('water', PO): 64,
           ('water', QZ): 3, ('walk', DZ): 44, ('walk', TZ): 24,
           ('walk', PO): 58, ('walk', QZ): 5}[shape, bas]
    n_dm = rng.choice([1, 1, 1, 2])
    if n_dm == 2:
        top = max(2, int(0.7 * top))
    kind = rng.choice(['jk', 'jk', 'jk', 'jk', 'j', 'k'])
    c = _jk('', shape, _log_int(rng, 2 if shape == 'walk' else 1, top), bas,
            n_dm=n_dm, j=kind != 'k', k=kind != 'j',
            fp32_cutoff=rng.choice([0., 0., 0., 1e-7, 1e-6]))
    del c['name']
    return c


# --------------------------------------------------------------- molecules --
def _atoms(shape, n, seed):
    if shape == 'water':
        return geom.water_cluster(n, box=max(14. * (n / 32.) ** (1. / 3.), 3.),
                                  seed=seed)
    return _displaced(geom.random_walk_molecule(n, seed=n), seed)


def _displaced(atoms, seed):
    """Another geometry of the same molecule (0.04 A per coordinate)."""
    rng = np.random.default_rng(seed)
    return [(s, tuple(np.asarray(x) + rng.normal(0., .04, 3)))
            for s, x in atoms]


def _mole(atoms, bas):
    if bas == QZ:
        bas = {s: basis.load(TZ, s) + ([] if s == 'H' else [[4, [1.2, 1.0]]])
               for s in {a[0] for a in atoms}}
    return Mole(atom=atoms, basis=bas).build()


def _density(mol, seed, n_dm=1):
    """Seeded closed-shell densities, orthonormal orbitals in the overlap."""
    s = mol.intor('int1e_ovlp')
    d = np.stack([geom.scf_like_density(s, max(mol.nelectron // 2 - m, 1),
                                        seed=seed + 101 * m)
                  for m in range(n_dm)])
    return d[0] if n_dm == 1 else d


def _inputs(case, seed):
    """Molecules and densities of a case."""
    seed = int(seed) % (1 << 20)
    if case['kind'] == 'batch':
        mols, dms = [], []
        for i in range(case['nmol']):
            natm = 3 + (case['atoms'] - 3) * i // max(case['nmol'] - 1, 1)
            mols.append(_mole(_displaced(geom.random_walk_molecule(
                natm, seed=7 * i + natm), seed + i), case['basis']))
            dms.append(_density(mols[-1], seed + i))
        return mols, dms
    mol = _mole(_atoms(case.get('shape', 'water'), case['n'], seed),
                case['basis'])
    dm = (_density(mol, seed + 1, case['n_dm']) if case['kind'] == 'jk'
          else None)
    return mol, dm


def prepare(case, seed):
    x, d = _inputs(case, seed)
    st = {'case': case}
    if case['kind'] == 'batch':
        st['batch'] = JKBatch(x)
        st['dm'] = [torch.as_tensor(v, device='cuda') for v in d]
    elif case['kind'] == 'jk':
        st['mol'] = x
        st['opt'] = hf._VHFOpt(x).build(1e-13)
        st['dm'] = torch.as_tensor(d, device='cuda')
    elif case['kind'] == 'eri':
        st['mol'] = x
        st['opt'] = hf._VHFOpt(x).build(diag_block_with_triu=True)
    else:
        aux = Mole(atom=_atoms('water', case['n'], int(seed) % (1 << 20)),
                   basis=DF_AUX).build()
        st['opt'] = int3c.VHFOpt3c(x, aux, 'int3c2e').build()
    return st


def run(st):
    case = st['case']
    if case['kind'] == 'jk':
        return hf.get_jk(st['mol'], st['dm'], vhfopt=st['opt'],
                         with_j=case['with_j'], with_k=case['with_k'],
                         fp32_cutoff=case['fp32_cutoff'], out='device')
    if case['kind'] == 'batch':
        return st['batch'].get_jk(st['dm'], out='device',
                                  fp32_cutoff=case['fp32_cutoff'])
    opt = st['opt']
    if case['kind'] == 'eri':
        return int4c.get_int4c(st['mol'], vhfopt=opt)
    blocks = [int3c.get_int3c(cp, ca, opt)[3] for cp in range(len(opt.log_qs))
              for ca in range(len(opt.aux_log_qs))]
    return blocks, int3c.get_int2c(opt)


# -------------------------------------------------------------------- work --
def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _quartet_flops(l, npp, dig):
    """Operations of one contracted quartet of class l with npp primitive
    quartets: Rys recursion and Cartesian products, and dig per integral for
    the digestion."""
    n = sum(l) // 2 + 1
    nm, mm = l[0] + l[1], l[2] + l[3]
    nf = math.prod(_ncart(x) for x in l)
    vrr = 4 * nm + 6 * (nm + 1) * mm
    hrr = 2 * sum((nm - j + 1) * (mm + 1) for j in range(1, l[1] + 1))
    hrr += 2 * (l[0] + 1) * (l[1] + 1) * sum(mm - x + 1
                                             for x in range(1, l[3] + 1))
    return npp * (30 + n * (76 + 3 * (vrr + hrr) + 3 * nf)) + dig * nf


def _jk_work(mol, dm, j, k):
    """Screened quartets of one build as the engine counts them."""
    opt = hf._VHFOpt(mol).build(1e-13)
    hf.get_jk(mol, torch.as_tensor(dm, device='cuda'), vhfopt=opt,
              with_j=j, with_k=k, out='device')
    lib = jklib.load_library()
    info = np.zeros(7, dtype=np.int32)
    jklib.check(lib.jk_basis_info(opt.handle, info.ctypes.data), 'info')
    ncq = int(info[6])
    cq = np.zeros((ncq, 8), dtype=np.int32)
    cnt = np.zeros(2 * ncq, dtype=np.int64)
    jklib.check(lib.jk_basis_cq_info(opt.handle, cq.ctypes.data), 'cq')
    jklib.check(lib.jk_last_counts(opt.handle, cnt.ctypes.data, None), 'cnt')
    n_dm = 1 if np.ndim(dm) == 2 else len(dm)
    dig = n_dm * (4 * j + 8 * k)
    fl = sum(float(c) * _quartet_flops([int(x) for x in r[2:6]],
                                       int(r[6]) * int(r[7]), dig)
             for c, r in zip(cnt, cq))
    opt.clear()
    return 8. * n_dm * mol.nao ** 2 * (1 + j + k), fl


def work(case):
    if case['kind'] == 'jk':
        mol, dm = _inputs(case, 1)
        b, f = _jk_work(mol, dm, case['with_j'], case['with_k'])
        return {'bytes': b, 'flops': f}
    if case['kind'] == 'batch':
        w = [_jk_work(m, d, True, True) for m, d in zip(*_inputs(case, 1))]
        return {'bytes': sum(b for b, _ in w), 'flops': sum(f for _, f in w)}
    # integrals: every unique quartet of the uncontracted working basis once
    mol, _ = _inputs(case, 1)
    sh = [(l, len(p)) for l, p, _ in _working(mol)]
    nao = sum(_ncart(l) for l, _ in sh)
    count = {}
    for s in sh:
        count[s] = count.get(s, 0) + 1
    pairs = {}
    ks = sorted(count, reverse=True)
    for i, a in enumerate(ks):
        for b in ks[i:]:
            n = count[a] * (count[a] + 1) / 2 if a == b else count[a] * count[b]
            pairs[a[0], b[0], a[1] * b[1]] = pairs.get(
                (a[0], b[0], a[1] * b[1]), 0) + n
    if case['kind'] == 'eri':
        f = sum(0.5 * n * m * _quartet_flops(p[:2] + q[:2], p[2] * q[2], 1)
                for p, n in pairs.items() for q, m in pairs.items())
        return {'bytes': 8. * nao ** 4, 'flops': f}
    aux = [s[0] for s in DF_AUX['O']] + 2 * [s[0] for s in DF_AUX['H']]
    f = sum(n * case['n'] * _quartet_flops(p[:2] + (a, 0), p[2], 1)
            for p, n in pairs.items() for a in aux)
    naux = case['n'] * sum(_ncart(a) for a in aux)
    return {'bytes': 8. * (nao * (nao + 1) / 2 * naux + naux ** 2), 'flops': f}


def tolerance(case):
    # FP64: 1e-15 to 3e-13 off ``exact`` (the integrals dropped by the 1e-13
    # Schwarz cutoff among it); mixed: the rounding of the FP32 quartets
    if case.get('fp32_cutoff'):
        return {'rel': 4e-12, 'max': 4e-10}
    return {'rel': 1e-12, 'max': 1e-10}


# ------------------------------------------------------------------- exact --
_FAC = {0: math.sqrt(0.25 / math.pi), 1: math.sqrt(0.75 / math.pi)}


def _powers(l):
    return [(a, b, l - a - b) for a in range(l, -1, -1)
            for b in range(l - a, -1, -1)]


def _radial_norm(l, e):
    return math.sqrt(2. * (2. * e) ** (l + 1.5) / math.gamma(l + 1.5))


def _shells(mol):
    """(l, centre, exponents, coefficients (nctr, nprim)) of a molecule."""
    for s in mol._bas:
        l, npr, nct = int(s[1]), int(s[2]), int(s[3])
        p = int(mol._atm[s[0], 1])
        yield (l, mol._env[p:p + 3], mol._env[s[5]:s[5] + npr],
               mol._env[s[6]:s[6] + npr * nct].reshape(nct, npr))


def _working(mol):
    """The working basis: shells with several contractions split into their
    primitives, sorted by (l, primitives)."""
    out = []
    for l, r, es, cs in _shells(mol):
        if len(cs) == 1:
            out.append((l, [(e, c) for e, c in zip(es, cs[0])], r))
        else:
            out += [(l, [(e, _radial_norm(l, e))], r) for e in es]
    return sorted(out, key=lambda s: (s[0], len(s[1])))


def _solid(l):
    """Real solid harmonics of degree l over the monomials of _powers(l),
    columns m = -l .. l (p: x, y, z)."""
    if l < 2:
        return np.eye(_ncart(l))
    at = {p: i for i, p in enumerate(_powers(l))}
    out = np.zeros((_ncart(l), 2 * l + 1))
    for m in range(l + 1):
        nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * (2 if m else 1)
                        * math.factorial(l - m) / math.factorial(l + m))
        for k in range((l - m) // 2 + 1):  # z^(l-2k-m) r^2k of the Legendre part
            c = (nrm * (-1) ** k * .5 ** l * math.comb(l, k)
                 * math.comb(2 * l - 2 * k, l) * math.factorial(l - 2 * k)
                 / math.factorial(l - 2 * k - m))
            for a in range(k + 1):         # r^2k = (x^2 + y^2 + z^2)^k
                for b in range(k - a + 1):
                    cr = c * math.factorial(k) / (
                        math.factorial(a) * math.factorial(b)
                        * math.factorial(k - a - b))
                    for q in range(m + 1):  # (x + iy)^m
                        v = cr * math.comb(m, q) * (-1) ** (q // 2)
                        p = (2 * a + m - q, 2 * b + q,
                             l - 2 * k - m + 2 * (k - a - b))
                        if q % 2 == 0:
                            out[at[p], l + m] += v
                        elif m:
                            out[at[p], l - m] += v
    return out


class _Prims:
    """Primitive Cartesian functions of a list of shells
    (l, [(exponent, coefficients over the contractions)], centre), grouped
    by l: exponents, centres, first function, and the (functions x
    contracted functions) map."""

    def __init__(self, shells, sph):
        by = {}
        nrow = sum(len(p) * _ncart(l) for l, p, _ in shells)
        ncol = sum(np.size(p[0][1]) * (2 * l + 1 if sph else _ncart(l))
                   for l, p, _ in shells)
        m = np.zeros((nrow, ncol))
        col = 0
        rows = {}
        for l, p, _ in shells:
            rows[l] = rows.get(l, 0) + len(p) * _ncart(l)
        start, acc = {}, 0
        for l in sorted(rows):
            start[l], acc = acc, acc + rows[l]
        for l, p, r in shells:
            t = _solid(l) if sph else np.eye(_ncart(l))
            g = by.setdefault(l, ([], []))
            nc = np.size(p[0][1])
            for e, c in p:
                r0 = start[l] + len(g[0]) * _ncart(l)
                m[r0:r0 + _ncart(l), col:col + nc * t.shape[1]] = np.kron(
                    np.reshape(c, (1, nc)) * _FAC.get(l, 1.), t)
                g[0].append(e)
                g[1].append(r)
            col += nc * t.shape[1]
        f = dict(dtype=torch.float64, device='cuda')
        self.map = torch.as_tensor(m, **f)
        self.groups = [(l, torch.as_tensor(np.array(by[l][0]), **f),
                        torch.as_tensor(np.array(by[l][1]), **f), start[l])
                       for l in sorted(by)]
        self.n = nrow


def _hermite(n):
    return [(t, u, s - t - u) for s in range(n + 1) for t in range(s, -1, -1)
            for u in range(s - t, -1, -1)]


def _pair(la, ea, ra, lb, eb, rb):
    """Exponent sums p, centres P and Hermite coefficients
    E[pair, component, hermite] of all pairs of two groups."""
    a, b = ea[:, None].expand(len(ea), len(eb)).reshape(-1), eb.repeat(len(ea))
    A = ra[:, None].expand(-1, len(eb), 3).reshape(-1, 3)
    B = rb.repeat(len(ea), 1)
    p = a + b
    P = (a[:, None] * A + b[:, None] * B) / p[:, None]
    axis = []
    for d in range(3):
        PA, PB = P[:, d] - A[:, d], P[:, d] - B[:, d]
        E = {(0, 0, 0): torch.exp(-a * b / p * (A[:, d] - B[:, d]) ** 2)}

        def get(i, j, t):
            return E.get((i, j, t), torch.zeros_like(p)) if 0 <= t <= i + j else 0.
        for i in range(la + 1):
            for j in range(lb + 1):
                for t in range(i + j + 1):
                    if i:
                        E[i, j, t] = (get(i - 1, j, t - 1) / (2 * p)
                                      + PA * get(i - 1, j, t)
                                      + (t + 1) * get(i - 1, j, t + 1))
                    elif j:
                        E[i, j, t] = (get(i, j - 1, t - 1) / (2 * p)
                                      + PB * get(i, j - 1, t)
                                      + (t + 1) * get(i, j - 1, t + 1))
        axis.append(E)
    herm = _hermite(la + lb)
    zero = torch.zeros_like(p)
    cols = [[(axis[0][x[0], y[0], h[0]] * axis[1][x[1], y[1], h[1]]
              * axis[2][x[2], y[2], h[2]])
             if all(h[d] <= x[d] + y[d] for d in range(3)) else zero
             for h in herm] for x in _powers(la) for y in _powers(lb)]
    return p, P, torch.stack([torch.stack(c, -1) for c in cols], 1), herm


def _eri_block(bra, ket):
    """(ab|cd) as [bra pair, ket pair, bra component, ket component]."""
    (p, P, E, hb), (q, Q, F, hk) = bra, ket
    L = sum(hb[-1]) + sum(hk[-1])
    pp, qq = p[:, None], q[None]
    al = pp * qq / (pp + qq)
    X, Y, Z = (P[:, None, d] - Q[None, :, d] for d in range(3))
    x = al * (X * X + Y * Y + Z * Z)
    ex = torch.exp(-x)
    xs = x.clamp_min(1e-12)
    f = 0.5 * math.gamma(L + .5) * torch.special.gammainc(
        torch.full_like(x, L + .5), xs) * xs ** -(L + .5)
    fm = {L: torch.where(x < 1e-12, torch.full_like(x, 1. / (2 * L + 1)), f)}
    for m in range(L, 0, -1):
        fm[m - 1] = (2 * x * fm[m] + ex) / (2 * m - 1)
    pre = 2 * math.pi ** 2.5 / (pp * qq * torch.sqrt(pp + qq))
    R = {(0, 0, 0, m): pre * (-2 * al) ** m * fm[m] for m in range(L + 1)}
    for s in range(1, L + 1):
        for h in _hermite(L):
            if sum(h) != s:
                continue
            d = next(i for i in range(3) if h[i])
            lo = tuple(h[i] - (i == d) for i in range(3))
            lo2 = tuple(h[i] - 2 * (i == d) for i in range(3))
            for m in range(L - s + 1):
                v = (X, Y, Z)[d] * R[lo + (m + 1,)]
                if lo[d]:
                    v = v + lo[d] * R[lo2 + (m + 1,)]
                R[h + (m,)] = v
        R = {k: v for k, v in R.items() if k[3] or sum(k[:3]) <= s}
    G = torch.stack([torch.stack([(-1) ** sum(u) * R[tuple(
        t[i] + u[i] for i in range(3)) + (0,)] for u in hk], -1)
        for t in hb], -2)  # [bra, ket, t, u]
    return E[:, None] @ G @ F.transpose(1, 2)[None]


def _blocks(gr_a, gr_b, gr_c, gr_d):
    """Integral blocks of all (a, b | c, d) group products, chunked over the
    functions of a: yields the slices of the four and the [a, b, c, d] block."""
    for la, ea, ra, ia in gr_a:
        for lb, eb, rb, ib in gr_b:
            for lc, ec, rc, ic in gr_c:
                for ld, ed, rd, id_ in gr_d:
                    ket = _pair(lc, ec, rc, ld, ed, rd)
                    na, nb, nc, nd = (_ncart(v) for v in (la, lb, lc, ld))
                    cost = (len(eb) * len(ec) * len(ed)
                            * (len(_hermite(la + lb)) * len(ket[3]) + 40))
                    step = max(1, int(3e8 // cost))
                    for a0 in range(0, len(ea), step):
                        sa = slice(a0, a0 + step)
                        v = _eri_block(_pair(la, ea[sa], ra[sa], lb, eb, rb),
                                       ket)
                        m = len(ea[sa])
                        v = v.view(m, len(eb), len(ec), len(ed), na, nb, nc, nd)
                        v = v.permute(0, 4, 1, 5, 2, 6, 3, 7).reshape(
                            m * na, len(eb) * nb, len(ec) * nc, len(ed) * nd)
                        s = [slice(o, o + n) for o, n in
                             zip((ia + a0 * na, ib, ic, id_), v.shape)]
                        yield s, v


def _exact_jk(mol, dm, j, k):
    sh = [(l, list(zip(es, cs.T)), r) for l, r, es, cs in _shells(mol)]
    b = _Prims(sh, True)
    C = b.map
    D = C @ torch.as_tensor(dm, device='cuda').reshape(-1, mol.nao, mol.nao) @ C.T
    J, K = torch.zeros_like(D), torch.zeros_like(D)
    g = b.groups
    for (sa, sb, sc, sd), v in _blocks(g, g, g, g):
        for m in range(len(D)):
            if j:
                J[m, sa, sb] += torch.einsum('abcd,cd->ab', v, D[m, sc, sd])
            if k:
                K[m, sa, sc] += torch.einsum('abcd,bd->ac', v, D[m, sb, sd])
    return tuple((C.T @ v @ C).reshape(np.shape(dm)) if on else None
                 for v, on in ((J, j), (K, k)))


def _exact_cost(mol):
    return sum(len(es) for _, _, es, _ in _shells(mol)) ** 4


def exact(case, seed):
    x, d = _inputs(case, seed)
    if case['kind'] == 'batch':
        if sum(_exact_cost(m) for m in x) > 1e9:
            return None
        return [_exact_jk(m, v, True, True) for m, v in zip(x, d)]
    if case['kind'] == 'jk':
        if _exact_cost(x) > 1.5e9 or case['basis'] == QZ and case['n'] > 2:
            return None
        return _exact_jk(x, d, case['with_j'], case['with_k'])
    b = _Prims(_working(x), False)
    C = b.map
    if case['kind'] == 'eri':
        if b.n > 130:
            return None
        out = torch.zeros((b.n,) * 4, dtype=torch.float64, device='cuda')
        for s, v in _blocks(b.groups, b.groups, b.groups, b.groups):
            out[s] = v
        if b.n != C.shape[1] or not torch.equal(C != 0, torch.eye(
                b.n, device='cuda') != 0):
            for _ in range(4):  # contract the last index, move it to the front
                out = (out @ C).permute(3, 0, 1, 2).contiguous()
            return out
        c = C.diagonal()
        return (out * c[:, None, None, None] * c[:, None, None] * c[:, None] * c)
    aux = Mole(atom=_atoms('water', case['n'], int(seed) % (1 << 20)),
               basis=DF_AUX).build()
    xb = _Prims(_working(aux), False)
    f = dict(dtype=torch.float64, device='cuda')
    one = [(0, torch.zeros(1, **f), torch.zeros(1, 3, **f), 0)]
    c, ca = C.diagonal(), xb.map.diagonal()  # all shells are single primitives
    full = torch.zeros((b.n, b.n, xb.n), **f)
    for (sa, sb, sc, _), v in _blocks(b.groups, b.groups, xb.groups, one):
        full[sa, sb, sc] = v[..., 0]
    full *= c[:, None, None] * c[:, None] * ca
    blocks = []
    starts = [g[3] for g in b.groups] + [b.n]
    astarts = [g[3] for g in xb.groups] + [xb.n]
    for i in range(len(b.groups)):
        for jj in range(i + 1):
            for a in range(len(xb.groups)):
                blocks.append(full[starts[i]:starts[i + 1],
                                   starts[jj]:starts[jj + 1],
                                   astarts[a]:astarts[a + 1]])
    met = torch.zeros((xb.n, xb.n), **f)
    for (sa, _, sc, _), v in _blocks(xb.groups, one, xb.groups, one):
        met[sa, sc] = v[:, 0, :, 0]
    met *= ca[:, None] * ca
    # the metric factor in the auxiliary molecule's spherical functions, in
    # its own order
    T = torch.zeros((xb.n, aux.nao), **f)
    col = 0
    used = {}
    for l, r, es, cs in _shells(aux):
        g = next(q for q in xb.groups if q[0] == l)
        i = used.get(l, 0)
        used[l] = i + 1
        t = torch.as_tensor(_solid(l), **f)
        r0 = g[3] + i * _ncart(l)
        T[r0:r0 + _ncart(l), col:col + t.shape[1]] = t
        col += t.shape[1]
    return blocks, torch.linalg.cholesky(T.T @ met @ T)
