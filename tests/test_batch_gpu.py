"""Batched J/K over molecules of uneven size: identical (to rounding) to
building each molecule alone, in FP64, in mixed precision and when replayed
from a captured CUDA graph."""
import numpy as np
import pytest

from byteqc_b200.gto import Mole, geom

pytestmark = pytest.mark.gpu


def _mols():
    out = []
    for i, n in enumerate((3, 7, 12, 5)):
        atoms = geom.random_walk_molecule(n, seed=40 + i)
        out.append(Mole(atom=atoms, basis='standin-6-31g*').build())
    return out


def _dms(mols, seed=0):
    rng = np.random.default_rng(seed)
    res = []
    for m in mols:
        d = rng.random((m.nao, m.nao))
        res.append(d + d.T)
    return res


def test_batch_matches_single_molecule_builds():
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()
    dms = _dms(mols)
    batch = JKBatch(mols)
    res = batch.get_jk(dms)
    for m, (mol, dm, opt) in enumerate(zip(mols, dms, batch.opts)):
        vj, vk = hf.get_jk(mol, dm, vhfopt=opt)
        scale = max(1.0, abs(vj).max())
        assert abs(res[m][0] - vj).max() <= 1e-10
        assert abs(res[m][1] - vk).max() <= 1e-10
    # mixed precision in the batch equals mixed precision alone
    mres = batch.get_jk(dms, fp32_cutoff=1e-6)
    for m, (mol, dm, opt) in enumerate(zip(mols, dms, batch.opts)):
        vj, vk = hf.get_jk(mol, dm, vhfopt=opt, fp32_cutoff=1e-6)
        assert abs(mres[m][0] - vj).max() <= 1e-9
        assert abs(mres[m][1] - vk).max() <= 1e-9


@pytest.mark.parametrize('solo', [None, 1])
def test_batch_with_a_repeated_basis(solo):
    """One basis handle several times in a batch, each time with a density of
    its own (other screening decisions among them: the third is tiny): every
    occurrence is screened into its own buffers."""
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    a, b = _mols()[:2]
    oa, ob = hf._VHFOpt(a).build(), hf._VHFOpt(b).build()
    mols = [a, b, a, a, b]
    dms = _dms(mols)
    dms[2] = 1e-11 * dms[2]
    dms[3] = _dms([a], seed=9)[0]
    batch = JKBatch(mols, vhfopts=[oa, ob, oa, oa, ob], solo_tasks=solo)
    for cutoff in (None, 1e-6):
        for rep in range(2):
            res = batch.get_jk(dms, fp32_cutoff=cutoff)
            for r, mol, dm, opt in zip(res, mols, dms, batch.opts):
                vj, vk = hf.get_jk(mol, dm, vhfopt=opt, fp32_cutoff=cutoff)
                tol = 1e-9 if cutoff else 1e-10
                assert abs(r[0] - vj).max() <= tol * min(1., abs(dm).max())
                assert abs(r[1] - vk).max() <= tol * min(1., abs(dm).max())
    batch.close()


def test_batch_with_a_larger_caller_basis_later():
    """jk_batch_get_jk at one n_dm with another caller basis than the first
    call's: spherical, then Cartesian (more functions), then spherical."""
    import ctypes
    import torch
    from byteqc_b200.cuobc import lib as jklib
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch, _ptrs
    lib = jklib.load_library()
    mols = []
    for i in range(3):
        mols.append(Mole(atom=geom.water_cluster(1 + i, box=5.0, seed=i),
                         basis='standin-def2-tzvp').build())
    batch = JKBatch(mols)
    rng = np.random.default_rng(2)
    o = batch._opts(True, None, None)
    for cart in (False, True, False):
        coeff = [torch.eye(op.nao, dtype=torch.float64, device='cuda') if cart
                 else op.coeff_dev for op in batch.opts]
        dms = []
        for c in coeff:
            d = rng.standard_normal((c.shape[1], c.shape[1]))
            dms.append(torch.as_tensor(d + d.T, device='cuda'))
        vj, vk = ([torch.zeros_like(d) for d in dms] for _ in range(2))
        assert lib.jk_batch_get_jk(
            batch.handle, _ptrs([c.data_ptr() for c in coeff]),
            (ctypes.c_int * 3)(*[c.shape[1] for c in coeff]),
            *(_ptrs([x.data_ptr() for x in y]) for y in (dms, vj, vk)), 1,
            ctypes.byref(o), None) == 0
        torch.cuda.synchronize()
        for m in range(3):
            op = batch.opts[m]
            rj, rk = torch.zeros_like(dms[m]), torch.zeros_like(dms[m])
            so = jklib.JKOpts()
            so.direct_scf_tol, so.nbins, so.prescreen = 1e-13, o.nbins, 1
            assert lib.jk_get_jk(op.handle, coeff[m].data_ptr(),
                                 coeff[m].shape[1], dms[m].data_ptr(), 1,
                                 rj.data_ptr(), rk.data_ptr(),
                                 ctypes.byref(so), None) == 0
            torch.cuda.synchronize()
            assert (vj[m] - rj).abs().max().item() <= 1e-10
            assert (vk[m] - rk).abs().max().item() <= 1e-10
    batch.close()


def test_batch_build_with_outputs_left_out():
    """jk_batch_build with null entries in the output arrays: J of the first
    molecule only, K of the second only, both of the third."""
    import ctypes
    import torch
    from byteqc_b200.cuobc import lib as jklib
    from byteqc_b200.cuobc.scf.batch import JKBatch, _ptrs
    lib = jklib.load_library()
    mols = _mols()[:3]
    batch = JKBatch(mols)
    rng = np.random.default_rng(4)
    dms = []
    for op in batch.opts:
        d = rng.standard_normal((op.nao, op.nao))
        dms.append(torch.as_tensor(d + d.T, device='cuda'))
    o = batch._opts(True, None, None)
    full = None
    for jn, kn in (((1, 1, 1), (1, 1, 1)), ((1, 0, 1), (0, 1, 1))):
        vj, vk = ([torch.zeros_like(d) for d in dms] for _ in range(2))
        assert lib.jk_batch_build(
            batch.handle, _ptrs([d.data_ptr() for d in dms]),
            _ptrs([v.data_ptr() if on else None for v, on in zip(vj, jn)]),
            _ptrs([v.data_ptr() if on else None for v, on in zip(vk, kn)]), 1,
            ctypes.byref(o), None) == 0
        torch.cuda.synchronize()
        if full is None:
            full = vj, vk
        for got, ref, on in ((vj, full[0], jn), (vk, full[1], kn)):
            for g, r, want in zip(got, ref, on):
                if want:
                    assert (g - r).abs().max().item() <= 1e-10
                else:
                    assert not g.any().item()
    batch.close()


def test_batch_build_after_one_that_did_not_fit():
    """A build whose workspace cannot be allocated (4 million densities asked
    for) is an error before any launch, and the next one of the old size makes
    its tables again."""
    import ctypes
    import torch
    from byteqc_b200.cuobc import lib as jklib
    from byteqc_b200.cuobc.scf.batch import JKBatch, _ptrs
    lib = jklib.load_library()
    batch = JKBatch(_mols())
    rng = np.random.default_rng(6)
    dms = []
    for op in batch.opts:
        d = rng.standard_normal((op.nao, op.nao))
        dms.append(torch.as_tensor(d + d.T, device='cuda'))
    vj, vk = ([torch.zeros_like(d) for d in dms] for _ in range(2))
    o = batch._opts(True, None, None)

    def build(n_dm):
        return lib.jk_batch_build(
            batch.handle, *(_ptrs([x.data_ptr() for x in y])
                            for y in (dms, vj, vk)), n_dm, ctypes.byref(o), None)
    assert build(1) == 0
    torch.cuda.synchronize()
    ref = [v.clone() for v in vj + vk]
    for v in vj + vk:
        v.zero_()
    assert build(1 << 22) == 1
    assert build(1) == 0
    torch.cuda.synchronize()
    for v, r in zip(vj + vk, ref):
        assert (v - r).abs().max().item() <= 1e-10
    batch.close()


def test_batch_graph_replay():
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()
    batch = JKBatch(mols)
    d0 = _dms(mols, seed=1)
    d1 = _dms(mols, seed=2)
    ref1 = batch.get_jk(d1)
    batch.capture(d0)
    for _ in range(2):
        got = batch.replay(d1)
    for (aj, ak), (bj, bk) in zip(ref1, got):
        assert abs(aj - bj).max() <= 1e-10
        assert abs(ak - bk).max() <= 1e-10


def test_batch_identical_molecules_keep_their_own_j():
    """Copies of one molecule in a batch: their segments of a class carry the
    same shell indices, so a warp that straddles two of them must not merge
    their J contributions (each copy has its own density)."""
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    atoms = geom.water_cluster(1, box=4.0, seed=3)
    mols = [Mole(atom=atoms, basis='standin-cc-pvdz').build() for _ in range(6)]
    dms = _dms(mols, seed=5)
    batch = JKBatch(mols)
    for cut in (None, 1e-6):
        res = batch.get_jk(dms, fp32_cutoff=cut)
        for m, (mol, dm, opt) in enumerate(zip(mols, dms, batch.opts)):
            vj, vk = hf.get_jk(mol, dm, vhfopt=opt, fp32_cutoff=cut)
            scale = max(1.0, abs(vj).max())
            assert abs(res[m][0] - vj).max() <= 1e-10, (cut, m)
            assert abs(res[m][1] - vk).max() <= 1e-10, (cut, m)


def test_batch_g_h_shells():
    """Batched builds of molecules with g and h shells (the generic kernel's
    segment-table launch) match the single-molecule builds."""
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    from byteqc_b200.gto import basis as basis_mod
    extra = {'O': [[4, [1.1, 1.0]], [5, [0.9, 1.0]]], 'H': [[4, [0.8, 1.0]]]}
    bas = {s: list(basis_mod.load('standin-cc-pvdz', s)) + extra[s]
           for s in ('O', 'H')}
    mols = [Mole(atom=geom.water_cluster(n, box=5.0, seed=s), basis=bas).build()
            for n, s in ((1, 1), (2, 2), (1, 3))]
    dms = _dms(mols, seed=5)
    batch = JKBatch(mols)
    for cut in (0., 1e-6):
        res = batch.get_jk(dms, fp32_cutoff=cut)
        for m, (mol, dm, opt) in enumerate(zip(mols, dms, batch.opts)):
            vj, vk = hf.get_jk(mol, dm, vhfopt=opt, fp32_cutoff=cut)
            scale = max(1.0, abs(vj).max())
            assert abs(res[m][0] - vj).max() <= 1e-10
            assert abs(res[m][1] - vk).max() <= 1e-10


def test_batch_molecules_vs_oracle():
    """The first eight molecules of the 256-molecule batched workload
    (random walks of 3-60 atoms, C:N:O:H = 3:1:1:5, 6-31G* stand-in, seed 4,
    SCF-like densities) built in one batch, each against the oracle at
    1e-10 absolute, FP64."""
    import os
    import sys
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    from byteqc_b200.cuobc.scf.batch import JKBatch
    from oracle import hf_oracle
    mols, dms = bench.batch_workload(8)
    batch = JKBatch(mols)
    res = batch.get_jk(dms)
    for m, (mol, dm) in enumerate(zip(mols, dms)):
        rj, rk = hf_oracle.get_jk(mol, dm)
        assert abs(res[m][0] - rj).max() <= 1e-10, m
        assert abs(res[m][1] - rk).max() <= 1e-10, m
    batch.close()


def test_batch_tune_keeps_results_and_cache(tmp_path):
    """The autotuner picks a launch shape per class launch (static chunks or
    a persistent grid with a device work counter); the batched J/K are the
    same before and after tuning, in FP64 and in the mixed mode, and a second
    tuning from the cache file times nothing again."""
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()
    dms = _dms(mols, seed=9)
    batch = JKBatch(mols)
    ref = batch.get_jk(dms)
    ref32 = batch.get_jk(dms, fp32_cutoff=1e-6)
    cache = str(tmp_path / 'tune.txt')
    info = batch.tune(dms, fp32_cutoff=1e-6, cache=cache)
    assert info and all(k['fp64']['ms'] is not None for k in info)
    assert all(k['fp32']['ms'] is not None for k in info)
    got = batch.get_jk(dms)
    got32 = batch.get_jk(dms, fp32_cutoff=1e-6)
    for (aj, ak), (bj, bk) in zip(ref, got):
        assert abs(aj - bj).max() <= 1e-10
        assert abs(ak - bk).max() <= 1e-10
    for (aj, ak), (bj, bk) in zip(ref32, got32):
        assert abs(aj - bj).max() <= 1e-10
        assert abs(ak - bk).max() <= 1e-10
    # every persistent shape also gives the same result in a captured graph
    batch.capture(dms)
    rep = batch.replay(dms)
    for (aj, ak), (bj, bk) in zip(ref, rep):
        assert abs(aj - bj).max() <= 1e-10
        assert abs(ak - bk).max() <= 1e-10
    lines = open(cache).read().splitlines()
    assert len(lines) > 1
    b2 = JKBatch(mols, vhfopts=batch.opts)
    info2 = b2.tune(dms, fp32_cutoff=1e-6, cache=cache)
    shapes = {(k['class'], k['np_ij'], k['np_kl']): (k['fp64']['grab'],
              k['fp64']['grid_mul']) for k in info}
    for k in info2:
        assert shapes[(k['class'], k['np_ij'], k['np_kl'])] == (
            k['fp64']['grab'], k['fp64']['grid_mul'])
    b2.close()
    batch.close()


def test_batch_persistent_shapes_match_static():
    """Every persistent launch shape gives the static result: the batch's
    class launches forced to each candidate grab size (through a cache file
    written by hand) on molecules of uneven size."""
    import os
    import tempfile
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()
    dms = _dms(mols, seed=10)
    batch = JKBatch(mols)
    ref = batch.get_jk(dms)
    info = batch.info()
    with tempfile.TemporaryDirectory() as d:
        for grab, gm in ((1, 1), (2, 2), (64, 1), (1024, 2)):
            path = os.path.join(d, 'c%d_%d.txt' % (grab, gm))
            with open(path, 'w') as f:
                for k in info:
                    lg = max(0, int(k['tasks']).bit_length() - 1)
                    f.write('%d %d %d 0 %d %d %d 1.0\n' % (
                        k['class'], k['np_ij'], k['np_kl'], lg, grab, gm))
            b = JKBatch(mols, vhfopts=batch.opts)
            b.tune(dms, cache=path)
            assert all(k['fp64']['grab'] == grab for k in b.info())
            got = b.get_jk(dms)
            for (aj, ak), (bj, bk) in zip(ref, got):
                assert abs(aj - bj).max() <= 1e-10, (grab, gm)
                assert abs(ak - bk).max() <= 1e-10, (grab, gm)
            b.close()
    batch.close()


def test_batch_tune_leaves_files_of_before_alone(tmp_path):
    """A cache file of the tuner whose grabs counted quartets (its first line
    carries no version) is timed anew and rewritten; entries that are no launch
    shape are passed over."""
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()[:2]
    dms = _dms(mols, seed=10)
    batch = JKBatch(mols)
    path = str(tmp_path / 'tune.txt')

    def write(head, grab, gm):
        with open(path, 'w') as f:
            f.write(head)
            for k in batch.info():
                f.write('%d %d %d 0 %d %d %d 1.0\n' % (
                    k['class'], k['np_ij'], k['np_kl'],
                    max(0, int(k['tasks']).bit_length() - 1), grab, gm))
    old = ('# byteqc_b200 batch launch shapes: cls np_ij np_kl part log2tasks '
           'grab grid_mul ms\n')
    for head, grab, gm in ((old, 1024, 1), ('', 4, 0), ('', -3, 1)):
        write(head, grab, gm)
        info = batch.tune(dms, cache=path)
        assert all(k['fp64']['grab'] in (0, 1, 2, 4, 8, 16, 32)
                   and k['fp64']['grid_mul'] in (1, 2) for k in info)
        assert not any(k['fp64']['ms'] == 1.0 for k in info)
    assert open(path).readline() != old
    again = batch.tune(dms, cache=path)
    for key in ('grab', 'grid_mul'):
        assert [k['fp64'][key] for k in again] == [k['fp64'][key] for k in info]
    batch.close()


def test_batch_solo_class_quartets():
    """Class quartets above the solo threshold run as their own launches
    (the single-molecule kernels), the rest merged: every split gives the
    single-molecule result, in FP64, in mixed precision and from a graph."""
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mols = _mols()
    dms = _dms(mols, seed=20)
    base = JKBatch(mols, solo_tasks=0)
    assert base.nsolo == 0
    ref = [hf.get_jk(m, d, vhfopt=o) for m, d, o in zip(mols, dms, base.opts)]
    ref32 = [hf.get_jk(m, d, vhfopt=o, fp32_cutoff=1e-6)
             for m, d, o in zip(mols, dms, base.opts)]
    nsolos = []
    for solo in (1, 64, 4096):
        b = JKBatch(mols, vhfopts=base.opts, solo_tasks=solo)
        nsolos.append(b.nsolo)
        if solo == 1:
            assert b.info() == []      # everything on its own
        for cut, want, tol in ((None, ref, 1e-10), (1e-6, ref32, 1e-9)):
            got = b.get_jk(dms, fp32_cutoff=cut)
            for (aj, ak), (bj, bk) in zip(want, got):
                assert abs(aj - bj).max() <= tol, (solo, cut)
                assert abs(ak - bk).max() <= tol, (solo, cut)
        b.capture(dms, fp32_cutoff=1e-6)
        got = b.replay(dms)
        for (aj, ak), (bj, bk) in zip(ref32, got):
            assert abs(aj - bj).max() <= 1e-9
            assert abs(ak - bk).max() <= 1e-9
        b.close()
    assert nsolos[0] >= nsolos[1] >= nsolos[2] and nsolos[0] > nsolos[2]
    base.close()
