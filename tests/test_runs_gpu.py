"""Run kernels (a warp walks up to 32 bra pairs of one shell against a chunk of
ket pairs, keeping sums over the walk) against the CPU oracle where the walk
and the chunks have edges: molecules whose runs are cut at each run length,
chunks of 1 to 32 live kets, J or K alone, several densities (the sums kept in
shared memory, and added per quartet when they no longer fit), split groups,
and the FP32 part of the mixed mode.  1e-10 absolute, as the other J/K tests
(1e-9 for the mixed mode at cutoff 1e-6, whose FP32 quartets are each bounded
by the cutoff times 2^-24)."""
import numpy as np
import pytest

from byteqc_b200.gto import Mole, geom

pytestmark = pytest.mark.gpu


def _dm(mol, n_dm, seed):
    s = mol.intor('int1e_ovlp')
    return np.stack([geom.scf_like_density(s, max(1, mol.nelectron // 2 - m),
                                           seed=seed + m)
                     for m in range(n_dm)])


@pytest.mark.parametrize('basis,nw,n_dm,group_size', [
    ('standin-cc-pvdz', 1, 1, None),   # shortest runs, one partial chunk
    ('standin-cc-pvdz', 3, 2, None),
    ('standin-cc-pvdz', 3, 1, 24),     # classes split into small groups
    ('standin-def2-tzvp', 1, 5, None),  # five densities: some classes add per quartet
    ('standin-def2-tzvp', 2, 1, None),
    ('standin-6-31g*', 4, 3, None),    # contracted: several primitives per pair
])
def test_run_kernels_vs_oracle(basis, nw, n_dm, group_size):
    from byteqc_b200.cuobc.scf import hf
    from oracle import hf_oracle
    mol = Mole(atom=geom.water_cluster(nw, box=3.0 + 2.0 * nw, seed=nw),
               basis=basis).build()
    dm = _dm(mol, n_dm, 3)
    opt = hf._VHFOpt(mol).build(group_size=group_size)
    rj, rk = zip(*(hf_oracle.get_jk(mol, d) for d in dm))
    rj, rk = np.stack(rj), np.stack(rk)
    vj, vk = hf.get_jk(mol, dm, vhfopt=opt)
    assert abs(vj - rj).max() <= 1e-10
    assert abs(vk - rk).max() <= 1e-10
    vj, none = hf.get_jk(mol, dm, vhfopt=opt, with_k=False)
    assert none is None and abs(vj - rj).max() <= 1e-10
    none, vk = hf.get_jk(mol, dm, vhfopt=opt, with_j=False)
    assert none is None and abs(vk - rk).max() <= 1e-10
    vj, vk = hf.get_jk(mol, dm, vhfopt=opt, fp32_cutoff=1e-6)
    assert abs(vj - rj).max() <= 1e-9
    assert abs(vk - rk).max() <= 1e-9
    opt.clear()


def test_single_pair_runs_of_contracted_classes_vs_oracle():
    """Two waters in a six-fold contracted minimal basis: 1296 primitive
    quartets each, too few items for runs of more than one bra pair."""
    from byteqc_b200.cuobc.scf import hf
    from oracle import hf_oracle
    six = [[a, 1. / (i + 1)] for i, a in enumerate((60., 20., 7., 2.5, .9, .3))]
    mol = Mole(atom=geom.water_cluster(2, box=5.0, seed=2),
               basis={'O': [[0] + six, [1] + six], 'H': [[0] + six]}).build()
    dm = _dm(mol, 2, 3)
    opt = hf._VHFOpt(mol).build()
    rj, rk = zip(*(hf_oracle.get_jk(mol, d) for d in dm))
    for d, j, k in zip(dm, rj, rk):
        vj, vk = hf.get_jk(mol, d, vhfopt=opt)
        assert abs(vj - j).max() <= 1e-10
        assert abs(vk - k).max() <= 1e-10
    vj, vk = hf.get_jk(mol, dm, vhfopt=opt)
    assert abs(vj - np.stack(rj)).max() <= 1e-10
    assert abs(vk - np.stack(rk)).max() <= 1e-10
    opt.clear()
