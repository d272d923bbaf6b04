"""The generic J/K kernel against the CPU oracle where its two ways of digesting
meet: classes whose integrals fit one range of components, classes of a few
ranges, and classes of many ranges, which are summed from the 2D blocks
directly -- contracted and uncontracted, with several batches of roots.  1e-10
absolute, as the other J/K tests."""
import numpy as np
import pytest

from byteqc_b200.gto import Mole

pytestmark = pytest.mark.gpu

S, P, D = [0, [1.3, 1.0]], [1, [0.9, 1.0]], [2, [0.8, .7], [.35, .5]]
F = [3, [0.7, 1.0]]


@pytest.mark.parametrize('shells,n_dm', [
    ([S, P, D, [4, [1.1, 0.6], [0.5, 0.5]]], 1),  # contracted (gg|gg), (gd|dd)
    ([S, D, F, [4, [0.9, 1.0]]], 3),              # (gf|fd): a few ranges
    ([S, P, [5, [0.8, 1.0]]], 2),                 # (hh|hh): 74 ranges
    ([S, [4, [0.9, 1.0]], [6, [0.7, 1.0]]], 1)])  # (ii|ii): 13 roots
def test_generic_kernel_vs_oracle(shells, n_dm):
    from byteqc_b200.cuobc.scf import hf
    from oracle import hf_oracle
    mol = Mole(atom=[('H', (0., 0., 0.)), ('H', (0.3, 0.5, 0.9))],
               basis={'H': shells}).build()
    rng = np.random.default_rng(len(shells))
    d = rng.standard_normal((n_dm, mol.nao, mol.nao))
    d = d + d.transpose(0, 2, 1)
    opt = hf._VHFOpt(mol).build()
    rj, rk = (np.stack(x) for x in zip(*(hf_oracle.get_jk(mol, x) for x in d)))
    vj, vk = hf.get_jk(mol, d, vhfopt=opt)
    assert abs(vj - rj).max() <= 1e-10
    assert abs(vk - rk).max() <= 1e-10
    vj, none = hf.get_jk(mol, d, vhfopt=opt, with_k=False)
    assert none is None and abs(vj - rj).max() <= 1e-10
    opt.clear()
