"""The ERI fill runs a class pair (ij|kl) whose kernel exists only for the
other order as (kl|ij), with the two sets of bins exchanged: both orders keep
the same quartets whenever both sets of bins start at pair 0.  Checked on the
host with jk_class_pair_tasks (the row prefixes the device uses) for random
bins, empty ones among them, and classes larger than the bins cover."""
import numpy as np
import pytest

from byteqc_b200.cuobc import lib as jklib


def _kept(lib, bij, bkl, nbins, n_ij, n_kl):
    q = np.zeros(n_ij + 1, dtype=np.int64)
    tot = np.zeros(1, dtype=np.int64)
    assert lib.jk_class_pair_tasks(bij.ctypes.data, bkl.ctypes.data, nbins,
                                   n_ij, 0, q.ctypes.data,
                                   tot.ctypes.data) == 0
    return np.arange(n_kl)[None, :] < np.diff(q)[:, None]


@pytest.mark.parametrize('seed', range(20))
def test_swapped_bins_keep_the_same_quartets(seed):
    lib = jklib.load_library()
    rng = np.random.default_rng(seed)
    nbins = int(rng.integers(1, 12))
    bij, bkl = (np.append(0, np.sort(rng.integers(0, 30, nbins))).astype(
        np.int32) for _ in range(2))
    n_ij = int(bij[-1] + rng.integers(0, 3))
    n_kl = int(bkl[-1] + rng.integers(0, 3))
    a = _kept(lib, bij, bkl, nbins, n_ij, n_kl)
    b = _kept(lib, bkl, bij, nbins, n_kl, n_ij)
    np.testing.assert_array_equal(a, b.T)
