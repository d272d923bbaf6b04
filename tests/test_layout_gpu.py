"""Layout of the raw J and K that the C-ABI accumulates (GINTbuild_jk's,
cuobc/lib/gvhf/nr_jk_driver.cu:227-284): element (a, b) at a + nao*b, for every
class -- run kernels, team kernels and the generic kernel -- and for every
entry that hands the raw matrices out.  A class pair (gi gj | gk gl) of four
different groups adds K_ik, K_il, K_jk and K_jl and nothing to their mirror
images, which is what a kernel that writes rows for columns gets wrong while
V + V^T stays right."""
import ctypes

import numpy as np
import pytest

from byteqc_b200.gto import Mole, basis, geom

pytestmark = pytest.mark.gpu


def _setup(n, bas, n_dm=1):
    import torch
    from byteqc_b200.cuobc.scf import hf
    if bas == 'tzvp+g':
        bas = {'O': basis.load('standin-def2-tzvp', 'O') + [[4, [1.2, 1.0]]],
               'H': basis.load('standin-def2-tzvp', 'H')}
    mol = Mole(atom=geom.water_cluster(n, box=min(3.0 + n, 11.0), seed=n),
               basis=bas).build()
    opt = hf._VHFOpt(mol).build()
    rng = np.random.default_rng(5)
    d = rng.standard_normal((n_dm, opt.nao, opt.nao))
    return opt, torch.as_tensor(d + d.transpose(0, 2, 1), device='cuda')


def _class_pairs(opt, d, fn, each=None):
    """Raw J and K of every class pair, all quartets kept; each(c, vj, vk)
    after every call on cleared matrices, else summed."""
    import torch
    vj, vk = torch.zeros_like(d), torch.zeros_like(d)
    for cij in range(len(opt.log_qs)):
        for ckl in range(cij + 1):
            bij, bkl = (np.array([0, len(opt.log_qs[c])], np.int32)
                        for c in (cij, ckl))
            rc = fn(opt.handle, vj.data_ptr(), vk.data_ptr(), d.data_ptr(),
                    opt.nao, len(d), bij.ctypes.data, bkl.ctypes.data, 1, cij,
                    ckl, None)
            assert rc == 0
            torch.cuda.synchronize()
            if each:
                each(cij, ckl, vj, vk)
                vj.zero_()
                vk.zero_()
    return vj, vk


def _opts(opt, cutoff=0.):
    from byteqc_b200.cuobc import lib as jklib
    o = jklib.JKOpts()
    o.direct_scf_tol = 1e-30  # every quartet
    o.nbins = 10
    o.prescreen = 0
    o.fp32_cutoff = cutoff
    return o


@pytest.mark.parametrize('entry', ['jk_build_class_pair',
                                   'jk_build_class_pair_noalloc'])
@pytest.mark.parametrize('n_dm', [1, 2])
def test_class_pair_k_blocks(entry, n_dm):
    from byteqc_b200.cuobc import lib as jklib
    lib = jklib.load_library()
    opt, d = _setup(1, 'tzvp+g', n_dm)
    gao = opt.mol.ao_loc_nr(cart=True)[opt.l_ctr_offsets]
    cls = [(i, j) for i in range(len(gao) - 1) for j in range(i + 1)]
    seen = set()

    def check(cij, ckl, vj, vk):
        g = cls[cij] + cls[ckl]
        if len(set(g)) < 4:
            return
        seen.add(g)
        pairs = {(a, b) for a in g[:2] for b in g[2:]}
        for a in set(g):
            for b in set(g):
                # element (x, y) at x + nao y: rows y, columns x of the tensor
                blk = vk[:, gao[b]:gao[b + 1], gao[a]:gao[a + 1]]
                assert (blk.abs().max().item() > 0) == ((a, b) in pairs), (g, a, b)
    _class_pairs(opt, d, getattr(lib, entry), check)
    assert len(seen) > 20


@pytest.mark.parametrize('bas,n', [
    ('standin-cc-pvdz', 3), ('tzvp+g', 1),
    ('standin-cc-pvdz', 22)])  # classes of more than 8192 pairs
@pytest.mark.parametrize('cutoff', [0., 1e-3])
def test_raw_entries_agree(bas, n, cutoff):
    """jk_build, the same without J as a captured build whose K buffer was
    never allocated, and jk_batch_build against the per-class-pair entry,
    element by element of the raw matrices (accumulated onto other values)."""
    import torch
    from byteqc_b200.cuobc import lib as jklib
    lib = jklib.load_library()
    opt, d = _setup(n, bas, 2)
    assert n < 22 or max(len(q) for q in opt.log_qs) > 8192
    rj, rk = _class_pairs(opt, d, lib.jk_build_class_pair)
    base = torch.randn_like(d)
    tol = 1e-10 if cutoff == 0. else 1e-4  # FP32 quartets up to 1e-3 each
    o = _opts(opt, cutoff)

    def build(vj, vk, stream=None):
        assert lib.jk_build(opt.handle, d.data_ptr(), len(d),
                            vj.data_ptr() if vj is not None else None,
                            vk.data_ptr() if vk is not None else None,
                            ctypes.byref(o), stream) == 0, lib.jk_last_error()
    vj, vk = base.clone(), base.clone()
    build(vj, None)  # launch tables, J workspaces
    torch.cuda.synchronize()
    assert (vj - base - rj).abs().max().item() <= tol
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        build(None, vk, ctypes.c_void_p(s.cuda_stream))
    g.replay()
    torch.cuda.synchronize()
    assert (vk - base - rk).abs().max().item() <= tol
    for _ in range(2):
        vj, vk = base.clone(), base.clone()
        build(vj, vk)
        torch.cuda.synchronize()
        assert (vj - base - rj).abs().max().item() <= tol
        assert (vk - base - rk).abs().max().item() <= tol
    h = ctypes.c_void_p()
    arr = (ctypes.c_void_p * 1)(opt.handle.value)
    assert lib.jk_batch_create(arr, 1, ctypes.byref(h)) == 0
    for with_j in (True, False):
        vj, vk = base.clone(), base.clone()
        pd, pj, pk = ((ctypes.c_void_p * 1)(x.data_ptr()) for x in (d, vj, vk))
        assert lib.jk_batch_build(h, pd, pj if with_j else None, pk, len(d),
                                  ctypes.byref(o), None) == 0
        torch.cuda.synchronize()
        if with_j:
            assert (vj - base - rj).abs().max().item() <= tol
        assert (vk - base - rk).abs().max().item() <= tol
    lib.jk_batch_destroy(h)
    opt.clear()


def test_class_pair_without_densities_adds_nothing():
    """n_dm = 0 is a call with nothing to do, on run and team classes alike
    (full-size buffers: a kernel that took it for one density stays inside)."""
    import torch
    from byteqc_b200.cuobc import lib as jklib
    lib = jklib.load_library()
    opt, d = _setup(1, 'standin-def2-tzvp')

    def fn(handle, vj, vk, dm, nao, n_dm, *a):
        return lib.jk_build_class_pair(handle, vj, vk, dm, nao, 0, *a)
    vj, vk = _class_pairs(opt, d, fn)
    assert not vj.any().item() and not vk.any().item()


@pytest.mark.parametrize('bas', ['standin-cc-pvdz', 'tzvp+g'])
def test_class_pair_call_is_two_launches(bas):
    """A per-class-pair call of a small molecule is one preparation and one
    class kernel: its latency is what such a call costs (five launches took
    1.6 times as long for 13 atoms / TZVP)."""
    import torch
    from cuda.bindings import runtime as cudart
    from byteqc_b200.cuobc import lib as jklib
    lib = jklib.load_library()
    opt, d = _setup(1, bas)
    vj, vk = torch.zeros_like(d), torch.zeros_like(d)
    _class_pairs(opt, d, lib.jk_build_class_pair)
    for cij in range(len(opt.log_qs)):
        bij = np.array([0, len(opt.log_qs[cij])], np.int32)
        g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(g, stream=s):
            assert lib.jk_build_class_pair(
                opt.handle, vj.data_ptr(), vk.data_ptr(), d.data_ptr(),
                opt.nao, 1, bij.ctypes.data, bij.ctypes.data, 1, cij, cij,
                ctypes.c_void_p(s.cuda_stream)) == 0
        err, _, n = cudart.cudaGraphGetNodes(
            cudart.cudaGraph_t(g.raw_cuda_graph()), 0)
        assert err == cudart.cudaError_t.cudaSuccess
        assert n == 2


def test_noalloc_entry_on_more_than_8192_bra_pairs():
    """Above 8192 bra pairs a call is prepared by several launches instead of
    one block: the no-alloc entry against the allocating one on the largest
    class of (H2O)22, with itself (diagonal) and with the smallest class, the
    bins cutting it off in the middle."""
    import torch
    from byteqc_b200.cuobc import lib as jklib
    from byteqc_b200.cuobc.scf import hf
    lib = jklib.load_library()
    opt, d = _setup(22, 'standin-cc-pvdz')
    sizes = [len(q) for q in opt.log_qs]
    big = int(np.argmax(sizes))
    assert sizes[big] > 8192
    small = min((n, i) for i, n in enumerate(sizes) if n)[1]
    for cij, ckl in ((big, big), (max(big, small), min(big, small))):
        bij, bkl = (hf._make_s_index_offsets(opt.log_qs[c], 10, 1e-9)
                    for c in (cij, ckl))
        out = []
        for fn in (lib.jk_build_class_pair, lib.jk_build_class_pair_noalloc):
            vj, vk = torch.zeros_like(d), torch.zeros_like(d)
            assert fn(opt.handle, vj.data_ptr(), vk.data_ptr(), d.data_ptr(),
                      opt.nao, 1, bij.ctypes.data, bkl.ctypes.data, 10, cij,
                      ckl, None) == 0
            torch.cuda.synchronize()
            out.append((vj, vk))
        assert out[0][0].abs().max().item() > 0
        for a, b in zip(*out):
            assert (a - b).abs().max().item() <= 1e-10
    opt.clear()
