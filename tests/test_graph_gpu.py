"""CUDA graphs captured from a basis handle stay valid whatever the handle
builds later: other splits of a sharded build, more densities.  And builds
that need no workspace of their own can be captured as the first of their
kind: the launch tables of the whole build come with the handle, and the first
build of a split inside a capture does without tables."""
import ctypes

import numpy as np
import pytest

from byteqc_b200.gto import Mole, geom

pytestmark = pytest.mark.gpu


def _case():
    import torch
    from byteqc_b200.cuobc.scf import hf
    mol = Mole(atom=geom.water_cluster(2, box=5.0, seed=4),
               basis='standin-def2-tzvp').build()
    opt = hf._VHFOpt(mol).build()
    rng = np.random.default_rng(8)
    d = rng.standard_normal((3, opt.nao, opt.nao))
    return opt, torch.as_tensor(d + d.transpose(0, 2, 1), device='cuda')


def _build(opt, d, vj, vk, shard=0, nshards=1, stream=None, cutoff=0.):
    from byteqc_b200.cuobc import lib as jklib
    lib = jklib.load_library()
    o = jklib.JKOpts()
    o.direct_scf_tol, o.nbins, o.prescreen = 1e-13, 10, 1
    o.shard, o.nshards, o.fp32_cutoff = shard, nshards, cutoff
    rc = lib.jk_build(opt.handle, d.data_ptr(), len(d),
                      vj.data_ptr() if vj is not None else None,
                      vk.data_ptr() if vk is not None else None,
                      ctypes.byref(o), stream)
    assert rc == 0, lib.jk_last_error()


def _capture(f):
    import torch
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        f(ctypes.c_void_p(s.cuda_stream))
    torch.cuda.current_stream().wait_stream(s)
    return g


def test_graphs_of_shards_outlive_other_splits():
    import torch
    opt, d3 = _case()
    d = d3[:1].contiguous()
    rj, rk = torch.zeros_like(d), torch.zeros_like(d)
    _build(opt, d, rj, rk)
    vj, vk = torch.zeros_like(d), torch.zeros_like(d)
    for sh in range(2):
        _build(opt, d, torch.zeros_like(d), torch.zeros_like(d), sh, 2)
    torch.cuda.synchronize()
    graphs = [_capture(lambda s: _build(opt, d, vj, vk, sh, 2, s))
              for sh in range(2)]
    # other splits, and buffers that grow
    wj, wk = torch.zeros_like(d3), torch.zeros_like(d3)
    for sh in range(3):
        _build(opt, d3, wj, wk, sh, 3)
    junk = [torch.full((1 << 18,), float('nan'), dtype=torch.float64,
                       device='cuda') for _ in range(64)]
    for rep in range(2):
        vj.zero_()
        vk.zero_()
        for g in graphs:
            g.replay()
        torch.cuda.synchronize()
        assert (vj - rj).abs().max().item() <= 1e-10
        assert (vk - rk).abs().max().item() <= 1e-10
    assert (wj[0] - rj[0]).abs().max().item() <= 1e-10
    assert (wk[0] - rk[0]).abs().max().item() <= 1e-10
    del junk


@pytest.mark.parametrize('cutoff', [0., 1e-3])
def test_first_builds_inside_a_capture(cutoff):
    import torch
    opt, d3 = _case()
    d = d3[:1].contiguous()
    tol = 1e-10 if cutoff == 0. else 1e-4  # FP32 quartets up to 1e-3 each
    # K alone, the handle's very first build
    vk = torch.zeros_like(d)
    torch.cuda.synchronize()
    g = _capture(lambda s: _build(opt, d, None, vk, 0, 1, s, cutoff))
    g.replay()
    torch.cuda.synchronize()
    rj, rk = torch.zeros_like(d), torch.zeros_like(d)
    _build(opt, d, rj, rk)
    assert (vk - rk).abs().max().item() <= tol
    # the first build of a split, the J workspace being there
    vj = torch.zeros_like(d)
    vk.zero_()
    torch.cuda.synchronize()
    for sh in range(3):
        g = _capture(lambda s: _build(opt, d, vj, vk, sh, 3, s, cutoff))
        g.replay()
    torch.cuda.synchronize()
    assert (vj - rj).abs().max().item() <= tol
    assert (vk - rk).abs().max().item() <= tol


def test_side_stream_right_after_set_up():
    """Builds on a non-blocking stream right after the basis, the tables of a
    split or those of a batch were made, with nothing in between that would
    wait for their uploads."""
    import torch
    from byteqc_b200.cuobc.scf import hf
    from byteqc_b200.cuobc.scf.batch import JKBatch
    mol = Mole(atom=geom.water_cluster(2, box=5.0, seed=4),
               basis='standin-def2-tzvp').build()
    rng = np.random.default_rng(8)
    dm = rng.standard_normal((mol.nao, mol.nao))
    d = torch.as_tensor(dm + dm.T, device='cuda')
    opt = hf._VHFOpt(mol).build()
    rj, rk = hf.get_jk(mol, d, vhfopt=opt, out='device')
    w = (opt.coeff_dev @ d @ opt.coeff_dev.T).contiguous()[None]
    raw = torch.zeros_like(w), torch.zeros_like(w)
    _build(opt, w, *raw)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    sp = ctypes.c_void_p(s.cuda_stream)
    for rep in range(10):
        with torch.cuda.stream(s):
            o = hf._VHFOpt(mol).build()
            vj, vk = hf.get_jk(mol, d, vhfopt=o, out='device')
            assert (vj - rj).abs().max().item() <= 1e-10
            assert (vk - rk).abs().max().item() <= 1e-10
            vj, vk = torch.zeros_like(w), torch.zeros_like(w)
            for sh in range(2):
                _build(o, w, vj, vk, sh, 2, sp)
            assert (vj - raw[0]).abs().max().item() <= 1e-10
            assert (vk - raw[1]).abs().max().item() <= 1e-10
            b = JKBatch([mol, mol], vhfopts=[o, opt])
            for vj, vk in b.get_jk([d, d], out='device'):
                assert (vj - rj).abs().max().item() <= 1e-10
                assert (vk - rk).abs().max().item() <= 1e-10
            b.close()
            o.clear()
