"""Builds whose class launches run on side streams (classes that cannot fill
the chip) keep the order of the caller's stream: back-to-back builds of
different densities into different outputs, nothing waited for in between,
equal the builds with all launches in turn (vlx_b200_fock_build_noalloc), also
replayed from a captured graph.  Both sum the same FP64 contributions in
another order: 1e-11 is 1e4 roundings of the largest elements (about 10)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _build(entry, scr, d, f, stream, symmetric):
    from veloxchem_b200 import _native as nat
    nat.check(getattr(nat.lib(), entry)(scr.handle, ctypes.c_void_p(d.data_ptr()), symmetric, b'2jk', 1.0, 0.0, 12,
                                        ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(stream.cuda_stream)), entry)


@pytest.mark.parametrize('n,basis,symmetric', [(1, 'def2-svp', 1), (3, 'def2-svp', 0), (2, 'def2-tzvp', 1),
                                               (13, 'def2-svp', 1)])
def test_overlapped_builds_keep_stream_order(n, basis, symmetric):
    import torch
    from veloxchem_b200 import MolecularBasis, T4CScreener
    from veloxchem_b200.geometry import water_cluster
    mol = water_cluster((3, 3, 2), 5, n)
    scr = T4CScreener()
    scr.partition(MolecularBasis.read(mol, basis), mol, 'eri')
    rng = np.random.default_rng(n)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        dens = []
        for _ in range(3):
            a = rng.standard_normal((scr.nao, scr.nao))
            dens.append(torch.from_numpy((a + a.T) / 2 if symmetric else a).cuda())
        d, outs = torch.empty_like(dens[0]), [torch.empty_like(x) for x in dens]
        for x, f in zip(dens, outs):
            d.copy_(x)  # the density is overwritten as soon as the stream allows
            _build('vlx_b200_fock_build_device', scr, d, f, stream, symmetric)
        refs = [torch.empty_like(x) for x in dens]
        for x, f in zip(dens, refs):
            _build('vlx_b200_fock_build_noalloc', scr, x, f, stream, symmetric)
    stream.synchronize()
    for f, r in zip(outs, refs):
        assert float((f - r).abs().max()) < TOL
    graph = torch.cuda.CUDAGraph()
    f = torch.empty_like(d)
    with torch.cuda.graph(graph, stream=stream):
        _build('vlx_b200_fock_build_device', scr, d, f, stream, symmetric)
    for x, r in zip(dens, refs):
        d.copy_(x)
        f.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert float((f - r).abs().max()) < TOL
