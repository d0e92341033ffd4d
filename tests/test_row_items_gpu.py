"""Row items (plain builds: lanes keep their ket pair, the bra pairs of one
second shell pass by) against pair items (the multi-density build of a single
density), over labels, symmetric and general densities, thresholds, elements,
basis sets and work-item lengths.  Both sum the same FP64 contributions in
another order: 1e-12 of the largest element is about 1e4 roundings."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

METHANE_AND_HF = """C 0.0 0.0 0.0
H 0.63 0.63 0.63
H -0.63 -0.63 0.63
H -0.63 0.63 -0.63
H 0.63 -0.63 -0.63
F 2.9 0.1 -0.2
H 3.8 0.2 -0.1"""


def _screener(which, basis):
    from veloxchem_b200 import MolecularBasis, Molecule, T4CScreener
    from veloxchem_b200.geometry import water_cluster
    mol = Molecule.read_str(METHANE_AND_HF) if which == 'mixed' else water_cluster((3, 2, 2) if which <= 12 else (4, 3, 2), 11, which)
    scr = T4CScreener()
    scr.partition(MolecularBasis.read(mol, basis), mol, 'eri')
    return scr


def _density(n, symmetric, seed=0):
    a = np.random.default_rng(seed).standard_normal((n, n))
    return (a + a.T) / 2 if symmetric else a


def _rows(scr, d, symmetric, label, ith, omega=0.3, rank=0, nodes=1):
    from veloxchem_b200 import _native as nat
    out = np.zeros_like(d)
    nat.check(nat.lib().vlx_b200_fock_build_local(scr.handle, rank, nodes, nat.dptr(d), symmetric, label.encode(), 0.25,
                                                  omega, ith, nat.dptr(out), None), 'fock_build')
    return out


def _pairs(scr, d, symmetric, label, ith, omega=0.3):
    from veloxchem_b200 import _native as nat
    out = np.zeros_like(d)
    dp = (ctypes.POINTER(ctypes.c_double) * 1)(nat.dptr(d))
    op = (ctypes.POINTER(ctypes.c_double) * 1)(nat.dptr(out))
    lp = (ctypes.c_char_p * 1)(label.encode())
    nat.check(nat.lib().vlx_b200_fock_build_multi(scr.handle, 0, 1, 1, dp, symmetric, lp, 0.25, omega, ith, op, None),
              'fock_build_multi')
    return out


def _close(a, b, tol=1e-12):
    return np.max(np.abs(a - b)) < tol * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize('which,basis', [(1, 'sto-3g'), (1, 'def2-tzvp'), (3, 'def2-svpd'), (7, 'def2-svp'),
                                         ('mixed', 'def2-tzvp'), ('mixed', 'def2-svp')])
@pytest.mark.parametrize('symmetric', [1, 0])
def test_row_items_equal_pair_items(which, basis, symmetric):
    scr = _screener(which, basis)
    d = _density(scr.nao, symmetric)
    for label in ('2jk', '2jkx', 'j', 'k', 'kx', 'j_rs', 'k_rs'):
        assert _close(_rows(scr, d, symmetric, label, 12), _pairs(scr, d, symmetric, label, 12)), label
    for ith in (0, 3, 7, 15):
        assert _close(_rows(scr, d, symmetric, '2jk', ith), _pairs(scr, d, symmetric, '2jk', ith)), ith


def _longest_rows(scr, ith):
    """Longest row of each compiled class of the cached plain list."""
    from veloxchem_b200 import _native as nat
    return {c: w.longest for c, w in nat.work_list(scr, ith).items() if w.rows}


@pytest.mark.parametrize('symmetric', [1, 0])
def test_row_lengths_filters_and_shares(symmetric):
    """Rows of up to 32, 8 and 4 bra pairs: a cluster large enough that the work of
    its s and p classes fills every SM at these lengths."""
    scr = _screener(24, 'def2-svp')
    d = _density(scr.nao, symmetric, 4)
    ref = {ith: _pairs(scr, d, symmetric, '2jk', ith) for ith in (6, 9, 12)}
    for factor, length in ((1, 32), (4, 8), (128, 4)):
        scr.set_block_size_factor(factor)
        assert _close(_rows(scr, d, symmetric, '2jk', 12), ref[12])
        longest = _longest_rows(scr, 12)
        assert max(longest.values()) == length
        assert all(longest[c] == length for c in ((0, 0, 0, 0), (0, 1, 0, 0), (0, 1, 0, 1), (1, 1, 0, 1))), longest
    scr.set_block_size_factor(1)
    scr.set_fp32_threshold(1e-6, float(np.max(np.abs(d))))  # rows of 32 cut at the FP32 boundary
    assert np.max(np.abs(_rows(scr, d, symmetric, '2jk', 12) - ref[12])) < 1e-8 + 1e-12 * np.max(np.abs(ref[12]))
    scr.set_fp32_threshold(0.0, 0.0)
    scr.set_work_threshold(14)  # one list, filtered at run time
    for ith, want in ref.items():
        assert _close(_rows(scr, d, symmetric, '2jk', ith), want)
    for partition in ('round_robin', 'balanced'):
        scr.set_partition(partition)
        assert _close(sum(_rows(scr, d, symmetric, '2jk', 12, rank=r, nodes=3) for r in range(3)), ref[12])


@pytest.mark.parametrize('symmetric', [1, 0])
def test_long_rows_of_large_classes(symmetric):
    """Rows of several bra pairs of the d and f classes whose blocks walk them in
    step, whole and cut at the FP32 boundary (tolerance as below)."""
    scr = _screener(24, 'def2-tzvp')
    d = _density(scr.nao, symmetric, 6)
    want = _pairs(scr, d, symmetric, '2jk', 12)
    assert _close(_rows(scr, d, symmetric, '2jk', 12), want)
    longest = _longest_rows(scr, 12)
    assert longest[0, 3, 1, 2] >= 8 and longest[1, 3, 0, 2] >= 8 and longest[1, 2, 1, 2] >= 4, longest
    scr.set_fp32_threshold(1e-6, float(np.max(np.abs(d))))
    assert np.max(np.abs(_rows(scr, d, symmetric, '2jk', 12) - want)) < 1e-8 + 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize('which,basis', [(7, 'def2-svp'), (2, 'def2-tzvp')])
def test_fp32_split_of_rows(which, basis):
    """The decade-bin split cuts rows at the FP32 boundary: each FP32 quartet's
    bound is below the cutoff and its relative error about 1e-6, so a hundredth
    of the cutoff leaves room for 1e4 such quartets per element."""
    scr = _screener(which, basis)
    d = _density(scr.nao, 1, 2)
    want = _pairs(scr, d, 1, '2jk', 12)
    fp64 = _rows(scr, d, 1, '2jk', 12)
    for cutoff in (1e-9, 1e-6, 1e-3):
        scr.set_fp32_threshold(cutoff, float(np.max(np.abs(d))))
        got = _rows(scr, d, 1, '2jk', 12)
        assert np.max(np.abs(got - want)) < 1e-2 * cutoff + 1e-12 * np.max(np.abs(want))
    # far above what another order of the additions changes
    assert np.max(np.abs(got - fp64)) > 1e3 * max(np.max(np.abs(fp64 - want)), 1e-13)
