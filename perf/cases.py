"""Performance cases: the work a user of this framework has it do, through its
public entry points, over the range of sizes, data types and options in use.

Kinds of a case (all on seeded water clusters, the framework's workloads):

* ``fock``      one Fock matrix through ``FockDriver.compute`` (host matrices);
* ``device``    the device-resident build of an SCF iteration
                (``vlx_b200_fock_build_device``), plain FP64;
* ``screened``  the same entry point with per-quartet density screening and
                mixed precision on a density difference, as the incremental
                (FP64 digestion) and the early (FP32 digestion) iterations of
                the SCF driver call it;
* ``multi``     several general densities in one ``FockDriver.compute``;
* ``batch``     ``FockBatch.build_device`` over clusters of uneven size;
* ``scf``       a whole restricted Hartree-Fock run;
* ``train``     one training step (forward, backward, Adam) of the guess network.

``exact`` restates the Fock matrices with the McMurchie-Davidson scheme and the
network step with plain formulas, in 64-bit torch, from the shell tables and
coordinates alone.
"""

import ctypes
import math

import numpy as np
import torch

from veloxchem_b200 import FockDriver, Matrices, MolecularBasis, T4CScreener, make_matrix, mat_t
from veloxchem_b200 import _native as nat
from veloxchem_b200.batch import FockBatch
from veloxchem_b200.geometry import random_density, water_cluster
from veloxchem_b200.guess_net import GuessMLP
from veloxchem_b200.scf import ScfRestrictedDriver

ITHRESHOLD = 12
NET_IN, NET_OUT = 134, 196  # the shipped guess network's input and output widths


def listed():
    return [
        # the smallest build: one molecule in the reference's API, latency of the call and its launches
        {'name': 'fock_1_svp', 'kind': 'fock', 'n': 1, 'basis': 'def2-svp', 'label': '2jk'},
        # BASELINE's first workload: a small cluster, Fock matrix through the reference's API
        {'name': 'fock_4_svp', 'kind': 'fock', 'n': 4, 'basis': 'def2-svp', 'label': '2jk'},
        # ordinary size in a triple-zeta basis (f shells), through the reference's API
        {'name': 'fock_8_tzvp', 'kind': 'fock', 'n': 8, 'basis': 'def2-tzvp', 'label': '2jk'},
        # Coulomb matrix alone, odd size, as density fitting checks and pure functionals need it
        {'name': 'j_13_svp', 'kind': 'fock', 'n': 13, 'basis': 'def2-svp', 'label': 'j'},
        # long-range exchange of a range-separated functional with a general (response) density
        {'name': 'krs_11_svp', 'kind': 'fock', 'n': 11, 'basis': 'def2-svp', 'label': 'k_rs', 'general': True},
        # the bench workload: one SCF iteration's build on resident matrices
        {'name': 'device_32_svp', 'kind': 'device', 'n': 32, 'basis': 'def2-svp', 'label': '2jk'},
        # the largest single build that is timed: triple zeta, 1161 functions
        {'name': 'device_27_tzvp', 'kind': 'device', 'n': 27, 'basis': 'def2-tzvp', 'label': '2jk'},
        # an incremental iteration of the mixed-precision SCF in triple zeta
        {'name': 'incremental_16_tzvp', 'kind': 'screened', 'n': 16, 'basis': 'def2-tzvp', 'ith': 12, 'early': False},
        # several response vectors digested in one pass (general densities)
        {'name': 'multi_6_svp', 'kind': 'multi', 'n': 6, 'basis': 'def2-svp', 'ndens': 3},
        # many independent molecules of uneven size in one call
        {'name': 'batch_48_svp', 'kind': 'batch', 'count': 48, 'nmax': 16, 'basis': 'def2-svp'},
        # a whole SCF from the SAD guess: integrals, builds, DIIS and diagonalisation
        {'name': 'scf_8_svp', 'kind': 'scf', 'n': 8, 'basis': 'def2-svp', 'mixed': False},
        # one training step of the guess network (batch of the shipped training)
        {'name': 'train_4096', 'kind': 'train', 'm': 4096},
    ]


def _between(rng, lo, hi):
    """Whole number spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(('fock', 'fock', 'device', 'device', 'screened', 'multi', 'batch', 'scf', 'train'))
    basis = rng.choice(('def2-svp', 'def2-tzvp'))
    svp = basis == 'def2-svp'
    if kind == 'fock':
        label = rng.choice(('2jk', '2jk', 'j', 'k', 'k_rs', '2jkx'))
        general = rng.random() < 0.25
        return {'kind': kind, 'n': _between(rng, 1, 24 if svp else 10), 'basis': basis, 'label': label,
                'general': general}
    if kind == 'device':
        return {'kind': kind, 'n': _between(rng, 6, 40 if svp else 22), 'basis': basis,
                'label': rng.choice(('2jk', '2jk', 'j', 'k'))}
    if kind == 'screened':
        early = rng.random() < 0.4
        return {'kind': kind, 'n': _between(rng, 4, 32 if svp else 16), 'basis': basis, 'ith': 8 if early else 12,
                'early': early}
    if kind == 'multi':
        return {'kind': kind, 'n': _between(rng, 1, 10 if svp else 4), 'basis': basis, 'ndens': rng.randint(2, 6)}
    if kind == 'batch':
        return {'kind': kind, 'count': _between(rng, 5, 40), 'nmax': rng.randint(2, 16), 'basis': 'def2-svp'}
    if kind == 'scf':
        return {'kind': kind, 'n': _between(rng, 1, 9 if svp else 4), 'basis': basis, 'mixed': rng.random() < 0.5}
    return {'kind': kind, 'm': _between(rng, 100, 4096)}


# ------------------------------------------------------------------- inputs

def _cluster(n, seed):
    """n waters on a near-cubic lattice (4, 4, 2 for the 32 of the bench workload)."""
    nx = math.ceil(n ** (1.0 / 3.0) - 1e-9)
    ny = math.ceil(math.sqrt(n / nx) - 1e-9)
    nz = math.ceil(n / (nx * ny))
    return water_cluster((4, 4, 2) if n == 32 else (nx, ny, nz), seed, n)


def _batch_sizes(case):
    """Waters of each cluster of a batch, uniform in 1..nmax."""
    return [int(v) for v in np.random.default_rng(7).integers(1, case['nmax'] + 1, size=case['count'])]


def _molecule(case, seed):
    mol = _cluster(case['n'], 1000 + seed)
    return mol, MolecularBasis.read(mol, case['basis'])


def _general_density(nao, nocc, seed):
    """A non-symmetric density of the size a response vector has."""
    d = random_density(nao, nocc, seed)
    return d + 0.1 * np.random.default_rng(seed + 77).standard_normal((nao, nao)) / math.sqrt(nao)


def _difference_density(mol, basis, seed, scale):
    """Symmetric density difference that falls off with the distance of its
    two functions, as between two SCF iterations."""
    nao = basis.get_dimensions_of_basis()
    centre = np.zeros((nao, 3))
    xyz = mol.get_coordinates_in_bohr()
    for shell, idx in zip(basis.shells, basis.ao_indices()):
        centre[idx] = xyz[shell.atom]
    r = np.sqrt(np.maximum(0.0, ((centre[:, None, :] - centre[None, :, :]) ** 2).sum(-1)))
    d = np.random.default_rng(seed).standard_normal((nao, nao)) * np.exp(-0.7 * r)
    return scale * 0.5 * (d + d.T)


def _host_inputs(case, seed):
    """The molecule, basis and host density matrices of a case."""
    mol, basis = _molecule(case, seed)
    nao, nocc = basis.get_dimensions_of_basis(), 5 * case['n']
    if case['kind'] == 'screened':
        return mol, basis, [_difference_density(mol, basis, seed + 5, 1e-2 if case['early'] else 1e-4)]
    if case['kind'] == 'multi':
        return mol, basis, [_general_density(nao, nocc, seed + 5 + k) for k in range(case['ndens'])]
    make = _general_density if case.get('general') else random_density
    return mol, basis, [make(nao, nocc, seed + 5)]


def _network(case, seed):
    net = GuessMLP(NET_IN, NET_OUT, seed=seed)
    g = torch.Generator(device='cpu').manual_seed(seed + 5)
    x = torch.randn(case['m'], NET_IN, generator=g)
    t = 0.1 * torch.randn(case['m'], NET_OUT, generator=g)
    mask = (torch.rand(case['m'], NET_OUT, generator=g) < 0.6).float()
    return net, x, t, mask


def prepare(case, seed):
    kind = case['kind']
    if kind == 'batch':
        screeners, dens = [], []
        for i, n in enumerate(_batch_sizes(case)):
            mol = water_cluster((3, 3, 2), 100000 + 1000 * seed + i, n)
            scr = T4CScreener()
            scr.partition(MolecularBasis.read(mol, case['basis']), mol, 'eri')
            screeners.append(scr)
            dens.append(random_density(scr.nao, 5 * n, seed + i))
        batch = FockBatch(screeners)
        d = torch.from_numpy(batch.pack(dens)).cuda()
        return {'case': case, 'batch': batch, 'd': d, 'f': torch.empty_like(d)}
    if kind == 'train':
        net, x, t, mask = _network(case, seed)
        return {'case': case, 'net': net, 'x': x.cuda(), 't': t.cuda(), 'mask': mask.cuda()}
    if kind == 'scf':
        mol, basis = _molecule(case, seed)
        return {'case': case, 'mol': mol, 'basis': basis}
    mol, basis, dens = _host_inputs(case, seed)
    scr = T4CScreener()
    scr.partition(basis, mol, 'eri')
    state = {'case': case, 'screener': scr}
    if kind in ('device', 'screened'):
        state['d'] = torch.from_numpy(dens[0]).cuda()
        state['f'] = torch.empty_like(state['d'])
        if kind == 'screened':
            # the cutoffs the SCF driver sets for such an iteration
            scr.set_work_threshold(ITHRESHOLD)
            scr.set_fp32_digestion(case['early'])
            scr.set_density_screening(1e-4, (1e-1 if case['early'] else 1e-2) * 10.0 ** -case['ith'])
        return state
    mtype = mat_t.general if (kind == 'multi' or case.get('general')) else mat_t.symmetric
    mats = []
    for d in dens:
        m = make_matrix(basis, mtype)
        m.set_values(d)
        mats.append(m)
    state['driver'] = FockDriver()
    if kind == 'multi':
        state['mats'] = Matrices()
        for k, m in enumerate(mats):
            state['mats'].add(m, k)
    else:
        state['mat'] = mats[0]
    return state


def _device_build(state, ith):
    stream = torch.cuda.current_stream().cuda_stream or 1  # 1: the legacy default stream
    nat.check(nat.lib().vlx_b200_fock_build_device(state['screener'].handle, ctypes.c_void_p(state['d'].data_ptr()),
                                                    1, state['case'].get('label', '2jk').encode(), 1.0, 0.0, ith,
                                                    ctypes.c_void_p(state['f'].data_ptr()),
                                                    ctypes.c_void_p(stream)), 'fock_build')
    return state['f']


OMEGA, XFAC = 0.33, 0.25


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'fock':
        f = state['driver'].compute(state['screener'], state['mat'], case['label'], XFAC, OMEGA, ITHRESHOLD)
        return f.to_numpy()
    if kind == 'multi':
        labels = ['2jk'] * case['ndens']
        f = state['driver'].compute(state['screener'], state['mats'], labels, XFAC, 0.0, ITHRESHOLD)
        return [f.matrix(k).to_numpy() for k in range(case['ndens'])]
    if kind == 'device':
        return _device_build(state, ITHRESHOLD)
    if kind == 'screened':
        return _device_build(state, case['ith'])
    if kind == 'batch':
        return state['batch'].build_device(state['d'], state['f'])
    if kind == 'scf':
        drv = ScfRestrictedDriver()
        drv.conv_thresh = 1.0e-7
        if case['mixed']:
            drv.fp32_cutoff = 1.0e-4
            drv.full_skip_factor = 1.0e-2
        res = drv.compute(state['mol'], state['basis'])
        return {'energy': res['scf_energy'], 'D': res['D_alpha'], 'F': res['F_alpha']}
    net = state['net']
    y, cache = net.forward(state['x'], keep=True)
    loss, dy = net.mse(y, state['t'], state['mask'])
    grads = net.backward(dy, cache)
    net.adam_step(grads, lr=2e-3)
    return {'y': y, 'loss': loss, 'grads': [g for pair in grads for g in pair], 'params': net.params()}


# ---------------------------------------------------------- work and tolerance

# Operations of one 2J-K build at integral threshold 1e-12 (recursions,
# transforms and digestion of the quartets that pass the Schwarz bins; adds and
# multiplies counted once each): a polynomial in log n through counts of
# clusters of 1 to 40 (def2-svp) and 1 to 27 waters (def2-tzvp).
_LOG_FLOPS = {'def2-svp': (15.693, 3.6032, -0.14615), 'def2-tzvp': (17.902, 3.4808, -0.11595)}
_NAO = {'def2-svp': 24, 'def2-tzvp': 43}


def _build_flops(n, basis):
    c = _LOG_FLOPS[basis]
    x = math.log(n)
    return math.exp(c[0] + c[1] * x + c[2] * x * x)


def work(case):
    kind = case['kind']
    if kind == 'train':
        shapes = [(NET_IN, 128), (128, 128), (128, NET_OUT)]
        flops = sum(2 * case['m'] * k * n * (3 if i else 2) for i, (k, n) in enumerate(shapes))
        par = sum(k * n + n for k, n in shapes)
        return {'bytes': 4.0 * (case['m'] * (NET_IN + 3 * NET_OUT) + 8 * par), 'flops': float(flops)}
    if kind == 'batch':
        ns = _batch_sizes(case)
        return {'bytes': sum(16.0 * (24 * n) ** 2 for n in ns), 'flops': sum(_build_flops(n, 'def2-svp') for n in ns)}
    nao = _NAO[case['basis']] * case['n']
    flops = _build_flops(case['n'], case['basis'])
    if kind == 'scf':
        return {'bytes': 14 * 16.0 * nao * nao, 'flops': 14 * flops + 14 * 30.0 * nao ** 3}
    ndens = case.get('ndens', 1)
    return {'bytes': 16.0 * ndens * nao * nao, 'flops': flops}


def tolerance(case):
    kind = case['kind']
    if kind == 'train':
        return {'rel': 1e-5, 'max': 0.05}
    if kind == 'scf':
        return {'rel': 1e-8, 'max': 1e-6}
    if kind == 'screened':
        return {'rel': 1e-6}
    return {'rel': 1e-12, 'max': 1e-10}


# ------------------------------------------------------- exact values (64 bits)

def _components(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


# real solid harmonics m = -l..l as {Cartesian exponents: factor}, up to a norm
_HARMONICS = {
    0: [{(0, 0, 0): 1}],
    1: [{(0, 1, 0): 1}, {(0, 0, 1): 1}, {(1, 0, 0): 1}],
    2: [{(1, 1, 0): 1}, {(0, 1, 1): 1}, {(0, 0, 2): 2, (2, 0, 0): -1, (0, 2, 0): -1}, {(1, 0, 1): 1},
        {(2, 0, 0): 1, (0, 2, 0): -1}],
    3: [{(2, 1, 0): 3, (0, 3, 0): -1}, {(1, 1, 1): 1}, {(0, 1, 2): 4, (2, 1, 0): -1, (0, 3, 0): -1},
        {(0, 0, 3): 2, (2, 0, 1): -3, (0, 2, 1): -3}, {(1, 0, 2): 4, (3, 0, 0): -1, (1, 2, 0): -1},
        {(2, 0, 1): 1, (0, 2, 1): -1}, {(3, 0, 0): 1, (1, 2, 0): -3}],
}


def _double_factorial(n):
    return 1.0 if n <= 0 else n * _double_factorial(n - 2)


def _normalised(l, exps, coefs):
    """Contraction coefficients and harmonic factors of a shell whose spherical
    functions have unit norm: ([nprim], [2l + 1, ncart])."""
    def moment(c, e):  # int x^i y^j z^k exp(-e r^2)
        if any(v % 2 for v in c):
            return np.zeros_like(e)
        f = np.prod([_double_factorial(v - 1) for v in c])
        return f * (np.pi / e) ** 1.5 / (2.0 * e) ** (sum(c) / 2)
    e2 = exps[:, None] + exps[None, :]
    carts = _components(l)
    sph = np.zeros((2 * l + 1, len(carts)))
    for m, terms in enumerate(_HARMONICS[l]):
        for c, f in terms.items():
            sph[m, carts.index(c)] = f
    # primitives of the file are normalised, then the contraction is
    own = np.zeros_like(exps)
    for i, ci in enumerate(carts):
        for j, cj in enumerate(carts):
            own += sph[0, i] * sph[0, j] * moment(tuple(np.add(ci, cj)), 2.0 * exps)
    w = coefs / np.sqrt(own)
    for m in range(2 * l + 1):
        norm = 0.0
        for i, ci in enumerate(carts):
            for j, cj in enumerate(carts):
                norm += sph[m, i] * sph[m, j] * float(w @ moment(tuple(np.add(ci, cj)), e2) @ w)
        sph[m] /= math.sqrt(norm)
    return w, sph


def _device():
    return torch.device('cuda' if torch.cuda.is_available() else 'cpu')


def _tensor(v):
    return torch.as_tensor(np.ascontiguousarray(v), device=_device())


def _shells_by_l(mol, basis):
    """Per angular momentum: the shells, and per shell its primitives' slice."""
    xyz = mol.get_coordinates_in_bohr()
    atom, lval, nprim, exps, coefs = basis.shell_table()
    start = np.concatenate([[0], np.cumsum(nprim)])
    ao = basis.ao_indices()
    groups = {}
    for s in range(len(atom)):
        e, c = exps[start[s]:start[s + 1]], coefs[start[s]:start[s + 1]]
        l = int(lval[s])
        w, sph = _normalised(l, e, c)
        groups.setdefault(l, []).append((s, e, w, sph, xyz[atom[s]], ao[s]))
    return groups


def _hermite(i_max, j_max, pa, pb, p, e00):
    """Hermite expansion coefficients E[i][j][t] of one axis."""
    half = 0.5 / p
    E = {(0, 0): [e00]}

    def raise_(prev, x):
        n = len(prev)
        out = []
        for t in range(n + 1):
            v = torch.zeros_like(p)
            if t > 0:
                v = v + half * prev[t - 1]
            if t < n:
                v = v + x * prev[t]
            if t + 1 < n:
                v = v + (t + 1) * prev[t + 1]
            out.append(v)
        return out

    for i in range(i_max + 1):
        if i > 0:
            E[(i, 0)] = raise_(E[(i - 1, 0)], pa)
        for j in range(1, j_max + 1):
            E[(i, j)] = raise_(E[(i, j - 1)], pb)
    return E


def _pairs(groups, la, lb):
    """Primitive pairs of all shell pairs (A of la, B of lb, A <= B for la =
    lb): exponents, centres, shell-pair index, Hermite coefficients
    [primitive pair, na nb, hermite], and the pairs' AO indices."""
    A, B = groups[la], groups[lb]
    ids = [(i, j) for i in range(len(A)) for j in range(i if la == lb else 0, len(B))]
    cols = {k: [] for k in ('a', 'b', 'w', 'ra', 'rb', 'pair')}
    sph_a, sph_b, pao, pbo = [], [], [], []
    for k, (i, j) in enumerate(ids):
        _, ea, wa, sa, ra, aoa = A[i]
        _, eb, wb, sb, rb, aob = B[j]
        n = len(ea) * len(eb)
        cols['a'].append(np.repeat(ea, len(eb)))
        cols['b'].append(np.tile(eb, len(ea)))
        cols['w'].append(np.outer(wa, wb).ravel())
        cols['ra'].append(np.tile(ra, (n, 1)))
        cols['rb'].append(np.tile(rb, (n, 1)))
        cols['pair'].append(np.full(n, k))
        sph_a.append(sa)
        sph_b.append(sb)
        pao.append(aoa)
        pbo.append(aob)
    t = {k: _tensor(np.concatenate(v)) for k, v in cols.items()}
    t['sph_a'], t['sph_b'] = _tensor(np.stack(sph_a)), _tensor(np.stack(sph_b))
    t['ao_a'], t['ao_b'] = _tensor(np.stack(pao)), _tensor(np.stack(pbo))
    t['p'] = t['a'] + t['b']
    t['P'] = (t['a'][:, None] * t['ra'] + t['b'][:, None] * t['rb']) / t['p'][:, None]
    mu = t['a'] * t['b'] / t['p']
    t['E'] = [_hermite(la, lb, t['P'][:, x] - t['ra'][:, x], t['P'][:, x] - t['rb'][:, x], t['p'],
                       torch.exp(-mu * (t['ra'][:, x] - t['rb'][:, x]) ** 2)) for x in range(3)]
    t['npairs'] = len(ids)
    return t


def _spherical(t, cart):
    """[primitive pair, ncart_a, ncart_b, ...] -> [primitive pair, na, nb, ...]
    with the contraction weights."""
    pair = t['pair']
    out = torch.einsum('pma,pab...->pmb...', t['sph_a'][pair], cart)
    out = torch.einsum('pnb,pmb...->pmn...', t['sph_b'][pair], out)
    return out * t['w'].reshape(-1, *([1] * (out.dim() - 1)))


def _orders(l):
    return [(a, b, c) for n in range(l + 1) for a in range(n, -1, -1) for b in range(n - a, -1, -1)
            for c in (n - a - b,)]


def _hermite_matrix(t, la, lb):
    """[primitive pair, na nb, hermite orders up to la + lb]."""
    orders = _orders(la + lb)
    ca, cb = _components(la), _components(lb)
    n = t['p'].shape[0]
    cart = torch.zeros((n, len(ca), len(cb), len(orders)), dtype=torch.float64, device=t['p'].device)
    for i, a in enumerate(ca):
        for j, b in enumerate(cb):
            ex = [t['E'][x][(a[x], b[x])] for x in range(3)]
            for h, o in enumerate(orders):
                if all(o[x] < len(ex[x]) for x in range(3)):
                    cart[:, i, j, h] = ex[0][o[0]] * ex[1][o[1]] * ex[2][o[2]]
    s = _spherical(t, cart)
    return s.reshape(n, -1, len(orders))


def _boys(m, T):
    """F_0..F_m(T): series for the highest order and downward recursion below
    T = 40, the asymptotic F_0 and upward recursion above."""
    Ts = T.clamp(max=40.0)
    term = torch.full_like(Ts, 1.0 / (2 * m + 1))
    total = term.clone()
    for k in range(1, 170):
        term = term * (2.0 * Ts / (2 * m + 2 * k + 1))
        total += term
    et = torch.exp(-Ts)
    F = [None] * (m + 1)
    F[m] = et * total
    for k in range(m - 1, -1, -1):
        F[k] = (2.0 * Ts * F[k + 1] + et) / (2 * k + 1)
    big = T > 40.0
    if bool(big.any()):
        Tb = T.clamp(min=40.0)
        eb = torch.exp(-Tb)
        g = 0.5 * torch.sqrt(math.pi / Tb)
        for k in range(m + 1):
            F[k] = torch.where(big, g, F[k])
            g = ((2 * k + 1) * g - eb) / (2.0 * Tb)
    return F


def _hermite_integrals(L, alpha, X, Y, Z):
    """R_tuv of all orders up to L (stacked in _orders(L))."""
    F = _boys(L, alpha * (X * X + Y * Y + Z * Z))
    R = {(0, 0, 0, n): (-2.0 * alpha) ** n * F[n] for n in range(L + 1)}
    for n in range(L - 1, -1, -1):
        for (t, u, v) in _orders(L - n):
            if t + u + v == 0:
                continue
            ax = 0 if t else (1 if u else 2)
            o = [t, u, v]
            o[ax] -= 1
            val = (X, Y, Z)[ax] * R[(*o, n + 1)]
            if o[ax] > 0:
                low = list(o)
                low[ax] -= 1
                val = val + o[ax] * R[(*low, n + 1)]
            R[(t, u, v, n)] = val
    return torch.stack([R[(*o, 0)] for o in _orders(L)])


def _eri(mol, basis, omega):
    """The full (nao)^4 tensor; omega > 0: erf(omega r) / r."""
    groups = _shells_by_l(mol, basis)
    nao = basis.get_dimensions_of_basis()
    dev = _device()
    G = torch.zeros((nao,) * 4, dtype=torch.float64, device=dev)
    ls = sorted(groups)
    classes = []
    for la in ls:
        for lb in ls:
            if la <= lb:
                t = _pairs(groups, la, lb)
                classes.append((la, lb, t, _hermite_matrix(t, la, lb) / t['p'][:, None, None]))
    for x, (la, lb, tb, Eb) in enumerate(classes):
        for (lc, ld, tk, Ek) in classes[:x + 1]:
            ob, ok = _orders(la + lb), _orders(lc + ld)
            L = la + lb + lc + ld
            pos = {o: i for i, o in enumerate(_orders(L))}
            idx = torch.tensor([[pos[tuple(np.add(o, q))] for q in ok] for o in ob], device=dev)
            sign = torch.tensor([(-1.0) ** sum(q) for q in ok], dtype=torch.float64, device=dev)
            Es = Ek * sign
            nk = tk['p'].shape[0]
            V = torch.zeros((tb['npairs'], Eb.shape[1], tk['npairs'], Ek.shape[1]), dtype=torch.float64, device=dev)
            step = max(1, int(4e7 // (nk * (len(pos) * 3 + 40))))
            for b0 in range(0, tb['p'].shape[0], step):
                sl = slice(b0, b0 + step)
                p, q = tb['p'][sl, None], tk['p'][None, :]
                alpha = p * q / (p + q)
                pref = 2.0 * math.pi ** 2.5 / torch.sqrt(p + q)
                if omega > 0.0:
                    s = omega ** 2 / (omega ** 2 + alpha)
                    pref = pref * torch.sqrt(s)
                    alpha = alpha * s
                d = [tb['P'][sl, None, c] - tk['P'][None, :, c] for c in range(3)]
                R = _hermite_integrals(L, alpha, *d) * pref
                half = torch.zeros((p.shape[0], len(ob), tk['npairs'], Ek.shape[1]), dtype=torch.float64, device=dev)
                for h in range(len(ob)):
                    prim = torch.einsum('hbk,kch->bkc', R[idx[h]], Es)
                    half[:, h].index_add_(1, tk['pair'], prim)
                V.index_add_(0, tb['pair'][sl], torch.einsum('bhkc,bah->bakc', half, Eb[sl]))
            na, nb, nc, nd = 2 * la + 1, 2 * lb + 1, 2 * lc + 1, 2 * ld + 1
            V = V.reshape(tb['npairs'], na, nb, tk['npairs'], nc, nd)
            i = tb['ao_a'][:, :, None, None, None, None]
            j = tb['ao_b'][:, None, :, None, None, None]
            k = tk['ao_a'][None, None, None, :, :, None]
            l = tk['ao_b'][None, None, None, :, None, :]
            for a, b in ((i, j), (j, i)):
                for c, d in ((k, l), (l, k)):
                    G[a, b, c, d] = V
                    G[c, d, a, b] = V
    return G


def _exact_fock(case, seed):
    mol, basis, dens = _host_inputs(case, seed)
    label = case.get('label', '2jk')
    G = _eri(mol, basis, OMEGA if label.endswith('_rs') else 0.0)
    out = []
    for d in dens:
        D = _tensor(d)
        F = torch.zeros_like(D)
        if label in ('j', '2jk', '2jkx'):
            J = torch.einsum('pqrs,rs->pq', G, D)
            F = J if label == 'j' else 2.0 * J
        if label in ('k', 'k_rs', '2jk', '2jkx'):
            K = torch.einsum('prqs,rs->pq', G, D)
            F = F + {'k': 1.0, 'k_rs': 1.0, '2jk': -1.0, '2jkx': -XFAC if case['kind'] == 'fock' else -1.0}[label] * K
        out.append(F)
    if case['kind'] == 'fock':
        return out[0].cpu().numpy()
    return [f.cpu().numpy() for f in out] if case['kind'] == 'multi' else out[0]


def _exact_train(case, seed):
    net, x, t, mask = _network(case, seed)
    W = [w.double() for w in net.W]
    b = [v.double() for v in net.b]
    x, t, mask = (v.cuda().double() for v in (x, t, mask))
    hs, zs = [x], []
    for i in range(3):
        z = hs[-1] @ W[i].T + b[i]
        zs.append(z)
        hs.append(z * torch.sigmoid(z) if i < 2 else z)
    y, count = hs[-1], mask.sum()
    loss = (mask * (y - t) ** 2).sum().reshape(1) / count
    g = 2.0 * mask * (y - t) / count
    grads = [None] * 3
    for i in (2, 1, 0):
        if i < 2:
            s = torch.sigmoid(zs[i])
            g = g * s * (1.0 + zs[i] * (1.0 - s))
        grads[i] = (g.T @ hs[i], g.sum(0))
        g = g @ W[i]
    flat = [v for pair in grads for v in pair]
    params = [v for pair in zip(W, b) for v in pair]
    return {'y': y, 'loss': loss, 'grads': flat,
            'params': [p - 2e-3 * v / (v.abs() + 1e-8) for p, v in zip(params, flat)]}


def exact(case, seed):
    kind = case['kind']
    if kind in ('fock', 'device', 'screened', 'multi'):
        # the full tensor of larger clusters takes too long and too much memory
        return _exact_fock(case, seed) if _NAO[case['basis']] * case['n'] <= 144 else None
    return _exact_train(case, seed) if kind == 'train' else None
