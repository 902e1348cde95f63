"""
The work that a user of mom25d_b200 has it do, as cases that can be timed and compared: one frequency of a board
solved in double and in mixed precision, a short sweep, the impedance matrix alone, the dense LU and its solves
through the C ABI and through the host LU backend, and the compiled-core seam on host arrays.

A board case's inputs are a board of this package's generators and a frequency drawn from the seed within 3% of the
case's; a matrix case's are a complex symmetric matrix of the kind the equilibrated impedance matrices are (unit
diagonal, a smooth oscillating kernel of the distance between jittered points of a board-sized rectangle).
"""
import ctypes
import math
import random

import numpy as np
import torch

import mom25d_b200.board as B
from mom25d_b200 import _lib, core
from mom25d_b200.backend import CudaBackend
from mom25d_b200.geometry import Geometry
from mom25d_b200.operator import DirectSolver
from mom25d_b200.sim import Simulation

C0 = 299792458.0
c_int, c_long, c_size_t = ctypes.c_int, ctypes.c_long, ctypes.c_size_t


def listed():
    return [
        # the smallest board that is solved in earnest: a 10 mm microstrip, N = 302; launches and host work
        dict(name='sparams_double_302', kind='sparams', board='microstrip', dmax=0.6e-3, length=10e-3,
             precision='double', f=3.0e9),
        # an ordinary board below the size where mixed precision is chosen: the 2-port through line, N = 2,921
        dict(name='currents_double_2921', kind='currents', board='microstrip', dmax=0.3e-3, length=30e-3,
             precision='double', f=3.5e9),
        # the drop-in at full size: every step of a double sweep of the routed board, N = 18,788
        dict(name='sparams_double_18788', kind='sparams', board='routed', n_traces=24, ncross=4, board_seed=1,
             precision='double', f=4.0e9),
        # a request of the serving loop: a mixed solve without kept factors on the stub filter, N = 4,977
        dict(name='currents_mixed_4977', kind='currents', board='stub', dmax=0.2e-3, precision='mixed', f=4.0e9),
        # the same on the routed board, the headline size
        dict(name='currents_mixed_18788', kind='currents', board='routed', n_traces=24, ncross=4, board_seed=1,
             precision='mixed', f=5.0e9),
        # a board whose double matrix is taken not to fit: complex64 fill, the matrix-free double operator
        dict(name='currents_matrix_free_5908', kind='currents', board='routed', n_traces=6, ncross=3, board_seed=1,
             precision='mixed', matrix_free=True, f=4.0e9),
        # a sweep of one board from cold: a fresh factor, then reused ones; S at every frequency
        dict(name='sweep_mixed_2553x6', kind='sweep', board='stub', dmax=0.3e-3, precision='mixed', f=2.0e9,
             f_stop=5.0e9, points=6),
        # the impedance matrix alone (tables, far fill, near field, vias), for a caller with its own solver
        dict(name='impedance_8520', kind='impedance', board='routed', n_traces=12, ncross=3, board_seed=1,
             precision='double', f=4.0e9),
        # the C ABI from another host program: factor a complex64 matrix, prepare the solves, solve 8 columns
        dict(name='lu_solve_c64_9601', kind='lu', n=9601, nrhs=8, single=True),
        # many solves with one kept factor (a preconditioner's use): one pair of triangular solves
        dict(name='solve_c64_12000', kind='solve', n=12000, nrhs=8, single=True),
        # the LU backend seam on host arrays: factor, solve, an odd size and column count
        dict(name='backend_c128_2001', kind='backend', n=2001, nrhs=3, single=False),
        # the compiled-core seam on host arrays: the far fill and the matrix-free product
        dict(name='core_861', kind='core', board='microstrip', dmax=0.6e-3, length=30e-3, nrhs=4, f=3.0e9),
    ]


def _loguniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _draw_board(rng, small=False):
    """A microstrip of 300 to 5,000 unknowns, a stub filter of 2,000 to 8,000, a routed board of 3,000 to 16,000."""
    pick = rng.choice(['microstrip', 'stub', 'routed'])
    if small or pick == 'microstrip':
        return dict(board='microstrip', dmax=round(_loguniform(rng, 0.25e-3, 0.6e-3), 7),
                    length=round(_loguniform(rng, 10e-3, 30e-3), 5))
    if pick == 'stub':
        return dict(board='stub', dmax=round(_loguniform(rng, 0.16e-3, 0.34e-3), 7))
    return dict(board='routed', n_traces=rng.randint(4, 18), ncross=3, board_seed=rng.randint(1, 6))


def draw(rng):
    kind = rng.choice(['sparams', 'currents', 'currents', 'currents', 'sweep', 'impedance', 'lu', 'lu', 'solve', 'solve',
                       'backend', 'core'])
    if kind in ('lu', 'solve'):
        return dict(kind=kind, n=int(_loguniform(rng, 300, 12000)), nrhs=rng.randint(1, 16),
                    single=rng.random() < 0.6)
    if kind == 'backend':
        return dict(kind=kind, n=int(_loguniform(rng, 200, 4500)), nrhs=rng.randint(1, 16), single=rng.random() < 0.5)
    if kind == 'core':
        return dict(kind=kind, nrhs=rng.randint(1, 16), f=rng.uniform(1e9, 8e9), **_draw_board(rng, small=True))
    # (from 1.5 GHz: below it a complex64 factor may not precondition its own frequency, and whether the refinement
    # then converges is a matter of rounding)
    case = dict(kind=kind, f=rng.uniform(1.5e9, 8e9), precision='double', **_draw_board(rng))
    if kind == 'currents' and case['board'] == 'routed':
        case['precision'] = 'mixed'
    if kind == 'currents' and rng.random() < 0.6:
        case['precision'] = 'mixed'
        if case['board'] != 'microstrip' and rng.random() < 0.3:
            case['matrix_free'] = True
    if kind == 'sweep':
        case = dict(case, f=rng.uniform(1.5e9, 3e9), f_stop=rng.uniform(3.5e9, 6e9), points=rng.randint(3, 7),
                    precision=rng.choice(['double', 'mixed']), **_draw_board(rng, small=True))
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------------
def _board(case):
    if case['board'] == 'microstrip':
        return B.microstrip_board(dmax=case['dmax'], length=case['length'])
    if case['board'] == 'stub':
        return B.stub_filter_board(dmax=case['dmax'])
    n = case['n_traces']
    full = n >= 24
    return B.routed_board(seed=case['board_seed'], n_traces=n, n_vias=16 if full else max(2, 2 * n // 3),
                          n_ports=8 if full else 4, ncross=case['ncross'])


def _freq(case, seed):
    return case['f'] * (1.0 + 0.03 * random.Random(seed).uniform(-1, 1))


def _matrix(n, seed, double):
    """A complex symmetric n x n matrix of unit diagonal: exp(-j k r) / (r + a) between jittered grid points of a
    60 x 40 mm board, times the cosine of the angle between two random directions, scaled by its diagonal."""
    gen = torch.Generator(device='cuda').manual_seed(1000003 * n + seed)

    def rand(*shape):
        return torch.rand(*shape, generator=gen, device='cuda', dtype=torch.float64)
    nx = max(1, int(math.ceil(math.sqrt(1.5 * n))))
    h = 60e-3 / nx
    i = torch.arange(n, device='cuda', dtype=torch.float64)
    x = (i % nx + 0.6 * rand(n)) * h
    y = (torch.div(i, nx, rounding_mode='floor') + 0.6 * rand(n)) * h
    th = 2 * math.pi * rand(n)
    k = 2 * math.pi * (3e9 + 3e9 * float(rand(1))) * math.sqrt(4.4) / C0
    Z = torch.empty(n, n, dtype=torch.complex128 if double else torch.complex64, device='cuda')
    a = 0.3 * h
    for r0 in range(0, n, 1024):
        s = slice(r0, min(n, r0 + 1024))
        r = torch.hypot(x[s, None] - x[None, :], y[s, None] - y[None, :])
        Z[s] = torch.polar(a / (r + a), -k * r) * torch.cos(th[s, None] - th[None, :])
    return Z


def _rhs(n, k, seed, dtype):
    gen = torch.Generator(device='cuda').manual_seed(seed + 77)
    return torch.randn(n, k, generator=gen, device='cuda', dtype=torch.complex128).to(dtype)


def _core_tables(geo, f):
    """The Green tables of one frequency as the compiled core takes them: one table an interface pair, the static
    singular coefficients of a dielectric half-space and a smooth oscillating remainder."""
    L = len(geo.layers)
    pairs = [(i, j) for i in range(L) for j in range(i, L)]
    tab = np.zeros((L, L), np.int32)
    for t, (i, j) in enumerate(pairs):
        tab[i, j] = tab[j, i] = t
    nt, nf = len(pairs), 8192
    dr = geo.rho_max / (nf - 1)
    rho = dr * np.arange(nf)
    k = 2 * np.pi * f / C0 * np.sqrt(3.0)
    A = np.stack([1e-7 * (np.exp(-1j * k * rho) - 1) / (rho + 1e-3 * (t + 1)) for t in range(nt)])
    Q = np.stack([4e9 * (np.exp(-1j * k * rho) - 0.6) / (rho + 2e-3 * (t + 1)) for t in range(nt)])
    one = np.ones(nt)
    z = [geo.st.z[kk] for kk in geo.layers]
    return dict(A=A, Q=Q, cA=1e-7 * one + 0j, cq=5e9 * one - 1e8j, cAi=-0.8e-7 * one + 0j, cqi=-4e9 * one + 2e7j,
                dr=dr * one, d=np.array([abs(z[i] - z[j]) for i, j in pairs], float), dimg=2.8e-3 * one, tab=tab,
                kind=np.array([0 if i == j else 1 for i, j in pairs], np.int32))


class _Plan:
    """What a caller of the C ABI keeps for a size: the factor's memory, pivots, workspace, solve data."""

    def __init__(self, n, nrhs, single):
        L, self.n, self.nrhs, self.single = _lib.lib(), n, nrhs, int(single)
        self.dtype = torch.complex64 if single else torch.complex128
        byte = dict(dtype=torch.uint8, device='cuda')
        self.ipiv = torch.empty(n, dtype=torch.int32, device='cuda')
        self.work = torch.empty(int(L.m25_getrf_workspace(n, self.single)), **byte)
        self.aux = torch.empty(int(L.m25_getrs_aux_bytes(n, self.single)), **byte)
        self.A = torch.empty(n, n, dtype=self.dtype, device='cuda')
        self.X = torch.empty(n, nrhs, dtype=self.dtype, device='cuda')

    def factor(self, Z):
        L, P, n, s = _lib.lib(), _lib.P, self.n, _lib.stream_ptr()
        self.A.copy_(Z)                                   # (the factorisation is in place)
        _lib.check(L.m25_getrf(P(self.A), c_long(n), n, P(self.ipiv), self.single, self.single, P(self.work),
                               c_size_t(self.work.numel()), s), 'm25_getrf')
        _lib.check(L.m25_getrs_prepare(P(self.A), c_long(n), n, P(self.ipiv), self.single, P(self.aux),
                                       c_size_t(self.aux.numel()), s), 'm25_getrs_prepare')

    def solve(self, R):
        L, P = _lib.lib(), _lib.P
        self.X.copy_(R)
        _lib.check(L.m25_getrs_aux(P(self.A), c_long(self.n), self.n, self.single, P(self.aux), P(self.X), self.nrhs,
                                   _lib.stream_ptr()), 'm25_getrs_aux')
        return self.X


def prepare(case, seed):
    kind = case['kind']
    s = dict(case=case)
    if kind in ('lu', 'solve'):
        s['Z'] = _matrix(case['n'], seed, not case['single'])
        s['plan'] = _Plan(case['n'], case['nrhs'], case['single'])
        s['R'] = _rhs(case['n'], case['nrhs'], seed, s['plan'].dtype)
        if kind == 'solve':
            s['plan'].factor(s.pop('Z'))
    elif kind == 'backend':
        s['Z'] = _matrix(case['n'], seed, not case['single']).cpu().numpy()
        s['R'] = _rhs(case['n'], case['nrhs'], seed, torch.complex128).cpu().numpy()
        s['be'] = CudaBackend()
    elif kind == 'core':
        geo = Geometry(_board(case))
        s['f'] = _freq(case, seed)
        s['g'], s['tb'] = geo.g, _core_tables(geo, s['f'])
        s['Z'] = np.zeros((geo.Ne, geo.Ne), complex)
        s['X'] = _rhs(geo.Ne, case['nrhs'], seed, torch.complex128).cpu().numpy()
    elif kind == 'impedance':
        s['f'] = _freq(case, seed)
        s['ds'] = DirectSolver(Geometry(_board(case)))
    else:
        s['f'] = _freq(case, seed)
        s['sim'] = Simulation.from_board(_board(case), precision=case['precision'])
        if case.get('matrix_free'):
            s['sim'].fast.hybrid = False
        if kind == 'currents':
            s['E'] = s['sim'].excitation()
        if kind == 'sweep':
            s['freqs'] = np.linspace(s['f'], case['f_stop'], case['points'])
    return s


def run(s):
    kind = s['case']['kind']
    if kind == 'lu':
        s['plan'].factor(s['Z'])
        return s['plan'].solve(s['R'])
    if kind == 'solve':
        return s['plan'].solve(s['R'])
    if kind == 'backend':
        s['be'].factor(s['Z'])
        return s['be'].solve(s['R'])
    if kind == 'core':
        w = 2 * np.pi * s['f']
        core.fill_far(s['Z'], s['g'], s['tb'], w)
        return dict(Z=s['Z'], Y=core.matvec_far_multi(s['X'], s['g'], s['tb'], w))
    if kind == 'impedance':
        return s['ds'].impedance(s['f'], s['case']['precision'])
    s['sim'].fast.forget()                                # a new sweep: no factor kept from the pass before
    if kind == 'sweep':
        return s['sim'].sweep(s['freqs'])
    if kind == 'sparams':
        return s['sim'].sparams(s['f'])
    return s['sim'].currents(s['f'], s['E'])


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _size(case):
    geo = Geometry(_board(case))
    return geo.N, len(geo.ports)


def work(case):
    kind = case['kind']
    if kind in ('lu', 'solve', 'backend'):
        n, k, e = case['n'], case['nrhs'], 8 if case['single'] else 16
        solve = 8.0 * n * n * k
        if kind == 'solve':
            return dict(bytes=1.0 * e * n * (n + 2 * k), flops=solve)
        return dict(bytes=1.0 * e * n * (n + 2 * k), flops=8.0 / 3 * n ** 3 + solve)
    N, k = _size(case)
    fill = 84.5 * N * N                                   # 56 flops an entry, 30 a kernel evaluation, 0.95 an entry
    if kind == 'core':
        k = case['nrhs']
        return dict(bytes=16.0 * N * (N + 2 * k), flops=fill + 8.0 * N * N * k)
    if kind == 'impedance':
        return dict(bytes=16.0 * N * N, flops=fill)
    lu = 8.0 / 3 * N ** 3 + 8.0 * N * N * k
    each = dict(bytes=16.0 * N * (N + k), flops=fill + lu)
    if kind == 'sweep':                                   # (mixed: one factor for the sweep)
        m = case['points']
        return dict(bytes=m * each['bytes'], flops=m * fill + (lu if case['precision'] == 'mixed' else m * lu))
    return each


def tolerance(case):
    """About four times what the path differed by from torch.linalg.solve of the same matrix (from exact() where there
    is one; S by the same currents; Z from the reference's compiled core, 3e-13 to 3e-12)."""
    kind = case['kind']
    if kind in ('lu', 'solve', 'backend'):                # 4e-7 and 2e-6; 7e-15 and 4e-14
        return dict(rel=2e-6, max=1e-5) if case['single'] else dict(rel=3e-14, max=2e-13)
    if kind == 'core':                                    # 6e-16 and 3e-14
        return dict(rel=3e-15, max=1.2e-13)
    if kind == 'impedance':
        return dict(rel=1.2e-11, max=5e-10)
    if case['precision'] == 'double':                     # S: 1.4e-9 and 5.4e-9; currents: 4.6e-9 and 2.4e-7
        return dict(rel=2e-8, max=1e-6) if kind == 'currents' else dict(rel=6e-9, max=2.4e-8)
    if kind == 'sweep':                                   # |dS| of mixed against double solves: up to 1.7e-5
        return dict(rel=7e-5, max=7e-5)
    return dict(rel=3e-4, max=5e-3)                       # 7e-5 and 1.4e-3 (residuals of 1e-6, ill-conditioned Z)


# ---- the same in 64 bits, by torch and numpy alone -------------------------------------------------------------------
def exact(case, seed):
    kind = case['kind']
    if kind in ('lu', 'solve', 'backend'):
        n, k = case['n'], case['nrhs']
        Z = _matrix(n, seed, not case['single']).to(torch.complex128)
        R = _rhs(n, k, seed, torch.complex64 if case['single'] else torch.complex128)
        return torch.linalg.solve(Z, R.to(torch.complex128))
    if kind == 'core':
        return _exact_core(case, seed)
    return None


def _exact_core(case, seed):
    geo = Geometry(_board(case))
    f = _freq(case, seed)
    g, tb, w = geo.g, _core_tables(geo, f), 2 * np.pi * f
    cent = np.asarray(g['cent'], float).reshape(-1, 2)
    r = np.hypot(cent[:, None, 0] - cent[None, :, 0], cent[:, None, 1] - cent[None, :, 1])
    t = tb['tab'][np.ix_(g['lt'], g['lt'])]
    u = np.minimum(r / tb['dr'][t], tb['A'].shape[1] - 1.000001)
    i = u.astype(int)
    fr = u - i
    far = np.where(r > 0, r, np.inf)
    same = tb['kind'][t] == 0
    image = 1 / np.sqrt(r * r + tb['dimg'][t] ** 2)
    cross = 1 / np.sqrt(np.where(same, 1.0, r * r + tb['d'][t] ** 2))
    G = []
    for T, c, ci in (('A', 'cA', 'cAi'), ('Q', 'cq', 'cqi')):
        rest = tb[T][t, i] * (1 - fr) + tb[T][t, i + 1] * fr
        G.append(rest + np.where(same, tb[c][t] / far + tb[ci][t] * image, tb[c][t] * cross))
    ap, am = np.asarray(g['ap'], float), np.asarray(g['am'], float)
    Z = 0
    halves = []
    for p, a, v in ((g['ep'], ap, g['vp']), (g['em'], am, g['vm'])):
        halves.append((p, a * np.asarray(g['area'])[p], cent[p] - np.asarray(v, float).reshape(-1, 2)))
    for p, a, d in halves:
        for q, b, e in halves:
            at = np.ix_(p, q)
            Z = Z + np.outer(a, b) * (1j * w * (d @ e.T) * G[0][at] + 4 * G[1][at] / (1j * w))
    X = _rhs(geo.Ne, case['nrhs'], seed, torch.complex128).cpu().numpy()
    return dict(Z=Z, Y=Z @ X)
