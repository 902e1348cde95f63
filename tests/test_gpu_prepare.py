"""What is prepared once per factor and per frequency, at the sizes where the split changes: the solves' row permutation
(interchanges resolved 256 at a time) and diagonal-block inverses (64 rows, joined from 16), the spline's tridiagonal
system (two, or up to ten, equations a thread)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


def _solve(LU, ipiv, B, single):
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    n, k = B.shape
    aux = torch.empty(int(lib().m25_getrs_aux_bytes(n, int(single))), dtype=torch.uint8, device='cuda')
    check(lib().m25_getrs_prepare(P(LU), ctypes.c_long(n), n, P(ipiv), int(single), P(aux), ctypes.c_size_t(aux.numel()),
                                  _lib.stream_ptr()), 'prepare')
    X = B.clone()
    check(lib().m25_getrs_aux(P(LU), ctypes.c_long(n), n, int(single), P(aux), P(X), k, _lib.stream_ptr()), 'solve')
    _lib.sync_check(what='solve')
    return X


@pytest.mark.parametrize('n', [1, 2, 15, 17, 63, 64, 65, 255, 256, 257, 511, 513, 1000])
@pytest.mark.parametrize('kind', ['down', 'any', 'none'])
def test_row_permutation(n, kind):
    """With L = U = I the solve is the permutation alone: the interchanges applied from the last to the first."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    piv = {'down': i + rng.integers(0, n - i), 'any': rng.integers(0, n, n), 'none': i}[kind].astype(np.int32)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    want = B.copy()
    for r in range(n - 1, -1, -1):
        want[[r, piv[r]]] = want[[piv[r], r]]
    LU = torch.eye(n, dtype=torch.complex128, device='cuda')
    X = _solve(LU, torch.from_numpy(piv).to('cuda'), torch.from_numpy(B).to('cuda'), False)
    assert np.array_equal(X.cpu().numpy(), want)


@pytest.mark.parametrize('n', [1, 15, 16, 17, 33, 63, 64, 65, 130])
@pytest.mark.parametrize('single', [True, False])
def test_block_inverses(n, single):
    """Solves by the diagonal-block inverses of a factor with full off-diagonal triangles, against the product."""
    rng = np.random.default_rng(n)
    F = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / max(4.0, n ** 0.5)
    F[np.arange(n), np.arange(n)] += 2.0
    dt = torch.complex64 if single else torch.complex128
    LU = torch.from_numpy(F.T.copy()).to('cuda').to(dt)                    # column-major F
    Fq = LU.T.to(torch.complex128).cpu().numpy()
    L, U = np.tril(Fq, -1) + np.eye(n), np.triu(Fq)
    X0 = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    Zt = (L @ U).T                                                         # Z X = B with A = Z^T = L U
    B = torch.from_numpy(Zt @ X0).to('cuda').to(dt)
    X = _solve(LU, torch.arange(n, dtype=torch.int32, device='cuda'), B, single).to(torch.complex128).cpu().numpy()
    eps = 2.0 ** -24 if single else 2.0 ** -53
    # |X - X0| <= c n eps cond(L) cond(U) |X0| with c = 16: forming B, the two inverses, the two products
    bound = 16 * n * eps * np.linalg.cond(L) * np.linalg.cond(U) * np.linalg.norm(X0)
    assert np.linalg.norm(X - X0) <= bound


@pytest.mark.parametrize('n', [4, 5, 6, 7, 200, 260, 514, 515, 1030, 2300])
def test_spline(n):
    from scipy.interpolate import CubicSpline
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    rng = np.random.default_rng(n)
    x = 0.07 * np.linspace(0, 1, n) ** 2 if n % 2 == 0 else np.cumsum(rng.uniform(0.2, 1.0, n))
    x = x - x[0]
    y = np.exp(-9j * x / x[-1]) / (1 + np.arange(3)[:, None] + x / x[-1])
    nf = 1000
    dx = np.linspace(0, x[-1], nf)[1]
    out = torch.empty((3, nf), dtype=torch.complex128, device='cuda')
    d_x, d_y = _lib.dev(x), _lib.dev(y)
    check(lib().m25_spline_uniform(P(d_x), P(d_y), 3, n, ctypes.c_double(dx), nf, P(out), 0,
                                   ctypes.c_long(nf), ctypes.c_long(0), 1, _lib.stream_ptr()), 'm25_spline_uniform')
    _lib.sync_check()
    want = np.array([CubicSpline(x, r)(np.linspace(0, x[-1], nf)) for r in y])
    # both solve the system to rounding: differences of a few hundred ulp of the largest sample (steep end pieces)
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-12


@pytest.mark.parametrize('f', [0.1e9, 1.0e9, 4.0e9, 10.0e9])
@pytest.mark.parametrize('board', ['microstrip', 'stub'])
def test_contour(board, f):
    """The device's contour against the host's: the same pieces, nodes and weights to rounding."""
    from mom25d_b200 import _lib, board as B, device
    from mom25d_b200._lib import P, check, lib
    bd = B.microstrip_board(dmax=0.6e-3, length=10e-3) if board == 'microstrip' else B.stub_filter_board(dmax=0.3e-3)
    rho_max = float(np.ptp(bd.nodes[:, 0]) + np.ptp(bd.nodes[:, 1]))
    kr, dk, K = device.sommerfeld_contour(f, bd.stack, rho_max)
    t1, alpha, K2, wid2, m1, n2 = device.contour_path(f, bd.stack, rho_max)
    assert K2 == K and (m1 + n2) * 8 == len(kr)
    xg, wg = device.GAUSS[8]
    out = torch.empty((2, len(kr)), dtype=torch.complex128, device='cuda')
    D = ctypes.c_double
    check(lib().m25_contour(D(t1), D(alpha), D(K), D(wid2), m1, n2, P(xg), P(wg), 8, P(out[0]), P(out[1]),
                            _lib.stream_ptr()), 'm25_contour')
    _lib.sync_check()
    got = out.cpu().numpy()
    # breakpoints of up to K = m1 + n2 steps: a few ulp of K in a node, relative to a piece's width in a weight
    assert np.abs(got[0] - kr).max() <= 8 * 2.0 ** -53 * K
    assert np.abs(got[1] - dk).max() <= 16 * 2.0 ** -53 * K
    assert np.array_equal(got[0].imag == 0, kr.imag == 0)


@pytest.mark.parametrize('nr', [1, 3, 148, 149, 260])
@pytest.mark.parametrize('ns,npts', [(1, 5), (4, 1025), (5, 300), (16, 700)])
def test_hankel(ns, npts, nr):
    """The sums split over four blocks a radius (up to 64 radii) and one, 4, 8 and 16 spectra a pass, complex and real;
    fewer points than threads too."""
    from scipy.special import j0, jv
    from mom25d_b200 import _lib, core
    from mom25d_b200._lib import P, check, lib
    rng = np.random.default_rng(nr + npts)
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    kr = np.linspace(1.0, 900.0, npts) * (1 + 0.02j)
    kr[npts // 2:] = kr[npts // 2:].real                                   # a contour's tail lies on the real axis
    dk, W, rho = c(npts), c(ns, npts), np.linspace(1e-4, 0.07, nr)
    d_kr, d_dk, d_W, d_rho = (_lib.dev(v) for v in (kr, dk, W, rho))
    out = torch.empty((ns, nr), dtype=torch.complex128, device='cuda')
    check(lib().m25_hankel(P(d_kr), P(d_dk), npts, P(d_W), ns, P(d_rho), nr, P(out), _lib.stream_ptr()), 'm25_hankel')
    _lib.sync_check()
    z = rho[:, None] * kr
    want = W @ (jv(0, z) * kr * dk).T / (2 * np.pi)
    # |J0| <= e^|Im z|: each term to 1e-13 of that (J0's accuracy on both sides), and npts additions
    size = np.abs(W) @ (np.exp(np.abs(z.imag)) * np.abs(kr * dk)).T / (2 * np.pi)
    assert (np.abs(out.cpu().numpy() - want) <= (2e-13 + npts * 2.0 ** -52) * size).all()
    got = core.hankel_real(rho, kr.real.copy(), W)
    want, size = W @ j0(rho[:, None] * kr.real).T, np.abs(W).sum(1)[:, None]
    assert (np.abs(got - want) <= (2e-13 + npts * 2.0 ** -52) * size).all()


@pytest.mark.parametrize('nr', [1, 64, 65, 100, 148])
@pytest.mark.parametrize('ns,npts', [(4, 1025), (16, 700), (8, 512), (8, 513), (16, 100)])
def test_hankel_blocks_a_radius(ns, npts, nr):
    """Up to 64 radii (7/16 of the SMs) of more than 512 points are summed by four blocks each, others by one: there a
    radius's sum is that of a call with many radii, bit for bit; else it is, to rounding."""
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    rng = np.random.default_rng(nr)
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    kr, dk, W = np.linspace(1.0, 900.0, npts) + 0j, c(npts), c(ns, npts)
    rho = np.linspace(1e-4, 0.07, 260)
    d_kr, d_dk, d_W = (_lib.dev(v) for v in (kr, dk, W))

    def sums(r):
        d_rho, out = _lib.dev(r), torch.empty((ns, len(r)), dtype=torch.complex128, device='cuda')
        check(lib().m25_hankel(P(d_kr), P(d_dk), npts, P(d_W), ns, P(d_rho), len(r), P(out), _lib.stream_ptr()), 'm25_hankel')
        _lib.sync_check()
        return out.cpu().numpy()
    got, many = sums(rho[:nr]), sums(rho)[:, :nr]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if npts <= 512 or 16 * nr > 7 * sms:
        assert np.array_equal(got, many)
    size = np.abs(W) @ np.abs(kr * dk) / (2 * np.pi)       # |J0| <= 1, npts additions in either order
    assert (np.abs(got - many) <= npts * 2.0 ** -52 * size[:, None]).all()
