"""The LU's cluster panel (csrc/panel.cu) at the sizes where its split changes: one CTA and several, a last panel and a
last column group that are short, the rows a thread holds, the largest cluster cut to two CTAs. Checked by P A = L U
(both products in complex128 here), by the pivots' rule (the largest |re| + |im|: every |l| <= sqrt 2) and, in
complex128, against LAPACK's pivots."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

SIZES = [1, 2, 15, 17, 63, 64, 65, 100, 127, 129, 257, 300, 513, 1000, 2049, 2500]


def _lu(Z, single):
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    n = Z.shape[0]
    A = Z.clone()
    piv = torch.empty(n, dtype=torch.int32, device='cuda')
    work = torch.empty(int(lib().m25_getrf_workspace(n, int(single))), dtype=torch.uint8, device='cuda')
    check(lib().m25_getrf(P(A), ctypes.c_long(n), n, P(piv), int(single), 0, P(work), ctypes.c_size_t(work.numel()),
                          _lib.stream_ptr()), 'm25_getrf')
    _lib.sync_check(what='m25_getrf')
    return A, piv.cpu().numpy()


def _check(n, single, order):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if order == 'graded':                                 # pivots from the far rows, columns of very unlike sizes
        M *= np.geomspace(1e-3, 1e3, n)[:, None]
    Z = torch.from_numpy(M.T.copy()).to('cuda').to(torch.complex64 if single else torch.complex128)
    A, piv = _lu(Z, single)
    assert np.all(piv >= np.arange(n)) and np.all(piv < n)
    perm = np.arange(n)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    F = A.T.to(torch.complex128)                          # the column-major factor as a matrix
    L = torch.tril(F, -1) + torch.eye(n, dtype=torch.complex128, device='cuda')
    U = torch.triu(F)
    PA = Z.T.to(torch.complex128)[torch.from_numpy(perm).to('cuda')]
    eps = 2.0 ** -24 if single else 2.0 ** -53
    # |PA - LU| <= gamma_n |L| |U| entry by entry, gamma_n = 4 n eps (four roundings a complex term); the norms of it
    bound = 4 * n * eps * torch.linalg.norm(L.abs() @ U.abs())
    assert float(torch.linalg.norm(PA - L @ U)) <= float(bound) + 1e-300
    assert float(L.abs().max()) <= 2 ** 0.5 * (1 + 8 * eps)
    if not single and n <= 1000:
        import scipy.linalg
        assert np.array_equal(piv, scipy.linalg.lu_factor(M)[1])


@pytest.mark.parametrize('n', SIZES)
@pytest.mark.parametrize('single', [True, False])
def test_cluster_panel(n, single):
    _check(n, single, 'random')


@pytest.mark.parametrize('n,single,cl', [(1100, True, 2), (2100, True, 2), (3000, True, 2), (1100, False, 2),
                                         (2047, False, 2), (1500, True, 3), (2900, True, 7)])
def test_cluster_panel_more_rows_a_thread(n, single, cl, monkeypatch):
    monkeypatch.setenv('M25_PANEL_CLUSTER_MAX', str(cl))
    _check(n, single, 'graded')


@pytest.mark.parametrize('single', [True, False])
def test_cluster_panel_singular(single):
    from mom25d_b200 import _lib
    n = 200
    Z = torch.zeros(n, n, dtype=torch.complex64 if single else torch.complex128, device='cuda')
    Z.diagonal().fill_(1.0)
    Z[100, 100] = 0.0                                     # an exactly zero pivot
    with pytest.raises(_lib.M25Error):
        _lu(Z, single)
    Z[100, 100] = 1.0
    Z[50, :] = float('nan')                               # column 50 of A has no pivot
    with pytest.raises(_lib.M25Error):
        _lu(Z, single)
    Z[50, :] = 0.0
    Z[50, 50] = 2.0
    A, piv = _lu(Z, single)                               # and the next factorisation is sound
    assert torch.equal(A, Z) and np.array_equal(piv, np.arange(n))
