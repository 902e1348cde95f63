"""The LU's outer blocks of 64 to 256 columns in one factorisation (each takes the width the tuning table has for the
size that is left): P A = L U, and the same bits with the look-ahead's streams as on one stream."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

TABLES = {'falling': [(100, 64), (250, 128), (500, 192), (1000, 256)],
          'mixed': [(150, 128), (300, 64), (600, 256), (900, 64)], 'committed': None}


@pytest.mark.parametrize('n', [64, 65, 129, 300, 449, 700, 1100])
@pytest.mark.parametrize('table', sorted(TABLES))
@pytest.mark.parametrize('single', [True, False])
def test_widths(n, table, single, monkeypatch):
    from mom25d_b200 import _lib, tune
    from mom25d_b200._lib import P, check, lib
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    Z = torch.from_numpy(M.T.copy()).to('cuda').to(torch.complex64 if single else torch.complex128)
    work = torch.empty(int(lib().m25_getrf_workspace(n, int(single))), dtype=torch.uint8, device='cuda')

    def factor():
        A, piv = Z.clone(), torch.empty(n, dtype=torch.int32, device='cuda')
        check(lib().m25_getrf(P(A), ctypes.c_long(n), n, P(piv), int(single), int(single), P(work),
                              ctypes.c_size_t(work.numel()), _lib.stream_ptr()), 'm25_getrf')
        _lib.sync_check(what='m25_getrf')
        return A.cpu().numpy(), piv.cpu().numpy()
    try:
        if TABLES[table]:
            tune.set_table([(a, w, 32) for a, w in TABLES[table]], single)
        A, piv = factor()
        monkeypatch.setenv('M25_LOOKAHEAD', '0')
        A1, piv1 = factor()
    finally:
        _lib.apply_tuning(lib())
    assert np.array_equal(A, A1) and np.array_equal(piv, piv1)
    perm = np.arange(n)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    F = A.T.astype(np.complex128)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    X = Z.cpu().numpy().T.astype(np.complex128)[perm]
    # each product to eps (3xTF32: 2^-22), n terms, a complex product's four: 8 n eps |L| |U| bounds |P A - L U|
    eps = 2.0 ** -22 if single else 2.0 ** -53
    assert np.linalg.norm(L @ U - X) <= 8 * n * eps * np.linalg.norm(np.abs(L) @ np.abs(U))


@pytest.mark.parametrize('n', [8448, 8391])
@pytest.mark.parametrize('tf32', [True, False])
def test_schedule_changes_in_the_middle(n, tf32, monkeypatch):
    """complex64 from more than 8,000 rows left to fewer: the critical path goes from a block's columns to a panel's, and
    the block's own interchanges from one stream to another. A matrix that pivots far off the diagonal; the same bits on
    one stream, in each of three factorisations."""
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    g = torch.Generator(device='cuda').manual_seed(n)
    Z = torch.complex(*torch.randn((2, n, n), generator=g, device='cuda'))
    work = torch.empty(int(lib().m25_getrf_workspace(n, 1)), dtype=torch.uint8, device='cuda')

    def factor():
        A, piv = Z.clone(), torch.empty(n, dtype=torch.int32, device='cuda')
        check(lib().m25_getrf(P(A), ctypes.c_long(n), n, P(piv), 1, int(tf32), P(work), ctypes.c_size_t(work.numel()),
                              _lib.stream_ptr()), 'm25_getrf')
        _lib.sync_check(what='m25_getrf')
        return A, piv
    many = [factor() for _ in range(3)]
    monkeypatch.setenv('M25_LOOKAHEAD', '0')
    A1, piv1 = factor()
    assert int((piv1 != torch.arange(n, device='cuda')).sum()) > 0.9 * n
    for A, piv in many:
        assert torch.equal(piv, piv1) and torch.equal(torch.view_as_real(A), torch.view_as_real(A1))
