"""The 256-row-block solves by their number of right-hand sides (2, 4 or 8 columns are computed), at sizes with a short
last block, an odd leading dimension (8-byte copies in complex64) and whole blocks, against the product."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n', [2051, 2304])
@pytest.mark.parametrize('single', [True, False])
def test_solve_columns(n, single):
    from mom25d_b200 import _lib
    from mom25d_b200._lib import P, check, lib
    dt = torch.complex64 if single else torch.complex128
    g = torch.Generator(device='cuda').manual_seed(n)
    Z = torch.randn(n, n, generator=g, device='cuda', dtype=dt)
    Z.diagonal().add_(4 * n ** 0.5)
    A = Z.clone()
    piv = torch.empty(n, dtype=torch.int32, device='cuda')
    work = torch.empty(int(lib().m25_getrf_workspace(n, int(single))), dtype=torch.uint8, device='cuda')
    aux = torch.empty(int(lib().m25_getrs_aux_bytes(n, int(single))), dtype=torch.uint8, device='cuda')
    s = _lib.stream_ptr()
    check(lib().m25_getrf(P(A), ctypes.c_long(n), n, P(piv), int(single), 0, P(work), ctypes.c_size_t(work.numel()), s))
    check(lib().m25_getrs_prepare(P(A), ctypes.c_long(n), n, P(piv), int(single), P(aux), ctypes.c_size_t(aux.numel()), s))
    X0 = torch.randn(n, 8, generator=g, device='cuda', dtype=torch.complex128)
    B = (Z.to(torch.complex128) @ X0).to(dt)
    eps = 2.0 ** -24 if single else 2.0 ** -53
    for k in range(1, 9):
        X = B[:, :k].contiguous()
        check(lib().m25_getrs_aux(P(A), ctypes.c_long(n), n, int(single), P(aux), P(X), k, s))
        _lib.sync_check()
        # the matrix is well conditioned (about 3): c n eps with c = 1 is far above what rounding leaves
        err = torch.linalg.norm(X.to(torch.complex128) - X0[:, :k]) / torch.linalg.norm(X0[:, :k])
        assert float(err) <= n * eps, k
